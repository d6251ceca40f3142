"""A device without room, for tests: a stand-in for cudaMalloc that answers
cudaErrorMemoryAllocation to requests of given sizes, loaded before
libmocca_gpu.so so that the library's calls find it first (a process of its own).

`python tests/no_room.py CASE` runs one case of test_gpu_no_room.py."""
import ctypes as C
import subprocess
import sys
import tempfile
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

SHIM = r"""
#include <cstddef>
#include <dlfcn.h>
#include <driver_types.h>
static size_t refused[8];
static int nrefused, count;
static cudaError_t pending = cudaSuccess;
template <class F> static F real(const char* name) { return (F)dlsym(RTLD_NEXT, name); }
extern "C" {
void refuse(size_t bytes) { if (bytes) refused[nrefused++] = bytes; else nrefused = 0; }
int refusals() { return count; }
cudaError_t cudaMalloc(void** p, size_t bytes) {
    for (int i = 0; i < nrefused; ++i)
        if (refused[i] == bytes) { ++count; return pending = cudaErrorMemoryAllocation; }
    return real<cudaError_t (*)(void**, size_t)>("cudaMalloc")(p, bytes);
}
cudaError_t cudaGetLastError() {   // keeps the refusal like the runtime's own errors
    const cudaError_t e = pending;
    pending = cudaSuccess;
    return e != cudaSuccess ? e : real<cudaError_t (*)()>("cudaGetLastError")();
}
}
"""


class NoRoom:
    def __init__(self):
        from mocca_gb300.build import nvcc
        d = Path(tempfile.mkdtemp())
        (d / "shim.cpp").write_text(SHIM)
        subprocess.run([nvcc(), "-shared", "-cudart", "shared", "-Xcompiler", "-fPIC",
                        "-Xlinker", "--no-as-needed", "-o", str(d / "shim.so"),
                        str(d / "shim.cpp"), "-ldl"], check=True)
        self.lib = C.CDLL(str(d / "shim.so"), mode=C.RTLD_GLOBAL)
        self.lib.refuse.argtypes = [C.c_size_t]
        self.lib.refuse.restype = None

    def refuse(self, *sizes):
        self.lib.refuse(0)
        for s in sizes:
            self.lib.refuse(int(s))

    def refusals(self):
        return self.lib.refusals()


def relative(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b))


def spinors(nwt, npts, seed):
    rng = np.random.default_rng(seed)
    psi = rng.normal(size=(nwt, npts))
    qn = np.ones((nwt, 4), dtype=np.int32)
    qn[: nwt // 2, 0] = -1
    return psi / np.linalg.norm(psi, axis=1)[:, None], qn, rng.normal(size=nwt)


def gram_schmidt(room, precision, bar):
    """Without room for one of its three buffers the Gram-Schmidt of the tensor
    cores gives way to the FP64 kernels; once there is room it is back."""
    from mocca_gb300 import SLY4, RunParams
    from mocca_gb300.mesh import MeshState
    nwt, n = 60, (9, 10, 8)
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=nwt, neutrons=2, protons=2,
                  precision=precision)
    npts = 4 * n[0] * n[1] * n[2]
    psi, qn, en = spinors(nwt, npts, 1)

    def run(g):
        g.set_spinors(psi, qn)
        g.set_energies(en)
        g.GramSchmidt()
        return g.get_spinors()

    with MeshState(p, SLY4) as g:
        want = run(g)
    chunks = -(-npts // 128)
    for size in (2 * chunks * 30 * 30 * 8, 2 * 8 * 80 * 80 * 2, 2 * 80 * 4):
        with MeshState(p, SLY4) as g:
            for _ in range(2):
                seen = room.refusals()
                room.refuse(size)
                got = run(g)
                room.refuse()
                assert room.refusals() == seen + 1, size
                assert relative(got, want) < bar and not np.array_equal(got, want)
            assert np.array_equal(run(g), want)


def canonical(room):
    """The FP64 pairing step without room for the digit planes or the exponents of
    its coefficients: the kernels of pairing.cu, the same spinors and gaps."""
    from mocca_gb300 import MG_CAN_BASIS, MG_FP64, SLY4, RunParams, _abi, synthetic
    from mocca_gb300.mesh import MeshState
    p = RunParams(nx=9, ny=8, nz=7, dx=0.9, nwt=96, neutrons=12, protons=12, precision=MG_FP64,
                  pairing=_abi.MG_PAIRING_HFB)
    psi, qn, en = synthetic.ho_basis(p, 48, seed=5)

    def run(sizes):
        with MeshState(p, SLY4) as g:
            g.set_spinors(psi, qn)
            g.set_energies(en)
            g.set_pairing()
            room.refuse(*sizes)
            g.SolvePairing()
            room.refuse()
            can = g.get_spinors(MG_CAN_BASIS).reshape(96, -1)
            return [g.get_hfb_block(b)[2] for b in range(4)], can

    gaps, can = run(())
    for size in (4 * 8 * 80 * 80 * 2, 4 * 80 * 4):
        seen = room.refusals()
        g2, c2 = run((size,))
        # the field's buffer and the canonical basis' are of the same size
        assert room.refusals() >= seen + 2, size
        for b in range(4):
            assert relative(g2[b], gaps[b]) < 1e-9
        # canonical states by their occupations: degenerate ones may mix, the span
        # of all of a block does not
        assert relative(c2.T @ c2, can.T @ can) < 1e-9


def refused(fn, status):
    from mocca_gb300 import _abi
    try:
        fn()
    except _abi.MgError as e:
        assert e.status == status, e
    else:
        raise AssertionError("not refused")


def retried(room):
    """Set-ups that fail half way: the call is an error each time it is made
    again, and once there is room it does its work."""
    from mocca_gb300 import MG_FP64, SLY4, RunParams, _abi
    from mocca_gb300.mesh import MeshState
    nwt, n = 60, (9, 10, 8)
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=nwt, neutrons=20, protons=20,
                  precision=MG_FP64, parameter_estimation=1)
    psi, qn, en = spinors(nwt, 4 * n[0] * n[1] * n[2], 2)

    def prepare(g):
        g.set_spinors(psi, qn)
        g.set_energies(en)
        g.GramSchmidt()
        g.DeriveAll()
        rng = np.random.default_rng(3)
        g.set_potentials(U=rng.normal(size=2 * p.V), B=rng.uniform(10.0, 20.0, 2 * p.V),
                         nablaB=rng.normal(size=6 * p.V), W=rng.normal(size=18 * p.V),
                         divW=rng.normal(size=6 * p.V))

    def step(g):
        g.GradDesc(0.01, 0.3)
        return g.get_spinors(), g.StepParameters()

    with MeshState(p, SLY4) as g:
        prepare(g)
        want, dt = step(g)
    lists = 4 * (2 + 1 + 2 * nwt)
    with MeshState(p, SLY4) as g:
        room.refuse(4 * 12 * nwt)           # the jobs sorted by their matrices
        for _ in range(2):
            refused(lambda: g.set_spinors(psi, qn), _abi.MG_ERR_CUDA)
            refused(lambda: g.DeriveBasis(), _abi.MG_ERR_STATE)
        room.refuse()
        g.set_spinors(psi, qn)
        g.set_energies(en)
        for size in (lists, 2 * 30 * 30 * 8):   # member lists, factors
            room.refuse(size)
            for _ in range(2):
                refused(g.GramSchmidt, _abi.MG_ERR_CUDA)
            room.refuse()
        prepare(g)
        for size in (4 * 48, 4 * 4):        # the probe's jobs, its quantum numbers
            room.refuse(size)
            for _ in range(2):
                refused(lambda: g.GradDesc(0.01, 0.3), _abi.MG_ERR_CUDA)
            room.refuse()
        got, dt2 = step(g)
        assert dt2 == dt and np.array_equal(got, want)


def multigrid(room):
    """A Coulomb multigrid that cannot be set up, for want of room or because the
    mesh has none, is refused as often as it is asked for."""
    from mocca_gb300 import MG_FP64, SLY4, RunParams, _abi
    from mocca_gb300.mesh import MeshState

    def state(n):
        p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=2, neutrons=20, protons=20,
                      precision=MG_FP64, coulomb_solver=2)
        g = MeshState(p, SLY4)
        g.set_densities(rho=np.random.default_rng(4).uniform(0.0, 0.08, 2 * p.V))
        g.CalculateAllMoments()
        return g

    with state((17, 17, 17)) as g:
        for _ in range(3):
            refused(g.SolveCoulomb, _abi.MG_ERR_ARG)
    n = (24, 20, 28)
    V = n[0] * n[1] * n[2]
    with state(n) as g:
        its = g.SolveCoulomb()
        want = g.get_potentials()["coulomb"]
    with state(n) as g:
        # a double per point, the levels' floats, the partials, the sweep matrix
        parts = max(3 * 3 * 7, 256)
        coarse = 6 * 5 * 7
        for size in (8 * V, 4 * 3 * (V + V // 8 + V // 64), 3 * 8 * parts, 4 * coarse ** 2):
            seen = room.refusals()
            room.refuse(size)
            for _ in range(2):
                refused(g.SolveCoulomb, _abi.MG_ERR_CUDA)
            room.refuse()
            assert room.refusals() == seen + 2, size
        assert g.SolveCoulomb() == its
        assert np.array_equal(g.get_potentials()["coulomb"], want)


CASES = {
    "multigrid": multigrid,
    "retried": retried,
    "gram_schmidt_fp64": lambda room: gram_schmidt(room, 0, 1e-13),
    "gram_schmidt_mixed": lambda room: gram_schmidt(room, 1, 1e-11),
    "canonical": canonical,
}

if __name__ == "__main__":
    CASES[sys.argv[1]](NoRoom())
    print("ok")
