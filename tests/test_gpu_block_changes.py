"""New quantum numbers on a live context: the Gram-Schmidt blocks change in number
and size, and with them every buffer that is sized for them (more blocks, larger
ones, chunks of 128 points after chunks of 256 when blocks of more than 64 shrink
below and the FP64 form follows the mixed one).

The kernels are deterministic and nothing carries over from the blocks before, so
a context that has seen other blocks gives the bits of a fresh one."""
import numpy as np
import pytest

from mocca_gb300 import MG_FP64, MG_MIXED, SLY4, RunParams
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu

N = (11, 9, 10)
NWT = 100
KEYS = [(it, par, sig) for it in (-1, 1) for par in (-1, 1) for sig in (-1, 1)]


def _blocks(sizes, seed):
    rng = np.random.default_rng(seed)
    keys = np.repeat(np.arange(len(sizes)), sizes)
    rng.shuffle(keys)
    qn = np.ones((NWT, 4), dtype=np.int32)
    qn[:, :3] = np.array(KEYS)[keys]
    npts = 4 * N[0] * N[1] * N[2]
    psi = rng.normal(size=(NWT, npts))
    return psi / np.linalg.norm(psi, axis=1)[:, None], qn, rng.normal(size=NWT)


def _params(precision):
    return RunParams(nx=N[0], ny=N[1], nz=N[2], dx=0.8, nwt=NWT, neutrons=2, protons=2,
                     precision=precision)


def _run(g, sizes, precision, seed):
    psi, qn, en = _blocks(sizes, seed)
    g.set_precision(precision)
    g.set_spinors(psi, qn)
    g.set_energies(en)
    g.GramSchmidt()
    return g.get_spinors()


@pytest.mark.parametrize("steps", [
    [((25, 25, 25, 25), MG_FP64), ((50, 50), MG_FP64), ((64, 36), MG_FP64)],
    [((50, 50), MG_FP64), ((24, 24, 24, 7, 7, 7, 7), MG_FP64), ((30, 40, 30), MG_FP64)],
    [((20, 20, 20, 20, 20), MG_MIXED), ((80, 20), MG_MIXED), ((13,) * 7 + (9,), MG_MIXED)],
    [((80, 20), MG_MIXED), ((64, 36), MG_FP64), ((16,) * 6 + (4,), MG_MIXED)],
    [((90, 10), MG_FP64), ((33, 33, 34), MG_FP64), ((90, 10), MG_FP64)],
])
def test_live_context_like_a_fresh_one(built, steps):
    live = MeshState(_params(steps[0][1]), SLY4)
    for k, (sizes, precision) in enumerate(steps):
        got = _run(live, sizes, precision, k)
        fresh = MeshState(_params(precision), SLY4)
        want = _run(fresh, sizes, precision, k)
        fresh.close()
        assert np.isfinite(want).all()
        assert np.array_equal(got, want), (k, sizes)
    live.close()
