"""Gram-Schmidt on blocks at the edges of its contractions' splits: one spinor,
one fewer and one more than the 16 columns of a matrix step up to the largest
block, blocks of very different size beside each other, a last point tile of less
than 128, more and fewer tiles than SMs.

Reference: the Cholesky form Psi R^-1 in numpy, energy-ordered blocks.  The input
is orthonormal up to 5% noise (condition number below 2).  Bars: the FP64 form
carries at most 80 + 4 V products of eps 1.1e-16 in a row, in random signs: 1e-13;
the mixed form's operands are rounded at 2^-47 = 7e-15 of a row's largest entry,
which is up to ~30 times its root mean square in both factors of the overlap:
1e-11."""
import numpy as np
import pytest

from mocca_gb300 import MG_FP64, MG_MIXED, SLY4, RunParams
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bar", [(MG_FP64, 1e-13), (MG_MIXED, 1e-11)])
@pytest.mark.parametrize("n,sizes", [((7, 5, 6), (1, 16, 17, 31)), ((6, 7, 9), (49, 33, 1, 15)),
                                     ((5, 9, 8), (64, 2, 65, 24)), ((11, 7, 5), (80, 79, 32, 3)),
                                     ((24, 23, 21), (48, 41, 47, 40)),
                                     ((22, 24, 24), (20, 80, 64, 5))])
def test_blocks(built, precision, bar, n, sizes):
    nwt = sum(sizes)
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=nwt, neutrons=2, protons=2,
                  precision=precision)
    rng = np.random.default_rng(nwt)
    npts = 4 * n[0] * n[1] * n[2]
    qn = np.ones((nwt, 4), dtype=np.int32)
    psi = np.empty((nwt, npts))
    keys = np.repeat(np.arange(4), sizes)
    rng.shuffle(keys)
    for b in range(4):
        rows = np.flatnonzero(keys == b)
        qn[rows, 0], qn[rows, 1] = (-1, 1)[b // 2], (-1, 1)[b % 2]
        q, _ = np.linalg.qr(rng.normal(size=(npts, len(rows))))
        psi[rows] = (q.T + 0.05 * rng.normal(size=q.T.shape) / np.sqrt(npts)) / np.sqrt(p.dv)
    en = rng.normal(size=nwt)
    g = MeshState(p, SLY4)
    g.set_spinors(psi, qn)
    g.set_energies(en)
    g.GramSchmidt()
    got = g.get_spinors().reshape(nwt, npts)
    g.close()
    for b in range(4):
        rows = np.flatnonzero(keys == b)
        rows = rows[np.argsort(en[rows], kind="stable")]
        s = p.dv * psi[rows] @ psi[rows].T
        want = np.linalg.solve(np.linalg.cholesky(s), psi[rows])
        err = np.linalg.norm(got[rows] - want, axis=1) / np.linalg.norm(want, axis=1)
        assert err.max() <= bar, (b, len(rows), err.max())


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("nb", [20, 30, 50])
def test_not_a_number_stays_behind(built, nb, value):
    """A NaN or an infinity in one spinor of an FP64 block: the spinors before it
    in energy are what they are without it, those from it on are not finite there
    (blocks of 20 go to the FP64 kernels, the others to the tensor cores)."""
    p = RunParams(nx=6, ny=7, nz=5, dx=0.8, nwt=nb, neutrons=2, protons=2, precision=MG_FP64)
    rng = np.random.default_rng(nb)
    npts = 4 * 6 * 7 * 5
    q, _ = np.linalg.qr(rng.normal(size=(npts, nb)))
    psi = q.T / np.sqrt(p.dv)
    qn = np.ones((nb, 4), dtype=np.int32)
    out = []
    for bad in (False, True):
        x = psi.copy()
        if bad:
            x[12, 17] = value
        g = MeshState(p, SLY4)
        g.set_spinors(x, qn)
        g.set_energies(np.arange(nb, dtype=float))
        g.GramSchmidt()
        out.append(g.get_spinors().reshape(nb, npts))
        g.close()
    clean, got = out
    assert np.array_equal(got[:12], clean[:12])
    assert not np.isfinite(got[12:, 17]).any()
