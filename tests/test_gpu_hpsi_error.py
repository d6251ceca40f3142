"""The rounding error of FP64 h.psi, from the derivatives and the fields that it
reads, against sums in extended precision: no larger than with the terms U, B and W
summed one by one (a fused multiply-add each, the W terms in a sum of their own),
evaluated here beside it.  Norm-wise over all spinors, where both are averages over
1e5 components or more."""
import numpy as np
import pytest

from mocca_gb300 import MG_FP64, SLY4, RunParams, synthetic
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu

X = np.longdouble


def _fma(a, b, c):
    """a b + c rounded to FP64 from extended precision."""
    return np.asarray(X(a) * X(b) + X(c), dtype=np.float64)


def _pauli(p, n):
    return {1: (p[2], p[3], p[0], p[1]), 2: (p[3], -p[2], -p[1], p[0]),
            3: (p[0], p[1], -p[2], -p[3])}[n]


def _both(psi, der, lap, kin, U, B, nB, W, dW):
    """(extended, one by one) h.psi of one spinor: psi, lap [4, V], der [3, 4, V]."""
    terms = [(mu, nu, W[nu, mu], _pauli(der[mu], nu + 1)) for mu in range(3) for nu in range(3)]
    terms += [(0, nu, 0.5 * dW[nu], _pauli(psi, nu + 1)) for nu in range(3)]
    w, we = np.zeros_like(psi), np.zeros(psi.shape, dtype=X)
    for _, _, f, s in terms:
        for l in range(4):
            w[l] = _fma(f, s[l], w[l])
            we[l] += X(f) * X(s[l])
    flip = lambda q: np.stack([q[1], -q[0], q[3], -q[2]])
    exact = (-(X(B) + X(kin)) * X(lap) - sum(X(nB[m]) * X(der[m]) for m in range(3))
             + X(U) * X(psi) + flip(we))
    t = _fma(-kin, lap, -(B * lap))
    sd = _fma(nB[2], der[2], _fma(nB[1], der[1], nB[0] * der[0]))
    return exact, _fma(U, psi, t - sd) + flip(w)


def _well(p, full, rng):
    """A Woods-Saxon well with its spin-orbit field and a small div W."""
    n = (p.nx, p.ny, p.nz)
    ax = [p.dx * (np.arange(k) + 0.5) - (0.5 * p.dx * k if full else 0.0) for k in n]
    Z, Y, Xg = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    r = np.sqrt(Xg ** 2 / 0.94 + Y ** 2 + Z ** 2 / 1.17)
    f = 1 / (1 + np.exp((r - 3.6) / 0.65))
    g = np.stack([Xg / 0.94, Y, Z / 1.17]).reshape(3, -1) * (-f * (1 - f) / 0.65 / r).reshape(-1)
    f, V = f.reshape(-1), p.V
    W = np.zeros((2, 3, 3, V))
    for k, m, q in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
        W[:, q, m], W[:, m, q] = -60 * g[k], 60 * g[k]
    return dict(U=np.stack([-52 * f, -48 * f]), B=np.stack([8 * f, 7.5 * f]),
                nablaB=np.stack([8 * g, 7.5 * g]), W=W, divW=0.1 * rng.normal(size=(2, 3, V)) * f)


@pytest.mark.parametrize("n,nwt,full", [((10, 9, 11), 40, False), ((8, 8, 8), 60, False),
                                        ((13, 12, 14), 16, True)])
def test_error(built, n, nwt, full):
    rng = np.random.default_rng(nwt)
    sym = 0 if full else 1
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=nwt, neutrons=12, protons=12, pc=sym,
                  sc=sym, tsc=sym, precision=MG_FP64)
    if full:
        ax = [0.8 * (np.arange(k) + 0.5) - 0.4 * k for k in n]
        psi = np.empty((nwt, 4, n[2], n[1], n[0]))
        for i in range(nwt):
            for c in range(4):
                fx, fy, fz = (np.exp(-0.5 * ((a - rng.uniform(-2, 2)) / rng.uniform(1.5, 3)) ** 2)
                              * (1 + rng.normal() * a) for a in ax)
                psi[i, c] = fz[:, None, None] * fy[None, :, None] * fx
        qn = np.zeros((nwt, 4), dtype=np.int32)
        qn[:, 0] = np.where(np.arange(nwt) < nwt // 2, -1, 1)
    else:
        psi, qn, _ = synthetic.ho_basis(p, nwt // 2, seed=3)
    pot = _well(p, full, rng)
    with MeshState(p, SLY4) as g:
        g.set_spinors(psi, qn)
        g.DeriveBasis()
        g.set_potentials(**pot)
        h, _, _ = g.hPsi()
        der, lap = g.get_derivatives()
    V = p.V
    force = SLY4.to_c()
    m = force.nucleonmass
    num = {"gpu": 0.0, "one by one": 0.0}
    for i in range(nwt):
        it = 0 if qn[i, 0] < 0 else 1
        red = 1 - m[it] / (12 * m[0] + 12 * m[1]) if force.com1body == 2 else 1.0
        exact, sums = _both(psi[i].reshape(4, V), der[i].reshape(3, 4, V), lap[i].reshape(4, V),
                            force.hbm / 2 * red, pot["U"][it], pot["B"][it], pot["nablaB"][it],
                            pot["W"][it], pot["divW"][it])
        num["gpu"] += float(((h[i].reshape(4, V) - exact) ** 2).sum())
        num["one by one"] += float(((sums - exact) ** 2).sum())
    assert num["gpu"] <= num["one by one"], num
    assert num["gpu"] > 0
