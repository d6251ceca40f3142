"""Moments and Dirichlet values of the Coulomb problem at the edges of their
kernels' splits: meshes shorter than a round of the moments' chains, with a
remainder of one, and longer than the words loaded ahead; points beyond the box
that fill no block.  The potential against the oracle's: both solve to
|r| <= 1e-12 |b| (the oracle, which stops by the reference's own rule, by solving on
from its solution), so they agree within twice the condition number (below
16/3 (4 n / pi)^2, 2.5e3 at n = 17) of that, 5e-9, where a wrong moment or boundary
value shows at its own size."""
import numpy as np
import pytest

import oracle as O
from conftest import rel
from mocca_gb300 import MG_FP64, SLY4, RunParams
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(3, 4, 5), (6, 7, 6), (16, 16, 16), (17, 13, 11)])
def test_potential(built, n):
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=2, neutrons=20, protons=20,
                  precision=MG_FP64, coulomb_prec=1e-12, coulomb_max=2000)
    rng = np.random.default_rng(n[0])
    ax = [0.4 + 0.8 * np.arange(k) for k in n]
    Z, Y, X = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    r = np.sqrt(X ** 2 / 0.9 + Y ** 2 + Z ** 2 / 1.2)
    rho = 0.08 / (1 + np.exp((r - 0.4 * 0.8 * min(n)) / 0.5)) * rng.uniform(0.9, 1.1, r.shape)
    out = []
    for cls in (MeshState, O.OracleState):
        s = cls(p, SLY4)
        s.set_densities(rho=np.concatenate([0.7 * rho.reshape(-1), rho.reshape(-1)]))
        s.CalculateAllMoments()
        for _ in range(1 if cls is MeshState else 20):
            s.SolveCoulomb()
        out.append(s.get_potentials()["coulomb"])
    assert rel(out[0], out[1]) <= 5e-9, rel(out[0], out[1])
