"""The FP64 conjugate-gradient Coulomb solve on boxes where its split over
blocks and threads has remainders or changes (one point, fewer points than a
warp, odd and unequal lengths, two and four points per thread), against the
direct separable solve (residual ~1e-14).

Both stop criteria: to |b - L phi| <= 1e-10 |b| the potential agrees with the
direct one within the condition number's share (largest over smallest
eigenvalue of the stored box's Laplacian: below 16/3 (4 n / pi)^2, 3.5e4 at
n = 64) of 1e-10, so 3.5e-6 at most and in practice far less; 1e-7 is asked
of boxes up to 36^3, 1e-8 of boxes up to 20 points."""
import numpy as np
import pytest

from conftest import rel
from mocca_gb300 import MG_FP64, MG_MIXED, SLY4, RunParams
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


def _state(n, precision, coulomb_prec, coulomb_max=1000):
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=2, neutrons=20, protons=20,
                  precision=precision, coulomb_prec=coulomb_prec, coulomb_max=coulomb_max)
    ax = [0.4 + 0.8 * np.arange(k) for k in n]
    Z, Y, X = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    r = np.sqrt(X ** 2 / 0.9 + Y ** 2 + Z ** 2 / 1.2)
    rho = 0.08 / (1 + np.exp((r - 0.4 * 0.8 * min(n)) / 0.5))
    g = MeshState(p, SLY4)
    g.set_densities(rho=np.concatenate([rho.reshape(-1)] * 2))
    g.CalculateAllMoments()
    return g


@pytest.mark.parametrize("n", [(3, 3, 3), (5, 2, 4), (10, 10, 10), (7, 16, 11), (20, 17, 19),
                               (36, 35, 36), (48, 50, 47)])
def test_cg_against_direct(built, n):
    g = _state(n, MG_FP64, 1e-10)
    it = g.SolveCoulomb()
    assert 0 < it < 1000
    assert g.CoulombResidual() <= 1.01e-10
    d = _state(n, MG_MIXED, 0.0)
    d.SolveCoulomb()
    got, want = g.get_potentials()["coulomb"], d.get_potentials()["coulomb"]
    assert rel(got, want) < (1e-8 if max(n) <= 20 else 1e-7)
    # the reference's own stop, and a second solve from the solution
    h = _state(n, MG_FP64, 0.0)
    first = h.SolveCoulomb()
    again = h.SolveCoulomb()
    assert again <= first
    for s in (g, d, h):
        s.close()


def test_cg_cap(built):
    """The iteration cap: MG_NOT_CONVERGED with the last iterate written."""
    g = _state((12, 12, 12), MG_FP64, 1e-10, coulomb_max=5)
    assert g.SolveCoulomb() == 5
    assert np.isfinite(g.get_potentials()["coulomb"]).all()
    assert g.CoulombResidual() > 1e-10
    g.close()
