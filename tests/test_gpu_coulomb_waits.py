"""Waits of the Coulomb CG that run out: with a limit of one clock for the waits for
the other clusters' sums from some iteration on, no solve decides anything from what
has come so far.  MG_ERR_TIMEOUT, from the solve or, where that does not wait for its
result, from the energy behind it; once the limit is back, the same context solves as
before.

The last iteration is the one where sums that did not all come, being too small,
would pass for a residual below the bound."""
import numpy as np
import pytest

import poke
from mocca_gb300 import MG_FP64, SLY4, RunParams, _abi
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


def _state(n, coulomb_prec):
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=2, neutrons=20, protons=20,
                  precision=MG_FP64, coulomb_prec=coulomb_prec, coulomb_max=1000)
    rng = np.random.default_rng(sum(n))
    V = n[0] * n[1] * n[2]
    g = MeshState(p, SLY4)
    g.set_densities(rho=rng.uniform(0.0, 0.08, 2 * V), tau=rng.uniform(0.01, 0.1, 2 * V))
    g.CalculateAllMoments()
    return g


@pytest.mark.parametrize("coulomb_prec", [0.0, 1e-8])
@pytest.mark.parametrize("n", [(16, 15, 17), (24, 24, 24), (33, 36, 35)])
def test_sums_that_do_not_come(built, n, coulomb_prec):
    g = _state(n, coulomb_prec)
    its = g.SolveCoulomb()
    want = g.get_potentials()["coulomb"]
    for start in (its, its // 2):
        g.reset_coulomb_guess()
        poke.load().poke_cg_sum_wait(g.h, 1, start)
        with pytest.raises(_abi.MgError) as e:
            g.SolveCoulomb()
        assert e.value.status == _abi.MG_ERR_TIMEOUT
        poke.load().poke_cg_sum_wait(g.h, 0, 0)
        g.reset_coulomb_guess()
        assert g.SolveCoulomb() == its
        assert np.array_equal(g.get_potentials()["coulomb"], want)
    # without its iteration count the solve is not waited for: the energy is
    g.reset_coulomb_guess()
    poke.load().poke_cg_sum_wait(g.h, 1, its)
    assert g.lib.mg_construct_potentials(g.h, None) == _abi.MG_OK
    with pytest.raises(_abi.MgError) as e:
        g.CompEnergy()
    assert e.value.status == _abi.MG_ERR_TIMEOUT
    g.CompEnergy()   # reported once
    g.close()
