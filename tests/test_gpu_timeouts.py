"""A wait of a tensor-core kernel that ran out (here a kernel that does nothing but
leave the word which such a kernel leaves behind) is reported by whichever call hands
out results next, in both forms, and by that one only."""
import ctypes as C

import numpy as np
import pytest

import poke
from mocca_gb300 import (MG_CAN_BASIS, MG_FP64, MG_HF_BASIS, MG_MIXED, SLY4, RunParams, _abi,
                         synthetic)
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[MG_FP64, MG_MIXED], ids=["fp64", "mixed"])
def state(request):
    import __graft_entry__
    __graft_entry__.build()
    p = RunParams(nx=10, ny=10, nz=10, dx=0.8, nwt=40, neutrons=12, protons=12,
                  pairing=_abi.MG_PAIRING_HFB, precision=request.param)
    psi, qn, en = synthetic.ho_basis(p, 20, seed=1234)
    g = MeshState(p, SLY4)
    g.set_spinors(psi, qn)
    g.set_energies(en)
    g.set_pairing()
    g.Start()
    yield g
    g.close()


CALLS = {
    "synchronize": lambda g: g.synchronize(),
    "spinors": lambda g: g.get_spinors(),
    "derivatives": lambda g: g.get_derivatives(),
    "occupations": lambda g: g.get_occupations(MG_CAN_BASIS),
    "energies": lambda g: g.get_energies(),
    "hpsi": lambda g: g.hPsi(),
    "hpsi_energies": lambda g: g.hPsi(want_spinors=False),
    "derive_all": lambda g: g.DeriveAll(),
    "densities": lambda g: g.get_densities(),
    "potentials": lambda g: g.get_potentials(),
    "coulomb": lambda g: g.SolveCoulomb(),
    "energy": lambda g: g.CompEnergy(),
    "pairing": lambda g: g.SolvePairing(),
    "pairing_field": lambda g: g.get_pairing_field(),
    "hfb_block": lambda g: g.get_hfb_block(0),
    "symmetries": lambda g: g.SymmetryOperators(),
    "angular_momentum": lambda g: g.AngularMomentum(),
    "evolve": lambda g: g.Evolve(1, 0.01, 0.3),
    "evolve_none": lambda g: g.Evolve(0, 0.01, 0.3),
    "constraint_fields": lambda g: g.get_constraint_fields(),
}


@pytest.mark.parametrize("call", sorted(CALLS))
def test_reported_once(state, call):
    assert poke.load().poke_tc_timeout(state.h) == 0
    # the calls that only queue work leave it to the next
    state.DeriveBasis(MG_HF_BASIS)
    state.UpdateDensities()
    with pytest.raises(_abi.MgError) as e:
        CALLS[call](state)
    assert e.value.status == _abi.MG_ERR_TIMEOUT
    CALLS[call](state)
    assert np.isfinite(state.get_spinors()).all()
