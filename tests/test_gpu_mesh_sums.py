"""Sums over the mesh at the edges of their blocks: h.psi energies and dispersions
(blocks of 128 points, a warp per spwf adding them) and the mesh integrals of the
total energy (rows of 256 points, a warp of them per block), on meshes below a
warp's 32 points, at 128 and 256 and one beyond, with more blocks than lanes.

Against the oracle, whose sums are as long: V products of eps 1.1e-16 in a row in
random signs stay below 1e-13 of the terms' sum of magnitudes, of which the
energies here keep more than a tenth: 1e-12."""
import numpy as np
import pytest

import oracle as O
from mocca_gb300 import MG_FP64, SLY4, RunParams, synthetic
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(3, 3, 3), (8, 8, 2), (43, 3, 2), (16, 8, 2), (5, 13, 4),
                               (21, 23, 19)])
def test_sums(built, n):
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.8, nwt=8, neutrons=4, protons=4,
                  precision=MG_FP64)
    V = n[0] * n[1] * n[2]
    rng = np.random.default_rng(V)
    psi = rng.uniform(0.2, 1.0, size=(8, 4 * V)) / np.sqrt(4 * V * p.dv)
    qn = np.ones((8, 4), dtype=np.int32)
    qn[:4, 0] = -1
    qn[::2, 1] = -1
    dens = dict(rho=rng.uniform(0.02, 0.08, 2 * V), tau=rng.uniform(0.01, 0.1, 2 * V),
                nablaj=rng.normal(size=2 * V) * 0.01, derrho=rng.normal(size=6 * V) * 0.01,
                laprho=rng.normal(size=2 * V) * 0.01)
    pot = dict(U=rng.uniform(-60.0, -20.0, 2 * V), B=rng.uniform(0.0, 10.0, 2 * V),
               nablaB=rng.normal(size=6 * V), W=rng.normal(size=18 * V),
               divW=rng.normal(size=6 * V))
    out = []
    for cls in (MeshState, O.OracleState):
        s = cls(p, SLY4)
        s.set_spinors(psi, qn)
        s.set_energies(np.arange(8.0))
        s.set_occupations(np.ones(8))
        s.DeriveAll()
        s.set_potentials(**pot)
        h, e, d = s.hPsi()
        s.set_densities(**dens)
        out.append((np.asarray(h), np.asarray(e), np.asarray(d), s.CompEnergy()))
    (h, e, d, t), (ho, eo, do, to) = out
    assert np.abs(h - ho).max() <= 1e-12 * np.abs(ho).max()
    scale = p.dv * np.abs(psi * ho.reshape(8, -1)).sum(1)
    assert (np.abs(e - eo) <= 1e-12 * scale).all()
    assert (np.abs(d - do) <= 1e-12 * (np.abs(do) + 2 * eo ** 2)).all()
    for k, x in to.items():
        if k == "sp_energy":   # half the energies last set or computed: no mesh sum
            continue
        x = np.asarray(x, dtype=float)
        assert (np.abs(np.asarray(t[k]) - x) <= 1e-11 * np.maximum(np.abs(x), 1.0)).all(), k
