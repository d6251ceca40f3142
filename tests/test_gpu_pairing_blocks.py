"""The FP64 pairing step's contractions on blocks at the edges of their splits: 26
spinors (near the 24 where the tensor cores begin), more than 32 and 48 columns, beyond
42 (another form of the sums), the largest of 64, a mesh with remainders of point
tiles and chunks.  Against the oracle with the bars of the small-block tests: the
pairing field 1e-12, the gaps 1e-11 of their norms."""
import numpy as np
import pytest

import oracle as O
from conftest import rel
from mocca_gb300 import MG_FP64, SLY4, RunParams, _abi, synthetic
from mocca_gb300.mesh import MeshState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nspwf", [((9, 8, 7), 48), ((8, 9, 8), 66), ((9, 9, 8), 98),
                                     ((7, 9, 10), 114)])
def test_field_and_gaps(built, n, nspwf):
    p = RunParams(nx=n[0], ny=n[1], nz=n[2], dx=0.9, nwt=2 * nspwf, neutrons=12, protons=12,
                  precision=MG_FP64, pairing=_abi.MG_PAIRING_HFB)
    psi, qn, en = synthetic.ho_basis(p, nspwf, seed=5)
    sizes = [int(((qn[:, 0] == a) & (qn[:, 1] == b)).sum()) for a in (-1, 1) for b in (-1, 1)]
    assert 24 <= max(sizes) <= 64, sizes
    out = []
    for cls in (MeshState, O.OracleState):
        s = cls(p, SLY4)
        s.set_spinors(psi, qn)
        s.set_energies(en)
        s.set_pairing()
        s.SolvePairing()
        out.append((s.get_pairing_field(), [s.get_hfb_block(b) for b in range(4)]))
    (fg, bg), (fo, bo) = out
    assert rel(fg[0], fo[0]) < 1e-12
    for b in range(4):
        assert rel(bg[b][2], bo[b][2]) < 1e-11, b
