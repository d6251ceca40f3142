"""Sizes of the batched eigensolver (mg_eigh_batched) where its seed kernel's
work split can go wrong: one rotation pair and none, odd sizes (a padding row),
rounds shorter and longer than the ring of rotations between its two CTAs, warp
and scratch limits, the largest size.  Each runs beside a 1 x 1 and an empty
neighbour.

Bars against LAPACK, from the solver's form (FP64 refinement and polish, sums of
n products): eigenvalues n eps |A| with a factor of 4, residual and
orthonormality 1e-12 and 1e-13 as for every size.
"""
import numpy as np
import pytest

from mocca_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9, 31, 33, 64, 65, 127, 128, 129, 159, 160])
def test_size(built, n):
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, n))
    sizes = np.array([n, 0, 1], dtype=np.int32)
    a = np.zeros((3, n, n))
    a[0] = x + x.T
    a[2, 0, 0] = -2.5
    w = np.zeros((3, n))
    z = np.zeros((3, n, n))
    st = _abi.load().mg_eigh_batched(3, sizes.ctypes.data_as(_abi._I), n,
                                     a.ctypes.data_as(_abi._D), w.ctypes.data_as(_abi._D),
                                     z.ctypes.data_as(_abi._D))
    assert st == 0
    m, v = a[0], z[0]
    nrm = np.linalg.norm(m)
    assert np.abs(w[0] - np.linalg.eigvalsh(m)).max() <= 4 * n * 2.3e-16 * nrm
    assert np.linalg.norm(m @ v - v * w[0]) <= 1e-12 * nrm
    assert np.abs(v.T @ v - np.eye(n)).max() <= 1e-13
    assert w[2, 0] == -2.5 and abs(z[2, 0, 0]) == 1.0
