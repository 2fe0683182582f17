"""Schur of one dense block at the edges of its elimination: blocks taken whole (up to 160
unknowns, register tiles of 96 and 160), then the blocked form: redundant counts around
the 128-wide pivot blocks and the 64 x 64 product tiles, skeleton counts of one and
around a tile, ragged both ways.

The block is strictly diagonally dominant (each diagonal entry 1.5 times its row's
absolute sum), so ||A22^{-1}||_inf ||A22||_inf <= (2.5 / 0.5) = 5 per unit of scaling and
elimination without pivoting grows nothing: every output is within a small multiple of
n u = 1200 * 1.1e-16 of numpy's, and 100 n u relative (Frobenius) is required.
"""
import numpy as np
import pytest

import hifde3d_b200 as hb
from hifde3d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r,s", [(1, 1), (15, 1), (16, 16), (17, 78), (95, 1), (96, 0),
                                 (80, 17), (100, 60), (160, 0), (3, 157), (161, 1), (127, 64), (128, 63), (129, 65), (191, 128),
                                 (192, 129), (255, 17), (256, 0), (257, 191), (384, 64),
                                 (650, 129), (1023, 130)])
def test_schur_edges(r, s):
    n = r + s
    A = synth.normal(100 + r, n * n).reshape(n, n)
    A[np.arange(n), np.arange(n)] = 0.0
    A[np.arange(n), np.arange(n)] = 1.5 * np.abs(A).sum(axis=1)
    order = np.argsort(synth.uniform(7 + s, n))
    red, skel = order[:r], order[r:]
    A22, inv, X, S = hb.Schur(A, red, skel)
    B = A[np.ix_(red, red)]
    ref = np.linalg.inv(B)
    tol = 100 * n * 1.1e-16
    np.testing.assert_array_equal(A22, B)

    def rel(a, b):
        return np.linalg.norm(a - b) / np.linalg.norm(b)

    assert rel(inv, ref) < tol
    if s:
        Xr = ref @ A[np.ix_(red, skel)]
        assert rel(X, Xr) < tol
        assert rel(S, -A[np.ix_(skel, red)] @ Xr) < tol
