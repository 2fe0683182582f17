"""The pivot block of the elimination on blocks that are ill-conditioned however they are
scaled: a smooth kernel's matrix with 10^-8 added to its diagonal (scaled condition number
about 2 10^9), whose 16-wide diagonal blocks are nearly singular too, as it stands and
graded over six decades.

Elimination of a symmetric positive definite matrix without pivoting, each pivot's row and
column substituted, leaves a backward error of at most n u sqrt(a_ii a_jj) in entry (i, j)
of the n x n block; the inverse in the scaling of its diagonal is then within n u times the
scaled condition number of the exact one, here from elimination in extended precision.
Products with explicit inverses of the diagonal blocks miss that by a factor of 1000.
"""
import numpy as np
import pytest

import hifde3d_b200 as hb
from hifde3d_b200 import synth

pytestmark = pytest.mark.gpu


def exact_inverse(A):
    n = len(A)
    M, X = A.astype(np.longdouble), np.eye(n, dtype=np.longdouble)
    for i in range(n):
        f = M[i + 1:, i] / M[i, i]
        M[i + 1:] -= f[:, None] * M[i]
        X[i + 1:] -= f[:, None] * X[i]
    for i in range(n - 1, -1, -1):
        X[i] = (X[i] - M[i, i + 1:] @ X[i + 1:]) / M[i, i]
    return X


@pytest.mark.parametrize("r,s", [(100, 70), (127, 40), (128, 33)])
@pytest.mark.parametrize("graded", [False, True])
def test_ill_conditioned_pivot_block(r, s, graded):
    n = r + s
    x = np.arange(r) / r
    A = np.eye(n)
    A[:r, :r] = np.exp(-((x[:, None] - x) / 0.1) ** 2) + 1e-8 * np.eye(r)
    if graded:
        g = 10.0 ** (6.0 * synth.uniform(3, n) - 3.0)
        A = A * g[:, None] * g
    _, inv, _, _ = hb.Schur(A, np.arange(r), np.arange(r, n))
    d = np.sqrt(np.diag(A)[:r])
    scaled = A[:r, :r] / d[:, None] / d
    exact = exact_inverse(scaled)
    err = np.linalg.norm((inv * d[:, None] * d - exact).astype(float))
    bound = r * 1.1e-16 * np.linalg.cond(scaled) * np.linalg.norm(exact.astype(float))
    assert err < bound
