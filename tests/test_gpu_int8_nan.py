"""A NaN in an operand of the FP64 product from int8 slices has no digits: the product is,
bit for bit, the one with a zero in its place, whatever else its row (or column) holds.
(The factorization meets NaNs in its pivots first and refuses them.)
"""
import numpy as np
import pytest

import hifde3d_b200 as hb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def product(A, B, ta, tb, S):
    m, k = A.shape
    n = B.shape[1]
    # column-major storage of A or A^T, B or B^T
    a = torch.from_numpy(np.ascontiguousarray(A if ta else A.T)).cuda()
    b = torch.from_numpy(np.ascontiguousarray(B if tb else B.T)).cuda()
    c = torch.zeros(n, m, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    hb.GemmInt8Device(ta, tb, m, n, k, 1.0, a.data_ptr(), k if ta else m, b.data_ptr(),
                      n if tb else k, 0.0, c.data_ptr(), m, S)
    return c.cpu().numpy().T


@pytest.mark.parametrize("S", [2, 5, 8])
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
def test_nan_counts_as_zero(ta, tb, S):
    rng = np.random.default_rng(S)
    A = rng.standard_normal((150, 100))
    B = rng.standard_normal((100, 70))
    for X in (A, B):
        X[rng.integers(0, X.shape[0], 40), rng.integers(0, X.shape[1], 40)] = np.nan
    A[3] = np.nan
    got = product(A, B, ta, tb, S)
    want = product(np.nan_to_num(A, nan=0.0), np.nan_to_num(B, nan=0.0), ta, tb, S)
    np.testing.assert_array_equal(got, want)
