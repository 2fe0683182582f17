"""The several-vector apply at the edges of its right-hand-side tiles (8, 16, 32, 64) and
beyond one, on a ragged grid, for both forms of the factor (explicit inverse; Cholesky,
with triangular blocks) and both directions, against the single-vector apply of the same
factor. The two sum in different orders: with at most 2000 terms and about 10 sweeps,
1e-12 relative is two orders above n u.
"""
import numpy as np
import pytest

import hifde3d_b200 as hb
from hifde3d_b200 import synth

pytestmark = pytest.mark.gpu

N = 27


@pytest.fixture(scope="module", params=[hb.ELIM_GAUSS_JORDAN, hb.ELIM_CHOLESKY])
def factor(request):
    a = synth.face_coefficients_lognormal(N, 3)
    f = hb.HIFFactor(N, 4, 1e-6, hb.PARTITION_CLIPPED)
    f.set_option(hb.OPT_ELIMINATION, request.param)
    hb.SetupStencilFaces(f, N, 1.0 / (N + 1), *a, np.zeros((N + 2,) * 3))
    f.Factor()
    U = np.asfortranarray(np.stack([synth.dof_vector(N, 40 + c) for c in range(130)], axis=1))
    one = {}
    for inverse in (True, False):
        one[inverse] = np.stack([f.Apply(U[:, c].copy(), inverse) for c in range(130)], axis=1)
    yield f, U, one
    f.close()


@pytest.mark.parametrize("nrhs", [2, 7, 8, 9, 16, 17, 32, 33, 64, 65, 130])
@pytest.mark.parametrize("inverse", [True, False])
def test_columns_match_single_vector(factor, nrhs, inverse):
    f, U, one = factor
    Y = f.Apply(np.asfortranarray(U[:, :nrhs].copy()), inverse)
    ref = one[inverse][:, :nrhs]
    err = np.linalg.norm(Y - ref, axis=0) / np.linalg.norm(ref, axis=0)
    assert err.max() < 1e-12
