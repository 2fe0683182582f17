"""A count of right-hand sides whose work vectors the device cannot hold is refused and
leaves the handle as it was: the next apply and the next solve give what they gave before.
"""
import numpy as np
import pytest
import torch

import hifde3d_b200 as hb
from hifde3d_b200 import synth

pytestmark = pytest.mark.gpu

N = 15
N3 = (N + 1) ** 3
TOO_MANY = 2 ** 26  # 4096 * 8 B * 2^26 = 2 TB a vector


def unread():  # refused before the vectors are read
    return torch.zeros(N3, dtype=torch.float64, device="cuda")


@pytest.fixture()
def factor():
    a = synth.face_coefficients_lognormal(N, 3)
    f = hb.HIFFactor(N, 4, 1e-6)
    hb.SetupStencilFaces(f, N, 1.0 / (N + 1), *a, np.zeros((N + 2,) * 3))
    f.Factor()
    yield f
    f.close()


@pytest.mark.parametrize("nrhs", [1, 3])
def test_refused_apply_keeps_handle(factor, nrhs):
    f = factor
    U = np.asfortranarray(np.stack([synth.dof_vector(N, c) for c in range(nrhs)], axis=1))
    before = f.Apply(U.copy(order="F"), True)
    with pytest.raises(hb.HIFError) as e:
        f.apply_device(unread().data_ptr(), TOO_MANY, N3, True)
    assert e.value.code == hb.HIF_ERR_NOMEM
    np.testing.assert_array_equal(f.Apply(U.copy(order="F"), True), before)


def test_refused_solve_keeps_handle(factor):
    f = factor
    b = synth.dof_vector(N, 1)
    x, it, _ = f.solve_pcg(b)
    with pytest.raises(hb.HIFError) as e:
        f.solve_pcg_device(unread().data_ptr(), unread().data_ptr(), TOO_MANY, N3, 1e-10, 10)
    assert e.value.code == hb.HIF_ERR_NOMEM
    y, it2, _ = f.solve_pcg(b)
    assert it2 == it
    np.testing.assert_array_equal(x, y)
