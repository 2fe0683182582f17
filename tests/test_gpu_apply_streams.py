"""The apply on streams that it cannot use, and its own CUDA graphs.

Inside a caller's stream capture every apply and every solve is refused, whether the sweep has a graph by
then or not, and on the legacy default stream, which cannot be captured, from the first
call on; the handle goes on as before. A sweep's graph is made at the 17th use of a count of
right-hand sides: results stay bit for bit those of the plain launches, after the work
vectors have grown and after new coefficients too.
"""
import numpy as np
import pytest
import torch

import hifde3d_b200 as hb
from hifde3d_b200 import synth

pytestmark = pytest.mark.gpu

N = 15
N3 = (N + 1) ** 3


def operator(f, seed):
    a = synth.face_coefficients_lognormal(N, seed)
    hb.SetupStencilFaces(f, N, 1.0 / (N + 1), *a, np.zeros((N + 2,) * 3))
    f.Factor()


@pytest.fixture()
def factor():
    f = hb.HIFFactor(N, 4, 1e-6)
    operator(f, 3)
    yield f
    f.close()


def vectors(nrhs):
    U = np.stack([synth.dof_vector(N, 10 + c) for c in range(nrhs)])
    return torch.from_numpy(U).cuda()


def apply(f, u, inverse=True):
    v = u.clone()
    torch.cuda.synchronize()
    f.apply_device(v.data_ptr(), v.shape[0], N3, inverse)
    torch.cuda.synchronize()
    return v


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
@pytest.mark.parametrize("nrhs", [1, 3])
@pytest.mark.parametrize("uses", [0, 1, 20])
def test_refused_inside_capture(factor, nrhs, uses):
    f = factor
    s = torch.cuda.Stream()
    hb.set_stream(f, s.cuda_stream)
    u = vectors(nrhs)
    for _ in range(uses):
        apply(f, u)
    v = u.clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="relaxed")
        try:
            with pytest.raises(hb.HIFError) as e:
                f.apply_device(v.data_ptr(), nrhs, N3, True)
        finally:
            g.capture_end()
    assert e.value.code == hb.HIF_ERR_CUDA
    del g
    hb.set_stream(f, 0)
    ref = hb.HIFFactor(N, 4, 1e-6)
    operator(ref, 3)
    assert torch.equal(apply(f, u), apply(ref, u))
    ref.close()


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
@pytest.mark.parametrize("solver", ["solve_pcg_device", "solve_gmres_device"])
def test_solve_refused_inside_capture(factor, solver):
    f = factor
    b, x = vectors(2), torch.zeros(2, N3, dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    hb.set_stream(f, s.cuda_stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="relaxed")
        try:
            with pytest.raises(hb.HIFError) as e:
                getattr(f, solver)(b.data_ptr(), x.data_ptr(), 2, N3, 1e-10, 50)
        finally:
            g.capture_end()
    assert e.value.code == hb.HIF_ERR_CUDA
    del g
    hb.set_stream(f, 0)
    ref = hb.HIFFactor(N, 4, 1e-6)
    operator(ref, 3)
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    its = [getattr(q, solver)(b.data_ptr(), v.data_ptr(), 2, N3, 1e-10, 50)[0].tolist()
           for q, v in ((f, x), (ref, y))]
    torch.cuda.synchronize()
    assert its[0] == its[1] and torch.equal(x, y)
    ref.close()


def test_refused_on_legacy_stream(factor):
    f = factor
    u = vectors(1)
    x = apply(f, u)
    hb.set_stream(f, 1)  # cudaStreamLegacy
    for _ in range(20):
        with pytest.raises(hb.HIFError) as e:
            f.apply_device(u.data_ptr(), 1, N3, True)
        assert e.value.code == hb.HIF_ERR_CUDA
    hb.set_stream(f, 0)
    assert torch.equal(apply(f, vectors(1)), x)


@pytest.mark.parametrize("inverse", [True, False])
@pytest.mark.parametrize("nrhs", [1, 3, 20])
def test_graph_repeats_plain_launches(factor, nrhs, inverse):
    f = factor
    ref = hb.HIFFactor(N, 4, 1e-6)  # applied too seldom to make a graph
    operator(ref, 3)
    u = vectors(nrhs)
    x = apply(ref, u, inverse)
    for _ in range(20):
        assert torch.equal(apply(f, u, inverse), x)
    apply(f, vectors(40), inverse)  # larger work vectors: the graphs are dropped
    for _ in range(20):
        assert torch.equal(apply(f, u, inverse), x)
    operator(f, 4)
    operator(ref, 4)
    y = apply(ref, u, inverse)
    assert not torch.equal(y, x)
    for _ in range(20):
        assert torch.equal(apply(f, u, inverse), y)
    ref.close()
