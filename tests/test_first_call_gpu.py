"""What the first call of a plan or correlator may still allocate: the scratch
of a four-step transform, the tables of its other forms and the flags of an
in-place correlation, nothing to zero and wait for.  A first call, and one of a batch above what the counters
were made for, give the results of the calls after them."""
import numpy as np
import pytest
import torch

from packed_b200 import fft_unit, fxcorr_unit
from tests._util import TOL, normal_cx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 4096, 16384])
def test_out_of_place_correlation_allocates_nothing(n):
    x = torch.randn(2 * 30000, device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    units = [fxcorr_unit(normal_cx(np.random.default_rng(i), n // 4), n) for i in range(8)]
    st, graphs = torch.cuda.Stream(), [torch.cuda.CUDAGraph() for _ in units]
    for unit, graph in zip(units, graphs):
        # the strictest capture refuses any allocation by the call
        with torch.cuda.graph(graph, stream=st, capture_error_mode="global"):
            unit.exec(y, x, 30000, stream=st, check=False)
        got = torch.empty_like(y)
        graph.replay()
        torch.cuda.synchronize()
        got.copy_(y)
        unit.exec(y, x, 30000)
        assert torch.equal(got, y)


def test_larger_batch_allocates_nothing():
    lg, n = 16, 1 << 16
    x = torch.randn(500, 2 * n, device="cuda")
    y, want = torch.zeros_like(x), torch.zeros_like(x)
    unit = fft_unit(n)
    unit.exec(y, x, batch=100)    # as much scratch as any batch of this size takes
    st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st, capture_error_mode="global"):
        unit.exec(y, x, batch=500, stream=st, check=False)
    graph.replay()
    unit.exec(want, x, batch=500)
    assert torch.equal(y, want)


@pytest.mark.parametrize("lg", [15, 20])
def test_first_call_of_another_pack_captured(lg):
    """The tables of the four-step's other forms are made by their first call; one that is being
    captured, where nothing may be allocated, does without them."""
    n, batch = 1 << lg, 3
    x = torch.randn(batch, 2 * n, device="cuda")
    y, direct = torch.zeros_like(x), torch.zeros_like(x)
    unit = fft_unit(n)
    unit.exec(y, x, batch=batch)    # the scratch is there
    st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st, capture_error_mode="global"):
        unit.exec(y, x, batch=batch, pack_src=1, stream=st, check=False)
    want = torch.fft.fft(torch.complex(*x.reshape(batch, n, 2).double().unbind(2)))
    for _ in range(2):
        y.fill_(float("nan"))
        graph.replay()
        unit.exec(direct, x, batch=batch, pack_src=1)
        for out in (y, direct):
            f = out.reshape(batch, -1, 2, 8).double()
            got = torch.complex(f[:, :, 0].reshape(batch, n), f[:, :, 1].reshape(batch, n))
            assert ((got - want).norm() / want.norm()).item() < TOL[np.float32]


def test_more_transforms_than_the_counters_were_made_for():
    lg, dtype = 14, torch.float64
    n, unit = 1 << lg, fft_unit(1 << lg, dtype=dtype)
    for batch in (3, 5000, 9000, 2):    # 4096 at creation, then twice what was asked for
        x = torch.randn(batch, 2 * n, dtype=dtype, device="cuda")
        y = torch.full_like(x, float("nan"))
        unit.exec(y, x, batch=batch)
        for i in {0, batch // 2, batch - 1}:
            z, w = (torch.complex(*v[i].reshape(-1, 2, 4).unbind(1)).reshape(-1) for v in (x, y))
            want = torch.fft.fft(z)
            assert ((w - want).norm() / want.norm()).item() < TOL[np.float64], (batch, i)
        del x, y
