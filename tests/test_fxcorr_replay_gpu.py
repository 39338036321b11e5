"""A captured in-place correlation gives the out-of-place result on every
replay, not only the first: blocks overlap (many taps, hundreds of blocks), so
a replay that did not wait for its own windows would read overwritten samples.
Bitwise: the two forms do the same arithmetic."""
import numpy as np
import pytest
import torch

from packed_b200 import fxcorr_unit, real_size
from tests._util import normal_cx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n,k,pack", [(torch.float32, 256, 129, 8), (torch.float32, 4096, 3001, 8),
                                            (torch.float32, 8192, 6001, 8), (torch.float32, 16384, 12001, 8),
                                            (torch.float32, 1024, 700, 1), (torch.float64, 1024, 700, 4)])
def test_replays(dtype, n, k, pack):
    channels, length = 4, 100008
    g = normal_cx(np.random.default_rng(n), k, sigma=1 / np.sqrt(k))
    unit = fxcorr_unit(g, n, dtype=dtype)
    x0 = torch.randn(channels * real_size(length, pack), device="cuda", dtype=dtype)
    want = torch.empty_like(x0)
    unit.exec(want, x0, length, channels=channels, pack=pack)
    x = x0.clone()
    unit.exec(x, x, length, channels=channels, pack=pack)    # allocates what the capture needs
    assert torch.equal(x, want)
    st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        unit.exec(x, x, length, channels=channels, pack=pack, stream=st, check=False)
    for i in range(5):
        x.copy_(x0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, want), i
        if i == 2:    # a direct call between two replays
            x.copy_(x0)
            unit.exec(x, x, length, channels=channels, pack=pack)
            assert torch.equal(x, want)
    unit.status()
