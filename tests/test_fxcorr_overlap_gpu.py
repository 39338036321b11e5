"""Out-of-place correlations of one handle that overlap on two streams, of
different lengths (and so different grids), each give the result of a call on
its own, and so do the calls after them.  Bitwise."""
import numpy as np
import pytest
import torch

from packed_b200 import fxcorr_unit, real_size
from tests._util import normal_cx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n,pack", [(torch.float32, 1024, 8), (torch.float32, 8192, 8), (torch.float32, 16384, 8),
                                          (torch.float32, 1024, 1), (torch.float64, 1024, 4), (torch.float64, 8192, 4)])
def test_overlapping_calls(dtype, n, pack):
    k = n // 4
    unit = fxcorr_unit(normal_cx(np.random.default_rng(n), k, sigma=1 / np.sqrt(k)), n, dtype=dtype)
    sizes = [(16, 200000), (1, 3 * n)]    # fills the device; a few blocks
    xs = [torch.randn(c * real_size(m, pack), device="cuda", dtype=dtype) for c, m in sizes]
    want = [torch.empty_like(x) for x in xs]
    for x, y, (c, m) in zip(xs, want, sizes):
        unit.exec(y, x, m, channels=c, pack=pack)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[torch.full_like(x, float("nan")) for _ in range(6)] for x in xs]
    torch.cuda.synchronize()
    for i in range(6):
        for x, ys, (c, m), st in zip(xs, got, sizes, streams):
            unit.exec(ys[i], x, m, channels=c, pack=pack, stream=st, check=False)
    torch.cuda.synchronize()
    for ys, w in zip(got, want):
        for y in ys:
            assert torch.equal(y, w)
    for x, w, (c, m) in zip(xs, want, sizes):    # the handle is as it was
        y = torch.full_like(x, float("nan"))
        unit.exec(y, x, m, channels=c, pack=pack)
        assert torch.equal(y, w)
    unit.status()
