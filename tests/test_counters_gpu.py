"""Counters that launches leave zero for one another start zero whatever becomes
of the first call: one that is only captured and never replayed must leave the
plan or handle usable by direct calls.  FP32 parity bar (2e-6 relative L2)."""
import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import fft_unit, fxcorr_unit, vector
from tests._util import TOL, normal_cx, rel_l2

pytestmark = pytest.mark.gpu
BAR = TOL[np.float32]


def _capture_only(call):
    """Capture `call(stream)` into a graph that is never replayed."""
    # memory that the allocations inside are likely to get back: not zero
    junk = torch.full((1 << 22,), 0x01010101, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    del junk
    torch.cuda.empty_cache()
    st = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
        call(st)
    torch.cuda.synchronize()


@pytest.mark.parametrize("lg", [15, 18])
def test_fourstep_after_an_unused_capture(lg):
    rng = np.random.default_rng(lg)
    z = normal_cx(rng, 3, 1 << lg)
    x = torch.as_tensor(O.pack(z, 8)).cuda()
    y = torch.zeros_like(x)
    unit = fft_unit(1 << lg)
    _capture_only(lambda st: unit.exec(y, x, batch=3, stream=st, check=False))
    for _ in range(2):
        y.zero_()
        unit.exec(y, x, batch=3)
        assert rel_l2(O.unpack(y.cpu().numpy(), 1 << lg, 8), np.fft.fft(z)) < BAR


@pytest.mark.parametrize("n", [256, 4096, 16384])
def test_correlator_after_an_unused_capture(n):
    rng = np.random.default_rng(n)
    length, k = 50000, n // 4 + 1
    z, g = normal_cx(rng, length), normal_cx(rng, k, sigma=1 / np.sqrt(k)).astype(np.complex64)
    x = torch.as_tensor(O.pack(z, 8)).cuda()
    fxcorr_unit.release_idle()
    unit = fxcorr_unit(vector.from_complex(g), n)
    _capture_only(lambda st: unit.exec(x, x, length, stream=st, check=False))
    m = 1 << (length + k).bit_length()
    for _ in range(2):
        y = x.clone()
        torch.cuda.synchronize()
        unit.exec(y, y, length)
        want = np.fft.ifft(np.fft.fft(z, m) * np.conj(np.fft.fft(g.astype(complex), m)))[:length]
        assert rel_l2(O.unpack(y.cpu().numpy(), length, 8), want) < BAR
