"""A correlator reads its kernel after whatever writes it, on any stream: made
with no synchronisation from reused memory, behind long work and a write of the
kernel on a side stream, it must hold the new kernel.  FP32 parity bar (2e-6
relative L2)."""
import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import fxcorr_unit, vector
from packed_b200.autograd import FxcorrFunction
from tests._util import TOL, normal_cx, rel_l2

pytestmark = pytest.mark.gpu
BAR = TOL[np.float32]
DELAY = 100_000_000    # cycles (about 50 ms) that the side stream is busy before the write


def _corr(x, g):
    m = 1 << (x.size + g.size).bit_length()
    return np.fft.ifft(np.fft.fft(x, m) * np.conj(np.fft.fft(g, m)))[: x.size]


@pytest.mark.parametrize("n,k", [(256, 50), (4096, 500), (16384, 4000)])
@pytest.mark.parametrize("warm", [False, True])
def test_kernel_written_on_a_side_stream(n, k, warm):
    rng = np.random.default_rng(n)
    z, old, new = normal_cx(rng, 20000), normal_cx(rng, k), normal_cx(rng, k)
    x = torch.as_tensor(O.pack(z, 8)).cuda()
    g, g_new = (torch.as_tensor(O.pack(v, 8)).cuda() for v in (old, new))
    fxcorr_unit.release_idle()
    if warm:
        for _ in range(2):
            unit = fxcorr_unit(vector(k, torch.float32, 8, data=g), n)
            unit.exec(torch.empty_like(x), x, z.size)
            del unit
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        torch.cuda._sleep(DELAY)
        g.copy_(g_new)
        unit = fxcorr_unit(vector(k, torch.float32, 8, data=g), n)
        y = torch.empty_like(x)
        unit.exec(y, x, z.size)
    assert rel_l2(O.unpack(y.cpu().numpy(), z.size, 8), _corr(z, new.astype(np.complex64).astype(complex))) < BAR


def test_training_loop_on_a_side_stream():
    rng = np.random.default_rng(1)
    n, k, length = 1024, 100, 20000
    z = normal_cx(rng, length)
    x = torch.as_tensor(O.pack(z, 8)).cuda()
    g = torch.as_tensor(O.pack(normal_cx(rng, k), 8)).cuda().requires_grad_(True)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        for _ in range(4):
            y = FxcorrFunction.apply(x, g, n, length, k, 1)
            want = _corr(z, O.unpack(g.detach().cpu().numpy(), k, 8))
            assert rel_l2(O.unpack(y.detach().cpu().numpy(), length, 8), want) < BAR
            g.grad = None
            y.backward(torch.ones_like(y))
            torch.cuda._sleep(DELAY)
            with torch.no_grad():
                g.sub_(1e-5 * g.grad)    # still queued when the next step makes its correlator
    torch.cuda.synchronize()    # the last write is done before its memory is given back
