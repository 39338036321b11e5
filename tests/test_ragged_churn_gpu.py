"""Ragged batches made, run many times back to back and destroyed one after
another, single-pass, four-step and correlation items following each other in
every block's ring: no item may see another's destination or length, and no
batch another's tensor maps.  Against FP64 on the device, FP32 parity bar."""
import numpy as np
import pytest
import torch

from packed_b200 import ragged_batch, vector
from tests._util import TOL, normal_cx

pytestmark = pytest.mark.gpu
BAR = TOL[np.float32]


def _cx(t):
    t = t.reshape(-1, 2, 8).double()
    return torch.complex(t[:, 0].reshape(-1), t[:, 1].reshape(-1))


def _bad(got, want):
    return ((got - want).norm() / want.norm()).item() >= BAR


@pytest.mark.parametrize("seed", range(4))
def test_churn(seed):
    rng = np.random.default_rng(seed)
    for _ in range(6):
        ffts, xcorrs, gs = [], [], []
        for _ in range(40):
            n = 1 << int(rng.integers(5, 17))
            x = torch.randn(2 * n, device="cuda")
            ffts.append((torch.zeros_like(x), x, n))
        for _ in range(12):
            length, k = int(rng.integers(600, 6000)) * 8, int(rng.integers(16, 1000))
            nf = 1 << int(rng.integers((2 * k).bit_length(), 15))
            g = normal_cx(rng, k, sigma=1 / np.sqrt(k)).astype(np.complex64)
            x = torch.randn(2 * length, device="cuda")
            xcorrs.append((torch.zeros_like(x), x, length, vector.from_complex(g), max(nf, 128)))
            gs.append(torch.as_tensor(g.astype(complex), device="cuda"))
        batch = ragged_batch(ffts, xcorrs)
        for _ in range(50):
            batch()
        torch.cuda.synchronize()
        batch.status()
        for y, x, n in ffts:
            assert not _bad(_cx(y), torch.fft.fft(_cx(x))), n
        for (y, x, length, _, nf), g in zip(xcorrs, gs):
            m = 1 << (length + g.numel()).bit_length()
            want = torch.fft.ifft(torch.fft.fft(_cx(x), m) * torch.fft.fft(g, m).conj())[:length]
            assert not _bad(_cx(y), want), (length, nf)
