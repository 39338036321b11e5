"""The whole-window correlator (FP32, up to 2^12 points, pack 8) and its adjoint
at the sizes where its tiles, windows and waits end: every FFT size, one tap to
all but seven of the block (steps of 8 outputs: hundreds of blocks overlap),
signals of one sample, around one block and around one tile of blocks, one and
several channels with padded rows, in place and out of place.  NaN fills what
must not be read or written.  Checked against FP64 sums by numpy's FFT with the
FP32 parity bar (2e-6 relative L2), and against the general kernel."""
import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import fxcorr_unit, vector
from tests._util import TOL, normal_cx, rel_l2

pytestmark = pytest.mark.gpu
BAR = TOL[np.float32]


def _corr(x, g):
    m = 1 << (x.shape[-1] + g.size).bit_length()
    return np.fft.ifft(np.fft.fft(x, m) * np.conj(np.fft.fft(g, m)))[..., : x.shape[-1]]


def _conv(x, g):
    m = 1 << (x.shape[-1] + g.size).bit_length()
    return np.fft.ifft(np.fft.fft(x, m) * np.fft.fft(g, m))[..., : x.shape[-1]]


def _cases(lg):
    n = 1 << lg
    tile = 4096 // n    # windows per tile
    for k in sorted({1, n // 8 + 3, n // 2, n - 7}):
        step = (n - (k - 1)) // 8 * 8
        lengths = {1, step - 1, step, step + 1, n, tile * step + 1, 3 * tile * step - 5}
        for length in sorted(v for v in lengths if 0 < v <= 40000):
            yield k, step, length


@pytest.mark.parametrize("lg", range(6, 13))
def test_forward(lg):
    n = 1 << lg
    rng = np.random.default_rng(lg)
    for k, step, length in _cases(lg):
        g = normal_cx(rng, k, sigma=1 / np.sqrt(k)).astype(np.complex64)
        unit = fxcorr_unit(vector.from_complex(g), n)
        for channels, pad in ((1, 0), (3, 8)):
            z = normal_cx(rng, channels, length).astype(np.complex64)
            want = _corr(z.astype(complex), g.astype(complex))
            packed = O.pack(z, 8)
            if length % 8:    # the places of the last pack beyond the signal
                packed[:, -16:].reshape(channels, 2, 8)[:, :, length % 8:] = np.nan
            x = torch.full((channels, packed.shape[1] + pad), float("nan"), device="cuda")
            x[:, : packed.shape[1]] = torch.as_tensor(packed).cuda()
            y = torch.full_like(x, float("nan"))
            unit.exec(y, x, length, channels=channels, src_stride=x.shape[1], dst_stride=x.shape[1])
            got = y.cpu().numpy()
            assert rel_l2(O.unpack(got, length, 8), want) < BAR, (k, length, channels)
            assert np.isnan(got).sum() == got.size - 2 * channels * length, (k, length, channels)
            unit.exec(x, x, length, channels=channels, src_stride=x.shape[1], dst_stride=x.shape[1])
            assert np.array_equal(O.unpack(x.cpu().numpy(), length, 8), O.unpack(got, length, 8)), (k, length, channels)


@pytest.mark.parametrize("lg", range(6, 13))
def test_adjoint(lg, monkeypatch):
    n = 1 << lg
    rng = np.random.default_rng(50 + lg)
    for k, step, length in _cases(lg):
        g = normal_cx(rng, k, sigma=1 / np.sqrt(k)).astype(np.complex64)
        unit = fxcorr_unit(vector.from_complex(g), n)
        monkeypatch.setenv("PCX_XC_GENERAL", "1")
        general = fxcorr_unit(vector.from_complex(g), n)
        monkeypatch.delenv("PCX_XC_GENERAL")
        for channels in (1, 2):
            z, w = (normal_cx(rng, channels, length).astype(np.complex64) for _ in range(2))
            xs, ws = (torch.as_tensor(O.pack(v, 8)).cuda() for v in (z, w))
            gx, gg = unit.vjp(ws, xs, length, channels=channels)
            gx2, gg2 = general.vjp(ws, xs, length, channels=channels)
            want_x = _conv(w.astype(complex), g.astype(complex))
            corr = sum(np.fft.ifft(np.fft.fft(z[c].astype(complex), 1 << (length + k).bit_length())
                                   * np.conj(np.fft.fft(w[c].astype(complex), 1 << (length + k).bit_length())))[:k]
                       for c in range(channels))
            assert rel_l2(O.unpack(gx.cpu().numpy().reshape(channels, -1), length, 8), want_x) < BAR, (k, length)
            got, old = (O.unpack(v.cpu().numpy(), k, 8) for v in (gg, gg2))
            # a short gradient is a sum of few products, its zeros the FFT's
            # rounding of the whole block: both forms are held to the block's energy
            scale = np.linalg.norm(z) * np.linalg.norm(w) / max(np.linalg.norm(corr), 1e-30)
            assert rel_l2(got, corr) < BAR * max(1.0, scale), (k, length, channels)
            assert rel_l2(got, old) < 2 * BAR * max(1.0, scale), (k, length, channels)
            assert rel_l2(O.unpack(gx2.cpu().numpy().reshape(channels, -1), length, 8), want_x) < BAR, (k, length)
        unit.status()
