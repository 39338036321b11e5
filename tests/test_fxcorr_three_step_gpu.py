"""The three-step correlator (FP32, 2^13 and 2^14 points, pack 8) and its adjoint
at the sizes where its windows, copies and waits end: one tap to all but seven
of the block, signals of one sample, around one block, several blocks and
partial packs, one and several channels with padded rows, in place and out of
place.  NaN fills what must not be read or written.  Checked against FP64 sums
by numpy's FFT with the FP32 parity bar (2e-6 relative L2), and against the
general kernel."""
import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import fxcorr_unit, vector
from tests._util import TOL, normal_cx, rel_l2

pytestmark = pytest.mark.gpu
BAR = TOL[np.float32]


def _spec(x, m):
    return np.fft.fft(x.astype(complex), m)


def _cases(lg):
    n = 1 << lg
    for k in (1, n // 4, n // 2 + 5, n - 7):
        step = (n - (k - 1)) // 8 * 8
        for length in sorted({1, step - 3, step, step + 1, n + 9, 3 * step + 13} | ({60000} if step > 100 else set())):
            if 0 < length <= 70000:
                yield k, length


@pytest.mark.parametrize("lg", [13, 14])
def test_forward(lg):
    n, rng = 1 << lg, np.random.default_rng(lg)
    for k, length in _cases(lg):
        g = normal_cx(rng, k, sigma=1 / np.sqrt(k)).astype(np.complex64)
        unit = fxcorr_unit(vector.from_complex(g), n)
        m = 1 << (length + k).bit_length()
        for channels, pad in ((1, 0), (3, 8)):
            z = normal_cx(rng, channels, length).astype(np.complex64)
            want = np.fft.ifft(_spec(z, m) * np.conj(_spec(g, m)))[:, :length]
            packed = O.pack(z, 8)
            if length % 8:
                packed[:, -16:].reshape(channels, 2, 8)[:, :, length % 8:] = np.nan
            x = torch.full((channels, packed.shape[1] + pad), float("nan"), device="cuda")
            x[:, : packed.shape[1]] = torch.as_tensor(packed).cuda()
            y = torch.full_like(x, float("nan"))
            kw = dict(channels=channels, src_stride=x.shape[1], dst_stride=x.shape[1])
            unit.exec(y, x, length, **kw)
            got = y.cpu().numpy()
            assert rel_l2(O.unpack(got, length, 8), want) < BAR, (k, length, channels)
            assert np.isnan(got).sum() == got.size - 2 * channels * length, (k, length, channels)
            unit.exec(x, x, length, **kw)
            assert np.array_equal(O.unpack(x.cpu().numpy(), length, 8), O.unpack(got, length, 8)), (k, length, channels)


@pytest.mark.parametrize("lg", [13, 14])
def test_adjoint(lg, monkeypatch):
    n, rng = 1 << lg, np.random.default_rng(50 + lg)
    for k, length in _cases(lg):
        g = normal_cx(rng, k, sigma=1 / np.sqrt(k)).astype(np.complex64)
        unit = fxcorr_unit(vector.from_complex(g), n)
        monkeypatch.setenv("PCX_XC_GENERAL", "1")
        general = fxcorr_unit(vector.from_complex(g), n)
        monkeypatch.delenv("PCX_XC_GENERAL")
        m = 1 << (length + k).bit_length()
        for channels in (1, 2):
            z, w = (normal_cx(rng, channels, length).astype(np.complex64) for _ in range(2))
            xs, ws = (torch.as_tensor(O.pack(v, 8)).cuda() for v in (z, w))
            gx, gg = unit.vjp(ws, xs, length, channels=channels)
            _, gg2 = general.vjp(ws, xs, length, channels=channels, want_signal_grad=False)
            want_x = np.fft.ifft(_spec(w, m) * _spec(g, m))[:, :length]
            corr = np.fft.ifft((_spec(z, m) * np.conj(_spec(w, m))).sum(0))[:k]
            assert rel_l2(O.unpack(gx.cpu().numpy().reshape(channels, -1), length, 8), want_x) < BAR, (k, length)
            # a gradient of few products is held to the rounding of the whole block
            scale = max(1.0, np.linalg.norm(z) * np.linalg.norm(w) / max(np.linalg.norm(corr), 1e-30))
            got, old = (O.unpack(v.cpu().numpy(), k, 8) for v in (gg, gg2))
            assert rel_l2(got, corr) < BAR * scale, (k, length, channels)
            assert rel_l2(got, old) < 2 * BAR * scale, (k, length, channels)
        unit.status()
