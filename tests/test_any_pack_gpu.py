"""The one-pass FFT at any pack widths and with short (zero-extended) rows, at
the sizes and lengths where its tiles, rows and copies end: every one-pass
size, widths from interleaved to wider than a thread group, odd batches, rows
of 1, half, odd and all but one elements, with NaN wherever nothing may be
read.  Checked against numpy in double precision; the bar is the parity bar of
the other transforms (FP32 2e-6, FP64 1e-13 relative L2)."""
import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import fft_order, fft_unit
from tests._util import TOL, normal_cx, rel_l2

pytestmark = pytest.mark.gpu


def _stride(n, pack, vec):
    reals = -(-n // pack) * 2 * pack
    return -(-reals // vec) * vec


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("lg", [5, 6, 7, 8, 9, 10, 11, 12, 13, 14])
@pytest.mark.parametrize("ps,pd", [(1, 8), (8, 1), (1, 1), (2, 4), (16, 2), (4, 16)])
def test_widths_and_short_rows(dtype, lg, ps, pd):
    npd = np.float32 if dtype == torch.float32 else np.float64
    if dtype == torch.float64:
        ps, pd = max(1, ps // 2), max(1, pd // 2)    # 4 is the default width
    n, vec = 1 << lg, 16 // np.dtype(npd).itemsize
    rng = np.random.default_rng(lg * 100 + ps * 10 + pd)
    unit = fft_unit(n, dtype=dtype)
    for batch, length in ((1, n), (5, n), (3, 1), (3, n // 2 + 1), (2, n - 1)):
        if length < n and lg > 12 and ps > (8 if npd == np.float32 else 4):
            continue    # refused: no short rows of packs wider than the two-pass kernels'
        ss = _stride(length, ps, vec)
        z = normal_cx(rng, batch, length)
        host = np.full((batch, ss), np.nan, npd)
        for e in range(length):
            o = (e // ps) * 2 * ps + e % ps
            host[:, o], host[:, o + ps] = z[:, e].real, z[:, e].imag
        x = torch.as_tensor(host).cuda()
        y = torch.full((batch, 2 * n), float("nan"), dtype=dtype, device="cuda")
        unit.exec(y, x, batch=batch, pack_dst=pd, pack_src=ps, src_len=length, src_stride=ss)
        want = np.fft.fft(z.astype(np.complex64 if npd == np.float32 else np.complex128).astype(complex), n)
        assert rel_l2(O.unpack(y.cpu().numpy(), n, pd), want) < TOL[npd], (batch, length)
        back = torch.full((batch, 2 * n), float("nan"), dtype=dtype, device="cuda")
        unit.exec(back, y, batch=batch, direction=1, pack_dst=ps, pack_src=pd)
        full = np.zeros((batch, n), complex)
        full[:, :length] = z
        assert rel_l2(O.unpack(back.cpu().numpy(), n, ps), full) < TOL[npd], (batch, length)


@pytest.mark.parametrize("order", [fft_order.bit_reversed, fft_order.unordered])
@pytest.mark.parametrize("lg", [5, 8, 12])
def test_permuted_orders_interleaved(order, lg):
    n, rng = 1 << lg, np.random.default_rng(lg)
    z = normal_cx(rng, 7, n)
    unit, plain = fft_unit(n, order=order), fft_unit(n, order=order)
    x8, x1 = (torch.as_tensor(O.pack(z, p)).cuda() for p in (8, 1))
    y8, y1, back = torch.empty_like(x8), torch.empty_like(x8), torch.empty_like(x8)
    plain.exec(y8, x8, batch=7)    # the default packs: another instantiation
    unit.exec(y1, x1, batch=7, pack_dst=1)
    assert rel_l2(O.unpack(y1.cpu().numpy(), n, 1), O.unpack(y8.cpu().numpy(), n, 8)) < TOL[np.float32]
    unit.exec(back, y1, batch=7, direction=1, pack_dst=1)
    assert rel_l2(O.unpack(back.cpu().numpy(), n, 1), z) < TOL[np.float32]
