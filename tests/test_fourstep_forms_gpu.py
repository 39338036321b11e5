"""The one-launch four-step FFT in its forms for other packs, short sources and
permuted orders, over every size that has them: one transform and an odd
batch, padded strides, in place, and short sources whose last row is empty,
whole or partial (NaN wherever nothing may be read).  Checked against numpy in
double precision with the parity bar (FP32 2e-6, FP64 1e-13 relative L2); the
position of a frequency comes from the oracle."""
import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import fft_order, fft_unit
from tests._util import TOL, normal_cx, rel_l2

pytestmark = pytest.mark.gpu

F32, F64 = torch.float32, torch.float64
# log2 of the row length N2 of each size's default split
ROW = {13: 6, 14: 7, 15: 8, 16: 8, 17: 9, 18: 9, 19: 9, 20: 10}
SIZES = [(F32, lg) for lg in range(13, 21)] + [(F64, lg) for lg in (14, 15, 16, 17, 18, 19, 20)]


def _np(dtype):
    return np.float32 if dtype == F32 else np.float64


def _dev(rows, stride, dtype):
    """Packed rows on the device, `stride` reals apart, NaN between them."""
    host = np.full((rows.shape[0], stride), np.nan, _np(dtype))
    host[:, : rows.shape[1]] = rows
    return torch.as_tensor(host).cuda()


@pytest.mark.parametrize("dtype,lg", SIZES)
@pytest.mark.parametrize("order", [fft_order.bit_reversed, fft_order.unordered])
def test_permuted_orders(dtype, lg, order):
    n, p, npd = 1 << lg, 8 if dtype == F32 else 4, _np(dtype)
    rng = np.random.default_rng(lg)
    unit = fft_unit(n, dtype=dtype, order=order)
    pos = O.order_pos(n, int(order))
    for batch, ps, pd, pad in ((1, p, p, 0), (3, 1, p, 16), (2, p, 1, 0), (5 if lg < 18 else 2, 2, 1, 8)):
        z = normal_cx(rng, batch, n)
        x = _dev(O.pack(z, ps, npd), 2 * n + pad, dtype)
        y = torch.full((batch, 2 * n + pad), float("nan"), dtype=dtype, device="cuda")
        unit.exec(y, x, batch=batch, pack_src=ps, pack_dst=pd, src_stride=2 * n + pad, dst_stride=2 * n + pad)
        want = np.zeros((batch, n), complex)
        want[:, pos] = np.fft.fft(z)
        assert rel_l2(O.unpack(y.cpu().numpy(), n, pd), want) < TOL[npd]
        unit.exec(y, y, batch=batch, direction=1, pack_src=pd, pack_dst=pd, src_stride=2 * n + pad,
                  dst_stride=2 * n + pad)    # in place
        assert rel_l2(O.unpack(y.cpu().numpy(), n, pd), z) < TOL[npd]
        s = _dev(O.pack(want, pd, npd), 2 * n, dtype)
        back = torch.full((batch, 2 * n), float("nan"), dtype=dtype, device="cuda")
        unit.exec(back, s, batch=batch, direction=1, normalize=False, pack_src=pd, pack_dst=ps)
        assert rel_l2(O.unpack(back.cpu().numpy(), n, ps), z * n) < TOL[npd]


@pytest.mark.parametrize("dtype,lg", SIZES)
def test_packs_and_short_sources(dtype, lg):
    n, p, npd, row = 1 << lg, 8 if dtype == F32 else 4, _np(dtype), 1 << ROW[lg]
    rng = np.random.default_rng(100 + lg)
    unit = fft_unit(n, dtype=dtype)
    if dtype == F32 and lg <= 14:    # the one-pass form would take it
        unit.set_tuning("one-launch four-step", split=(128, n // 128), blocks_per_sm=2, stages=3)
    for batch, ps, pd, length in ((1, 1, 1, n), (3, 1, p, n), (2, 2, 2, n), (2, p, 1, n), (1, 1, p, row), (3, 1, p, row + 1),
                                  (2, p, p, n // 2 + 3), (2, 2, 1, n - 1), (1, p, p, row - 1)):
        z = normal_cx(rng, batch, length)
        packed = O.pack(z, ps, npd)
        if length % ps:    # the last pack's places beyond the end hold NaN
            tail = packed[:, -2 * ps:].reshape(batch, 2, ps)
            tail[:, :, length % ps:] = np.nan
        x = _dev(packed, -(-packed.shape[1] // 4) * 4 + 4, dtype)
        y = torch.full((batch, 2 * n), float("nan"), dtype=dtype, device="cuda")
        unit.exec(y, x, batch=batch, pack_src=ps, pack_dst=pd, src_len=length, src_stride=x.shape[1])
        want = np.fft.fft(z, n)
        assert rel_l2(O.unpack(y.cpu().numpy(), n, pd), want) < TOL[npd], (batch, ps, pd, length)
        if length == n:
            unit.exec(y, y, batch=batch, direction=1, pack_src=pd, pack_dst=ps)    # in place, other packs
            assert rel_l2(O.unpack(y.cpu().numpy(), n, ps), z) < TOL[npd], (batch, ps, pd)
