"""Error of the faster FFT forms against FP64, on the same data as the
forms that they stand beside: it may be no larger."""
import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import default_pack_size, fft_order, fft_unit

pytestmark = pytest.mark.gpu

F32, F64 = torch.float32, torch.float64


def _cx(t, n, p):
    f = t.reshape(t.shape[0], -1, 2, p).double()
    return torch.complex(f[:, :, 0].reshape(-1, n), f[:, :, 1].reshape(-1, n))


def _error(unit, x, n, ps, pd, pos=None):
    y = torch.empty_like(x)
    unit.exec(y, x, batch=x.shape[0], pack_src=ps, pack_dst=pd)
    want, got = torch.fft.fft(_cx(x, n, ps)), _cx(y, n, pd)
    if pos is not None:    # frequency k is at position pos[k]
        got = got[:, pos]
    return ((got - want).norm() / want.norm()).item()


@pytest.mark.parametrize("lg", [9, 10, 13])
def test_radix_32_stages(lg):
    """32 points a thread against 16 (which the permuted orders run)."""
    n = 1 << lg
    x = torch.randn((1 << 22) >> lg, 2 * n, device="cuda", generator=torch.Generator("cuda").manual_seed(lg))
    pos = torch.as_tensor(np.asarray(O.order_pos(n, 1)).astype(np.int64), device="cuda")
    wide = _error(fft_unit(n), x, n, 8, 8)
    assert wide <= _error(fft_unit(n, order=fft_order.bit_reversed), x, n, 8, 8, pos)


@pytest.mark.parametrize("dtype,lg", [(F32, lg) for lg in range(7, 14)] + [(F64, lg) for lg in range(7, 13)])
@pytest.mark.parametrize("order", [fft_order.normal, fft_order.unordered])
def test_other_packs(dtype, lg, order):
    """Packs other than the default have full twiddle tables, as the general kernel had: a
    smaller error than the default pack's, whose twiddles are products."""
    n, p = 1 << lg, default_pack_size(dtype)
    pos = torch.as_tensor(np.asarray(O.order_pos(n, int(order))).astype(np.int64), device="cuda")
    x = torch.randn((1 << 21) >> lg, 2 * n, device="cuda", dtype=dtype, generator=torch.Generator("cuda").manual_seed(lg))
    xp = x.reshape(x.shape[0], -1, 2, p).transpose(2, 3).reshape(x.shape).contiguous()    # the same elements interleaved
    unit = fft_unit(n, dtype=dtype, order=order)
    plain = _error(unit, x, n, p, p, pos)
    for ps, pd in ((1, p), (p, 1), (1, 1)):
        assert _error(unit, xp if ps == 1 else x, n, ps, pd, pos) < 0.998 * plain, (ps, pd)


@pytest.mark.parametrize("lg", range(15, 21))
@pytest.mark.parametrize("order", [fft_order.normal, fft_order.unordered])
def test_fourstep_forms(lg, order, monkeypatch):
    """The one-launch four-step's forms against the general two-launch kernels, whose twiddles are
    one entry or the product of two (0.4 % for the data's chance)."""
    n = 1 << lg
    pos = torch.as_tensor(np.asarray(O.order_pos(n, int(order))).astype(np.int64), device="cuda")
    x = torch.randn((1 << 22) >> lg, 2 * n, device="cuda", generator=torch.Generator("cuda").manual_seed(lg))
    unit = fft_unit(n, order=order)
    one = _error(unit, x, n, 1, 1, pos)
    monkeypatch.setenv("PCX_FOURSTEP", "chunked")
    assert one < 1.004 * _error(unit, x, n, 1, 1, pos)
