"""Error of the faster FFT forms against FP64, on the same data as the
forms that they stand beside: it may be no larger."""
import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import default_pack_size, fft_order, fft_unit, fxcorr_unit

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


@pytest.mark.parametrize("lg", range(7, 13))
@pytest.mark.parametrize("part", [4, 2])
def test_correlators(lg, part, monkeypatch):
    """The whole-window correlator and its signal gradient against the general kernel that ran these
    sizes before it, which has full twiddle tables (0.4 % for the data's chance)."""
    n, channels, length = 1 << lg, 16, 1 << 16
    k, m = n // part, 1 << 17
    rng = np.random.default_rng(lg)
    g = ((rng.standard_normal(k) + 1j * rng.standard_normal(k)) / np.sqrt(2 * k)).astype(np.complex64)
    unit = fxcorr_unit(g, n)
    monkeypatch.setenv("PCX_XC_GENERAL", "1")
    general = fxcorr_unit(g, n)
    x = torch.randn(channels, 2 * length, device="cuda", generator=torch.Generator("cuda").manual_seed(lg))
    spec, gs = torch.fft.fft(_cx(x, length, 8), m), torch.fft.fft(torch.as_tensor(g.astype(complex), device="cuda"), m)
    for want, run in ((torch.fft.ifft(spec * gs.conj()), lambda u, y: u.exec(y, x, length, channels=channels)),
                      (torch.fft.ifft(spec * gs),
                       lambda u, y: y.copy_(u.vjp(x, x, length, channels=channels, want_kernel_grad=False)[0]))):
        want, err = want[:, :length], []
        for u in (unit, general):
            y = torch.empty_like(x)
            run(u, y)
            err.append(((_cx(y, length, 8) - want).norm() / want.norm()).item())
        assert err[0] < 1.004 * err[1], err
