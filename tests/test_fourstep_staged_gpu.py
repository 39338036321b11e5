"""The one-launch four-step FFT with its outputs staged in shared memory and
stored by TMA, which batches of at least 12 tiles a block take: batches just
above that line, for every size and form that has the kernel (plain, other
packs, short sources, into and out of permuted orders), in place and into rows
with gaps, which stay untouched.  Every row against FP64 on the device, parity
bar (FP32 2e-6, FP64 1e-13 relative L2), and against the register-stored kernel
that half the batch takes."""
import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import fft_order, fft_unit
from tests._util import TOL

pytestmark = pytest.mark.gpu

F32, F64 = torch.float32, torch.float64
# log2 N: (log2 N1, log2 N2, blocks per SM) of the default split
SPLIT = {(F32, 17): (8, 9, 2), (F32, 18): (9, 9, 2), (F32, 19): (10, 9, 1), (F32, 20): (10, 10, 1),
         (F64, 14): (7, 7, 2), (F64, 15): (8, 7, 2), (F64, 16): (8, 8, 2), (F64, 17): (9, 8, 2), (F64, 18): (9, 9, 2)}
SIZES = sorted(SPLIT, key=str)
# the autotuner's other FP32 variants with the kernel
VARIANTS = [(6, 9, 2), (7, 9, 2), (9, 7, 2), (6, 10, 1), (9, 8, 2), (10, 7, 1), (9, 8, 1), (7, 10, 1), (8, 10, 1),
            (10, 8, 1), (9, 9, 1), (9, 10, 1)]


def _batch(dtype, split):
    """Transforms from which a launch has 12 tiles a block or more."""
    l1, l2, per_sm = split
    eb = 8 if dtype == F32 else 16
    tile, least = 65536 // per_sm // eb, 64 // eb
    tiles = (1 << l2) // max(tile >> l1, least) + (1 << l1) // max(tile >> l2, least)
    blocks = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    return -(-12 * blocks // tiles)


def _cx(t, n, p):
    """Complex128 [rows, n] of packed rows."""
    f = t[:, : -(-n // p) * 2 * p].reshape(t.shape[0], -1, 2, p).double()
    return torch.complex(f[:, :, 0].reshape(t.shape[0], -1), f[:, :, 1].reshape(t.shape[0], -1))[:, :n]


def _worst(got, want):
    """Largest relative error of a row (NaN counts as infinite)."""
    e = [((g - w).norm() / w.norm()).item() for g, w in zip(got, want)]
    return max(v if v == v else float("inf") for v in e)


def _nan(rows, stride, dtype):
    return torch.full((rows, stride), float("nan"), dtype=dtype, device="cuda")


def _check(unit, dtype, lg, ps, pd, want_of, length=None, inverse=0, pad=0, in_place=False, split=None):
    n, tol = 1 << lg, TOL[np.float32 if dtype == F32 else np.float64]
    b, length = _batch(dtype, split or SPLIT[dtype, lg]) + 1, length or n
    ss = (-(-length // ps) * 2 * ps + 3) // 4 * 4 + pad
    ds = 2 * n + pad
    x = torch.randn(b, ss, dtype=dtype, device="cuda")
    want = want_of(_cx(x, length, ps))
    y = x.clone() if in_place else _nan(b, ds, dtype)
    kw = dict(direction=inverse, normalize=True, pack_src=ps, pack_dst=pd, src_len=length, src_stride=ss, dst_stride=ds)
    unit.exec(y, y if in_place else x, batch=b, **kw)
    assert _worst(_cx(y, n, pd), want) < tol
    if pad and not in_place:
        assert torch.isnan(y[:, 2 * n:]).all()
    half = _nan(b, ds, dtype)
    for r in range(0, b, b // 2):    # short batches: outputs from registers
        m = min(b // 2, b - r)
        unit.exec(half[r:r + m], x[r:r + m], batch=m, **kw)
    assert _worst(_cx(y, n, pd), _cx(half, n, pd)) < tol


@pytest.mark.parametrize("dtype,lg", SIZES)
def test_natural_order(dtype, lg):
    n, p, unit = 1 << lg, 8 if dtype == F32 else 4, fft_unit(1 << lg, dtype=dtype)
    row = 1 << SPLIT[dtype, lg][1]

    def fwd(z):
        return torch.fft.fft(z, n)

    for ps, pd, kw in ((p, p, {}), (p, p, dict(pad=16)), (p, p, dict(in_place=True)), (1, p, dict(pad=8)), (p, 1, {}),
                       (2, 2, dict(in_place=True)), (1, 1, dict(length=n // 2 + 3)), (p, p, dict(length=row)),
                       (p, 2, dict(length=n - 1, pad=16))):
        _check(unit, dtype, lg, ps, pd, fwd, **kw)
    for ps, pd, kw in ((p, p, {}), (p, 1, dict(in_place=True)), (2, p, dict(pad=16))):
        _check(unit, dtype, lg, ps, pd, torch.fft.ifft, inverse=1, **kw)


@pytest.mark.parametrize("dtype,lg", SIZES)
@pytest.mark.parametrize("order", [fft_order.bit_reversed, fft_order.unordered])
def test_permuted_orders(dtype, lg, order):
    n, p, unit = 1 << lg, 8 if dtype == F32 else 4, fft_unit(1 << lg, dtype=dtype, order=order)
    pos = torch.as_tensor(np.asarray(O.order_pos(n, int(order))).astype(np.int64), device="cuda")

    def fwd(z):
        out = torch.empty(z.shape[0], n, dtype=torch.complex128, device="cuda")
        out[:, pos] = torch.fft.fft(z, n)
        return out

    def inv(z):
        return torch.fft.ifft(z[:, pos])

    for ps, pd, kw in ((p, p, {}), (1, p, dict(pad=16)), (p, 1, dict(in_place=True)), (2, p, dict(length=n // 2 + 3))):
        _check(unit, dtype, lg, ps, pd, fwd, **kw)
    for ps, pd, kw in ((p, p, {}), (1, 1, dict(in_place=True)), (p, 2, dict(pad=16))):
        _check(unit, dtype, lg, ps, pd, inv, inverse=1, **kw)


@pytest.mark.parametrize("l1,l2,per_sm", VARIANTS)
def test_variants(l1, l2, per_sm):
    unit = fft_unit(1 << (l1 + l2))
    unit.set_tuning("one-launch four-step", split=(1 << l1, 1 << l2), blocks_per_sm=per_sm, stages=3)
    for kw in ({}, dict(in_place=True), dict(pad=16)):
        _check(unit, F32, l1 + l2, 8, 8, torch.fft.fft, split=(l1, l2, per_sm), **kw)
