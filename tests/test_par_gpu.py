"""Transforms across vectors: every size of the one-pass kernel and the first
beyond it, lengths at the ends of a block's positions, other packs, orders,
both types, in place, and vectors that overlap so that the one-pass kernel may
not run.  Checked against numpy in double precision with the parity bar (FP32
2e-6, FP64 1e-13 relative L2)."""
import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import fft_order, fft_unit_par, real_size, vector
from tests._util import TOL, normal_cx, rel_l2

pytestmark = pytest.mark.gpu


def _vectors(z, pack, dtype):
    npd = np.float32 if dtype == torch.float32 else np.float64
    rows = torch.as_tensor(O.pack(z, pack, npd)).cuda()
    return [vector(z.shape[1], dtype, pack, data=r) for r in rows]


def _values(vs):
    return np.stack([v.to_complex() for v in vs])


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("lg", range(1, 12))
def test_sizes_lengths_packs_orders(dtype, lg):
    n, tol = 1 << lg, TOL[np.float32 if dtype == torch.float32 else np.float64]
    block = max(8, 256 // max(1, n // 16))
    rng = np.random.default_rng(lg)
    cases = [(1, 8, 8, 0), (block - 1, 8, 4, 0), (block, 1, 8, 0), (2 * block + 3, 16, 1, 0), (block + 1, 8, 8, 1)]
    if n >= 16:
        cases.append((block + 5, 4, 4, 2))
    for length, ps, pd, order in cases:
        z = normal_cx(rng, n, length)
        unit = fft_unit_par(n, dtype=dtype, order=fft_order(order))
        src = _vectors(z, ps, dtype)
        dst = [vector(length, dtype, pd) for _ in range(n)]
        unit(dst, src)
        want = np.empty((n, length), complex)
        want[O.order_pos(n, order) if order else np.arange(n)] = np.fft.fft(z, axis=0)
        assert rel_l2(_values(dst), want) < tol, (length, ps, pd, order)
        unit(dst, dst, inverse=True)    # in place
        assert rel_l2(_values(dst), z) < tol, (length, ps, pd, order)
        for v in dst:    # nothing beyond the elements is written
            assert v.to_complex().size == length and v.data.numel() == real_size(length, pd)


@pytest.mark.parametrize("n,length,pack", [(64, 100, 8), (1024, 40, 16), (16, 300, 4)])
def test_overlapping_vectors(n, length, pack):
    rng = np.random.default_rng(n)
    z = normal_cx(rng, n, length)
    want = np.fft.fft(z, axis=0)
    unit = fft_unit_par(n)
    vs = _vectors(z, pack, torch.float32)    # outputs into the inputs' storage in another order
    unit(vs[::-1], vs)
    assert rel_l2(_values(vs[::-1]), want) < TOL[np.float32]
    vs = _vectors(z, pack, torch.float32)    # outputs one vector further on
    room = torch.zeros((n + 1, real_size(length, pack)), device="cuda")
    room[:n] = torch.stack([v.data for v in vs])
    src = [vector(length, torch.float32, pack, data=r) for r in room[:n]]
    dst = [vector(length, torch.float32, pack, data=r) for r in room[1:]]
    unit(dst, src)
    assert rel_l2(_values(dst), want) < TOL[np.float32]
    # in place from one pack width to another, wider than the block's positions at 1024 points
    vs = _vectors(z, pack, torch.float32)
    out = [vector(length, torch.float32, 1, data=v.data) for v in vs]
    unit(out, vs)
    assert rel_l2(_values(out), want) < TOL[np.float32]
