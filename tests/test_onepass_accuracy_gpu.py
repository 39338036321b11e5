"""Error of the one-pass FFT's faster forms against FP64, on the same data as the
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
