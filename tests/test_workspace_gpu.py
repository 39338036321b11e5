"""A workspace smaller than pcx_plan_workspace_size is refused whichever form a
size above 4096 points runs, and one of that size is taken."""
import ctypes

import numpy as np
import pytest
import torch

from packed_b200 import _lib, fft_unit
from tests._util import TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,lg,ps,refused", [(torch.float32, 13, 8, False), (torch.float32, 13, 1, True),
                                                 (torch.float32, 14, 8, True), (torch.float64, 13, 4, True),
                                                 (torch.float64, 13, 1, True), (torch.float32, 16, 8, True)])
def test_small_workspace(dtype, lg, ps, refused):
    n, batch, lib = 1 << lg, 3, _lib.lib()
    p = 8 if dtype == torch.float32 else 4
    unit = fft_unit(n, dtype=dtype)
    x = torch.randn(batch, 2 * n, device="cuda", dtype=dtype)
    y, ws = torch.full_like(x, float("nan")), torch.empty(1 << 24, dtype=torch.uint8, device="cuda")
    lib.pcx_plan_workspace_size.restype = ctypes.c_size_t
    need = lib.pcx_plan_workspace_size(unit._plan, batch)

    def run(nbytes):
        return lib.pcx_fft_exec_ws(unit._plan, ctypes.c_void_p(y.data_ptr()), ctypes.c_void_p(x.data_ptr()), 0, p, ps, 0, 1,
                                   batch, 2 * n, 2 * n, ctypes.c_void_p(ws.data_ptr()), nbytes,
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))

    assert need <= ws.numel()
    assert (run(256) != 0) == refused
    torch.cuda.synchronize()
    assert torch.isnan(y).all() == refused
    assert run(need) == 0
    f = x.reshape(batch, -1, 2, ps).double()
    want = torch.fft.fft(torch.complex(f[:, :, 0].reshape(batch, n), f[:, :, 1].reshape(batch, n)))
    g = y.reshape(batch, -1, 2, p).double()
    got = torch.complex(g[:, :, 0].reshape(batch, n), g[:, :, 1].reshape(batch, n))
    assert ((got - want).norm() / want.norm()).item() < TOL[np.float32 if dtype == torch.float32 else np.float64]
