"""Short rows are read no further than the caller's storage goes: the copied bytes
at compile time (no GPU), the results of what then comes another way on one."""
import subprocess

import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import build as B
from packed_b200 import fft_order, fft_unit
from tests._util import TOL, normal_cx, rel_l2


def test_copied_bytes(tmp_path):
    src = B.ROOT / "tests" / "cpp" / "short_rows.cu"
    cmd = [B.nvcc(), *B.ARCH, "-std=c++20", "--expt-relaxed-constexpr", f"-I{B.ROOT / 'include'}", f"-I{B.CSRC}", "-c", str(src),
           "-o", str(tmp_path / "short_rows.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("lg", [5, 6, 7, 9, 12])
@pytest.mark.parametrize("order", list(fft_order))
def test_odd_interleaved_rows(lg, order):
    n, rng = 1 << lg, np.random.default_rng(lg)
    unit, pos = fft_unit(n, order=order), O.order_pos(n, int(order))
    for batch, length in ((1, 1), (3, 1), (5, 3), (300, n // 2 + 1), (7, n - 1), (2, n - 2)):
        z = normal_cx(rng, batch, length)
        ss = (2 * length + 3) // 4 * 4
        host = np.full((batch, ss), np.nan, np.float32)
        host[:, 0:2 * length:2], host[:, 1:2 * length:2] = z.real, z.imag
        # the last row ends with its last element
        flat = torch.as_tensor(host.reshape(-1)[: (batch - 1) * ss + 2 * length].copy()).cuda()
        y = torch.full((batch, 2 * n), float("nan"), device="cuda")
        unit.exec(y, flat, batch=batch, pack_src=1, src_len=length, src_stride=ss)
        want = np.empty((batch, n), complex)
        want[:, pos] = np.fft.fft(z.astype(np.complex64).astype(complex), n)
        assert rel_l2(O.unpack(y.cpu().numpy(), n, 8), want) < TOL[np.float32], (batch, length)
