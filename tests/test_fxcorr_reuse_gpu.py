"""Correlator handles made one after another reuse the destroyed ones' memory:
each must give its own kernel's results, whatever the last owner left running,
on which stream, of which size or form, and with which error flag; what is kept
is bounded and can be given back.  FP32 parity bar (2e-6 relative L2)."""
import gc
import threading

import numpy as np
import pytest
import torch

import oracle as O
from packed_b200 import fxcorr_unit, vector
from tests._util import TOL, normal_cx, rel_l2

pytestmark = pytest.mark.gpu
BAR = TOL[np.float32]


def _corr(x, g):
    m = 1 << (x.shape[-1] + g.size).bit_length()
    return np.fft.ifft(np.fft.fft(x, m) * np.conj(np.fft.fft(g, m)))[..., : x.shape[-1]]


def _one(rng, k, n, length, stream, unit_out=None):
    z, g = normal_cx(rng, length), normal_cx(rng, k, sigma=1 / np.sqrt(k)).astype(np.complex64)
    x = torch.as_tensor(O.pack(z, 8)).cuda()
    torch.cuda.synchronize()
    unit = fxcorr_unit(vector.from_complex(g), n)
    with torch.cuda.stream(stream):
        unit.exec(x, x, length, stream=stream, check=False)    # still running when the unit goes
    if unit_out is not None:
        unit_out.append(unit)
    return z, g, x


def test_each_owner_gets_its_own_kernel():
    rng = np.random.default_rng(0)
    streams = [torch.cuda.default_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    done = []
    for i in range(24):
        n = (4096, 1024, 4096, 16384, 8192)[i % 5]
        done.append(_one(rng, 17 + 13 * i, n, 60000 + 8 * i, streams[i % 3]))
    torch.cuda.synchronize()
    for z, g, x in done:
        assert rel_l2(O.unpack(x.cpu().numpy(), z.size, 8), _corr(z, g.astype(complex))) < BAR


def test_one_handle_on_two_streams_then_reused():
    rng = np.random.default_rng(1)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    z, g = normal_cx(rng, 200000), normal_cx(rng, 100).astype(np.complex64)
    xs = [torch.as_tensor(O.pack(z, 8)).cuda() for _ in range(2)]
    torch.cuda.synchronize()
    unit = fxcorr_unit(vector.from_complex(g), 1024)
    for x, st in zip(xs, (a, b)):
        y = torch.empty_like(x)
        torch.cuda.synchronize()
        unit.exec(y, x, 200000, stream=st, check=False)
        xs.append(y)
    del unit
    gc.collect()
    later = _one(rng, 300, 1024, 50000, b)
    torch.cuda.synchronize()
    for y in xs[2:]:
        assert rel_l2(O.unpack(y.cpu().numpy(), z.size, 8), _corr(z, g.astype(complex))) < BAR
    assert rel_l2(O.unpack(later[2].cpu().numpy(), later[0].size, 8), _corr(later[0], later[1].astype(complex))) < BAR


def test_threads():
    bad = []

    def work(seed):
        rng, st = np.random.default_rng(seed), torch.cuda.Stream()
        for i in range(8):
            z, g, x = _one(rng, 50 + i, 2048, 30000, st)
            st.synchronize()
            if rel_l2(O.unpack(x.cpu().numpy(), z.size, 8), _corr(z, g.astype(complex))) >= BAR:
                bad.append((seed, i))

    ts = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_kept_memory_is_bounded_and_given_back():
    fxcorr_unit.release_idle()
    g = vector.from_complex(np.ones(9))
    keep = [fxcorr_unit(g, 128) for _ in range(2)]    # whatever the first use loads
    del keep
    fxcorr_unit.release_idle()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    units = [fxcorr_unit(g, 16384) for _ in range(12)]
    del units
    gc.collect()
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] < 80 << 20
    fxcorr_unit.release_idle()
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= 4 << 20
