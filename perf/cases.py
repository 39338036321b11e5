"""Workloads of the FFT / correlation framework, one per way that it is used.

Every case goes through the package's public entry points.  Data are packed
split-complex reals: at pack width P, element i of a row has its real part at
``i + (i // P) * P`` and its imaginary part P reals further (P = 1 is plain
interleaved complex).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import packed_b200 as pb
from packed_b200.autograd import FxcorrFunction

DEV = "cuda"
KINDS = {"f32": torch.float32, "f64": torch.float64}
ORDERS = {"normal": 0, "bit_reversed": 1, "unordered": 2}


def listed():
    return [
        # A few short transforms there and back (a filter step on a small frame):
        # launches and latency are all there is.
        {"name": "frames_1024", "kind": "roundtrip", "dtype": "f32", "order": "normal", "n": 1024, "batch": 64},
        # The spectrogram kind of batch: very many short transforms.
        {"name": "batch_256", "kind": "forward", "dtype": "f32", "n": 256, "batch": 262144},
        # Middle sizes beyond what one block's shared memory transforms in one
        # pass, an odd batch.
        {"name": "batch_65536", "kind": "forward", "dtype": "f32", "n": 65536, "batch": 511},
        # The largest transforms, normalised inverse.
        {"name": "inverse_1m", "kind": "inverse", "dtype": "f32", "n": 1 << 20, "batch": 33},
        # Double precision.
        {"name": "double_4096", "kind": "forward", "dtype": "f64", "n": 4096, "batch": 2001},
        # To the frequency domain and back with no interest in the order there
        # (fast convolution): the reference's `unordered` plans.
        {"name": "unordered_32768", "kind": "roundtrip", "dtype": "f32", "order": "unordered", "n": 32768,
         "batch": 301},
        # Samples as they come (interleaved std::complex, a row shorter than the
        # transform: zero-extended) into packed spectra, and packed spectra back
        # into interleaved samples.
        {"name": "interleaved_2048", "kind": "convert", "dtype": "f32", "n": 2048, "length": 1500, "batch": 5003},
        # Long signals filtered in place by overlap-save (pulse compression with
        # a chirp of 4096 taps).
        {"name": "correlate_4096", "kind": "correlate", "dtype": "f32", "channels": 32, "length": 1 << 20,
         "taps": 4096},
        # A training step of a learned filter: correlation, signal gradient and
        # kernel gradient.
        {"name": "train_filter", "kind": "train", "dtype": "f32", "channels": 16, "length": 250008, "taps": 504},
        # Transforms across an array of receivers: one transform per sample.
        {"name": "across_64", "kind": "across", "dtype": "f32", "n": 64, "length": 250007},
        # The tensor-core form at full FP32 accuracy.
        {"name": "tensor_core_4096", "kind": "tensor_core", "dtype": "f32", "n": 4096, "batch": 4096,
         "precision": "bf16x6"},
        # Requests of mixed sizes served together.
        {"name": "requests", "kind": "requests", "dtype": "f32", "ffts": 1500, "correlations": 40, "mix": 5},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["roundtrip", "forward", "forward", "inverse", "roundtrip", "convert", "correlate", "train",
                       "across", "tensor_core", "requests"])
    dtype = "f64" if rng.random() < 0.25 and kind not in ("tensor_core", "requests") else "f32"
    case = {"kind": kind, "dtype": dtype}
    most = 23 if dtype == "f64" else 25
    if kind in ("forward", "inverse", "roundtrip"):
        lg = rng.randint(6, 20)
        case.update(n=1 << lg, batch=_log_uniform(rng, max(1, 2 ** (16 - lg)), 2 ** (most - lg)))
        if kind == "roundtrip":
            case["order"] = rng.choice(["normal", "bit_reversed", "unordered"])
    elif kind == "convert":
        lg = rng.randint(6, 15)
        case.update(n=1 << lg, length=rng.randint(1 << (lg - 1), 1 << lg),
                    batch=_log_uniform(rng, max(1, 2 ** (16 - lg)), 2 ** (most - 1 - lg)))
    elif kind == "correlate":
        channels = _log_uniform(rng, 1, 32)
        case.update(channels=channels, length=_log_uniform(rng, 4096, min(1 << 20, 2 ** (most - 1) // channels)),
                    taps=_log_uniform(rng, 16, 4096))
    elif kind == "train":
        channels = _log_uniform(rng, 1, 16)
        case.update(channels=channels, length=_log_uniform(rng, 512, 2 ** (most - 3) // channels // 8) * 8,
                    taps=_log_uniform(rng, 4, 512) * 8)
    elif kind == "across":
        lg = rng.randint(3, 10)
        case.update(n=1 << lg, length=_log_uniform(rng, max(8, 2 ** (16 - lg)), 2 ** (most - 1 - lg)))
    elif kind == "tensor_core":
        lg = rng.randint(8, 16)
        case.update(n=1 << lg, batch=_log_uniform(rng, 2 ** (18 - lg), 2 ** (24 - lg)),
                    precision=rng.choice(["bf16", "tf32", "bf16x6"]))
    else:
        case.update(ffts=_log_uniform(rng, 50, 1500), correlations=rng.randint(0, 40), mix=rng.randint(0, 1 << 20))
    return case


# ------------------------------------------------------------------- helpers
def _pack(case):
    return pb.default_pack_size(KINDS[case["dtype"]])


def _eb(case):
    return 16 if case["dtype"] == "f64" else 8    # bytes of a complex element


def _randn(case, seed, *shape):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(*shape, device=DEV, dtype=KINDS[case["dtype"]], generator=g)


def _rows(t, rows, stride, n, p):
    """Complex128 [rows, n] of packed rows `stride` reals apart."""
    full = t.reshape(rows, stride)[:, : (n + p - 1) // p * 2 * p].reshape(rows, -1, 2, p).double()
    return torch.complex(full[:, :, 0, :].reshape(rows, -1), full[:, :, 1, :].reshape(rows, -1))[:, :n]


def _packed(z, p, like=None):
    """Packed reals of complex [rows, n]; what a last pack has beyond n is `like`'s, or zero."""
    rows, n = z.shape
    m = (n + p - 1) // p
    out = torch.zeros(rows, m * p, dtype=torch.complex128, device=z.device)
    if like is not None:
        out = _rows(like, rows, m * 2 * p, m * p, p).clone()
    out[:, :n] = z
    return torch.stack([out.real.reshape(rows, m, p), out.imag.reshape(rows, m, p)], dim=2).reshape(-1)


def _frequencies(n, order):
    """The frequency at each position of a length-n spectrum in this order."""
    pos = np.arange(n)
    if order == "unordered":    # bits (0, 1, 2, 3) of the position go to (2, 1, 3, 0)
        pos = ((pos & ~15) | ((pos & 1) << 2) | (pos & 2) | (((pos >> 2) & 1) << 3) | ((pos >> 3) & 1))
    if order != "normal":
        bits = n.bit_length() - 1
        rev = np.zeros_like(pos)
        for b in range(bits):
            rev |= ((pos >> b) & 1) << (bits - 1 - b)
        pos = rev
    return torch.as_tensor(pos, device=DEV)


def _fft_size(case):
    """Block size of a correlation: four times the taps for long signals in
    place, the library's own choice in the trained filter."""
    most = 8192 if case["dtype"] == "f64" else 16384
    if case["kind"] == "train":
        return pb.correlation_fft_size(case["taps"], most)
    return min(most, max(128, 1 << (4 * case["taps"] - 1).bit_length()))


def _taps(case, seed):
    """Filter taps, complex128: a chirp for the matched filter, else noise of unit energy."""
    k = case["taps"]
    if case["kind"] == "correlate":
        i = np.arange(k)
        return 0.8 / math.sqrt(k) * np.exp(1j * math.pi * i * i / k + 1j * 0.37 * (seed % 16))
    r = np.random.default_rng(seed + 77)
    return (r.standard_normal(k) + 1j * r.standard_normal(k)) / math.sqrt(2 * k)


def _stride(case):
    """Row stride in reals of the interleaved short rows: whole 16-byte units."""
    return (2 * case["length"] + 3) // 4 * 4


def _mix(case):
    """Sizes of the requests: transforms of 2^8..2^18 and correlations of 2^12..2^20 samples."""
    r = np.random.default_rng(case["mix"])
    lgs = np.floor(r.uniform(8, 19, case["ffts"])).astype(int)
    lengths = np.floor(2 ** r.uniform(12, 20, case["correlations"])).astype(int) // 8 * 8
    taps = np.floor(2 ** r.uniform(6, 13, case["correlations"])).astype(int)
    return {lg: int((lgs == lg).sum()) for lg in sorted(set(lgs.tolist()))}, lengths.tolist(), taps.tolist()


def _request_taps(k, seed):
    r = np.random.default_rng(seed)
    return ((r.standard_normal(k) + 1j * r.standard_normal(k)) / math.sqrt(2 * k)).astype(np.complex64)


# ------------------------------------------------------------------- prepare
def prepare(case, seed):
    kind, dt, p = case["kind"], KINDS[case["dtype"]], _pack(case)
    s = {"case": case}
    if kind in ("forward", "inverse", "roundtrip", "tensor_core"):
        s["unit"] = pb.fft_unit(case["n"], dtype=dt, order=pb.fft_order(ORDERS[case.get("order", "normal")]))
        s["x"] = _randn(case, seed, case["batch"] * 2 * case["n"])
        s["y"] = torch.empty_like(s["x"])
        if kind == "roundtrip":
            s["z"] = torch.empty_like(s["x"])
    elif kind == "convert":
        s["unit"] = pb.fft_unit(case["n"], dtype=dt)
        s["x"] = _randn(case, seed, case["batch"] * _stride(case))
        s["y"] = torch.empty(case["batch"] * 2 * case["n"], dtype=dt, device=DEV)
        s["z"] = torch.empty_like(s["y"])
    elif kind == "correlate":
        s["unit"] = pb.fxcorr_unit(_taps(case, seed), _fft_size(case), dtype=dt)
        s["x"] = _randn(case, seed, case["channels"] * pb.real_size(case["length"], p))
    elif kind == "train":
        s["nf"] = _fft_size(case)
        rs = pb.real_size(case["length"], p)
        s["x"] = _randn(case, seed, case["channels"] * rs).requires_grad_(True)
        s["gy"] = _randn(case, seed + 1000003, case["channels"] * rs)
        taps = torch.as_tensor(_taps(case, seed), device=DEV).reshape(1, -1)
        s["g"] = _packed(taps, p).to(dt).requires_grad_(True)
    elif kind == "across":
        s["unit"] = pb.fft_unit_par(case["n"], dtype=dt)
        rs = pb.real_size(case["length"], p)
        s["x"] = _randn(case, seed, case["n"], rs)
        s["y"] = torch.zeros_like(s["x"])
        s["src"] = [pb.vector(case["length"], dt, p, data=r) for r in s["x"]]
        s["dst"] = [pb.vector(case["length"], dt, p, data=r) for r in s["y"]]
    else:
        sizes, lengths, taps = _mix(case)
        s["x"], s["y"], ffts, xcorrs = {}, {}, [], []
        for lg, count in sizes.items():
            n = 1 << lg
            x = _randn(case, seed + lg, count, 2 * n)
            y = torch.empty_like(x)
            s["x"][lg], s["y"][lg] = x, y
            ffts += [(y[i], x[i], n) for i in range(count)]
        total = 2 * sum(lengths)
        s["xs"], s["ys"], at = _randn(case, seed + 100, total), torch.zeros(total, device=DEV), 0
        for i, (length, k) in enumerate(zip(lengths, taps)):
            g = pb.vector.from_complex(_request_taps(k, seed + i))
            xcorrs.append((s["ys"][at:at + 2 * length], s["xs"][at:at + 2 * length], length, g,
                           pb.correlation_fft_size(k)))
            at += 2 * length
        s["batch"] = pb.ragged_batch(ffts, xcorrs)
    return s


# ----------------------------------------------------------------------- run
def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind in ("forward", "inverse"):
        s["unit"].exec(s["y"], s["x"], batch=case["batch"], direction=int(kind == "inverse"), check=False)
        return s["y"]
    if kind == "roundtrip":
        s["unit"].exec(s["y"], s["x"], batch=case["batch"], check=False)
        s["unit"].exec(s["z"], s["y"], batch=case["batch"], direction=1, check=False)
        return s["y"], s["z"]
    if kind == "tensor_core":
        s["unit"].exec_tensor_core(s["y"], s["x"], batch=case["batch"], precision=case["precision"], check=False)
        return s["y"]
    if kind == "convert":
        s["unit"].exec(s["y"], s["x"], batch=case["batch"], pack_src=1, src_len=case["length"],
                       src_stride=_stride(case), check=False)
        s["unit"].exec(s["z"], s["y"], batch=case["batch"], direction=1, pack_dst=1, pack_src=_pack(case),
                       check=False)
        return s["y"], s["z"]
    if kind == "correlate":
        s["unit"].exec(s["x"], s["x"], case["length"], channels=case["channels"], check=False)
        return s["x"]
    if kind == "train":
        s["x"].grad = s["g"].grad = None
        y = FxcorrFunction.apply(s["x"], s["g"], s["nf"], case["length"], case["taps"], case["channels"])
        y.backward(s["gy"])
        return y.detach(), s["x"].grad, s["g"].grad
    if kind == "across":
        s["unit"](s["dst"], s["src"])
        return s["y"]
    s["batch"]()
    return {"transforms": [s["y"][lg] for lg in sorted(s["y"])], "correlations": s["ys"]}


# ---------------------------------------------------------------------- work
def _fft_flops(n):
    return 5.0 * n * math.log2(n)


def work(case):
    kind, eb = case["kind"], _eb(case)
    if kind in ("forward", "inverse", "tensor_core"):
        return {"bytes": 2 * eb * case["n"] * case["batch"], "flops": case["batch"] * _fft_flops(case["n"])}
    if kind == "roundtrip":
        return {"bytes": 4 * eb * case["n"] * case["batch"], "flops": 2 * case["batch"] * _fft_flops(case["n"])}
    if kind == "convert":
        return {"bytes": eb * case["batch"] * (case["length"] + 3 * case["n"]),
                "flops": 2 * case["batch"] * _fft_flops(case["n"])}
    if kind in ("correlate", "train"):
        points = case["channels"] * case["length"]
        nf = _fft_size(case)
        blocks = case["channels"] * -(-case["length"] // (nf - case["taps"] + 1))
        if kind == "correlate":
            return {"bytes": 2 * eb * points, "flops": 2 * blocks * _fft_flops(nf)}
        # x, y, the output's gradient and the signal's
        return {"bytes": 4 * eb * points, "flops": 6 * blocks * _fft_flops(nf)}
    if kind == "across":
        return {"bytes": 2 * eb * case["n"] * case["length"], "flops": case["length"] * _fft_flops(case["n"])}
    sizes, lengths, taps = _mix(case)
    points = sum(c << lg for lg, c in sizes.items()) + sum(lengths)
    flops = sum(c * _fft_flops(1 << lg) for lg, c in sizes.items())
    for length, k in zip(lengths, taps):
        nf = pb.correlation_fft_size(k)
        flops += 2 * -(-length // (nf - k + 1)) * _fft_flops(nf)
    return {"bytes": 2 * eb * points, "flops": flops}


# --------------------------------------------------------------------- exact
def _correlate(x, g):
    """y[m] = sum_j x[m + j] conj(g[j]) of complex rows, and zero beyond the end."""
    n = 1 << (x.shape[1] + g.shape[-1]).bit_length()
    return torch.fft.ifft(torch.fft.fft(x, n) * torch.fft.fft(g, n).conj())[:, : x.shape[1]]


def _by_rows(f, x, rows=8):
    return torch.cat([f(x[i:i + rows]) for i in range(0, x.shape[0], rows)])


def exact(case, seed):
    kind, p, s = case["kind"], _pack(case), {}
    if kind != "requests":
        s = prepare(case, seed)
    n, b = case.get("n"), case.get("batch")
    if kind in ("forward", "inverse", "tensor_core"):
        x = _rows(s["x"], b, 2 * n, n, p)
        return _packed(torch.fft.ifft(x) if kind == "inverse" else torch.fft.fft(x), p)
    if kind == "roundtrip":
        x = _rows(s["x"], b, 2 * n, n, p)
        return _packed(torch.fft.fft(x)[:, _frequencies(n, case["order"])], p), _packed(x, p)
    if kind == "convert":
        x = _rows(s["x"], b, _stride(case), case["length"], 1)
        x = torch.nn.functional.pad(x, (0, n - case["length"]))
        return _packed(torch.fft.fft(x), p), _packed(x, 1)
    if kind == "correlate":
        ch, length = case["channels"], case["length"]
        x = _rows(s["x"], ch, pb.real_size(length, p), length, p)
        g = torch.as_tensor(_taps(case, seed), device=DEV).to(torch.complex64 if _eb(case) == 8 else torch.complex128)
        return _packed(_by_rows(lambda r: _correlate(r, g.to(torch.complex128)), x), p, s["x"])
    if kind == "train":
        ch, length, k = case["channels"], case["length"], case["taps"]
        rs = pb.real_size(length, p)
        x, gy = _rows(s["x"].detach(), ch, rs, length, p), _rows(s["gy"], ch, rs, length, p)
        g = _rows(s["g"].detach(), 1, pb.real_size(k, p), k, p)[0]
        m = 1 << (length + k).bit_length()
        gx = _by_rows(lambda r: torch.fft.ifft(torch.fft.fft(r, m) * torch.fft.fft(g, m))[:, :length], gy)
        spec = sum(torch.fft.fft(x[c], m) * torch.fft.fft(gy[c], m).conj() for c in range(ch))
        return _packed(_by_rows(lambda r: _correlate(r, g), x), p), _packed(gx, p), _packed(
            torch.fft.ifft(spec)[:k].reshape(1, -1), p)
    if kind == "across":
        x = _rows(s["x"], n, s["x"].shape[1], case["length"], p)
        y = torch.fft.fft(x, dim=0)
        return _packed(y, p).reshape(n, -1)
    sizes, lengths, taps = _mix(case)
    ys, at, out = _randn(case, seed + 100, 2 * sum(lengths)), 0, []
    for i, (length, k) in enumerate(zip(lengths, taps)):
        g = torch.as_tensor(_request_taps(k, seed + i).astype(np.complex128), device=DEV)
        out.append(_packed(_correlate(_rows(ys[at:at + 2 * length], 1, 2 * length, length, 8), g), 8))
        at += 2 * length
    transforms = [_packed(torch.fft.fft(_rows(_randn(case, seed + lg, c, 2 << lg), c, 2 << lg, 1 << lg, 8)), 8)
                  .reshape(c, 2 << lg) for lg, c in sizes.items()]
    return {"transforms": transforms,
            "correlations": torch.cat(out) if out else torch.zeros(0, dtype=torch.float64, device=DEV)}
