// FFT across a set of vectors (reference fft_unit_par, fft.hpp:2167-2572):
// for every element position p < len, the n-point transform of
// src[0][p], src[1][p], ..., src[n-1][p] goes to dst[0][p], ..., dst[n-1][p].
//
// Up to 1024 points one kernel does it all (k_par).  Above, and where vectors
// overlap in a way that needs every input read first, a tiled transpose
// gathers the vectors into `len` contiguous rows of n points (default pack),
// the batched FFT of the plan transforms those rows in place, and a second
// tiled transpose scatters the rows back; both transposes read and write 32
// consecutive elements per warp.
#include "pcx_fft_v2.cuh"
#include "pcx_host.hpp"

#include <algorithm>
#include <string>
#include <vector>

using namespace pcxg;

namespace {

constexpr int TD = 32;    // tile edge
constexpr int TR = 8;     // thread rows

// rows[i][p] (pack 2^lps) -> buf[p][i] (pack 2^lpb, row stride rs reals)
template<class T>
__global__ void k_par_gather(const T* const* __restrict__ rows, int lps, T* __restrict__ buf, int lpb, long long rs,
                             long long n, long long len) {
    __shared__ T re[TD][TD + 1], im[TD][TD + 1];
    const long long i0 = (long long)blockIdx.y * TD, p0 = (long long)blockIdx.x * TD;
    const int       tx = threadIdx.x, ty = threadIdx.y;
    const long long ps = 1LL << lps, pb = 1LL << lpb;
    for (int r = ty; r < TD; r += TR) {
        const long long i = i0 + r, p = p0 + tx;
        if (i < n && p < len) {
            const T*        v = rows[i];
            const long long o = ((p >> lps) << (lps + 1)) + (p & (ps - 1));
            re[r][tx]         = v[o];
            im[r][tx]         = v[o + ps];
        }
    }
    __syncthreads();
    for (int r = ty; r < TD; r += TR) {
        const long long p = p0 + r, i = i0 + tx;
        if (i < n && p < len) {
            const long long o = p * rs + ((i >> lpb) << (lpb + 1)) + (i & (pb - 1));
            buf[o]            = re[tx][r];
            buf[o + pb]       = im[tx][r];
        }
    }
}

// buf[p][i] -> rows[i][p] (pack 2^lpd)
template<class T>
__global__ void k_par_scatter(T* const* __restrict__ rows, int lpd, const T* __restrict__ buf, int lpb, long long rs,
                              long long n, long long len) {
    __shared__ T re[TD][TD + 1], im[TD][TD + 1];
    const long long i0 = (long long)blockIdx.y * TD, p0 = (long long)blockIdx.x * TD;
    const int       tx = threadIdx.x, ty = threadIdx.y;
    const long long pd = 1LL << lpd, pb = 1LL << lpb;
    for (int r = ty; r < TD; r += TR) {
        const long long p = p0 + r, i = i0 + tx;
        if (i < n && p < len) {
            const long long o = p * rs + ((i >> lpb) << (lpb + 1)) + (i & (pb - 1));
            re[r][tx]         = buf[o];
            im[r][tx]         = buf[o + pb];
        }
    }
    __syncthreads();
    for (int r = ty; r < TD; r += TR) {
        const long long i = i0 + r, p = p0 + tx;
        if (i < n && p < len) {
            T*              v = rows[i];
            const long long o = ((p >> lpd) << (lpd + 1)) + (p & (pd - 1));
            v[o]              = re[tx][r];
            v[o + pd]         = im[tx][r];
        }
    }
}

// One pass: a block transforms C neighbouring element positions of all n
// vectors.  Neighbouring threads hold neighbouring positions, so every load
// and store of a warp covers whole 32-byte sectors of one or a few vectors
// (C >= 8 positions; 32 and more up to 128 vectors), and nothing but the
// stage exchanges goes through shared memory.  The vectors' addresses are
// kernel parameters (16 bytes a vector, at most 16 KB), so a call copies
// nothing to the device and needs no workspace.
// HBM-bound: 16 bytes per point where gather + transform + scatter moved 48.
// 64 vectors of 250007 elements: 187 us before, 53.5 us with three blocks an
// SM in FP32 (two: 61.4, four: 55.3; loads in flight hide the latency, four
// blocks leave too few registers).
template<class T, int LOGN>
struct par_cfg {
    using P                  = splan<LOGN>;
    static constexpr int N   = P::L;
    static constexpr int C   = 256 / P::TT > 8 ? 256 / P::TT : 8;    // positions per block
    static constexpr int NT  = C * P::TT;
    using X                  = xch_interleaved<N, C>;
    static constexpr int SMEM = P::NST > 1 ? X::size * (int)sizeof(cpx<T>) : 0;
};
template<int N>
struct par_args {
    const void* src[N];
    void*       dst[N];
    const void* stw;    // stage twiddles
    long long   len;
    int         lps, lpd;
    int         order_in, order_out;
    int         conj;
    double      scale;
};

template<class T, int LOGN>
__global__ void __launch_bounds__(par_cfg<T, LOGN>::NT, par_cfg<T, LOGN>::NT > 256 ? 1 : (sizeof(T) == 8 ? 2 : 3))
    k_par(const __grid_constant__ par_args<(1 << LOGN)> a) {
    using F          = par_cfg<T, LOGN>;
    using P          = typename F::P;
    constexpr int E  = P::E;
    constexpr int TT = P::TT;
    extern __shared__ __align__(16) unsigned char smem[];
    const int       c    = threadIdx.x % F::C;
    const int       t    = threadIdx.x / F::C;
    const long long p    = (long long)blockIdx.x * F::C + c;
    const bool      live = p < a.len;
    const long long os   = ((p >> a.lps) << (a.lps + 1)) + (p & ((1LL << a.lps) - 1));
    const long long od   = ((p >> a.lpd) << (a.lpd + 1)) + (p & ((1LL << a.lpd) - 1));
    const int       ps   = 1 << a.lps, pd = 1 << a.lpd;
    cpx<T>          v[E];
    static_for<E>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        const T*      x = static_cast<const T*>(a.src[order_pos(t + i * TT, a.order_in, LOGN)]) + os;
        v[i]            = {T(0), T(0)};
        if (live) v[i] = {x[0], x[ps]};
    });
    if (a.conj) static_for<E>([&](auto ic) { v[decltype(ic)::value].im = -v[decltype(ic)::value].im; });
    const auto* stw = static_cast<const cpx<T>*>(a.stw);
    stage_compute_tab<P, 0>(v, t, stw);
    // every input of the block is in registers before any output is written
    // (the exchanges' barriers, or this one)
    if constexpr (P::NST > 1) run_stages_tab<P, typename F::X>(v, reinterpret_cast<cpx<T>*>(smem), c, t, stw);
    else __syncthreads();
    const T sc = T(a.scale), sim = a.conj ? -sc : sc;
    if (live) {
        static_for<E>([&](auto ic) {    // frequency t + i*TT
            constexpr int i = decltype(ic)::value;
            T*            y = static_cast<T*>(a.dst[order_pos(t + i * TT, a.order_out, LOGN)]) + od;
            y[0]            = v[i].re * sc;
            y[pd]           = v[i].im * sim;
        });
    }
}

template<class T, int LOGN>
int launch_par(const pcx_plan_s* p, void* const* dst, const void* const* src, size_t len, int pd, int ps, bool inv,
               double scale, cudaStream_t st) {
    using F = par_cfg<T, LOGN>;
    par_args<F::N> a{};
    std::copy(src, src + F::N, a.src);
    std::copy(dst, dst + F::N, a.dst);
    a.stw       = p->stwL;
    a.len       = (long long)len;
    a.lps       = __builtin_ctz(ps);
    a.lpd       = __builtin_ctz(pd);
    a.order_in  = inv ? p->order : 0;
    a.order_out = inv ? 0 : p->order;
    a.conj      = inv;
    a.scale     = scale;
    auto kern   = k_par<T, LOGN>;
    if (F::SMEM > 0) PCX_CUDA_TRY(smem_attr_cached(reinterpret_cast<const void*>(kern), F::SMEM));
    kern<<<(unsigned)((len + F::C - 1) / F::C), F::NT, F::SMEM, st>>>(a);
    PCX_CUDA_TRY(cudaGetLastError());
    return PCX_OK;
}

template<class T>
int dispatch_par(const pcx_plan_s* p, void* const* dst, const void* const* src, size_t len, int pd, int ps, bool inv,
                 double scale, cudaStream_t st) {
    switch (p->log_n) {
    case 1: return launch_par<T, 1>(p, dst, src, len, pd, ps, inv, scale, st);
    case 2: return launch_par<T, 2>(p, dst, src, len, pd, ps, inv, scale, st);
    case 3: return launch_par<T, 3>(p, dst, src, len, pd, ps, inv, scale, st);
    case 4: return launch_par<T, 4>(p, dst, src, len, pd, ps, inv, scale, st);
    case 5: return launch_par<T, 5>(p, dst, src, len, pd, ps, inv, scale, st);
    case 6: return launch_par<T, 6>(p, dst, src, len, pd, ps, inv, scale, st);
    case 7: return launch_par<T, 7>(p, dst, src, len, pd, ps, inv, scale, st);
    case 8: return launch_par<T, 8>(p, dst, src, len, pd, ps, inv, scale, st);
    case 9: return launch_par<T, 9>(p, dst, src, len, pd, ps, inv, scale, st);
    default: return launch_par<T, 10>(p, dst, src, len, pd, ps, inv, scale, st);
    }
}

// Whether a block may write its outputs while other blocks still read: no
// destination row may overlap a source row, except a vector transformed in
// place, whose block reads and writes the same places as long as both pack
// widths keep a position's group inside the block.
bool par_one_pass(void* const* dst, const void* const* src, size_t n, size_t len, int pd, int ps, size_t es) {
    if (n > 1024) return false;
    const size_t c  = std::max<size_t>(8, 256 / std::max<size_t>(1, n / 16));
    const size_t sb = (len + ps - 1) / ps * 2 * ps * es, db = (len + pd - 1) / pd * 2 * pd * es;
    struct span {
        uintptr_t lo, hi;
        bool      dst;
    };
    uintptr_t slo = ~uintptr_t(0), shi = 0, dlo = ~uintptr_t(0), dhi = 0;
    for (size_t i = 0; i < n; ++i) {
        const uintptr_t s = reinterpret_cast<uintptr_t>(src[i]), d = reinterpret_cast<uintptr_t>(dst[i]);
        slo = std::min(slo, s);
        shi = std::max(shi, s + sb);
        dlo = std::min(dlo, d);
        dhi = std::max(dhi, d + db);
    }
    if (shi <= dlo || dhi <= slo) return true;
    const bool        in_place = pd == ps || (size_t)std::max(pd, ps) <= c;
    std::vector<span> v;
    v.reserve(2 * n);
    for (size_t i = 0; i < n; ++i) {
        const uintptr_t s = reinterpret_cast<uintptr_t>(src[i]), d = reinterpret_cast<uintptr_t>(dst[i]);
        if (s == d && in_place) {
            v.push_back({s, s + std::max(sb, db), true});    // one span for both: may touch no other
            continue;
        }
        v.push_back({s, s + sb, false});
        v.push_back({d, d + db, true});
    }
    std::sort(v.begin(), v.end(), [](const span& x, const span& y) { return x.lo < y.lo; });
    uintptr_t any_hi = 0, dst_hi = 0;    // ends of the spans so far: all, and the written ones
    for (const span& x: v) {
        if (x.lo < (x.dst ? any_hi : dst_hi)) return false;
        any_hi = std::max(any_hi, x.hi);
        if (x.dst) dst_hi = std::max(dst_hi, x.hi);
    }
    return true;
}

int check_pack(int pack, const char* what) {
    if (pack < 1 || (pack & (pack - 1)) != 0) {
        return pcx_fail(PCX_ERR_INVALID, std::string(what) + " pack size (which is " + std::to_string(pack) +
                                             ") is not a power of two");
    }
    return PCX_OK;
}

}    // namespace

extern "C" int pcx_fft_par_exec(pcx_plan plan, void* const* dst, const void* const* src, size_t count, size_t len,
                                int pack_dst, int pack_src, int direction, int normalize, void* stream) {
    return pcx_guard([&]() -> int {
        if (!plan) return pcx_fail(PCX_ERR_INVALID, "plan is null");
        pcx_plan_s* p = plan;
        // reference fft.hpp:2197-2211
        if (count != p->n) {
            return pcx_fail(PCX_ERR_INVALID, "destination size (which is " + std::to_string(count) +
                                                 " is not equal to fft size (which is " + std::to_string(p->n) + ")");
        }
        if (int rc = check_pack(pack_dst, "destination")) return rc;
        if (int rc = check_pack(pack_src, "source")) return rc;
        if (direction != PCX_FORWARD && direction != PCX_INVERSE) return pcx_fail(PCX_ERR_INVALID, "unknown direction");
        if (len == 0) return PCX_OK;
        if (!dst || !src) return pcx_fail(PCX_ERR_INVALID, "null vector array");
        for (size_t i = 0; i < count; ++i) {
            if (!dst[i] || !src[i]) return pcx_fail(PCX_ERR_INVALID, "null vector pointer");
        }
        const bool   f64  = p->dtype == PCX_F64;
        const size_t es   = f64 ? sizeof(double) : sizeof(float);
        if (par_one_pass(dst, src, count, len, pack_dst, pack_src, es)) {
            const bool   inv   = direction == PCX_INVERSE;
            const double scale = inv && normalize ? 1.0 / (double)p->n : 1.0;
            const auto   run   = f64 ? dispatch_par<double> : dispatch_par<float>;
            return run(p, dst, src, len, pack_dst, pack_src, inv, scale, static_cast<cudaStream_t>(stream));
        }
        int          lpb  = f64 ? 2 : 3;    // default pack, at most the row length
        while ((size_t(1) << lpb) > p->n) --lpb;
        const size_t pb   = size_t(1) << lpb;
        const size_t rs   = (p->n + pb - 1) / pb * 2 * pb;    // reals per gathered row
        const size_t need = 2 * count * sizeof(void*) + len * rs * es;
        cudaStream_t st   = static_cast<cudaStream_t>(stream);
        std::lock_guard<std::mutex> g(p->par_mu);
        if (p->par_bytes < need) {
            if (p->par_buf) cudaFree(p->par_buf);
            p->par_buf   = nullptr;
            p->par_bytes = 0;
            PCX_CUDA_TRY(cudaMalloc(&p->par_buf, need));
            p->par_bytes = need;
        }
        void** dptr = static_cast<void**>(p->par_buf);
        void** sptr = dptr + count;
        void*  buf  = sptr + count;
        // the pointer arrays are host memory: the copies return once staged
        PCX_CUDA_TRY(cudaMemcpyAsync(dptr, dst, count * sizeof(void*), cudaMemcpyHostToDevice, st));
        PCX_CUDA_TRY(cudaMemcpyAsync(sptr, src, count * sizeof(void*), cudaMemcpyHostToDevice, st));
        const dim3 blk(TD, TR);
        const dim3 grd((unsigned)((len + TD - 1) / TD), (unsigned)((count + TD - 1) / TD));
        const int  lps = __builtin_ctz(pack_src), lpd = __builtin_ctz(pack_dst);
        if (f64) {
            k_par_gather<double><<<grd, blk, 0, st>>>(reinterpret_cast<const double* const*>(sptr), lps,
                                                      static_cast<double*>(buf), lpb, (long long)rs, (long long)count,
                                                      (long long)len);
        } else {
            k_par_gather<float><<<grd, blk, 0, st>>>(reinterpret_cast<const float* const*>(sptr), lps,
                                                     static_cast<float*>(buf), lpb, (long long)rs, (long long)count,
                                                     (long long)len);
        }
        PCX_CUDA_TRY(cudaGetLastError());
        if (int rc = pcx_fft_run(p, buf, buf, p->n, (int)pb, (int)pb, direction, normalize, len, rs, rs, nullptr, 0,
                                 st, 1.0)) {
            return rc;
        }
        if (f64) {
            k_par_scatter<double><<<grd, blk, 0, st>>>(reinterpret_cast<double* const*>(dptr), lpd,
                                                       static_cast<const double*>(buf), lpb, (long long)rs,
                                                       (long long)count, (long long)len);
        } else {
            k_par_scatter<float><<<grd, blk, 0, st>>>(reinterpret_cast<float* const*>(dptr), lpd,
                                                      static_cast<const float*>(buf), lpb, (long long)rs,
                                                      (long long)count, (long long)len);
        }
        PCX_CUDA_TRY(cudaGetLastError());
        return PCX_OK;
    });
}
