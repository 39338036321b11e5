// Host side of the overlap-save correlator: handle creation (kernel spectrum
// computed on the device), the fused correlation launch and its adjoint.
#include "pcx_fxcorr3.cuh"
#include "pcx_fxcorr_ip.cuh"
#include "pcx_fxcorr_kernels.cuh"
#include "pcx_host.hpp"
#include "pcx_v2_launch.cuh"

#include <algorithm>
#include <cstdlib>
#include <list>
#include <mutex>
#include <string>
#include <vector>

using namespace pcxg;

struct pcx_fxcorr_s {
    int         dtype  = PCX_F32;
    size_t      k      = 0;
    size_t      n      = 0;
    int         log_n  = 0;
    int         pack_g = 8;
    pcx_plan_s* plan   = nullptr;    // natural-order N-point FFT (kernel spectrum, gradient inverse)
    void*       tw     = nullptr;    // W_N^i, i < N
    void*       kspec  = nullptr;    // FFT(g)/N, interleaved complex, natural order
    int*        err    = nullptr;    // error flag (host memory, see flag_words)
    unsigned*   ctl    = nullptr;    // in-place calls: [0] work counter, [1..] "window loaded" flags
    size_t      flags_cap = 0;
    void*       gscratch  = nullptr;    // kernel-gradient accumulators
    size_t      gscratch_bytes = 0;
    int         sms            = 0;
    int         device         = 0;
    bool        x3             = false;      // FP32, N <= 2^12: pcx_fxcorr3.cuh (tables: plan->stwL)
    // FP32, N = 2^13 or 2^14: three-step form (pcx_fxcorr_ip.cuh)
    void*       xi             = nullptr;    // one allocation: K in its order | twiddles
    const void* xi_tw          = nullptr;
    bool        general        = false;    // created with PCX_XC_GENERAL
};

namespace {

constexpr int XC_SINGLE_NT = 256;

template<class T, int LOGN>
struct xcfg {
    static constexpr int EPT = LOGN >= 14 ? 32 : 16;
    using P                  = splan<LOGN, EPT>;
    static constexpr int M   = P::TT >= XC_SINGLE_NT ? 1 : XC_SINGLE_NT / P::TT;
    static constexpr int NT  = M * P::TT;
};

template<class T, int LOGN>
int launch_xc(const xc_args& a, const void* tw, cudaStream_t st, int sms, bool attr_only) {
    using C             = xcfg<T, LOGN>;
    constexpr int bytes = fxcorr_smem_bytes<T, LOGN, C::EPT, C::M>();
    auto          kern  = k_fxcorr<T, LOGN, C::EPT, C::M>;
    if (attr_only) {
        PCX_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        return PCX_OK;
    }
    int per_sm = 0;
    PCX_CUDA_TRY(occupancy_cached(reinterpret_cast<const void*>(kern), C::NT, bytes, &per_sm));
    const long long groups = (a.total + C::M - 1) / C::M;
    const long long grid   = std::max<long long>(1, std::min<long long>(groups, (long long)std::max(per_sm, 1) * sms));
    kern<<<(unsigned)grid, C::NT, bytes, st>>>(a, reinterpret_cast<const cpx<T>*>(tw));
    PCX_CUDA_TRY(cudaGetLastError());
    return PCX_OK;
}

template<class T, int LOGN>
int launch_kg(const kg_args& a, const void* tw, cudaStream_t st, int grid, bool attr_only) {
    using C             = xcfg<T, LOGN>;
    constexpr int bytes = fxcorr_smem_bytes<T, LOGN, C::EPT, 1>();
    auto          kern  = k_fxcorr_kgrad<T, LOGN, C::EPT>;
    if (attr_only) {
        PCX_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        return PCX_OK;
    }
    kern<<<(unsigned)grid, C::P::TT, bytes, st>>>(a, reinterpret_cast<const cpx<T>*>(tw));
    PCX_CUDA_TRY(cudaGetLastError());
    return PCX_OK;
}

template<class T>
int dispatch_xc(int log_n, const xc_args& a, const void* tw, cudaStream_t st, int sms, bool attr_only) {
    switch (log_n) {
    case 6: return launch_xc<T, 6>(a, tw, st, sms, attr_only);
    case 7: return launch_xc<T, 7>(a, tw, st, sms, attr_only);
    case 8: return launch_xc<T, 8>(a, tw, st, sms, attr_only);
    case 9: return launch_xc<T, 9>(a, tw, st, sms, attr_only);
    case 10: return launch_xc<T, 10>(a, tw, st, sms, attr_only);
    case 11: return launch_xc<T, 11>(a, tw, st, sms, attr_only);
    case 12: return launch_xc<T, 12>(a, tw, st, sms, attr_only);
    case 13: return launch_xc<T, 13>(a, tw, st, sms, attr_only);
    case 14:
        if constexpr (sizeof(T) == 4) return launch_xc<T, 14>(a, tw, st, sms, attr_only);
        [[fallthrough]];
    default: return pcx_fail(PCX_ERR_UNSUPPORTED, "fft size not supported by the fused correlator");
    }
}

template<class T>
int dispatch_kg(int log_n, const kg_args& a, const void* tw, cudaStream_t st, int grid, bool attr_only) {
    switch (log_n) {
    case 6: return launch_kg<T, 6>(a, tw, st, grid, attr_only);
    case 7: return launch_kg<T, 7>(a, tw, st, grid, attr_only);
    case 8: return launch_kg<T, 8>(a, tw, st, grid, attr_only);
    case 9: return launch_kg<T, 9>(a, tw, st, grid, attr_only);
    case 10: return launch_kg<T, 10>(a, tw, st, grid, attr_only);
    case 11: return launch_kg<T, 11>(a, tw, st, grid, attr_only);
    case 12: return launch_kg<T, 12>(a, tw, st, grid, attr_only);
    case 13: return launch_kg<T, 13>(a, tw, st, grid, attr_only);
    case 14:
        if constexpr (sizeof(T) == 4) return launch_kg<T, 14>(a, tw, st, grid, attr_only);
        [[fallthrough]];
    default: return pcx_fail(PCX_ERR_UNSUPPORTED, "fft size not supported by the fused correlator");
    }
}

template<class T>
__global__ void k_scale_pack(const cpx<T>* __restrict__ src, int k, int lp, T* __restrict__ dst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= k) return;
    const int P = 1 << lp;
    const int o = ((i >> lp) << (lp + 1)) + (i & (P - 1));
    dst[o]      = src[i].re;
    dst[o + P]  = src[i].im;
}

// K / N from natural order k = k1 + N1*k2 to row-major [k1][k2].
__global__ void k_perm_spectrum(const cpx<float>* __restrict__ ks, cpx<float>* __restrict__ kp, int log_n1,
                                int log_n2) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (1 << (log_n1 + log_n2))) return;
    const int k1 = q >> log_n2, k2 = q & ((1 << log_n2) - 1);
    kp[q]        = ks[k1 + (k2 << log_n1)];
}

}    // namespace

// The spectrum K[k1 + N1*k2] stored at [k1*N2 + k2] (the (k1, k2) order of the
// in-CTA four-step correlator's rows), on `st`.
cudaError_t pcx_xc2_perm_spectrum(const void* ks, void* kp, int log_n1, int log_n2, cudaStream_t st) {
    const int n = 1 << (log_n1 + log_n2);
    k_perm_spectrum<<<(n + 255) / 256, 256, 0, st>>>(static_cast<const cpx<float>*>(ks), static_cast<cpx<float>*>(kp),
                                                      log_n1, log_n2);
    return cudaGetLastError();
}

namespace {

template<int LOGN>
int launch_xci(const xci_args& a, cudaStream_t st, int sms, bool attr_only) {
    using C   = xci_cfg<LOGN>;
    auto kern = a.base.inplace ? k_fxcorr_ip<LOGN, true> : k_fxcorr_ip<LOGN, false>;
    PCX_CUDA_TRY(smem_attr_cached(reinterpret_cast<const void*>(kern), C::SMEM));
    if (attr_only) return PCX_OK;
    const long long grid = std::max<long long>(1, std::min<long long>(a.base.total, (long long)C::MINB * sms));
    kern<<<(unsigned)grid, C::NT, C::SMEM, st>>>(a);
    PCX_CUDA_TRY(cudaGetLastError());
    return PCX_OK;
}

// grid: given a.acc == nullptr only returned (the rows of the accumulator)
template<int LOGN>
int launch_xci_kg(const xci_kg_args& a, cudaStream_t st, int sms, int* grid) {
    using C   = xci_cfg<LOGN>;
    auto kern = k_fxcorr_ip_kgrad<LOGN>;
    PCX_CUDA_TRY(smem_attr_cached(reinterpret_cast<const void*>(kern), xci_kg_cfg<LOGN>::SMEM));
    *grid = (int)std::max<long long>(1, std::min<long long>(a.base.total, (long long)C::MINB * sms));
    if (!a.base.acc) return PCX_OK;
    kern<<<(unsigned)*grid, C::NT, xci_kg_cfg<LOGN>::SMEM, st>>>(a);
    PCX_CUDA_TRY(cudaGetLastError());
    return PCX_OK;
}

// The whole-window form (pcx_fxcorr3.cuh): blocks of a launch over `total` windows.
// Two blocks per SM by shared memory and registers (xc3_cfg); the occupancy
// query answers one for a kernel that allocates tensor memory, whatever it
// needs of the 512 columns (64 and 128 here).  Out of place, one block an SM and
// two: 4096 points, 16 x 250008 samples, 504 taps 41.7 and 35.4 us, 32 x 2^20,
// 1024 taps 335 and 265 us; 1024 points, 32 x 250000, 250 taps 89 and 73 us.
template<int LOGN, class K>
int grid_xc3(K kern, long long total, int sms, int* grid) {
    using C = xc3_cfg<LOGN>;
    PCX_CUDA_TRY(smem_attr_cached(reinterpret_cast<const void*>(kern), C::SMEM));
    const long long tiles = (total + C::M - 1) / C::M;
    *grid = (int)std::max<long long>(1, std::min<long long>(tiles, 2LL * sms));
    return PCX_OK;
}
template<int LOGN>
int launch_xc3(const xc_args& a, const void* stw, const void* full, cudaStream_t st, int sms) {
    using C  = xc3_cfg<LOGN>;
    int grid = 0;
    if (int rc = grid_xc3<LOGN>(k_fxcorr3<LOGN>, a.total, sms, &grid)) return rc;
    if (a.total == 0) return PCX_OK;    // launch attributes only
    k_fxcorr3<LOGN><<<(unsigned)grid, C::NT, C::SMEM, st>>>(a, stw, full);
    PCX_CUDA_TRY(cudaGetLastError());
    return PCX_OK;
}
// grid: given a.acc == nullptr only returned (the rows of the accumulator)
template<int LOGN>
int launch_xc3_kg(const kg_args& a, const void* stw, cudaStream_t st, int sms, int* grid) {
    using C = xc3_cfg<LOGN>;
    if (int rc = grid_xc3<LOGN>(k_fxcorr3_kgrad<LOGN>, a.total, sms, grid)) return rc;
    if (!a.acc) return PCX_OK;
    k_fxcorr3_kgrad<LOGN><<<(unsigned)*grid, C::NT, C::SMEM, st>>>(a, stw);
    PCX_CUDA_TRY(cudaGetLastError());
    return PCX_OK;
}
int dispatch_xc3(int log_n, const xc_args& a, const void* stw, const void* full, cudaStream_t st, int sms) {
    switch (log_n) {
    case 6: return launch_xc3<6>(a, stw, full, st, sms);
    case 7: return launch_xc3<7>(a, stw, full, st, sms);
    case 8: return launch_xc3<8>(a, stw, full, st, sms);
    case 9: return launch_xc3<9>(a, stw, full, st, sms);
    case 10: return launch_xc3<10>(a, stw, full, st, sms);
    case 11: return launch_xc3<11>(a, stw, full, st, sms);
    default: return launch_xc3<12>(a, stw, full, st, sms);
    }
}
int dispatch_xc3_kg(int log_n, const kg_args& a, const void* stw, cudaStream_t st, int sms, int* grid) {
    switch (log_n) {
    case 6: return launch_xc3_kg<6>(a, stw, st, sms, grid);
    case 7: return launch_xc3_kg<7>(a, stw, st, sms, grid);
    case 8: return launch_xc3_kg<8>(a, stw, st, sms, grid);
    case 9: return launch_xc3_kg<9>(a, stw, st, sms, grid);
    case 10: return launch_xc3_kg<10>(a, stw, st, sms, grid);
    case 11: return launch_xc3_kg<11>(a, stw, st, sms, grid);
    default: return launch_xc3_kg<12>(a, stw, st, sms, grid);
    }
}

// Tables and launch attributes of the three-step form.
template<int LOGN>
int init_xci(pcx_fxcorr_s* h) {
    using C = xci_cfg<LOGN>;
    PCX_CUDA_TRY(cudaMalloc(&h->xi, (size_t)(C::N + C::TABLE) * sizeof(cpx<float>)));
    auto* tw = static_cast<cpx<float>*>(h->xi) + C::N;
    k_xci_twiddles<<<(C::TABLE + 255) / 256, 256>>>(tw, LOGN);
    PCX_CUDA_TRY(cudaGetLastError());
    h->xi_tw = tw;
    int grid = 0;
    if (int rc = launch_xci_kg<LOGN>(xci_kg_args{}, 0, h->sms, &grid)) return rc;
    xci_args a{};
    if (int rc = launch_xci<LOGN>(a, 0, 0, true)) return rc;
    a.base.inplace = 1;
    return launch_xci<LOGN>(a, 0, 0, true);
}

int check_pack(int pack) {
    if (pack < 1 || (pack & (pack - 1)) != 0) {
        return pcx_fail(PCX_ERR_INVALID, "pack size (which is " + std::to_string(pack) + ") is not a power of two");
    }
    return PCX_OK;
}

int ensure_flags(pcx_fxcorr_s* h, size_t items) {
    if (h->ctl && h->flags_cap >= items) return PCX_OK;
    if (h->ctl) cudaFree(h->ctl);
    h->ctl       = nullptr;
    h->flags_cap = 0;
    const size_t cap = std::max<size_t>(items, 1024);
    PCX_CUDA_TRY(cudaMalloc(&h->ctl, (cap + 1) * sizeof(unsigned)));
    h->flags_cap = cap;
    return PCX_OK;
}

int run_xc(pcx_fxcorr_s* h, void* dst, const void* src, size_t len, int pack, size_t channels, size_t dstride,
           size_t sstride, bool convolve, cudaStream_t st) {
    if (int rc = check_pack(pack)) return rc;
    const size_t n = h->n;
    if ((size_t)pack > n) return pcx_fail(PCX_ERR_UNSUPPORTED, "pack size larger than fft size");
    const size_t step = (n - (h->k - 1)) / pack * pack;
    if (step == 0) {
        return pcx_fail(PCX_ERR_INVALID, "kernel size (which is " + std::to_string(h->k) +
                                             ") leaves no output per block for fft size " + std::to_string(n));
    }
    if (len == 0 || channels == 0) return PCX_OK;
    if (!dst || !src) return pcx_fail(PCX_ERR_INVALID, "null data pointer");
    const size_t row = (len + pack - 1) / pack * 2 * pack;
    if (channels > 1 && (dstride < row || sstride < row)) return pcx_fail(PCX_ERR_INVALID, "channel stride smaller than a row");
    const size_t nblk  = (len + step - 1) / step;
    const size_t total = nblk * channels;
    if (total >= (size_t(1) << 31)) return pcx_fail(PCX_ERR_UNSUPPORTED, "too many blocks in one call");
    const bool inplace = dst == src;
    if (inplace && convolve) return pcx_fail(PCX_ERR_INVALID, "the adjoint needs distinct input and output buffers");
    if (inplace) {
        // The flags (and the counter before them) are cleared on the call's own
        // stream, so that every run of a captured call finds them clear too: a
        // flag value that the host chooses per call is the same in each run.
        if (int rc = ensure_flags(h, total)) return rc;
        PCX_CUDA_TRY(cudaMemsetAsync(h->ctl, 0, (1 + total) * sizeof(unsigned), st));
    }

    xc_args a{};
    a.src         = src;
    a.dst         = dst;
    a.src_stride  = (long long)sstride;
    a.dst_stride  = (long long)dstride;
    a.len         = (long long)len;
    a.lp          = __builtin_ctz(pack);
    a.step        = (int)step;
    a.nblk        = (int)nblk;
    a.total       = (long long)total;
    // convolution (the adjoint): window b starts `shift` samples before
    // output b*step, and output m of the block is circular index m + shift.
    // Any shift >= K-1 with step + shift <= N gives the same outputs; at pack 8
    // K-1 rounded up to whole packs is one (step = N - shift), and it keeps
    // the windows on whole packs, as the forms below need.
    const size_t shift = pack == 8 ? (h->k - 1 + 7) / 8 * 8 : h->k - 1;
    a.in_shift    = convolve ? (int)shift : 0;
    a.out_shift   = convolve ? (int)shift : 0;
    a.conj_kernel = convolve ? 0 : 1;
    a.inplace     = inplace ? 1 : 0;
    a.hwait       = (int)((n + step - 1) / step) - 1;
    a.flags       = inplace ? h->ctl + 1 : nullptr;
    a.counter     = h->ctl;
    a.error       = h->err;
    a.kspec       = h->kspec;
    // whole-window and three-step forms: FP32, pack 8, windows on whole
    // packs, rows of packs 16-byte aligned
    const bool rows = pack == 8 && a.in_shift % 8 == 0 && (channels == 1 || sstride % 4 == 0) &&
                      reinterpret_cast<uintptr_t>(src) % 16 == 0;
    if (h->x3 && rows) return dispatch_xc3(h->log_n, a, h->plan->stwL, h->plan->s3_any, st, h->sms);
    if (h->xi && rows) {
        xci_args b{};
        b.base  = a;
        b.kperm = h->xi;
        b.tw    = h->xi_tw;
        return h->log_n == 14 ? launch_xci<14>(b, st, h->sms, false) : launch_xci<13>(b, st, h->sms, false);
    }
    return h->dtype == PCX_F64 ? dispatch_xc<double>(h->log_n, a, h->tw, st, h->sms, false)
                               : dispatch_xc<float>(h->log_n, a, h->tw, st, h->sms, false);
}

}    // namespace

namespace {

// Error flags of the handles: words of page-locked host memory that a kernel
// writes only when a wait gives up, so that neither clearing one for a new owner
// nor reading it takes a copy (3 and 8 us of a training step).
class flag_words {
public:
    cudaError_t take(int** out) {
        std::lock_guard<std::mutex> g(mu_);
        if (free_.empty()) {
            int*              block = nullptr;
            const cudaError_t e     = cudaHostAlloc(&block, 1024 * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
            if (e != cudaSuccess) return e;
            for (int i = 0; i < 1024; i += 16) free_.push_back(block + i);    // a cache line each
        }
        *out = free_.back();
        free_.pop_back();
        return cudaSuccess;
    }
    void give(int* p) {
        std::lock_guard<std::mutex> g(mu_);
        free_.push_back(p);
    }

private:
    std::mutex        mu_;
    std::vector<int*> free_;
};
flag_words& flags() {
    static flag_words* f = new flag_words;    // never destroyed, as the pool below
    return *f;
}

// Its memory goes after the frees, which wait for the device.
void free_handle(pcx_fxcorr_s* h) {
    if (h->plan) pcx_plan_destroy(h->plan);
    if (h->tw) cudaFree(h->tw);
    if (h->kspec) cudaFree(h->kspec);
    if (h->ctl) cudaFree(h->ctl);
    if (h->gscratch) cudaFree(h->gscratch);
    if (h->xi) cudaFree(h->xi);
    if (h->err) flags().give(h->err);
    delete h;
}

// Handles that were destroyed, kept for the next create of the same kind
// (device, type, FFT size, form).  A correlation whose kernel changes with
// every call (a trained filter) creates a handle per call, and seven device
// allocations and frees, each of which waits for the device, cost it more than
// ten times its kernels.  What is reused is memory and the tables that depend
// on the size alone; a handle has one owner at a time, and the kernel's
// spectrum is computed anew for each.  At most 4 idle handles and 64 MB of
// their growing buffers are kept, the oldest goes first, and all go when making
// a handle fails for want of memory.
class handle_pool {
public:
    static constexpr size_t MAX_IDLE  = 4;
    static constexpr size_t MAX_BYTES = size_t(64) << 20;

    // An idle handle of this kind, or null.
    pcx_fxcorr_s* take(int device, int dtype, size_t n, bool general) {
        std::lock_guard<std::mutex> g(mu_);
        for (auto it = idle_.begin(); it != idle_.end(); ++it) {
            pcx_fxcorr_s* h = *it;
            if (h->device == device && h->dtype == dtype && h->n == n && h->general == general) {
                idle_.erase(it);
                return h;
            }
        }
        return nullptr;
    }
    void give(pcx_fxcorr_s* h) {
        std::list<pcx_fxcorr_s*> out;
        {
            std::lock_guard<std::mutex> g(mu_);
            idle_.push_back(h);
            size_t sum = 0;
            for (auto it = idle_.end(); it != idle_.begin();) {    // newest first
                --it;
                sum += bytes(*it);
                if (sum > MAX_BYTES || (size_t)std::distance(it, idle_.end()) > MAX_IDLE) {
                    out.splice(out.begin(), idle_, idle_.begin(), std::next(it));
                    break;
                }
            }
        }
        for (pcx_fxcorr_s* o: out) free_handle(o);
    }
    void drain() {
        std::list<pcx_fxcorr_s*> out;
        {
            std::lock_guard<std::mutex> g(mu_);
            out.swap(idle_);
        }
        for (pcx_fxcorr_s* o: out) free_handle(o);
    }

private:
    static size_t bytes(const pcx_fxcorr_s* h) {
        return h->flags_cap * sizeof(unsigned) + h->gscratch_bytes + (h->plan ? h->plan->scratch_bytes : 0);
    }
    std::mutex               mu_;
    std::list<pcx_fxcorr_s*> idle_;
};
// never destroyed: at process exit the CUDA context may be gone first
handle_pool& pool() {
    static handle_pool* p = new handle_pool;
    return *p;
}

// K = FFT(g zero-padded to N) / N, natural order, interleaved (fxcorr.hpp:62-69),
// and its reordered copy for the three-step form.
int set_kernel(pcx_fxcorr_s* h, const void* g) {
    if (int rc = pcx_fft_run(h->plan, h->kspec, g, h->k, 1, h->pack_g, PCX_FORWARD, 0, 1, 2 * h->n,
                             (h->k + h->pack_g - 1) / h->pack_g * 2 * h->pack_g, nullptr, 0, 0, 1.0 / (double)h->n)) {
        return rc;
    }
    if (h->xi) {
        k_xci_spectrum<<<(unsigned)(h->n / 256), 256>>>(static_cast<const cpx<float>*>(h->kspec),
                                                       static_cast<cpx<float>*>(h->xi), h->log_n);
        PCX_CUDA_TRY(cudaGetLastError());
    }
    return PCX_OK;
}

// Device memory, tables and launch attributes of a new handle.
int init_handle(pcx_fxcorr_s* h) {
    const int    log_n = h->log_n;
    const bool   f64   = h->dtype == PCX_F64;
    const size_t eb    = f64 ? 16 : 8;
    PCX_CUDA_TRY(cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, h->device));
    if (int rc = pcx_plan_create(&h->plan, h->n, h->dtype, PCX_ORDER_NORMAL, 2048)) return rc;
    // K rounds as the windows' transforms do where it has their stages, and part
    // of the error cancels (1024 points at pack 1: 2.035e-7 so, 2.059e-7 with K
    // in 32-point stages)
    h->plan->narrow = log_n <= 12;
    PCX_CUDA_TRY(cudaMalloc(&h->tw, h->n * eb));
    PCX_CUDA_TRY(cudaMalloc(&h->kspec, h->n * eb));
    PCX_CUDA_TRY(flags().take(&h->err));
    PCX_CUDA_TRY(pcx_gen_twiddles(h->tw, (int)h->n, log_n, 1, f64, 0));
    if (int rc = f64 ? dispatch_xc<double>(log_n, xc_args{}, nullptr, 0, 0, true)
                     : dispatch_xc<float>(log_n, xc_args{}, nullptr, 0, 0, true)) {
        return rc;
    }
    if (int rc = f64 ? dispatch_kg<double>(log_n, kg_args{}, nullptr, 0, 0, true)
                     : dispatch_kg<float>(log_n, kg_args{}, nullptr, 0, 0, true)) {
        return rc;
    }
    if (!f64 && log_n <= 12 && !h->general) {
        // its launch attributes now, not in a call that may be captured
        int grid = 0;
        if (int rc = dispatch_xc3_kg(log_n, kg_args{}, nullptr, 0, h->sms, &grid)) return rc;
        if (int rc = dispatch_xc3(log_n, xc_args{}, nullptr, nullptr, 0, h->sms)) return rc;
        h->x3 = true;
    }
    if (!f64 && log_n >= 13 && !h->general) return log_n == 14 ? init_xci<14>(h) : init_xci<13>(h);
    return PCX_OK;
}

}    // namespace

extern "C" int pcx_fxcorr_create(pcx_fxcorr* out, const void* g, size_t k, int pack_g, size_t n_fft, int dtype) {
    return pcx_guard([&]() -> int {
        if (!out) return pcx_fail(PCX_ERR_INVALID, "handle pointer is null");
        *out = nullptr;
        if (n_fft <= 1 || (n_fft & (n_fft - 1)) != 0) {
            return pcx_fail(PCX_ERR_INVALID, "fft_size (which is " + std::to_string(n_fft) +
                                                 ") is not a power of two or less than 2");
        }
        if (dtype != PCX_F32 && dtype != PCX_F64) return pcx_fail(PCX_ERR_INVALID, "unknown dtype");
        if (int rc = check_pack(pack_g)) return rc;
        if (k == 0 || k > n_fft) {
            return pcx_fail(PCX_ERR_INVALID, "kernel size (which is " + std::to_string(k) +
                                                 ") must be in 1..fft size (which is " + std::to_string(n_fft) + ")");
        }
        const int log_n = __builtin_ctzll(n_fft);
        const int maxlog = dtype == PCX_F64 ? 13 : 14;
        if (log_n < 6 || log_n > maxlog) {
            return pcx_fail(PCX_ERR_UNSUPPORTED, "fused correlator supports fft sizes 2^6..2^" + std::to_string(maxlog));
        }
        if (!g) return pcx_fail(PCX_ERR_INVALID, "null kernel pointer");
        const bool general = std::getenv("PCX_XC_GENERAL") != nullptr;
        int        device  = 0;
        PCX_CUDA_TRY(cudaGetDevice(&device));
        auto make = [&](pcx_fxcorr_s*& h) -> int {
            h = pool().take(device, dtype, n_fft, general);
            if (!h) {
                h          = new pcx_fxcorr_s{};
                h->dtype   = dtype;
                h->n       = n_fft;
                h->log_n   = log_n;
                h->device  = device;
                h->general = general;
                if (int rc = init_handle(h)) return rc;
            }
            h->k      = k;
            h->pack_g = pack_g;
            // g may have been written on any stream, and a reused handle's last
            // owner may still be running: what follows is on the default
            // stream, which no non-blocking stream is ordered with
            PCX_CUDA_TRY(cudaDeviceSynchronize());
            *h->err = 0;
            if (int rc = set_kernel(h, g)) return rc;
            PCX_CUDA_TRY(cudaStreamSynchronize(0));    // g is read, the tables and K are there
            return PCX_OK;
        };
        pcx_fxcorr_s* h  = nullptr;
        int           rc = make(h);
        if (rc == PCX_ERR_CUDA) {
            // out of memory, perhaps: once more without the idle handles' memory
            (void)cudaGetLastError();
            if (h) free_handle(h);
            h = nullptr;
            pool().drain();
            rc = make(h);
        }
        if (rc) {
            if (h) free_handle(h);
            return rc;
        }
        *out = h;
        return PCX_OK;
    });
}

extern "C" int pcx_fxcorr_destroy(pcx_fxcorr h) {
    return pcx_guard([&]() -> int {
        if (h) pool().give(h);
        return PCX_OK;
    });
}

extern "C" int pcx_fxcorr_release_idle(void) {
    return pcx_guard([&]() -> int {
        pool().drain();
        return PCX_OK;
    });
}

extern "C" int pcx_fxcorr_exec(pcx_fxcorr h, void* dst, const void* src, size_t len, int pack, size_t channels,
                               size_t dst_stride, size_t src_stride, void* stream) {
    return pcx_guard([&]() -> int {
        if (!h) return pcx_fail(PCX_ERR_INVALID, "handle is null");
        return run_xc(h, dst, src, len, pack, channels, dst_stride, src_stride, false,
                      static_cast<cudaStream_t>(stream));
    });
}

extern "C" int pcx_fxcorr_status(pcx_fxcorr h) {
    return pcx_guard([&]() -> int {
        if (!h) return pcx_fail(PCX_ERR_INVALID, "handle is null");
        PCX_CUDA_TRY(cudaStreamSynchronize(0));
        if (*static_cast<volatile int*>(h->err)) {
            *h->err = 0;
            return pcx_fail(PCX_ERR_TIMEOUT, "a correlation block gave up a bounded wait (for its input copy or, in place, for its predecessor)");
        }
        return PCX_OK;
    });
}

static int run_vjp(pcx_fxcorr_s* h, void* gx, void* gg, const void* gy, const void* x, size_t len, int pack,
                   size_t channels, size_t stride, cudaStream_t st) {
    // d/dx: convolution of gy with g
    if (gx) {
        int rc = run_xc(h, gx, gy, len, pack, channels, stride, stride, true, st);
        if (rc) return rc;
    }
    if (!gg) return PCX_OK;
    if (!x) return pcx_fail(PCX_ERR_INVALID, "kernel gradient needs the forward input x");
    if (int rc = check_pack(pack)) return rc;
    const size_t n    = h->n;
    const size_t step = (n - (h->k - 1)) / pack * pack;
    if (step == 0 || len == 0 || channels == 0) return pcx_fail(PCX_ERR_INVALID, "nothing to differentiate");
    const size_t nblk  = (len + step - 1) / step;
    const size_t total = nblk * channels;
    const size_t eb    = h->dtype == PCX_F64 ? 16 : 8;
    // FP32 at pack 8 on 16-byte aligned rows: the whole-window form up to
    // 2^12 points, the three-step form at 2^13 and 2^14
    const bool rows = pack == 8 && (channels == 1 || stride % 4 == 0) &&
                      (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gy)) % 16 == 0;
    const bool x3 = h->x3 && rows, xi = h->xi && rows;
    kg_args    a{};
    a.total  = (long long)total;
    int grid = (int)std::min<size_t>(total, (size_t)h->sms);
    const auto run_xci = [&]() -> int {
        xci_kg_args b{};
        b.base = a;
        b.tw   = h->xi_tw;
        return h->log_n == 14 ? launch_xci_kg<14>(b, st, h->sms, &grid) : launch_xci_kg<13>(b, st, h->sms, &grid);
    };
    if (x3) {
        if (int rc = dispatch_xc3_kg(h->log_n, a, nullptr, st, h->sms, &grid)) return rc;
    } else if (xi) {
        if (int rc = run_xci()) return rc;
    }
    // sums of the blocks, the general form's spectra, the sum and its inverse
    const size_t rows_s = (size_t)grid * (x3 || xi ? 1 : 2);
    const size_t need   = (rows_s + 2) * n * eb;
    if (h->gscratch_bytes < need) {
        if (h->gscratch) cudaFree(h->gscratch);
        h->gscratch       = nullptr;
        h->gscratch_bytes = 0;
        PCX_CUDA_TRY(cudaMalloc(&h->gscratch, need));
        h->gscratch_bytes = need;
    }
    char* base = static_cast<char*>(h->gscratch);
    a.x       = x;
    a.gy      = gy;
    a.stride  = (long long)stride;
    a.len     = (long long)len;
    a.lp      = __builtin_ctz(pack);
    a.step    = (int)step;
    a.nblk    = (int)nblk;
    a.error   = h->err;
    a.acc     = base;
    a.xspec   = base + (size_t)grid * n * eb;
    void* sum = base + rows_s * n * eb;
    void* inv = base + (rows_s + 1) * n * eb;
    int rc;
    if (x3) {
        rc = dispatch_xc3_kg(h->log_n, a, h->plan->stwL, st, h->sms, &grid);
    } else if (xi) {
        rc = run_xci();
    } else {
        rc = h->dtype == PCX_F64 ? dispatch_kg<double>(h->log_n, a, h->tw, st, grid, false)
                                 : dispatch_kg<float>(h->log_n, a, h->tw, st, grid, false);
    }
    if (rc) return rc;
    if (h->dtype == PCX_F64) {
        k_kgrad_reduce<double><<<(unsigned)((n + 15) / 16), 256, 0, st>>>(
            static_cast<const cpx<double>*>(a.acc), grid, (int)n, static_cast<cpx<double>*>(sum));
    } else {
        k_kgrad_reduce<float><<<(unsigned)((n + 15) / 16), 256, 0, st>>>(
            static_cast<const cpx<float>*>(a.acc), grid, (int)n, static_cast<cpx<float>*>(sum));
    }
    PCX_CUDA_TRY(cudaGetLastError());
    // gg[j] = (1/N) sum_k S[k] e^{+2 pi i jk/N}, j < K
    rc = pcx_fft_run(h->plan, inv, sum, 0, 1, 1, PCX_INVERSE, 1, 1, 2 * n, 2 * n, nullptr, 0, st, 1.0);
    if (rc) return rc;
    const int lpg = __builtin_ctz(h->pack_g);
    if (h->dtype == PCX_F64) {
        k_scale_pack<double><<<(unsigned)((h->k + 255) / 256), 256, 0, st>>>(
            static_cast<const cpx<double>*>(inv), (int)h->k, lpg, static_cast<double*>(gg));
    } else {
        k_scale_pack<float><<<(unsigned)((h->k + 255) / 256), 256, 0, st>>>(
            static_cast<const cpx<float>*>(inv), (int)h->k, lpg, static_cast<float*>(gg));
    }
    PCX_CUDA_TRY(cudaGetLastError());
    return PCX_OK;
}

extern "C" int pcx_fxcorr_vjp(pcx_fxcorr h, void* gx, void* gg, const void* gy, const void* x, size_t len, int pack,
                              size_t channels, size_t stride, void* stream) {
    return pcx_guard([&]() -> int {
        if (!h) return pcx_fail(PCX_ERR_INVALID, "handle is null");
        return run_vjp(h, gx, gg, gy, x, len, pack, channels, stride, static_cast<cudaStream_t>(stream));
    });
}
