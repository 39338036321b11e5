// Overlap-save correlation for FP32 blocks of N = 2^13 or 2^14 points at pack 8
// (reference fxcorr.hpp:102-136): one block's window in shared memory,
// transformed in place in three register-sized steps each way.
//
// With B = N / 512, sample n = a*16B + b*16 + c (a < 32, b < B, c < 16) and
// frequency k = ka + 32*kb + 32B*kc,
//   W_N^(nk) = W_32^(a ka) * W_N^(ka(16b+c)) * W_B^(b kb) * W_16B^(c kb) * W_16^(c kc),
// so the forward transform is 32-point DFTs over a, B-point over b and
// 16-point over c with a twiddle between, each step reading and writing the
// same places (frequency ka, kb, kc where a, b, c were).  Nothing needs the
// spectrum in natural order: the product with the kernel's spectrum is taken in
// the last step's registers, and the inverse (as the forward transform of the
// conjugate) runs the steps backwards with the same twiddles.
//
// A thread holds 32 points in registers (N / 32 threads), so the three steps
// each way are seven passes over the window in shared memory where two
// steps of 128-point transforms with exchanges took thirteen, without an
// exchange buffer, and six block barriers.  Rows of 16 points are padded to
// 18: the three access patterns (stride 16B, stride 16 and whole rows in
// 16-byte units) are free of bank conflicts.  A thread's W_N^(ka(16b+c)) and
// its kernel-spectrum values are the same for every window: 128 words in its
// tensor-memory lane, otherwise idle here.  The packed window lands by bulk
// copies in the same memory (it is in registers before the first step writes),
// the next one as soon as the last step has read this one.
// Bound by issue and the shared-memory pipe.  32 channels x 2^20 samples, 4096
// taps, in place: 395 us with the two-step form, 260 us; relative error against
// FP64 4.0e-7 and 2.8e-7.  8192 points, 16 x 2^20, 2048 taps: 220 and 121 us.
//
// Out of place, windows go round the blocks: calls that overlap share nothing
// (claimed from a counter 260 us, so 272 us, 18.6 rounds being 19).  In place
// (compiled apart: in one kernel 264 us), a window's outputs overwrite samples
// that earlier blocks' windows read: they are claimed in order, each block
// publishes "window loaded" (flags[item], cleared before each launch), and every
// warp waits (bounded, about a second) for its predecessors before it writes, as
// in the other forms.
#pragma once

#include "pcx_fft_v2.cuh"
#include "pcx_fxcorr_kernels.cuh"
#include "pcx_tmem.cuh"

namespace pcxg {

template<int LOGN>
struct xci_cfg {
    static constexpr int N    = 1 << LOGN;
    static constexpr int B    = N / 512;
    static constexpr int NT   = 16 * B;
    static constexpr int RL   = 18;                   // padded row of 16 points (complex)
    static constexpr int WIN  = 32 * B * RL * 8;
    static constexpr int SMEM = WIN + 16 * B * 8;     // window, W_16B^(c kb)
    static constexpr int MINB = 512 / NT;
    static constexpr int TCOLS = NT;                  // tensor-memory columns: 128 words a thread
    static constexpr int TABLE = N + 16 * B;          // entries of the two twiddle tables
    static_assert(LOGN == 13 || LOGN == 14, "B is 16 or 32");
    static_assert(MINB * (SMEM + 1024 + 256) <= 233472, "blocks per SM");
};

// Twiddles: [ka][16b+c] W_N^(ka(16b+c)), then [kb][c] W_16B^(c kb).
__global__ void k_xci_twiddles(cpx<float>* out, int log_n) {
    const int n = 1 << log_n, m = n / 32, q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n + m) return;
    const long long e = q < n ? (long long)(q / m) * (q % m) : (long long)((q - n) / 16) * ((q - n) % 16) * 32;
    double          s, c;
    sincospi(2.0 * (double)(e & (n - 1)) / (double)n, &s, &c);
    out[q] = {(float)c, (float)-s};
}

// K[ka + 32*kb + 32B*kc] in the order of the threads' registers: value
// j*16 + kc of thread t (row t + j*NT = ka*B + kb) at [(j*16 + kc)*NT + t].
__global__ void k_xci_spectrum(const cpx<float>* __restrict__ ks, cpx<float>* __restrict__ kp, int log_n) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= 1 << log_n) return;
    const int b = 1 << (log_n - 9), nt = 16 * b;
    const int t = q % nt, i = q / nt, kc = i % 16, r = t + i / 16 * nt;
    kp[q] = ks[r / b + 32 * (r % b) + 32 * b * kc];
}

struct xci_args {
    xc_args     base;
    const void* kperm;    // k_xci_spectrum's order
    const void* tw;       // k_xci_twiddles
};

// 32 values times the thread's 64 words of tensor memory at `col`: conj(v)*K or
// conj(v)*conj(K) with CJ, plain product without.
template<bool CJ>
__device__ __forceinline__ void xci_mul(cpx<float> (&v)[32], uint32_t col, bool conj_k) {
    __syncwarp();
    static_for<4>([&](auto hc) {
        constexpr int h = decltype(hc)::value;
        uint32_t      w[16];
        tmem_ld16(col + 16 * h, w);
        static_for<8>([&](auto jc) {
            constexpr int    j = decltype(jc)::value, i = 8 * h + j;
            const cpx<float> k = {__uint_as_float(w[2 * j]), __uint_as_float(w[2 * j + 1])};
            if constexpr (CJ) {
                const cpx<float> c = {v[i].re, -v[i].im};
                v[i]               = conj_k ? cmul(c, k) : cmulc(c, k);
            } else {
                v[i] = cmul(v[i], k);
            }
        });
    });
}

// 32 values from global memory (`stride` apart) into 64 words of tensor memory.
__device__ __forceinline__ void xci_keep(uint32_t col, const cpx<float>* g, int stride) {
    static_for<2>([&](auto hc) {
        constexpr int h = decltype(hc)::value;
        uint32_t      w[32];
        static_for<16>([&](auto jc) {
            constexpr int    j = decltype(jc)::value;
            const cpx<float> k = ldg_cpx(g + (16 * h + j) * stride);
            w[2 * j]           = __float_as_uint(k.re);
            w[2 * j + 1]       = __float_as_uint(k.im);
        });
        tmem_st32(col + 32 * h, w);
    });
}

// The B-point DFTs over b of the (ka, c) columns a thread owns.
template<int B>
__device__ __forceinline__ void xci_dft_b(cpx<float> (&v)[32]) {
    if constexpr (B == 32) {
        dft<32, 1, 0>(v);
    } else {
        dft<16, 1, 0>(v);
        dft<16, 1, 16>(v);
    }
}

template<int LOGN, bool INPLACE>
__global__ void __launch_bounds__(xci_cfg<LOGN>::NT, xci_cfg<LOGN>::MINB) k_fxcorr_ip(xci_args A) {
    using F            = xci_cfg<LOGN>;
    constexpr int N    = F::N;
    constexpr int B    = F::B;
    constexpr int NT   = F::NT;
    constexpr int RL   = F::RL;
    const xc_args& a   = A.base;
    extern __shared__ __align__(128) unsigned char smem[];
    cpx<float>*         win = reinterpret_cast<cpx<float>*>(smem);
    float*              raw = reinterpret_cast<float*>(smem);    // the packed window as it lands
    cpx<float>*         tw2 = reinterpret_cast<cpx<float>*>(smem + F::WIN);
    __shared__ uint64_t full;
    __shared__ unsigned s_item;
    __shared__ uint32_t s_tmem;
    const int           tid   = threadIdx.x;
    const int           lane  = tid % 32;
    const float*        src   = reinterpret_cast<const float*>(a.src);
    float*              dst   = reinterpret_cast<float*>(a.dst);
    const unsigned      total = (unsigned)a.total, nblk = (unsigned)a.nblk;    // < 2^31 (host check)

    if (tid < 32) {
        tmem_alloc(&s_tmem, F::TCOLS);
        tmem_relinquish();
    }
    tw2[tid] = ldg_cpx(reinterpret_cast<const cpx<float>*>(A.tw) + N + tid);
    if (tid == 0) {
        s_item = INPLACE ? atomicAdd(a.counter, 1u) : blockIdx.x;
        mbar_init(&full, 1);
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = s_tmem;
    const uint32_t tcol  = tbase + ((uint32_t)(32 * ((tid / 32) % 4)) << 16) + (uint32_t)(tid / 128) * 128;

    // window elements [lo, hi) of an item lie inside the signal
    auto range = [&](unsigned item, unsigned& ch, long long& b0, int& lo, int& hi) {
        ch = item / nblk;
        b0 = (long long)(item - ch * nblk) * a.step - a.in_shift;
        lo = (int)max(0LL, min((long long)N, -b0));
        hi = (int)max((long long)lo, min((long long)N, a.len - b0));
    };
    // warp 0: the item's packed samples, in pieces of 32 KB
    auto copy = [&](unsigned item) {
        if (item >= total) return;
        unsigned  ch;
        long long b0;
        int       lo, hi;
        range(item, ch, b0, lo, hi);
        const uint32_t bytes = (uint32_t)((hi - lo + 7) / 8) * 64;
        if (lane == 0) mbar_arrive_expect_tx(&full, bytes);
        __syncwarp();
        const uint32_t off = lane * 32768u;
        if (off < bytes) {
            bulk_g2s(smem + 8 * lo + off, reinterpret_cast<const char*>(src + ch * a.src_stride + 2 * (b0 + lo)) + off,
                     min(32768u, bytes - off), &full);
        }
    };
    if (tid < 32) copy(s_item);
    xci_keep(tcol, reinterpret_cast<const cpx<float>*>(A.tw) + tid, NT);
    xci_keep(tcol + 64, reinterpret_cast<const cpx<float>*>(A.kperm) + tid, NT);

    const int  c   = tid % 16;
    cpx<float>* p1 = win + tid + 2 * (tid / 16);                  // (b, c) = tid: ka at 18B apart
    cpx<float>* p2 = win + (tid / 16) * (B * RL) + c;             // (ka, c): b at 18 apart
    cpx<float>* p3 = win + tid * RL;                              // row (ka, kb) = tid, then tid + NT
    constexpr int J2 = 32 / B;                                    // columns (ka, c) per thread, NT/16 apart in ka
    unsigned   item  = s_item;
    uint32_t   phase = 0;
    bool       bad   = false;    // this warp gave up a wait
    while (item < total) {
        unsigned  ch;
        long long b0;
        int       lo, hi;
        range(item, ch, b0, lo, hi);
        const bool ok = mbar_wait_bounded(&full, phase);
        cpx<float> v[32];
        // ---------------- forward, 32-point DFTs over a, times W_N^(ka(16b+c))
        static_for<32>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            v[i]            = lds_swapped<float, 16>(raw, 2 * i * 16 * B + pk<3>(tid), 8);
        });
        if (lo > 0 || hi < N) {
            static_for<32>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                const int     n = i * 16 * B + tid;
                if (n < lo || n >= hi) v[i] = {0.f, 0.f};
            });
        }
        if (__syncthreads_or(!ok || bad)) {    // the window is in registers
            // give up: record it and let the copies in flight land first
            if (tid == 0) {
                atomicExch(a.error, 1);
                mbar_wait_bounded(&full, phase, 100000000ull);
            }
            break;    // every thread leaves together; nothing else is in flight
        }
        phase ^= 1;
        if (INPLACE && tid == 0) {
            st_release(a.flags + item, 1u);    // this window is loaded
            s_item = atomicAdd(a.counter, 1u);
        }
        dft<32, 1, 0>(v);
        xci_mul<false>(v, tcol, false);
        static_for<32>([&](auto ic) { p1[decltype(ic)::value * B * RL] = v[decltype(ic)::value]; });
        __syncthreads();
        // ---------------- over b, times W_16B^(c kb)
        static_for<32>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            v[i]            = p2[(i / B) * (NT / 16) * (B * RL) + (i % B) * RL];
        });
        xci_dft_b<B>(v);
        static_for<32>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            p2[(i / B) * (NT / 16) * (B * RL) + (i % B) * RL] = i % B ? cmul(v[i], tw2[(i % B) * 16 + c]) : v[i];
        });
        static_assert(J2 == 1 || J2 == 2, "columns per thread");
        __syncthreads();
        // ---------------- over c; times K; back over kc
        static_for<16>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            const float4  x = *reinterpret_cast<const float4*>(p3 + (i / 8) * NT * RL + 2 * (i % 8));
            v[2 * i]        = {x.x, x.y};
            v[2 * i + 1]    = {x.z, x.w};
        });
        dft<16, 1, 0>(v);
        dft<16, 1, 16>(v);
        xci_mul<true>(v, tcol + 64, a.conj_kernel != 0);
        dft<16, 1, 0>(v);
        dft<16, 1, 16>(v);
        static_for<16>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            *reinterpret_cast<float4*>(p3 + (i / 8) * NT * RL + 2 * (i % 8)) =
                make_float4(v[2 * i].re, v[2 * i].im, v[2 * i + 1].re, v[2 * i + 1].im);
        });
        // in place: the first look at the flags, so that the wait below rarely has to read one
        const unsigned blk  = item - ch * nblk;
        bool           seen = true;
        if (INPLACE && lane < a.hwait && lane < blk) seen = ld_acquire(a.flags + (item - 1 - lane)) != 0u;
        __syncthreads();
        // ---------------- times W_16B^(c kb), back over kb
        static_for<32>([&](auto ic) {
            constexpr int    i = decltype(ic)::value;
            const cpx<float> x = p2[(i / B) * (NT / 16) * (B * RL) + (i % B) * RL];
            v[i]               = i % B ? cmul(x, tw2[(i % B) * 16 + c]) : x;
        });
        xci_dft_b<B>(v);
        static_for<32>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            p2[(i / B) * (NT / 16) * (B * RL) + (i % B) * RL] = v[i];
        });
        __syncthreads();
        // ---------------- times W_N^(ka(16b+c)), back over ka: v[i] = conj(y) at i*16B + tid
        static_for<32>([&](auto ic) { v[decltype(ic)::value] = p1[decltype(ic)::value * B * RL]; });
        fence_proxy_async_smem();
        __syncthreads();    // the window is read: the next one may land
        const unsigned next = INPLACE ? s_item : item + gridDim.x;
        if (tid < 32) copy(next);
        xci_mul<false>(v, tcol, false);
        dft<32, 1, 0>(v);
        if constexpr (INPLACE) {
            // the outputs overwrite samples of the hwait previous blocks' windows;
            // a warp that gives up stores nothing, and the block leaves at the
            // next vote
            bool late = false;
            for (unsigned d = lane; d < (unsigned)a.hwait && d < blk && !late; d += 32) {
                const unsigned* f = a.flags + (item - 1 - d);
                if ((d == (unsigned)lane && seen) || ld_acquire(f) != 0u) continue;
                const unsigned long long t0 = globaltimer_ns();
                while (ld_acquire(f) == 0u) {
                    if (globaltimer_ns() - t0 > XC_WAIT_NS) {
                        late = true;
                        break;
                    }
                    __nanosleep(128);
                }
            }
            if (__any_sync(0xffffffffu, late)) {
                if (lane == 0) atomicExch(a.error, 1);
                bad = true;
            }
        }
        if (!bad) {
            // element n of the window is written when out_shift <= n < out_shift + step and it is
            // inside the signal; e0 is whole packs
            const long long e0 = b0 + a.in_shift - a.out_shift;
            const int       w0 = a.out_shift;
            const int       w1 = (int)max(0LL, min(min((long long)a.out_shift + a.step, a.len - e0), (long long)N));
            float*          d  = dst + ch * a.dst_stride + 2 * e0 + pk<3>(tid);
            static_for<32>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                const int     n = i * 16 * B + tid;
                if (n >= w0 && n < w1) {
                    __stcs(d + 2 * i * 16 * B, v[i].re);
                    __stcs(d + 2 * i * 16 * B + 8, -v[i].im);
                }
            });
        }
        item = next;
    }
    tc_fence_before();
    __syncthreads();
    if (tid < 32) tmem_dealloc(tbase, F::TCOLS);
}

// ---------------------------------------------------------------------------
// Kernel gradient in the same form: per block the gy block (zero beyond its
// outputs) and then the x window are transformed by the three forward steps.
// A thread's 32 values of FFT(gy) and of the running sum of FFT(x) *
// conj(FFT(gy)) fill its 128 words of tensor memory; its W_N^(ka(16b+c)) are
// products of two of ten factors (u^1..u^3, u^4, u^8..u^28, u = W_N^(16b+c)) in
// shared memory.  Both inputs land in the same window, the next one once the
// last step has read its rows.  Blocks go round the launch, so the sums do not
// depend on timing.  16 channels x 2^20, blocks of 16384 and 8192 points: 271 and
// 318 us in the two-step form, 190 and 157 us.
struct xci_kg_args {
    kg_args     base;
    const void* tw;    // k_xci_twiddles
};

template<int LOGN>
struct xci_kg_cfg {
    using F                   = xci_cfg<LOGN>;
    static constexpr int UB   = 10 * F::NT * 8;    // factors of the first twiddle
    static constexpr int SMEM = F::SMEM + UB;
    static_assert(F::MINB * (SMEM + 1024 + 256) <= 233472, "blocks per SM");
};

template<int LOGN>
__global__ void __launch_bounds__(xci_cfg<LOGN>::NT, xci_cfg<LOGN>::MINB) k_fxcorr_ip_kgrad(xci_kg_args A) {
    using F            = xci_cfg<LOGN>;
    constexpr int N    = F::N;
    constexpr int B    = F::B;
    constexpr int NT   = F::NT;
    constexpr int RL   = F::RL;
    const kg_args& a   = A.base;
    extern __shared__ __align__(128) unsigned char smem[];
    cpx<float>*         win = reinterpret_cast<cpx<float>*>(smem);
    float*              raw = reinterpret_cast<float*>(smem);
    cpx<float>*         tw2 = reinterpret_cast<cpx<float>*>(smem + F::WIN);
    cpx<float>*         uf  = tw2 + 16 * B;    // [10][NT]
    __shared__ uint64_t full;
    __shared__ uint32_t s_tmem;
    const int           tid   = threadIdx.x;
    const int           lane  = tid % 32;
    const unsigned      total = (unsigned)a.total, nblk = (unsigned)a.nblk;    // < 2^31 (host check)
    const cpx<float>*   tw    = reinterpret_cast<const cpx<float>*>(A.tw);

    if (tid < 32) {
        tmem_alloc(&s_tmem, F::TCOLS);
        tmem_relinquish();
    }
    tw2[tid] = ldg_cpx(tw + N + tid);
    static_for<10>([&](auto qc) {
        constexpr int q   = decltype(qc)::value;
        uf[q * NT + tid] = ldg_cpx(tw + (q < 3 ? q + 1 : 4 * (q - 2)) * NT + tid);    // row ka of the table: u^ka
    });
    if (tid == 0) {
        mbar_init(&full, 1);
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = s_tmem;
    const uint32_t tcol  = tbase + ((uint32_t)(32 * ((tid / 32) % 4)) << 16) + (uint32_t)(tid / 128) * 128;
    {
        uint32_t z[32];
        static_for<32>([&](auto jc) { z[decltype(jc)::value] = 0u; });
        tmem_st32(tcol + 64, z);
        tmem_st32(tcol + 96, z);
    }
    // elements of input s (0: gy block, 1: x window) of an item that count
    auto valid = [&](unsigned item, int s, long long& off) -> int {
        const unsigned  ch = item / nblk;
        const long long b  = (long long)(item - ch * nblk) * a.step;
        off                = ch * a.stride + 2 * b;
        return (int)min((long long)(s ? N : a.step), a.len - b);
    };
    // warp 0: the packed samples, in pieces of 32 KB
    auto copy = [&](unsigned item, int s) {
        if (item >= total) return;
        long long      off;
        const uint32_t bytes = (uint32_t)((valid(item, s, off) + 7) / 8) * 64;
        if (lane == 0) mbar_arrive_expect_tx(&full, bytes);
        __syncwarp();
        const uint32_t q = lane * 32768u;
        if (q < bytes) {
            bulk_g2s(smem + q, reinterpret_cast<const char*>(reinterpret_cast<const float*>(s ? a.x : a.gy) + off) + q,
                     min(32768u, bytes - q), &full);
        }
    };
    if (tid < 32) copy(blockIdx.x, 0);

    const int   c  = tid % 16;
    cpx<float>* p1 = win + tid + 2 * (tid / 16);
    cpx<float>* p2 = win + (tid / 16) * (B * RL) + c;
    cpx<float>* p3 = win + tid * RL;
    uint32_t    phase = 0;
    bool        fail  = false;
    for (unsigned item = blockIdx.x; item < total && !fail; item += gridDim.x) {
        for (int s = 0; s < 2; ++s) {
            long long  off;
            const int  n  = valid(item, s, off);
            const bool ok = mbar_wait_bounded(&full, phase);
            cpx<float> v[32];
            static_for<32>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                v[i]            = lds_swapped<float, 16>(raw, 2 * i * 16 * B + pk<3>(tid), 8);
            });
            if (n < N) {
                static_for<32>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    if (i * 16 * B + tid >= n) v[i] = {0.f, 0.f};
                });
            }
            if (__syncthreads_or(!ok)) {
                // give up: record it and let the copies in flight land first
                if (tid == 0) {
                    atomicExch(a.error, 1);
                    mbar_wait_bounded(&full, phase, 100000000ull);
                }
                fail = true;
                break;
            }
            phase ^= 1;
            dft<32, 1, 0>(v);
            static_for<31>([&](auto ic) {
                constexpr int i = decltype(ic)::value + 1, lo = i & 3, hi = i >> 2;
                cpx<float>    w;
                if constexpr (hi == 0) w = uf[(lo - 1) * NT + tid];
                else if constexpr (lo == 0) w = uf[(2 + hi) * NT + tid];
                else w = cmul(uf[(2 + hi) * NT + tid], uf[(lo - 1) * NT + tid]);
                v[i] = cmul(v[i], w);
            });
            static_for<32>([&](auto ic) { p1[decltype(ic)::value * B * RL] = v[decltype(ic)::value]; });
            __syncthreads();
            static_for<32>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                v[i]            = p2[(i / B) * (NT / 16) * (B * RL) + (i % B) * RL];
            });
            xci_dft_b<B>(v);
            static_for<32>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                p2[(i / B) * (NT / 16) * (B * RL) + (i % B) * RL] = i % B ? cmul(v[i], tw2[(i % B) * 16 + c]) : v[i];
            });
            __syncthreads();
            static_for<16>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                const float4  x = *reinterpret_cast<const float4*>(p3 + (i / 8) * NT * RL + 2 * (i % 8));
                v[2 * i]        = {x.x, x.y};
                v[2 * i + 1]    = {x.z, x.w};
            });
            fence_proxy_async_smem();
            __syncthreads();    // the window is read: the next input may land
            if (tid < 32) copy(s ? item + gridDim.x : item, s ^ 1);
            dft<16, 1, 0>(v);
            dft<16, 1, 16>(v);
            __syncwarp();
            if (s == 0) {
                static_for<2>([&](auto hc) {
                    constexpr int h = decltype(hc)::value;
                    uint32_t      r[32];
                    static_for<16>([&](auto jc) {
                        constexpr int j = decltype(jc)::value;
                        r[2 * j]        = __float_as_uint(v[16 * h + j].re);
                        r[2 * j + 1]    = __float_as_uint(v[16 * h + j].im);
                    });
                    tmem_st32(tcol + 32 * h, r);
                });
            } else {
                // sum += X * conj(GY), eight values at a time
                static_for<4>([&](auto hc) {
                    constexpr int h = decltype(hc)::value;
                    uint32_t      gq[16], sq[16];
                    tmem_ld16(tcol + 16 * h, gq);
                    tmem_ld16(tcol + 64 + 16 * h, sq);
                    static_for<8>([&](auto jc) {
                        constexpr int    j = decltype(jc)::value;
                        const cpx<float> p = cmulc(v[8 * h + j], cpx<float>{__uint_as_float(gq[2 * j]),
                                                                             __uint_as_float(gq[2 * j + 1])});
                        sq[2 * j]          = __float_as_uint(__uint_as_float(sq[2 * j]) + p.re);
                        sq[2 * j + 1]      = __float_as_uint(__uint_as_float(sq[2 * j + 1]) + p.im);
                    });
                    tmem_st16(tcol + 64 + 16 * h, sq);
                });
            }
        }
    }
    if (!fail) {
        // this block's sums in natural order: k = ka + 32*kb + 32B*kc, row r = ka*B + kb
        cpx<float>* acc = reinterpret_cast<cpx<float>*>(a.acc) + (long long)blockIdx.x * N;
        __syncwarp();
        static_for<2>([&](auto hc) {
            constexpr int h = decltype(hc)::value;
            uint32_t      sq[32];
            tmem_ld32(tcol + 64 + 32 * h, sq);
            const int r = tid + h * NT;
            static_for<16>([&](auto jc) {
                constexpr int kc                           = decltype(jc)::value;
                acc[r / B + 32 * (r % B) + 32 * B * kc] = {__uint_as_float(sq[2 * kc]), __uint_as_float(sq[2 * kc + 1])};
            });
        });
    }
    tc_fence_before();
    __syncthreads();
    if (tid < 32) tmem_dealloc(tbase, F::TCOLS);
}

}    // namespace pcxg
