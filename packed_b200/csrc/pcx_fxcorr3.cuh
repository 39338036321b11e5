// Overlap-save correlation and its kernel gradient for FP32 blocks of
// N = 2^6..2^12 points at pack 8 (reference fxcorr.hpp:102-136): whole windows
// transformed in shared memory, M = 4096 / N of them per tile.
//
// As in the one-pass FFT (k_single3), persistent blocks of 256 threads bring
// tiles in by bulk copies through a two-stage ring (a window is one
// contiguous run of packed samples, cut at the signal's ends), 16 points per
// thread, stage factors in shared memory; three things are a correlator's own:
//  * the forward transform leaves frequency t + i*TT in v[i], the pattern the
//    inverse starts from, so nothing is exchanged between the two;
//  * a thread's 16 kernel-spectrum values are the same for every window: they
//    stay in its tensor-memory lane (otherwise idle here), 32 columns;
//  * outputs go from registers to HBM, neighbouring threads on neighbouring
//    samples.
// What bounds it: the shared-memory pipe and issue, as two k_single3 passes
// would be, against 16 bytes of HBM per sample.  16 channels x 250008 samples,
// 504 taps, 4096-point windows: the general kernel (plain loads, no copy in
// flight during a block, sub-transform twiddles and kernel spectrum from
// global memory) 98 us, this one 34 us; kernel gradient 182 and
// 34 us (device times).
// Accuracy: full tables for all stages would leave room for one block an SM.
// With factors in all of them and butterflies by halves the error is 5 % above
// the general kernel's; a full table for the second stage (small) and radix-16
// butterflies as 4 x 4 bring it below at the same speed.  4096 points, 1024
// taps, against FP64: general 2.469e-7, by halves 2.649e-7, this 2.403e-7.  (The
// kernel gradient's sums differ anyway: 3.25e-7 in the general form, 2.78e-7.)
//
// In place, a tile's outputs overwrite samples that the windows of earlier
// tiles still read, so tiles are claimed in order from a counter, a block
// publishes "tile loaded" (flags[tile], cleared before each launch) as it starts
// on a tile and, before it writes, waits (bounded, about a second) for the tiles
// that hold the hwait blocks before its own.  A block's claimed tiles are
// published in order and every wait is for lower tiles, so the lowest
// unpublished tile always gets there.  Out of place, tiles go round the
// blocks without a counter.
#pragma once

#include "pcx_fft_v2.cuh"
#include "pcx_fxcorr_kernels.cuh"
#include "pcx_tmem.cuh"

namespace pcxg {

template<int LOGN>
struct xc3_cfg {
    using P                   = splan<LOGN>;
    static constexpr int N    = P::L;
    static constexpr int NT   = 256;
    static constexpr int TT   = P::TT;
    static constexpr int M    = NT / TT;                    // windows per tile
    static constexpr int RS   = 2 * N + single3_pad<TT>();  // shared window stride (reals)
    static constexpr int TILE = M * RS;
    static constexpr int SW   = TT >= 32 ? 16 : 0;
    using X                   = xch_blocked<N, M>;
    // twiddles: the correlator's second stage reads a full table (from 128
    // points on: FULL entries), later ones factors
    static constexpr int FULL = LOGN > 6 ? 1 << (4 + P::rbits(1)) : 0;
    static constexpr int TAB  = smem_align16(stage_tw_smem_bytes<P, float>());
    static constexpr int SKIP = FULL ? stage_tw_offset<P>(2) : 0;    // factors that the full table stands for
    static constexpr int TAB2 = (FULL + stage_tw_size<P>() - SKIP) * 8;
    static constexpr int BASE = 2 * TILE * 4 + X::size * 8;
    static constexpr int SMEM = BASE + (TAB > TAB2 ? TAB : TAB2);
    static_assert((RS * 4) % 16 == 0 && (X::size * 8) % 16 == 0, "16-byte sections");
    static_assert(P::E == 16 && P::NST > 1, "16 points per thread");
    static_assert(2 * (SMEM + 1024 + 256) <= 233472, "two blocks per SM");
};

// One window of a tile: where its samples come from and its outputs go.
struct xc3_window {
    long long dst;    // offset in reals of output 0
    int       lo;     // window elements [lo, hi) lie inside the signal
    int       hi;
    int       nout;   // outputs (0: no window)
};

// Zero the elements of a thread outside [lo, hi).
template<int TT>
__device__ __forceinline__ void xc3_clip(cpx<float> (&v)[16], int t, int lo, int hi) {
    static_for<16>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        if (t + i * TT < lo || t + i * TT >= hi) v[i] = {0.f, 0.f};
    });
}

// A window's transform, frequency t + i*TT into v[i].
template<int LOGN, int BAR>
__device__ __forceinline__ void xc3_transform(cpx<float> (&v)[16], cpx<float>* xch, int m, int t, const cpx<float>* tab) {
    using F = xc3_cfg<LOGN>;
    using P = typename F::P;
    using X = typename F::X;
    stage_compute_tab<P, 0, true>(v, t, tab);
    static_for<P::NST - 1>([&](auto sc) {
        constexpr int S = decltype(sc)::value;
        stage_exchange<P, S, X, BAR>(v, xch, m, t);
        if constexpr (S == 0 && F::FULL > 0) {
            stage_apply_rows<P, 1, true, true>(v, t, tab);
        } else {
            cpx<float> f[(16 >> P::rbits(S + 1)) * stw_q(P::rbits(S + 1))];
            load_stage_tw<P, S + 1, true>(f, t, tab + F::FULL - F::SKIP);
            stage_apply_tw<P, S + 1, true>(v, f);
        }
    });
}

// full_g: the second stage's full table (not read below 128 points).
template<int LOGN>
__global__ void __launch_bounds__(256, 2) k_fxcorr3(xc_args a, const void* stw_g, const void* full_g) {
    using F           = xc3_cfg<LOGN>;
    using P           = typename F::P;
    using X           = typename F::X;
    constexpr int N   = F::N;
    constexpr int NT  = F::NT;
    constexpr int TT  = F::TT;
    constexpr int M   = F::M;
    constexpr int RS  = F::RS;
    constexpr int BAR = TT <= 32 ? -1 : 0;    // a window's threads share a warp: its exchanges are private
    extern __shared__ __align__(128) unsigned char smem[];
    float*                in0 = reinterpret_cast<float*>(smem);
    cpx<float>*           xch = reinterpret_cast<cpx<float>*>(in0 + 2 * F::TILE);
    cpx<float>*           stw = xch + X::size;
    __shared__ uint64_t   full[2];
    __shared__ long long  s_tile[2];
    __shared__ xc3_window win[2][M];
    __shared__ uint32_t   s_tmem;
    const int             tid   = threadIdx.x;
    const int             m     = tid / TT;
    const int             t     = tid - m * TT;
    const float*          src   = reinterpret_cast<const float*>(a.src);
    float*                dst   = reinterpret_cast<float*>(a.dst);
    const long long       ntile = (a.total + M - 1) / M;
    const int             htile = (a.hwait + M - 1) / M;    // earlier tiles to wait for, in place

    if constexpr (F::FULL > 0) copy_table_to_smem<F::FULL * 8>(stw, full_g, tid, NT);
    if constexpr (stage_tw_size<P>() > F::SKIP) {
        copy_table_to_smem<(stage_tw_size<P>() - F::SKIP) * 8>(stw + F::FULL, static_cast<const cpx<float>*>(stw_g) + F::SKIP,
                                                               tid, NT);
    }
    if (tid < 32) {
        tmem_alloc(&s_tmem, 64);
        tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = s_tmem;
    const uint32_t tcol  = tbase + ((uint32_t)(32 * ((tid / 32) % 4)) << 16) + (uint32_t)(tid / 128) * 32;
    {
        const cpx<float>* ks = reinterpret_cast<const cpx<float>*>(a.kspec);
        uint32_t          kr[32];
        static_for<16>([&](auto ic) {
            constexpr int    i = decltype(ic)::value;
            const cpx<float> k = ldg_cpx(ks + t + i * TT);
            kr[2 * i]          = __float_as_uint(k.re);
            kr[2 * i + 1]      = __float_as_uint(k.im);
        });
        tmem_st32(tcol, kr);
    }

    // warp 0: the tile `next` into stage s (its lanes take the windows in
    // turn), then the tile after it, requested now and used at the next call
    long long next  = 0;
    auto      claim = [&](long long last) -> long long {
        return a.inplace ? (long long)atomicAdd(a.counter, 1u) : last + gridDim.x;
    };
    auto issue = [&](int s) {
        const long long tile = __shfl_sync(0xffffffffu, next, 0);
        uint32_t        sum  = 0;
        for (int w = tid; w < M; w += 32) {
            const long long item = tile * M + w;
            xc3_window      x{0, 0, 0, 0};
            if (tile < ntile && item < a.total) {
                const long long ch = item / a.nblk, b = (item - ch * a.nblk) * a.step, b0 = b - a.in_shift;
                x.lo   = (int)max(0LL, min((long long)N, -b0));
                x.hi   = (int)max((long long)x.lo, min((long long)N, a.len - b0));
                x.nout = (int)min((long long)a.step, a.len - b);
                x.dst  = ch * a.dst_stride + 2 * b;
                sum += (uint32_t)((x.hi - x.lo + 7) / 8) * 64;
            }
            win[s][w] = x;
        }
        sum = __reduce_add_sync(0xffffffffu, sum);
        if (tid == 0) {
            s_tile[s] = tile;
            if (tile < ntile) mbar_arrive_expect_tx(&full[s], sum);
        }
        __syncwarp();
        if (tile < ntile) {
            for (int w = tid; w < M; w += 32) {
                const long long item = tile * M + w;
                const int       lo = win[s][w].lo, hi = win[s][w].hi;
                if (hi > lo) {
                    const long long ch = item / a.nblk, b0 = (item - ch * a.nblk) * a.step - a.in_shift;
                    bulk_g2s(in0 + s * F::TILE + w * RS + 2 * lo, src + ch * a.src_stride + 2 * (b0 + lo),
                             (uint32_t)((hi - lo + 7) / 8) * 64, &full[s]);
                }
            }
        }
        if (tid == 0) next = claim(tile);
    };
    if (tid < 32) {
        if (tid == 0) next = a.inplace ? (long long)atomicAdd(a.counter, 1u) : blockIdx.x;
        issue(0);
        issue(1);
    }
    __syncthreads();

    bool bad = false;    // this warp gave up a wait
    for (int k = 0;; ++k) {
        const int       s    = k & 1;
        const long long tile = s_tile[s];
        if (tile >= ntile) break;    // claims only grow: nothing is in flight
        const bool ok = mbar_wait_bounded(&full[s], (uint32_t)((k >> 1) & 1));
        if (__syncthreads_or(!ok || bad)) {
            // give up: record it, let the copies in flight land, leave together
            if (tid == 0) {
                atomicExch(a.error, 1);
                mbar_wait_bounded(&full[s], (uint32_t)((k >> 1) & 1), 100000000ull);
                if (s_tile[s ^ 1] < ntile) mbar_wait_bounded(&full[s ^ 1], (uint32_t)(((k + 1) >> 1) & 1), 100000000ull);
            }
            break;
        }
        if (a.inplace && tid == 0) {
            st_release(a.flags + tile, 1u);    // this tile's windows are loaded
        }
        const xc3_window x  = win[s][m];
        const float*     in = in0 + s * F::TILE + m * RS;
        cpx<float>       v[16];
        static_for<16>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            v[i]            = lds_swapped<float, F::SW>(in, pk<3>(t + i * TT), 8);
        });
        if (x.lo > 0 || x.hi < N) xc3_clip<TT>(v, t, x.lo, x.hi);
        fence_proxy_async_smem();
        __syncthreads();    // stage s and its windows are read: refill them
        if (tid < 32) issue(s);
        xc3_transform<LOGN, BAR>(v, xch, m, t, stw);
        // conj(X * conj(K)) or conj(X * K), K eight values at a time
        __syncwarp();
        static_for<2>([&](auto hc) {
            constexpr int h = decltype(hc)::value;
            uint32_t      kq[16];
            tmem_ld16(tcol + 16 * h, kq);
            static_for<8>([&](auto jc) {
                constexpr int    j = decltype(jc)::value, i = 8 * h + j;
                const cpx<float> kv = {__uint_as_float(kq[2 * j]), __uint_as_float(kq[2 * j + 1])};
                const cpx<float> c  = {v[i].re, -v[i].im};
                v[i]                = a.conj_kernel ? cmul(c, kv) : cmulc(c, kv);
            });
        });
        // in place: the first look at the flags, so that the wait below rarely
        // has to read one
        const int lane = tid % 32;
        bool      seen = true;
        if (a.inplace && lane < htile && lane < tile) seen = ld_acquire(a.flags + (tile - 1 - lane)) != 0u;
        xc3_transform<LOGN, BAR>(v, xch, m, t, stw);
        if (a.inplace) {
            // every warp waits for itself, so that no barrier holds the outputs
            // of those that are done; one that gives up stores nothing, and the
            // block leaves at the next tile's vote
            bool late = false;
            for (long long d = lane; d < htile && d < tile && !late; d += 32) {
                const unsigned* f = a.flags + (tile - 1 - d);
                if ((d == lane && seen) || ld_acquire(f) != 0u) continue;
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
                continue;
            }
        }
        // v[i] = conj of circular output t + i*TT, output t + i*TT - out_shift of the block
        float* d = dst + x.dst - 2 * a.out_shift;    // out_shift is whole packs
        static_for<16>([&](auto ic) {
            constexpr int i  = decltype(ic)::value;
            const int     mo = t + i * TT - a.out_shift;
            if (mo >= 0 && mo < x.nout) {
                __stcs(d + pk<3>(t + i * TT), v[i].re);
                __stcs(d + pk<3>(t + i * TT) + 8, -v[i].im);
            }
        });
    }
    tc_fence_before();
    __syncthreads();
    if (tid < 32) tmem_dealloc(tbase, 64);
}

// ---------------------------------------------------------------------------
// Kernel gradient: per tile the gy blocks (stage 0, zero beyond a block's
// outputs) and the x windows (stage 1) are transformed one after the other
// while the next tile's are on their way; a thread's 16 values of FFT(gy) and
// of the running sum of FFT(x) * conj(FFT(gy)) stay in tensor memory, 32
// columns each.  Tiles go round the blocks, so the sums do not depend on
// timing.  At the end the block adds its M windows' sums and writes them in
// natural order to acc[blockIdx.x].
template<int LOGN>
__global__ void __launch_bounds__(256, 2) k_fxcorr3_kgrad(kg_args a, const void* stw_g) {
    using F           = xc3_cfg<LOGN>;
    using P           = typename F::P;
    using X           = typename F::X;
    constexpr int N   = F::N;
    constexpr int NT  = F::NT;
    constexpr int TT  = F::TT;
    constexpr int M   = F::M;
    constexpr int RS  = F::RS;
    constexpr int BAR = TT <= 32 ? -1 : 0;
    extern __shared__ __align__(128) unsigned char smem[];
    float*              in0 = reinterpret_cast<float*>(smem);
    cpx<float>*         xch = reinterpret_cast<cpx<float>*>(in0 + 2 * F::TILE);
    cpx<float>*         stw = xch + X::size;
    __shared__ uint64_t full[2];
    __shared__ int      valid[2][M];    // window elements that count
    __shared__ uint32_t s_tmem;
    const int           tid   = threadIdx.x;
    const int           m     = tid / TT;
    const int           t     = tid - m * TT;
    const long long     ntile = (a.total + M - 1) / M;

    stage_tw_to_smem<P, float>(stw, stw_g, tid, NT);
    if (tid < 32) {
        tmem_alloc(&s_tmem, 128);
        tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tbase = s_tmem;
    const uint32_t tcol  = tbase + ((uint32_t)(32 * ((tid / 32) % 4)) << 16) + (uint32_t)(tid / 128) * 64;
    {
        uint32_t z[32];
        static_for<32>([&](auto jc) { z[decltype(jc)::value] = 0u; });
        tmem_st32(tcol + 32, z);
    }
    // warp 0: the gy blocks (s = 0) or x windows (s = 1) of a tile into stage s
    auto issue = [&](long long tile, int s) {
        const float* base = reinterpret_cast<const float*>(s ? a.x : a.gy);
        uint32_t     sum  = 0;
        for (int w = tid; w < M; w += 32) {
            const long long item = tile * M + w;
            int             n    = 0;
            if (item < a.total) {
                const long long b = (item % a.nblk) * a.step;
                n                 = (int)min((long long)(s ? N : a.step), a.len - b);
                sum += (uint32_t)((n + 7) / 8) * 64;
            }
            valid[s][w] = n;
        }
        sum = __reduce_add_sync(0xffffffffu, sum);
        if (tid == 0) mbar_arrive_expect_tx(&full[s], sum);
        __syncwarp();
        for (int w = tid; w < M; w += 32) {
            const long long item = tile * M + w;
            if (item < a.total) {
                const long long ch = item / a.nblk, b = (item - ch * a.nblk) * a.step;
                bulk_g2s(in0 + s * F::TILE + w * RS, base + ch * a.stride + 2 * b,
                         (uint32_t)((valid[s][w] + 7) / 8) * 64, &full[s]);
            }
        }
    };
    if (tid < 32 && blockIdx.x < ntile) {
        issue(blockIdx.x, 0);
        issue(blockIdx.x, 1);
    }
    __syncthreads();

    uint32_t par  = 0;
    bool     fail = false;
    for (long long tile = blockIdx.x; tile < ntile && !fail; tile += gridDim.x, par ^= 1) {
        for (int s = 0; s < 2; ++s) {
            const bool ok = mbar_wait_bounded(&full[s], par);
            if (__syncthreads_or(!ok)) {
                // give up: record it and let the copies in flight land first
                if (tid == 0) {
                    atomicExch(a.error, 1);
                    mbar_wait_bounded(&full[s], par, 100000000ull);
                    if (s == 0 || tile + gridDim.x < ntile) mbar_wait_bounded(&full[s ^ 1], s ? par ^ 1 : par, 100000000ull);
                }
                fail = true;
                break;
            }
            const int    n  = valid[s][m];
            const float* in = in0 + s * F::TILE + m * RS;
            cpx<float>   v[16];
            static_for<16>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                v[i]            = lds_swapped<float, F::SW>(in, pk<3>(t + i * TT), 8);
            });
            if (n < N) xc3_clip<TT>(v, t, 0, n);
            fence_proxy_async_smem();
            __syncthreads();    // stage s is read: refill it
            if (tid < 32 && tile + gridDim.x < ntile) issue(tile + gridDim.x, s);
            stage_compute_tab<P, 0>(v, t, stw);
            run_stages_tab<P, X, true, BAR>(v, xch, m, t, stw);
            __syncwarp();
            if (s == 0) {
                uint32_t r[32];
                static_for<16>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    r[2 * i]        = __float_as_uint(v[i].re);
                    r[2 * i + 1]    = __float_as_uint(v[i].im);
                });
                tmem_st32(tcol, r);
            } else {
                // sum += X * conj(GY), eight values at a time
                static_for<2>([&](auto hc) {
                    constexpr int h = decltype(hc)::value;
                    uint32_t      gq[16], sq[16];
                    tmem_ld16(tcol + 16 * h, gq);
                    tmem_ld16(tcol + 32 + 16 * h, sq);
                    static_for<8>([&](auto jc) {
                        constexpr int    j = decltype(jc)::value;
                        const cpx<float> p = cmulc(v[8 * h + j], cpx<float>{__uint_as_float(gq[2 * j]),
                                                                             __uint_as_float(gq[2 * j + 1])});
                        sq[2 * j]          = __float_as_uint(__uint_as_float(sq[2 * j]) + p.re);
                        sq[2 * j + 1]      = __float_as_uint(__uint_as_float(sq[2 * j + 1]) + p.im);
                    });
                    tmem_st16(tcol + 32 + 16 * h, sq);
                });
            }
        }
    }
    if (!fail) {
        cpx<float>* acc = reinterpret_cast<cpx<float>*>(a.acc) + (long long)blockIdx.x * N;
        uint32_t    sq[32];
        tmem_ld32(tcol + 32, sq);
        if constexpr (M == 1) {
            static_for<16>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                acc[t + i * TT] = {__uint_as_float(sq[2 * i]), __uint_as_float(sq[2 * i + 1])};
            });
        } else {
            __syncthreads();    // the exchange buffer is no longer read
            static_for<16>([&](auto ic) {
                constexpr int i             = decltype(ic)::value;
                xch[X::idx(m, t + i * TT)] = {__uint_as_float(sq[2 * i]), __uint_as_float(sq[2 * i + 1])};
            });
            __syncthreads();
            for (int q = tid; q < N; q += NT) {
                cpx<float> sum = {0.f, 0.f};
                for (int w = 0; w < M; ++w) sum = sum + xch[X::idx(w, q)];
                acc[q] = sum;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (tid < 32) tmem_dealloc(tbase, 128);
}

}    // namespace pcxg
