// One persistent launch for a whole batch of four-step transforms N = N1*N2.
//
// The column and row passes of every transform are work items of a single
// grid: for transform r there are TC = N2/C column tiles (C columns of N1
// points, TMA tensor copies of the source, twiddled, written to a scratch
// slot) and TR = N1/CR row tiles (CR rows of N2 points read back from the
// slot, written to the destination).  Items are ordered
//     col(0..lag-1), [col(r+lag), row(r)] for r = 0.., row(batch-lag..)
// and CTA b takes items b, b + grid, b + 2*grid, ...  A row tile waits until
// all column tiles of its transform are written (col_done[r] == TC); a column
// tile of transform r writes slot r & (nslot-1) only after every row tile of
// transform r - nslot has read it (row_done[r - nslot] == TR).  Every
// dependency points to an earlier item, so the smallest unfinished item can
// always run.
//
// Each CTA has NT compute threads and two helper warps, so that no wait sits
// on the compute warps' path except their own tile landing:
//  * the producer warp walks the CTA's items, waits for a ring stage to be
//    free and for the item's dependency on other CTAs, and issues the TMA
//    copies into the ST-stage ring (for a column tile it also tells the
//    compute warps when the slot may be written);
//  * the publisher warp walks the same items and publishes each completion as
//    soon as it happens (col_done once a column tile is written; row_done once
//    a row tile's scratch rows have landed in shared memory and their L2 lines
//    are dropped unwritten).  Where outputs are stored by TMA (fs_cfg::TS) it
//    also issues those copies, a column tile's once its slot may be written
//    (a wait for earlier items, as every wait is); else it never waits on
//    another CTA.
// A stage is refilled after the compute warps are done with it and the
// publisher has passed its item (empty[s] counts both), so no barrier phase is
// ever overtaken.  With three stages the exchanges of the sub-transforms run
// in place in the item's own stage buffer (the tile is in registers by the
// first exchange barrier), which keeps the ring within the shared memory of
// two stages plus an exchange buffer while the producer runs two items ahead.
//
// Compared with one launch per pass per scratch chunk this removes the ramp
// and tail of every short launch (the SMs were idle ~30% of each chunk).
#pragma once

#include "pcx_fft_v2.cuh"

namespace pcxg {

struct fs_args {
    const void* src;
    void*       dst;
    long long   src_stride;    // reals between transforms
    long long   dst_stride;
    long long   batch;
    int         conj_in;
    int         conj_out;
    double      scale;
    const void* stw1;     // full stage tables of the N1 and N2 sub-transforms (fs_full_tw_*)
    const void* stw2;
    const void* tw_hi;    // W_N^(i*N2), i < N1 (FS_PLAIN, as tw_lo and tw_b)
    const void* tw_lo;    // W_N^i, i < N2
    const void* tw_b;     // W_{16*N2}^m
    const void* tw;       // other forms: four-step twiddles (k_fs_twiddles), [row][n2], FS_IN: [row][bitrev(n2)]
    void*       scratch;  // nslot slots of N complex
    int         nslot;    // a power of two: transform r uses slot r & (nslot - 1)
    int         lag;      // transforms between a column pass and its row pass
    int*        col_done;    // one per transform, zero at the start and at the end of a launch
    int*        row_done;    // the same, right behind col_done
    int*        ticket;      // blocks that are done with the counters, likewise zero outside a launch
    int*        error;
    // forms other than FS_PLAIN only
    int         lp_src;     // log2 pack widths
    int         lp_dst;
    int         src_len;    // valid source elements per transform, at least N2 (zero-extended to N)
    int         order;      // FS_OUT: the output's order; FS_IN: the input's
};

// Forms of the kernel.  FS_PLAIN is the hot one: default packs, whole rows,
// natural order on both sides.  The others run the same items in the same
// order (one built variant per size, the size's default):
//  * FS_ANY: source and destination packs of 1 up to the default width, and
//    short sources.  A column tile's row segment and a row tile's output
//    segment are the same contiguous reals at every such width, so only the
//    per-thread base and the distance of the imaginary part change.  Source
//    rows n1 that are whole come by TMA (the tensor map ends there and fills
//    the rest with zeros); the one partial row is read by its threads.
//  * FS_OUT (forward into bit_reversed / unordered order): frequency
//    k = k2*N1 + k1 goes to position bitrev(k1)*N2 + bitrev(k2), so a row tile's
//    outputs are whole contiguous rows, and the 16 values of a thread
//    (k2 = t + i*TT) are 16 consecutive positions of one: they are staged in
//    the tile's stage with 16-byte stores (8 rows on 8 bank groups by an XOR)
//    and leave as 16-byte stores, a quarter of the store instructions of the
//    transposed natural-order output.
//  * FS_IN (inverse from such an order): the N1 inputs of column n2 are the
//    contiguous run r = bitrev(n2), so a column tile is C whole source rows
//    brought in by bulk copies, each thread's 16 inputs one run of it.
//    The scratch keeps the columns in the order r, and a row tile reads its
//    n2 from bitrev(n2), again one run of 16 per thread.
// 2^15, 301 transforms, forward into `unordered` and inverse back: two
// launches per chunk of general kernels 427 us, these 121 us.
constexpr int FS_PLAIN = 0;
constexpr int FS_ANY   = 1;
constexpr int FS_OUT   = 2;
constexpr int FS_IN    = 3;

// Items a block from which outputs are stored by TMA (fs_cfg::TS).
constexpr int FS_TS_ROUNDS = 12;

// Register i of the 16 a thread holds (element t + i*TT) at place q of its run
// of 16 consecutive positions: i = bitrev4(q), or bitrev4(sigma(q)) in the
// unordered order (sigma moves bits (0,1,2,3) to (2,1,3,0)).
__host__ __device__ constexpr int run_reg(int q, bool unordered) {
    const int s = unordered ? (((q & 1) << 2) | (q & 2) | (((q >> 2) & 1) << 3) | ((q >> 3) & 1)) : q;
    return ((s & 1) << 3) | ((s & 2) << 1) | ((s & 4) >> 1) | ((s & 8) >> 3);
}

// Real f (0..31) of a run of 16 packed elements at pack width 2^LPX.
template<int LPX, bool UNORD, class T>
__device__ __forceinline__ T& run_real(cpx<T> (&v)[16], int f) {
    const int q = ((f >> (LPX + 1)) << LPX) | (f & ((1 << LPX) - 1));
    cpx<T>&   x = v[run_reg(q, UNORD)];
    return (f >> LPX) & 1 ? x.im : x.re;
}
template<class T>
struct alignas(16) vec16 {
    T x[16 / sizeof(T)];
};
// The 16 elements of the run at `p` (16-byte aligned) into the registers they belong to.
template<int LPX, bool UNORD, class T>
__device__ __forceinline__ void run_load(cpx<T> (&v)[16], const T* p) {
    constexpr int W = 16 / (int)sizeof(T);
    static_for<32 / W>([&](auto jc) {
        constexpr int  j = decltype(jc)::value;
        const vec16<T> w = *reinterpret_cast<const vec16<T>*>(p + j * W);
        static_for<W>([&](auto uc) {
            constexpr int u                       = decltype(uc)::value;
            run_real<LPX, UNORD>(v, j * W + u) = w.x[u];
        });
    });
}
// The run into 16-byte unit j ^ key of its 32 / W units at `p`.
template<int LPX, bool UNORD, class T>
__device__ __forceinline__ void run_store(cpx<T> (&v)[16], T* p, int key) {
    constexpr int W = 16 / (int)sizeof(T);
    static_for<32 / W>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        vec16<T>      w;
        static_for<W>([&](auto uc) {
            constexpr int u = decltype(uc)::value;
            w.x[u]          = run_real<LPX, UNORD>(v, j * W + u);
        });
        *reinterpret_cast<vec16<T>*>(p + (j ^ key) * W) = w;
    });
}

// Variant of the one-launch four-step: split N = 2^LOGN1 * 2^LOGN2, MINB
// resident blocks per SM (tiles of 64 KB / MINB: two blocks of 32 KB tiles
// let one block issue while the other waits at a barrier, and need both
// sub-transforms <= 512 points so that a tile still spans whole 32-byte
// sectors of its rows), and ST ring stages (3: the exchanges run in place in
// the item's stage; 2: a separate exchange buffer).  pcx_plan_tune times the
// variants that are built for a size and keeps the fastest.
template<class T, int LOGN1, int LOGN2, int MINB_ = (LOGN1 <= 9 ? 2 : 1), int ST_ = 3>
struct fs_cfg {
    static constexpr int N1   = 1 << LOGN1;
    static constexpr int N2   = 1 << LOGN2;
    static constexpr int MINB = MINB_;
    static constexpr int TILE = 65536 / MINB / (int)sizeof(cpx<T>);
    static constexpr int G8   = 64 / (2 * (int)sizeof(T));
    static constexpr int LP   = G8 == 8 ? 3 : 2;
    static constexpr int C    = (TILE >> LOGN1) > G8 ? (TILE >> LOGN1) : G8;    // columns per column tile
    static constexpr int CR   = (TILE >> LOGN2) > G8 ? (TILE >> LOGN2) : G8;    // rows per row tile
    using P1                  = splan<LOGN1>;
    using P2                  = splan<LOGN2>;
    static constexpr int NT   = C * P1::TT;
    static_assert(NT == CR * P2::TT, "both passes use the same block");
    static constexpr int TC   = N2 / C;
    static constexpr int TR   = N1 / CR;
    static constexpr int RSI  = N2 + 2;    // padded shared row of a row tile (complex)
    static constexpr int COLB = N1 * 2 * C * (int)sizeof(T);
    static constexpr int ROWB = CR * RSI * (int)sizeof(cpx<T>);
    using X1                  = xch_interleaved<N1, C>;
    using X2                  = xch_grouped<N2, CR, G8>;
    static constexpr int XB   = smem_align16((X1::size > X2::size ? X1::size : X2::size) * (int)sizeof(cpx<T>));
    static constexpr int ST   = ST_;
    static constexpr bool IP  = ST == 3;
    // Outputs of both passes staged in the item's stage and stored by TMA.  A
    // row tile's transposed stores are four 32-byte sectors in four lines per
    // instruction, 32 instructions a thread, and held the load/store queue
    // (lg_throttle the first stall at 2^20).  The exchange layout is a TMA box
    // already: 17 rows of 64 bytes (or of the columns) per 16, the 17th, the
    // bank padding, outside the tensor view and so not written; each thread
    // puts its outputs over values that it (row tiles: a lane beside it) read
    // last, without a block barrier, and the publisher issues one to eight
    // copies a tile.  The stage is held until its copy has read it, which costs
    // the short tiles more than it saves, and the two tensor maps cost a call
    // 3.5 us on the host: launch_fs takes it from FS_TS_ROUNDS items a block on.
    // GB/s at 512 MB, from registers and
    // staged: FP32 2^14 3405 3261, 2^15 3459 3249, 2^16 3313 3015, 2^17 2947
    // 3043, 2^18 2867 2950, 2^19 2523 2818, 2^20 2541 2830; FP64 2^14 3429 3502,
    // 2^15 3372 3399, 2^16 3351 3508, 2^17 2691 3254, 2^18 2429 2928.
    static constexpr bool TS  = IP && (sizeof(T) == 8 || LOGN1 >= 9 || LOGN2 >= 9);
    static_assert(ST == 2 || ST == 3, "two or three ring stages");
    static constexpr int TILEB = COLB > ROWB ? COLB : ROWB;
    static constexpr int STAGE = ((IP ? (TILEB > XB ? TILEB : XB) : TILEB) + 127) / 128 * 128;
    static constexpr int BASE = ST * STAGE + (IP ? 0 : XB);
    // one stage table for both passes when the larger sub-transform's serves
    // the smaller one (equal halves, or 512 with 1024 points): room for it
    // beside a three-stage ring of 64 KB tiles
    using PL                  = std::conditional_t<(LOGN1 >= LOGN2), P1, P2>;
    static constexpr bool ONE = full_tab_serves<P1, PL>() && full_tab_serves<P2, PL>();
    using PT1                 = std::conditional_t<ONE, PL, P1>;
    using PT2                 = std::conditional_t<ONE, PL, P2>;
    static constexpr int TB1  = fs_full_tw_size<PT1>() * (int)sizeof(cpx<T>);
    static constexpr int TB2  = ONE ? 0 : fs_full_tw_size<P2>() * (int)sizeof(cpx<T>);
    static constexpr bool SH  = stw_fits(BASE, TB1 + TB2, MINB);
    static constexpr int SMEM = SH ? BASE + TB1 + TB2 : BASE;
    static constexpr int BOXY = N1 < 256 ? N1 : 256;
    // FS_IN: padded shared row of a column tile (reals); 16 bytes in FP32, so
    // the 16-byte reads of 8 neighbouring columns fall on 8 bank groups
    static constexpr int RSC  = 2 * N1 + 4;
};

__device__ __forceinline__ void fence_proxy_async_global() {
    asm volatile("fence.proxy.async.global;" ::: "memory");
}

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Bounded wait for *p >= target (about one second); false on timeout.
__device__ __forceinline__ bool fs_wait(const int* p, int target) {
    if (ld_acquire(p) >= target) return true;
    const unsigned long long t0 = timer_ns();
    while (true) {
        if (ld_acquire(p) >= target) return true;
        if (timer_ns() - t0 > 1000000000ull) return false;
        __nanosleep(64);
    }
}

struct fs_item {
    int row;     // 0: column tile, 1: row tile
    int r;       // transform
    int tile;
};

// counter += 1 with release semantics at GPU scope: this thread's earlier
// writes, and those it has observed, are visible to whoever acquires the count
__device__ __forceinline__ void red_release_add(int* p, int v) {
    asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Twiddles of the forms other than FS_PLAIN: W_N^(k1*n2), k1 = t + i*TT, i =
// B*a + b, as W_N^((t + B*a*TT)*n2) (row a*TT + t) times u^b, u = W_N^(TT*n2)
// (row N1/B + b - 1), all generated in FP64 and rounded once; a row of N2 entries
// is read by neighbouring columns at once.  The fewer of them are products the
// smaller the error and the larger the table: B = 2 (9 entries a thread) where 4
// (7 entries) would be less accurate than the general kernels, whose twiddles
// are products of two half-size tables' entries; 8 and 16 (9 and 16) where the
// table would pass 2 MB, whose allocation takes 0.35 ms.
// Error against FP64, interleaved to packed, general kernels, one entry times
// powers of u (up to three products), B = 4, B = 2: 2^15 1.439e-7 1.472e-7
// 1.447e-7 1.434e-7; 2^17 1.573e-7 1.597e-7 1.573e-7 -; 2^20 1.691e-7 1.711e-7
// 1.69e-7 - (B = 8 1.69e-7).  GB/s, 512 MB: 2^15 - 3292 3231 3210, 2^20 - 2800
// 2672 - (2604).
template<class T>
__host__ __device__ constexpr int fs_tw_group(int log_n) {
    return sizeof(T) == 4 ? (log_n <= 16 ? 2 : log_n <= 19 ? 4 : 8) : (log_n <= 18 ? 4 : log_n <= 19 ? 8 : 16);
}
template<class T>
__host__ __device__ constexpr int fs_tw_rows(int log_n1, int log_n) {
    return (1 << log_n1) / fs_tw_group<T>(log_n) + fs_tw_group<T>(log_n) - 1;
}
template<class T>
__global__ void k_fs_twiddles(cpx<T>* out, int log_n1, int log_n2, int permuted) {
    const int log_n = log_n1 + log_n2, tt = 1 << (log_n1 - 4), grp = fs_tw_group<T>(log_n);
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= fs_tw_rows<T>(log_n1, log_n) << log_n2) return;
    const int       row = q >> log_n2, r = q & ((1 << log_n2) - 1), bases = 16 / grp * tt;
    const long long n2   = permuted ? (int)brev(r, log_n2) : r;
    const long long mult = row < bases ? row % tt + grp * tt * (row / tt) : tt * (row - bases + 1);
    const long long e    = (n2 * mult) & ((1LL << log_n) - 1);
    double          s, c;
    sincospi(2.0 * (double)e / (double)(1LL << log_n), &s, &c);
    out[q] = {T(c), T(-s)};
}

// Item j of the queue (32-bit: the launch holds fewer than 2^31 items).  TC
// and TR are powers of two, TC + TR a constant: no division is a real one.
template<int TC, int TR>
__device__ __forceinline__ fs_item fs_decode(uint32_t j, uint32_t batch, uint32_t lag) {
    const uint32_t A = lag * TC;
    if (j < A) return {0, (int)(j / TC), (int)(j % TC)};
    j -= A;
    constexpr uint32_t G      = TC + TR;
    const uint32_t     steady = (batch - lag) * G;
    if (j < steady) {
        const uint32_t q = j / G;
        const int      w = (int)(j - q * G);
        return w < TC ? fs_item{0, (int)(q + lag), w} : fs_item{1, (int)q, w - TC};
    }
    j -= steady;
    return {1, (int)(batch - lag + j / TR), (int)(j % TR)};
}

template<class T, int LOGN1, int LOGN2, int MINB, int ST_, int FORM, bool TS>
__global__ void __launch_bounds__(fs_cfg<T, LOGN1, LOGN2, MINB, ST_>::NT + 64, MINB)
    k_fourstep(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap tscr,
               const __grid_constant__ CUtensorMap tdst, fs_args a) {
    using F            = fs_cfg<T, LOGN1, LOGN2, MINB, ST_>;
    using P1           = typename F::P1;
    using P2           = typename F::P2;
    constexpr int N1   = F::N1;
    constexpr int N2   = F::N2;
    constexpr int NT   = F::NT;    // compute threads; then the producer warp, then the publisher warp
    constexpr int NW   = NT / 32;
    constexpr int ST   = F::ST;
    constexpr bool IP  = F::IP;
    constexpr int C    = F::C;
    constexpr int CR   = F::CR;
    constexpr int TC   = F::TC;
    constexpr int TR   = F::TR;
    constexpr int LP   = F::LP;
    constexpr int PK   = 1 << LP;
    constexpr int G8   = F::G8;
    constexpr int SEG  = 2 * C;
    constexpr int SW   = sizeof(T) == 8 ? 8 : 16;
    constexpr int RSI  = F::RSI;
    constexpr int RROW = N2 * (int)sizeof(cpx<T>);
    constexpr bool SH  = F::SH;
    static_assert(!TS || F::TS, "outputs staged in the item's stage and stored by TMA");
    constexpr bool TSR = TS && FORM != FS_OUT;       // row tiles too (FS_OUT stores whole rows itself)
    static_assert(FORM != FS_IN || C * F::RSC * (int)sizeof(T) <= F::STAGE, "a column tile of whole rows fits a stage");
    static_assert(FORM != FS_OUT || CR * 2 * N2 * (int)sizeof(T) <= (IP ? F::STAGE : F::XB), "a staged row tile fits");
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char*      ring = smem;
    cpx<T>*             tws1 = reinterpret_cast<cpx<T>*>(smem + F::BASE);
    cpx<T>*             tws2 = F::ONE ? tws1 : tws1 + F::TB1 / (int)sizeof(cpx<T>);
    // with one table it is the larger sub-transform's
    const void*         gtab1 = F::ONE && LOGN2 > LOGN1 ? a.stw2 : a.stw1;
    const void*         gtab2 = F::ONE && LOGN1 > LOGN2 ? a.stw1 : a.stw2;
    __shared__ uint64_t full[ST];      // TMA bytes landed
    __shared__ uint64_t empty[ST];     // the stage may be refilled
    __shared__ uint64_t slotok[ST];    // !TS, column tile: its scratch slot may be written
    __shared__ uint64_t written[ST];   // TS: outputs staged (FS_OUT rows: stored); !TS: column tile written
    cpx<T>*             scr   = reinterpret_cast<cpx<T>*>(a.scratch);
    const int           tid   = threadIdx.x;
    const uint32_t      items = (uint32_t)a.batch * (uint32_t)(TC + TR);    // < 2^31 (host check)
    const uint32_t      batch = (uint32_t)a.batch;
    const uint32_t      lag   = (uint32_t)a.lag;
    const uint32_t      G     = gridDim.x;
    const long long     mask  = a.nslot - 1;

    if constexpr (SH) {
        copy_table_to_smem<F::TB1>(tws1, gtab1, tid, NT + 64);
        if constexpr (!F::ONE) copy_table_to_smem<F::TB2>(tws2, a.stw2, tid, NT + 64);
    }
    if (tid == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], TS ? 1 : NW + 1);
            mbar_init(&slotok[s], 1);
            mbar_init(&written[s], NW);
        }
        fence_barrier_init();
    }
    __syncthreads();

    if (tid >= NT + 32) {
        // ======================= publisher warp
        const int lane    = tid - NT - 32;
        const uint64_t pol = l2_evict_first_policy();    // outputs are written once
        uint32_t  colpar  = 0;    // !TS, bit s: parity of the next `written` wait on stage s
        bool      fail    = false;
        int       s       = 0;
        uint32_t  par     = 0;
        for (uint32_t j = blockIdx.x; j < items && !fail; j += G, s = s + 1 == ST ? 0 : s + 1, par ^= s == 0) {
            const fs_item  it  = fs_decode<TC, TR>(j, batch, lag);
            int            ok  = 1;
            if (it.row) {
                // the tile's scratch rows are in shared memory: drop their L2
                // lines unwritten and count the tile
                if (lane == 0) ok = mbar_wait_bounded(&full[s], par) ? 1 : 0;
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (ok) {
                    const char* g = reinterpret_cast<const char*>(scr + (it.r & mask) * (long long)(N1 * N2) +
                                                                  (long long)it.tile * CR * N2);
                    for (int q = lane; q < CR * RROW / 128; q += 32) l2_discard(g + (size_t)q * 128);
                    __syncwarp();
                    if (lane == 0) red_release_add(a.row_done + it.r, 1);
                }
            }
            if constexpr (TS) {
                // the compute warps' staged outputs leave by TMA: a column
                // tile to its scratch slot once that may be written (counted
                // when the copy is complete), a row tile to the destination
                if (lane == 0 && ok) {
                    ok = mbar_wait_bounded(&written[s], par) ? 1 : 0;
                    const unsigned char* buf = ring + s * F::STAGE;
                    if (ok && !it.row) {
                        ok = it.r < a.nslot || fs_wait(a.row_done + (it.r - a.nslot), TR);
                        if (ok) {
                            fence_proxy_async_global();
                            tma_store_4d(&tscr, buf, 2 * it.tile * C, 0, 0, (int)(it.r & mask));
                            bulk_commit();
                            bulk_wait();
                            fence_proxy_async_global();
                            red_release_add(a.col_done + it.r, 1);
                        }
                    } else if (ok && TSR) {
#pragma unroll
                        for (int h = 0; h < CR / G8; ++h) {
                            tma_store_4d_hint(&tdst, buf + h * F::X2::LP * G8 * (int)sizeof(cpx<T>),
                                              2 * (it.tile * CR + h * G8), 0, 0, it.r, pol);
                        }
                        bulk_commit();
                        bulk_wait_read();
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
            } else if (!it.row) {
                // the compute warps' stores of the tile are done: make them
                // visible to other CTAs' TMA reads, then count the tile
                if (lane == 0) ok = mbar_wait_bounded(&written[s], (colpar >> s) & 1u) ? 1 : 0;
                ok = __shfl_sync(0xffffffffu, ok, 0);
                colpar ^= 1u << s;
                if (ok && lane == 0) {
                    fence_proxy_async_global();
                    red_release_add(a.col_done + it.r, 1);
                }
            }
            if (!ok) {
                fail = true;
                if (lane == 0) atomicExch(a.error, 1);
            } else if (lane == 0) {
                mbar_arrive(&empty[s]);
            }
        }
        // nothing is in flight when the block exits; the last block to get
        // here (every one does, also after giving up) leaves the counters zero
        // for the next launch, which a memset before each call did for one more
        // launch and 2-3 us of a short call
        int last = 0;
        if (lane == 0) {
            if (TS) bulk_wait();
            __threadfence();
            last = atomicAdd(a.ticket, 1) == (int)gridDim.x - 1;
            __threadfence();
        }
        if (__shfl_sync(0xffffffffu, last, 0)) {
#pragma unroll 4
            for (uint32_t q = lane; q < 2 * batch; q += 32) a.col_done[q] = 0;
            if (lane == 0) *a.ticket = 0;
        }
        return;
    }

    if (tid >= NT) {
        // ======================= producer warp
        const int      lane   = tid - NT;
        const uint64_t pol    = l2_evict_first_policy();    // column tiles are read once
        bool           fail   = false;
        long long      issued = 0;    // items whose copies were issued
        long long      k      = 0;
        // bounded wait for *ctr >= target by lane 0, the answer shared by the warp
        auto need = [&](const int* ctr, int target) -> bool {
            int ok = 1;
            if (lane == 0) ok = fs_wait(ctr, target) ? 1 : 0;
            return __shfl_sync(0xffffffffu, ok, 0) != 0;
        };
        int            s      = 0;
        uint32_t       par    = 0;
        for (uint32_t j = blockIdx.x; j < items && !fail; j += G, ++k, s = s + 1 == ST ? 0 : s + 1, par ^= s == 0) {
            if (k >= ST) {
                int ok = 1;
                if (lane == 0) ok = mbar_wait_bounded(&empty[s], par ^ 1u) ? 1 : 0;
                if (!__shfl_sync(0xffffffffu, ok, 0)) {
                    fail = true;
                    break;
                }
            }
            const fs_item  it  = fs_decode<TC, TR>(j, batch, lag);
            unsigned char* buf = ring + s * F::STAGE;
            if (!it.row) {
                // the source tile does not depend on anything: copy it first
                if constexpr (FORM == FS_IN) {
                    if (lane == 0) mbar_arrive_expect_tx(&full[s], F::COLB);
                    __syncwarp();
                    const T* g = reinterpret_cast<const T*>(a.src) + it.r * a.src_stride + (long long)it.tile * C * 2 * N1;
                    for (int q = lane; q < C; q += 32) {
                        bulk_g2s(reinterpret_cast<T*>(buf) + q * F::RSC, g + (long long)q * 2 * N1,
                                 2 * N1 * (int)sizeof(T), &full[s]);
                    }
                } else if (lane == 0) {
                    mbar_arrive_expect_tx(&full[s], F::COLB);
#pragma unroll
                    for (int y = 0; y < N1; y += F::BOXY) {
                        tma_load_3d_hint(buf + y * SEG * (int)sizeof(T), &tmap, 2 * it.tile * C, y, (int)it.r,
                                         &full[s], pol);
                    }
                }
                issued = k + 1;
                if constexpr (!TS) {
                    // the acquire of the slot's counter (or a first use of the
                    // slot) orders the compute warps' writes after the earlier
                    // row tiles' reads, through this arrive and their wait
                    if (!(it.r < a.nslot || need(a.row_done + (it.r - a.nslot), TR))) {
                        fail = true;
                        break;
                    }
                    if (lane == 0) mbar_arrive(&slotok[s]);
                }
            } else {
                if (!need(a.col_done + it.r, TC)) {
                    fail = true;
                    break;
                }
                // one bulk copy per row, issued by as many lanes
                if (lane == 0) {
                    fence_proxy_async_global();    // column-pass writes -> TMA reads
                    mbar_arrive_expect_tx(&full[s], CR * RROW);
                }
                __syncwarp();
                const cpx<T>* g = scr + (it.r & mask) * (long long)(N1 * N2) + (long long)it.tile * CR * N2;
                for (int q = lane; q < CR; q += 32) {
                    bulk_g2s(reinterpret_cast<cpx<T>*>(buf) + q * RSI, g + (long long)q * N2, RROW, &full[s]);
                }
                issued = k + 1;
            }
            __syncwarp();
        }
        if (fail && lane == 0) {
            // no copy may still be landing when the block exits: wait
            // (bounded) for the last ST issued items' copies
            atomicExch(a.error, 1);
            for (long long q = issued - 1; q >= 0 && q >= issued - ST; --q) {
                mbar_wait_bounded(&full[(int)(q % ST)], (uint32_t)((q / ST) & 1), 100000000ull);
            }
        }
        __syncwarp();
        return;
    }

    // ======================= compute warps
    // A bounded wait that gives up (tile copy or slot hand-off) is recorded
    // in `bad`; the work of that item goes on with whatever the stage holds,
    // nothing is stored, and at the next exchange barrier, which doubles as
    // a vote, every compute thread leaves together (run_stages_full).
    const int lane   = tid % 32;
    uint32_t  colpar = 0;    // bit s: parity of the next slot hand-off on stage s
    bool      bad    = false;
    int       s      = 0;
    uint32_t  par    = 0;
    cpx<T>*   xsep   = reinterpret_cast<cpx<T>*>(smem + ST * F::STAGE);    // exchange buffer when !IP
    for (uint32_t j = blockIdx.x; j < items; j += G, s = s + 1 == ST ? 0 : s + 1, par ^= s == 0) {
        const fs_item it = fs_decode<TC, TR>(j, batch, lag);
        cpx<T>*        xch = IP ? reinterpret_cast<cpx<T>*>(ring + s * F::STAGE) : xsep;
        // the stage is no longer read: it may be refilled (the publisher adds
        // its own arrival once it has passed the item)
        auto release_stage = [&]() {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
        };
        // TS: this warp's part of the staged outputs is in place
        auto staged = [&]() {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && !bad) mbar_arrive(&written[s]);
        };
        // column tile: the four-step twiddle inputs are requested before the
        // tile's data is waited for, and used after the stages
        constexpr int B = fs_tw_group<T>(LOGN1 + LOGN2), NE = 16 / B + B - 1;
        cpx<T> th{}, tl{}, tu[FORM == FS_PLAIN ? 1 : NE]{};
        if (!it.row) {
            const int n2 = it.tile * C + tid % C;    // FS_IN: the column's place in the scratch
            if constexpr (FORM == FS_PLAIN) {
                const uint32_t e0 = (uint32_t)(tid / C) * (uint32_t)n2;
                th                = ldg_cpx(reinterpret_cast<const cpx<T>*>(a.tw_hi) + (e0 >> LOGN2));
                tl                = ldg_cpx(reinterpret_cast<const cpx<T>*>(a.tw_lo) + (e0 & (N2 - 1)));
                tu[0]             = ldg_cpx(reinterpret_cast<const cpx<T>*>(a.tw_b) + n2);
            } else {
                const cpx<T>* tw = reinterpret_cast<const cpx<T>*>(a.tw) + n2;
                static_for<NE>([&](auto qc) {
                    constexpr int q = decltype(qc)::value;
                    tu[q] = ldg_cpx(tw + (q < 16 / B ? q * P1::TT + tid / C : 16 / B * P1::TT + q - 16 / B) * N2);
                });
            }
        }
        if (!mbar_wait_bounded(&full[s], par)) {
            bad = true;
            atomicExch(a.error, 1);
        }
        if (!it.row) {
            // ---------------- column tile: N1-point DFTs down C columns
            constexpr int E    = P1::E;
            constexpr int TT   = P1::TT;
            const int     c    = tid % C;
            const int     t    = tid / C;
            const int     n2   = it.tile * C + c;    // FS_IN: the column's place in the scratch
            const T*      in   = reinterpret_cast<const T*>(ring + s * F::STAGE);
            const auto*   stw1 = SH ? tws1 : reinterpret_cast<const cpx<T>*>(gtab1);
            cpx<T>        v[E];
            if constexpr (FORM == FS_IN) {
                const T* run = in + c * F::RSC + 32 * (int)brev(t, LOGN1 - 4);
                if (a.lp_src == 0) {
                    if (a.order == 2) run_load<0, true>(v, run);
                    else run_load<0, false>(v, run);
                } else {
                    if (a.order == 2) run_load<LP, true>(v, run);
                    else run_load<LP, false>(v, run);
                }
                static_for<E>([&](auto ic) { v[decltype(ic)::value].im = -v[decltype(ic)::value].im; });
            } else if constexpr (FORM != FS_PLAIN) {
                const int pks = 1 << a.lp_src;
                const int o   = t * SEG + (int)pk_re(c, a.lp_src);
                static_for<E>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    cpx<T>        x = lds_swapped<T, SW>(in, o + i * TT * SEG, pks);
                    v[i]            = {x.re, a.conj_in ? -x.im : x.im};
                });
                if (a.src_len < N1 * N2) {    // rows from src_len / N2 on arrived as zeros
                    const int q = a.src_len >> LOGN2;
                    static_for<E>([&](auto ic) {
                        constexpr int i = decltype(ic)::value;
                        const int     e = q * N2 + n2;
                        if (t + i * TT == q && e < a.src_len) {
                            const T* g = reinterpret_cast<const T*>(a.src) + it.r * a.src_stride + pk_re(e, a.lp_src);
                            v[i]       = {g[0], g[pks]};    // forward: no conjugate
                        }
                    });
                }
            } else {
                static_for<E>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    cpx<T>        x = lds_swapped<T, SW>(in, (t + i * TT) * SEG + pk<LP>(c), PK);
                    v[i]            = {x.re, a.conj_in ? -x.im : x.im};
                });
            }
            if constexpr (!IP) release_stage();
            stage_compute_tab<P1, 0>(v, t, stw1);
            if (run_stages_full<P1, typename F::X1, SH, NT, typename F::PT1>(v, xch, c, t, stw1, bad)) return;
            if constexpr (IP && !TS) release_stage();
            if constexpr (TS) {
                // each output over the value this thread read last: the
                // exchange layout is the box the publisher stores
                auto put = [&](auto ic, cpx<T> o) { xch[F::X1::idx(c, t + decltype(ic)::value * TT)] = o; };
                if constexpr (FORM == FS_PLAIN) apply_fourstep_tw(v, cmul(th, tl), tu[0], put);
                else apply_fourstep_ent<B>(v, tu, put);
                staged();
            } else {
                if (!mbar_wait_bounded(&slotok[s], (colpar >> s) & 1u)) {
                    // the producer gave up on this slot: nothing is written, and
                    // the compute warps leave at the next item's vote
                    bad = true;
                    atomicExch(a.error, 1);
                }
                colpar ^= 1u << s;
                if (!bad) {
                    cpx<T>* dst = scr + (it.r & mask) * (long long)(N1 * N2) + (long long)t * N2 + n2;
                    auto    put = [&](auto ic, cpx<T> o) {
                        constexpr int i             = decltype(ic)::value;
                        dst[(long long)i * TT * N2] = o;
                    };
                    if constexpr (FORM == FS_PLAIN) apply_fourstep_tw(v, cmul(th, tl), tu[0], put);
                    else apply_fourstep_ent<B>(v, tu, put);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&written[s]);
                }
            }
        } else {
            // ---------------- row tile: N2-point DFTs along CR rows
            constexpr int E    = P2::E;
            constexpr int TT   = P2::TT;
            const int     mlo  = tid % G8;
            const int     t    = (tid / G8) % TT;
            const int     mhi  = tid / (G8 * TT);
            const int     m    = mhi * G8 + mlo;
            const int     k1   = it.tile * CR + m;
            const auto*   stw2 = SH ? tws2 : reinterpret_cast<const cpx<T>*>(gtab2);
            const cpx<T>* in   = reinterpret_cast<const cpx<T>*>(ring + s * F::STAGE) + m * RSI +
                                 (FORM == FS_IN ? 16 * (int)brev(t, LOGN2 - 4) : t);
            cpx<T>        v[E];
            if constexpr (FORM == FS_IN) {
                run_load<0, false>(v, reinterpret_cast<const T*>(in));
            } else {
                static_for<E>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    v[i]            = in[i * TT];
                });
            }
            if constexpr (!IP) release_stage();
            stage_compute_tab<P2, 0>(v, t, stw2);
            if (run_stages_full<P2, typename F::X2, SH, NT, typename F::PT2>(v, xch, m, t, stw2, bad)) return;
            const T sc  = T(a.scale);
            const T sim = a.conj_out ? -sc : sc;
            if constexpr (FORM == FS_OUT) {
                // rows staged in output order, then copied out whole
                constexpr int W   = 16 / (int)sizeof(T);
                constexpr int U   = 32 / W;         // 16-byte units per run
                constexpr int KT  = 8 / G8;         // threads t per bank group turn
                T*            stg = reinterpret_cast<T*>(xch);
                auto          key = [](int row, int tt) { return row % G8 + G8 * (tt % KT); };
                static_for<E>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    v[i]            = {v[i].re * sc, v[i].im * sim};
                });
                xch_sync<NT>();    // the exchange buffer is no longer read
                T* run = stg + m * 2 * N2 + 32 * (int)brev(t, LOGN2 - 4);
                if (a.lp_dst == 0) {
                    if (a.order == 2) run_store<0, true>(v, run, key(m, t));
                    else run_store<0, false>(v, run, key(m, t));
                } else {
                    if (a.order == 2) run_store<LP, true>(v, run, key(m, t));
                    else run_store<LP, false>(v, run, key(m, t));
                }
                xch_sync<NT>();
                T* dst = reinterpret_cast<T*>(a.dst) + it.r * a.dst_stride;
                for (int q = tid; q < CR * (2 * N2 / W); q += NT) {
                    const int      row = q / (2 * N2 / W), u = q % (2 * N2 / W);
                    const int      tt  = (int)brev(u / U, LOGN2 - 4);
                    const vec16<T> w   = *reinterpret_cast<const vec16<T>*>(
                        stg + row * 2 * N2 + (u / U) * 32 + ((u % U) ^ key(row, tt)) * W);
                    const int      k   = (int)brev(it.tile * CR + row, LOGN1);
                    __stcs(reinterpret_cast<float4*>(dst + (long long)k * 2 * N2 + u * W),
                           *reinterpret_cast<const float4*>(&w));
                }
                // the stage is read: it may be refilled
                if constexpr (TS) staged();
                else if constexpr (IP) release_stage();
            } else if constexpr (TS) {
                // row k2 of the exchange layout is 8 (FP64: 4) elements of the
                // transposed output, one segment of 64 bytes, last read by
                // neighbouring lanes of this warp: they put their values there
                // in packed order, the box the publisher stores
                const int lpd = FORM == FS_PLAIN ? LP : a.lp_dst;
                T*        seg = reinterpret_cast<T*>(xch + F::X2::idx(m - mlo, 0)) + (int)pk_re(mlo, lpd);
                __syncwarp();
                static_for<E>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    const int     l = t + i * TT;
                    sts_swapped<T, SW>(seg, (l + (l >> 4)) * 2 * G8, 1 << lpd, v[i].re * sc, v[i].im * sim);
                });
                staged();
            } else if constexpr (FORM != FS_PLAIN) {
                if constexpr (IP) release_stage();
                T* dst = reinterpret_cast<T*>(a.dst) + it.r * a.dst_stride + pk_re(t * N1 + k1, a.lp_dst);
                if (a.lp_dst == 0) {
                    using V2 = std::conditional_t<sizeof(T) == 4, float2, double2>;
                    static_for<E>([&](auto ic) {
                        constexpr int i = decltype(ic)::value;
                        __stcs(reinterpret_cast<V2*>(dst + 2 * i * TT * N1), V2{v[i].re * sc, v[i].im * sim});
                    });
                } else {
                    T* dim = dst + (1 << a.lp_dst);
                    static_for<E>([&](auto ic) {
                        constexpr int i = decltype(ic)::value;
                        __stcs(dst + 2 * i * TT * N1, v[i].re * sc);
                        __stcs(dim + 2 * i * TT * N1, v[i].im * sim);
                    });
                }
            } else {
                if constexpr (IP) release_stage();
                T* dst = reinterpret_cast<T*>(a.dst) + it.r * a.dst_stride + pk<LP>(t * N1 + k1);
                static_for<E>([&](auto ic) {
                    constexpr int i = decltype(ic)::value;
                    __stcs(dst + 2 * i * TT * N1, v[i].re * sc);
                    __stcs(dst + 2 * i * TT * N1 + PK, v[i].im * sim);
                });
            }
        }
    }
}

}    // namespace pcxg
