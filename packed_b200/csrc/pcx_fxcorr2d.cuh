// Geometry of the in-CTA four-step correlation windows of the ragged batch
// (2^14 points on its whole ring): the window as N1 rows of N2 samples, column
// and row sub-FFTs by groups of TT threads inside one warp, 16 points per
// thread, exchanging through a private padded buffer.
#pragma once

#include "pcx_fft_v2.cuh"

namespace pcxg {

template<int LOGN>
struct xc2_cfg {
    static constexpr int LOGN1 = (LOGN + 1) / 2;
    static constexpr int LOGN2 = LOGN / 2;
    static constexpr int N1    = 1 << LOGN1;
    static constexpr int N2    = 1 << LOGN2;
    static constexpr int N     = N1 * N2;
    using P1                   = splan<LOGN1>;
    using P2                   = splan<LOGN2>;
    static constexpr int NT    = 512;
    static constexpr int TT1   = P1::TT;
    static constexpr int TT2   = P2::TT;
    static constexpr int G1    = NT / TT1;    // column groups per round
    static constexpr int G2    = NT / TT2;    // row groups per round
    static constexpr int R1    = N2 / G1;     // column rounds
    static constexpr int R2    = N1 / G2;     // row rounds
    static constexpr int RS    = N2 + 2;      // window row stride (complex), 2 mod 16
    static constexpr int WIN   = N1 * RS * 8;
    using X1                   = xch_blocked<N1, G1>;
    using X2                   = xch_blocked<N2, G2>;
    static constexpr int XB    = (X1::size > X2::size ? X1::size : X2::size) * 8;
    static constexpr int TB1   = smem_align16(fs_full_tw_size<P1>() * 8);    // full stage tables
    static constexpr int TB2   = smem_align16(fs_full_tw_size<P2>() * 8);
    static constexpr int NB    = N / 16;      // W_N^e, e < N/16 (= TT1*N2 = TT2*N1)
    // in shared memory entry e sits at e + e/16: the threads of a warp read
    // e = t*n2 for eight t, which would share banks whenever n2 is a multiple of 16
    static constexpr int NBP   = NB + NB / 16;
    static constexpr int SMEM  = WIN + XB + TB1 + TB2 + (NBP + N2 + N1) * 8;
    static_assert(P1::E == 16 && P2::E == 16, "16 points per thread");
    static_assert(TT1 <= 32 && TT2 <= 32 && TT2 >= 2, "sub-FFT groups inside one warp");
    static_assert(R1 >= 1 && R2 >= 1 && G1 * R1 == N2 && G2 * R2 == N1, "rounds");
    static_assert(TT1 * N2 == NB && TT2 * N1 == NB, "twiddle split");
    static_assert(NBP % 2 == 0, "16-byte offset of the tables behind it");
    static_assert(WIN % 16 == 0 && XB % 16 == 0 && TB1 % 16 == 0 && TB2 % 16 == 0, "16-byte sections");
};

}    // namespace pcxg
