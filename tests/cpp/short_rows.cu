// The copy of a short row stays inside the caller's storage: whole packs of
// (len + p - 1) / p * 2 * p reals.  Checked at compile time.
#include "pcx_fft_v2.cuh"

template<class T>
constexpr bool inside() {
    for (int lp = 0; lp <= 5; ++lp) {
        for (int len = 1; len <= 300; ++len) {
            const unsigned stored = (unsigned)(((len - 1) >> lp) + 1) * (2u << lp) * (unsigned)sizeof(T);
            const unsigned bytes  = pcxg::single3_row_bytes<T>(len, lp);
            const unsigned last   = (unsigned)(((len - 1) >> lp) << (lp + 1)) + ((len - 1) & ((1 << lp) - 1)) + (1u << lp);
            if (bytes % 16 != 0 || bytes > stored) return false;
            // all of the row, or (width 1) all but one element
            const unsigned need = (last + 1) * (unsigned)sizeof(T);
            if (bytes < need && !(lp == 0 && need - bytes == 2 * sizeof(T))) return false;
        }
    }
    return true;
}
static_assert(inside<float>() && inside<double>());
