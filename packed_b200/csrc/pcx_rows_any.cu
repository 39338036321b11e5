// Instantiations and launch of the register-fed single-pass kernel (k_rows), any packs and short rows.
#include "pcx_v2_launch.cuh"

namespace pcxg {

template<class T>
static cudaError_t dispatch_rows(int log_n, const v3_args& a, cudaStream_t st, bool attr_only) {
    switch (log_n) {
    case 7: return launch_rows<T, 7, true>(a, st, attr_only);
    case 8: return launch_rows<T, 8, true>(a, st, attr_only);
    case 9: return launch_rows<T, 9, true>(a, st, attr_only);
    case 10: return launch_rows<T, 10, true>(a, st, attr_only);
    case 11: return launch_rows<T, 11, true>(a, st, attr_only);
    case 12: return launch_rows<T, 12, true>(a, st, attr_only);
    case 13: return launch_rows<T, 13, true>(a, st, attr_only);
    case 14:
        if constexpr (sizeof(T) == 4) return launch_rows<T, 14, true>(a, st, attr_only);
        return cudaErrorNotSupported;
    default: return cudaErrorNotSupported;
    }
}

}    // namespace pcxg

cudaError_t pcx_rows_any(bool f64, int log_n, const pcxg::v3_args& a, cudaStream_t st, bool attr_only) {
    return f64 ? pcxg::dispatch_rows<double>(log_n, a, st, attr_only)
               : pcxg::dispatch_rows<float>(log_n, a, st, attr_only);
}
