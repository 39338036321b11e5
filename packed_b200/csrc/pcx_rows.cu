// Instantiations and launch of the register-fed single-pass kernel (k_rows).
#include "pcx_v2_launch.cuh"

namespace pcxg {

template<class T>
static cudaError_t dispatch_rows(int log_n, const v3_args& a, cudaStream_t st, bool attr_only) {
    switch (log_n) {
    case 7: return launch_rows<T, 7, false>(a, st, attr_only);
    case 8: return launch_rows<T, 8, false>(a, st, attr_only);
    case 9: return launch_rows<T, 9, false>(a, st, attr_only);
    case 10: return launch_rows<T, 10, false>(a, st, attr_only);
    case 11: return launch_rows<T, 11, false>(a, st, attr_only);
    case 12: return launch_rows<T, 12, false>(a, st, attr_only);
    case 13: return launch_rows<T, 13, false>(a, st, attr_only);
    default: return cudaErrorNotSupported;
    }
}

}    // namespace pcxg

cudaError_t pcx_rows(bool f64, int log_n, const pcxg::v3_args& a, cudaStream_t st, bool attr_only) {
    return f64 ? pcxg::dispatch_rows<double>(log_n, a, st, attr_only)
               : pcxg::dispatch_rows<float>(log_n, a, st, attr_only);
}
