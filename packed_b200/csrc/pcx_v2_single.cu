// Instantiations and launch of the TMA-fed single-pass kernel (k_single3).
#include "pcx_v2_launch.cuh"

namespace pcxg {

template<class T>
static cudaError_t dispatch3(int log_n, const v3_args& a, cudaStream_t st, int sms, bool attr_only) {
    switch (log_n) {
    case 5: return launch_single3<T, 5, false>(a, st, sms, attr_only);
    case 6: return launch_single3<T, 6, false>(a, st, sms, attr_only);
    case 7: return launch_single3<T, 7, false>(a, st, sms, attr_only);
    case 8: return launch_single3<T, 8, false>(a, st, sms, attr_only);
    case 9: return launch_single3<T, 9, false>(a, st, sms, attr_only);
    case 10: return launch_single3<T, 10, false>(a, st, sms, attr_only);
    case 11: return launch_single3<T, 11, false>(a, st, sms, attr_only);
    case 12: return launch_single3<T, 12, false>(a, st, sms, attr_only);
    case 13:
        if constexpr (sizeof(T) == 4) return launch_single3<T, 13, false>(a, st, sms, attr_only);    // 64 KB per row
        return cudaErrorNotSupported;
    default: return cudaErrorNotSupported;
    }
}

}    // namespace pcxg

cudaError_t pcx_v3_single(bool f64, int log_n, const pcxg::v3_args& a, cudaStream_t st, int sms, bool attr_only) {
    return f64 ? pcxg::dispatch3<double>(log_n, a, st, sms, attr_only)
               : pcxg::dispatch3<float>(log_n, a, st, sms, attr_only);
}
