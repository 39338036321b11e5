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
    case 14:
        if constexpr (sizeof(T) == 4) return launch_rows<T, 14, false>(a, st, attr_only);
        return cudaErrorNotSupported;
    default: return cudaErrorNotSupported;
    }
}

// Full tables of plan P at `out`.
template<class P, class T>
static cudaError_t full_tables(cpx<T>* out, cudaStream_t st) {
    for (int s = 1; s < P::NST; ++s) {
        const int nsb = P::nsbits(s), rb = P::rbits(s);
        k_rows_twiddles<T><<<((1 << (nsb + rb)) + 255) / 256, 256, 0, st>>>(out + rows_tw_offset<P>(s), nsb, rb);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
template<class T, int LOGL>
static cudaError_t rows_twiddles(void* out, cudaStream_t st, rows_sections* at) {
    using F = rows_cfg<T, LOGL>;
    using P = typename F::P;
    *at     = {F::FULL + rows_tw_size<P>(), F::W, F::FULL16, F::FULL};
    if (!out) return cudaSuccess;
    auto* o = static_cast<cpx<T>*>(out);
    if constexpr (F::W) {
        for (int s = 1; s < P::NST; ++s) {
            const int ns = 1 << P::nsbits(s), rb = P::rbits(s), nq = stw_q(rb) * ns;
            k_stage_twiddles<T><<<(nq + 255) / 256, 256, 0, st>>>(o + stage_tw_offset<P>(s), ns, rb, P::nsbits(s) + rb);
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return e;
        }
        const cudaError_t e = full_tables<splan<LOGL>>(o + F::FULL16, st);
        if (e != cudaSuccess) return e;
    }
    return full_tables<P>(o + F::FULL, st);
}
template<class T>
static cudaError_t dispatch_twiddles(int log_n, void* out, cudaStream_t st, rows_sections* at) {
    *at = {};
    switch (log_n) {
    case 7: return rows_twiddles<T, 7>(out, st, at);
    case 8: return rows_twiddles<T, 8>(out, st, at);
    case 9: return rows_twiddles<T, 9>(out, st, at);
    case 10: return rows_twiddles<T, 10>(out, st, at);
    case 11: return rows_twiddles<T, 11>(out, st, at);
    case 12: return rows_twiddles<T, 12>(out, st, at);
    case 13: return rows_twiddles<T, 13>(out, st, at);
    case 14: return rows_twiddles<T, 14>(out, st, at);
    default: return cudaSuccess;
    }
}

}    // namespace pcxg

cudaError_t pcx_rows_twiddles(bool f64, int log_n, void* out, cudaStream_t st, pcxg::rows_sections* at) {
    return f64 ? pcxg::dispatch_twiddles<double>(log_n, out, st, at)
               : pcxg::dispatch_twiddles<float>(log_n, out, st, at);
}

cudaError_t pcx_rows(bool f64, int log_n, const pcxg::v3_args& a, cudaStream_t st, bool attr_only) {
    return f64 ? pcxg::dispatch_rows<double>(log_n, a, st, attr_only)
               : pcxg::dispatch_rows<float>(log_n, a, st, attr_only);
}
