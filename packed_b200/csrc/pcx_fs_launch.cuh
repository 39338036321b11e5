// Launch of one variant of the one-launch four-step kernel (k_fourstep), and
// the macro the variant translation units (pcx_fs_part*.cu) instantiate it
// with.  The variants are split over several files only to build in parallel.
#pragma once

#include "pcx_fourstep.cuh"
#include "pcx_host.hpp"
#include "pcx_v2_launch.cuh"

#include <type_traits>

namespace pcxg {

template<class T, int LOGN1, int LOGN2, int MINB, int ST, int FORM = FS_PLAIN>
cudaError_t launch_fs(const fs_args& a, cudaStream_t st, int sms, bool attr_only, int* tc, int* tr, int* per_sm) {
    using F = fs_cfg<T, LOGN1, LOGN2, MINB, ST>;
    static_assert(F::SMEM <= 232448, "shared memory per block");
    static_assert(F::MINB * (F::SMEM + 1024 + 256) <= 233472, "blocks per SM fit the shared memory");
    static_assert(F::STAGE % 128 == 0, "TMA destinations stay 128-byte aligned");
    auto kern = k_fourstep<T, LOGN1, LOGN2, MINB, ST, FORM, false>;
    if (tc) *tc = F::TC;
    if (tr) *tr = F::TR;
    if (attr_only) {
        cudaError_t e = smem_attr_cached(reinterpret_cast<const void*>(kern), F::SMEM);
        if constexpr (F::TS) {
            if (e == cudaSuccess) {
                e = smem_attr_cached(reinterpret_cast<const void*>(k_fourstep<T, LOGN1, LOGN2, MINB, ST, FORM, true>), F::SMEM);
            }
        }
        if (e == cudaSuccess && per_sm) e = occupancy_cached(reinterpret_cast<const void*>(kern), F::NT + 64, F::SMEM, per_sm);
        return e;
    }
    const long long items = a.batch * (F::TC + F::TR);
    if (items == 0) return cudaSuccess;
    if (items >= (1LL << 31)) return cudaErrorInvalidValue;    // the kernel counts items in 32 bits
    // 3-D view of the source: [transform][n1][2*N2 reals], box = 2*C reals x min(N1, 256) rows; a
    // short source has as many rows n1 as it fills (the rest reads as zeros)
    CUtensorMap      map;
    const cuuint64_t dims[3]    = {(cuuint64_t)2 << LOGN2, (cuuint64_t)(FORM == FS_ANY || FORM == FS_OUT ? a.src_len >> LOGN2 : 1 << LOGN1),
                                   (cuuint64_t)a.batch};
    const long long  ss         = a.batch > 1 ? a.src_stride : (2LL << (LOGN1 + LOGN2));    // unused when 1 row
    const cuuint64_t strides[2] = {((cuuint64_t)2 << LOGN2) * sizeof(T), (cuuint64_t)ss * sizeof(T)};
    const cuuint32_t box[3]     = {(cuuint32_t)(2 * F::C), (cuuint32_t)F::BOXY, 1};
    const cuuint32_t estr[3]    = {1, 1, 1};
    cudaError_t      e = encode_tensor_map(&map, sizeof(T) == 8, 3, const_cast<void*>(a.src), dims, strides, box, estr);
    if (e != cudaSuccess) return FORM == FS_PLAIN ? e : cudaErrorNotSupported;    // the caller has another path
    unsigned grid = 0;
    e             = persistent_grid(kern, F::NT + 64, F::SMEM, items, sms, &grid);
    if (e != cudaSuccess) return e;
    // outputs through TMA: F::TS and enough items for the load/store queue to matter
    CUtensorMap tscr{}, tdst{};
    if constexpr (F::TS) {
        if (items >= (long long)FS_TS_ROUNDS * grid) {
            // 4-D views that the outputs are stored through, [.][16-row block][row of it][reals]: the scratch
            // (rows k1 of slot .) and the destination (rows k2 of transform .).  Boxes are 17 rows high: the
            // 17th, outside the view, is the padding row of the shared layout and is not written.
            const cuuint32_t estr4[4]    = {1, 1, 1, 1};
            const cuuint64_t sdims[4]    = {(cuuint64_t)2 << LOGN2, 16, (cuuint64_t)F::N1 / 16, (cuuint64_t)a.nslot};
            const cuuint64_t sstr[3]     = {((cuuint64_t)2 << LOGN2) * sizeof(T), ((cuuint64_t)32 << LOGN2) * sizeof(T),
                                            ((cuuint64_t)2 << (LOGN1 + LOGN2)) * sizeof(T)};
            const cuuint32_t sbox[4]     = {(cuuint32_t)(2 * F::C), 17, (cuuint32_t)F::N1 / 16, 1};
            const long long  ds          = a.batch > 1 ? a.dst_stride : (2LL << (LOGN1 + LOGN2));
            const cuuint64_t ddims[4]    = {(cuuint64_t)2 << LOGN1, 16, (cuuint64_t)F::N2 / 16, (cuuint64_t)a.batch};
            const cuuint64_t dstr[3]     = {((cuuint64_t)2 << LOGN1) * sizeof(T), ((cuuint64_t)32 << LOGN1) * sizeof(T),
                                            (cuuint64_t)ds * sizeof(T)};
            const cuuint32_t dbox[4]     = {(cuuint32_t)(2 * F::G8), 17, (cuuint32_t)F::N2 / 16, 1};
            e = encode_tensor_map(&tscr, sizeof(T) == 8, 4, a.scratch, sdims, sstr, sbox, estr4);
            if (e == cudaSuccess) e = encode_tensor_map(&tdst, sizeof(T) == 8, 4, a.dst, ddims, dstr, dbox, estr4);
            if (e != cudaSuccess) return FORM == FS_PLAIN ? e : cudaErrorNotSupported;
            k_fourstep<T, LOGN1, LOGN2, MINB, ST, FORM, true><<<grid, F::NT + 64, F::SMEM, st>>>(map, tscr, tdst, a);
            return cudaGetLastError();
        }
    }
    kern<<<grid, F::NT + 64, F::SMEM, st>>>(map, tscr, tdst, a);
    return cudaGetLastError();
}

}    // namespace pcxg

// Inside a part function (f64, v, a, st, sms, attr_only, tc, tr, per_sm in scope).
#define PCX_FS_VARIANT(T, L1, L2, M, S)                                                                    \
    if (f64 == std::is_same<T, double>::value && v.l1 == L1 && v.l2 == L2 && v.minb == M && v.st == S) { \
        return pcxg::launch_fs<T, L1, L2, M, S>(a, st, sms, attr_only, tc, tr, per_sm);                   \
    }

// The other forms: one variant per size.  FP32 2^13..2^20, FP64 2^14..2^20,
// the first of each size in kFsVariantsF32 / kFsVariantsF64.
#define PCX_FS_FORM_VARIANT(T, L1, L2, M, S)                                                              \
    if (f64 == std::is_same<T, double>::value && v.l1 == L1 && v.l2 == L2 && v.minb == M && v.st == S) { \
        return pcxg::launch_fs<T, L1, L2, M, S, FORM>(a, st, sms, attr_only, nullptr, nullptr, nullptr);  \
    }
#define PCX_FS_FORM(NAME, FORM_)                                                                              \
    cudaError_t NAME(bool f64, const pcxg::fs_variant& v, const pcxg::fs_args& a, cudaStream_t st, int sms, \
                     bool attr_only) {                                                                        \
        constexpr int FORM = pcxg::FORM_;                                                                     \
        PCX_FS_FORM_VARIANT(float, 7, 6, 2, 3)                                                                \
        PCX_FS_FORM_VARIANT(float, 7, 7, 2, 3)                                                                \
        PCX_FS_FORM_VARIANT(float, 7, 8, 2, 3)                                                                \
        PCX_FS_FORM_VARIANT(float, 8, 8, 2, 3)                                                                \
        PCX_FS_FORM_VARIANT(float, 8, 9, 2, 3)                                                                \
        PCX_FS_FORM_VARIANT(float, 9, 9, 2, 3)                                                                \
        PCX_FS_FORM_VARIANT(float, 10, 9, 1, 3)                                                               \
        PCX_FS_FORM_VARIANT(float, 10, 10, 1, 3)                                                              \
        PCX_FS_FORM_VARIANT(double, 7, 7, 2, 3)                                                               \
        PCX_FS_FORM_VARIANT(double, 8, 7, 2, 3)                                                               \
        PCX_FS_FORM_VARIANT(double, 8, 8, 2, 3)                                                               \
        PCX_FS_FORM_VARIANT(double, 9, 8, 2, 3)                                                               \
        PCX_FS_FORM_VARIANT(double, 9, 9, 2, 3)                                                               \
        PCX_FS_FORM_VARIANT(double, 10, 9, 1, 2)                                                              \
        PCX_FS_FORM_VARIANT(double, 10, 10, 1, 2)                                                             \
        return cudaErrorNotSupported;                                                                         \
    }

#define PCX_FS_PART(NAME)                                                                                     \
    cudaError_t NAME(bool f64, const pcxg::fs_variant& v, const pcxg::fs_args& a, cudaStream_t st, int sms, \
                     bool attr_only, int* tc, int* tr, int* per_sm)
