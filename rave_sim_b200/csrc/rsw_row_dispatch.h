// Row-pass dispatch by row length and samples per thread, shared by the
// instantiation units of the plain row passes (rsw_row_f32.cu, rsw_row_f64.cu)
// and of their batched variants (rsw_row_f32_batch.cu, rsw_row_f64_batch.cu).
#pragma once

#include "rsw_passes.cuh"

namespace rsw {
// rows of convolution plans (a table product), every length of the per-sample form
template <typename Real> cudaError_t row_table_dispatch(const PassArgs &a, cudaStream_t s) {
    switch (a.log_n2) {
    case 4: return row_table<Real, 4>(a, s);
    case 5: return row_table<Real, 5>(a, s);
    case 6: return row_table<Real, 6>(a, s);
    case 7: return row_table<Real, 7>(a, s);
    case 8: return row_table<Real, 8>(a, s);
    case 9: return row_table<Real, 9>(a, s);
    case 10: return row_table<Real, 10>(a, s);
    case 11: return row_table<Real, 11>(a, s);
    case 12: return row_table<Real, 12>(a, s);
    case 13: return row_table<Real, 13>(a, s);
    case 14:
        if constexpr (sizeof(Real) == 4) return row_table<Real, 14>(a, s);
        [[fallthrough]];
    default: return cudaErrorInvalidValue;
    }
}

// two-level rows (chirp form): 2^7 .. 2^13 (c128) / 2^14 (c64), 16 or 32 elements per thread;
// single-level rows (per-sample form): 2^4 .. 2^13 / 2^14, 16 elements per thread. A count that a
// length has no kernel for is an error: the plan's tables are laid out for it.
#define RSW_ROW_E(R, L, E, CH) (e == E ? row_impl<R, L, E, CH, BT>(a, s) : cudaErrorInvalidValue)
#define RSW_ROW_CASE(R, L) \
    case L: return chirp && e == 32 ? row_impl<R, L, 32, true, BT>(a, s) \
                                    : chirp ? RSW_ROW_E(R, L, 16, true) : RSW_ROW_E(R, L, 16, false);
#define RSW_ROW_CASE16(R, L) \
    case L: return chirp ? RSW_ROW_E(R, L, 16, true) : RSW_ROW_E(R, L, 16, false);
// rows with 8 samples per thread (radix-8 stages, twice the threads)
#define RSW_ROW_CASE8(R, L) \
    case L: return chirp && e == 8 ? row_impl<R, L, 8, true, BT>(a, s) \
                   : chirp && e == 32 ? row_impl<R, L, 32, true, BT>(a, s) \
                                      : chirp ? RSW_ROW_E(R, L, 16, true) : RSW_ROW_E(R, L, 16, false);
#define RSW_ROW_CASE_S(R, L) \
    case L: return chirp ? cudaErrorInvalidValue : RSW_ROW_E(R, L, 16, false);

// multi-level rows take the chirp form of the Fresnel kernel; the exact
// kernel, single-level rows and the rows of short two-level plans (no chirp
// table) work per sample.
// BT: the batched kernels (chirp form only; the others return an error)
static inline bool row_chirp(const PassArgs &a) {
    return a.log_n1 > 0 && !a.pr.exact && (a.pr.chirp || !a.pr.has_h);
}
template <bool BT> cudaError_t row_dispatch_f64(const PassArgs &a, int e, cudaStream_t s) {
    const bool chirp = row_chirp(a);
    switch (a.log_n2) {
        RSW_ROW_CASE_S(double, 4) RSW_ROW_CASE_S(double, 5) RSW_ROW_CASE_S(double, 6)
        RSW_ROW_CASE16(double, 7) RSW_ROW_CASE16(double, 8) RSW_ROW_CASE(double, 9)
        RSW_ROW_CASE(double, 10) RSW_ROW_CASE8(double, 11) RSW_ROW_CASE8(double, 12) RSW_ROW_CASE8(double, 13)
    default: return cudaErrorInvalidValue;
    }
}
template <bool BT> cudaError_t row_dispatch_f32(const PassArgs &a, int e, cudaStream_t s) {
    const bool chirp = row_chirp(a);
    switch (a.log_n2) {
        RSW_ROW_CASE_S(float, 4) RSW_ROW_CASE_S(float, 5) RSW_ROW_CASE_S(float, 6) RSW_ROW_CASE16(float, 7)
        RSW_ROW_CASE16(float, 8) RSW_ROW_CASE(float, 9) RSW_ROW_CASE(float, 10) RSW_ROW_CASE8(float, 11)
        RSW_ROW_CASE8(float, 12) RSW_ROW_CASE8(float, 13) RSW_ROW_CASE(float, 14)
    default: return cudaErrorInvalidValue;
    }
}
#undef RSW_ROW_E
#undef RSW_ROW_CASE
#undef RSW_ROW_CASE16
#undef RSW_ROW_CASE8
#undef RSW_ROW_CASE_S
}  // namespace rsw
