// Column-pass dispatch by column length, samples per thread and columns per
// CTA, shared by the plain column pass (rsw_col.cu) and its detection
// variant (rsw_col_det.cu).
#pragma once

#include "rsw_passes.cuh"

namespace rsw {
// A count that a length has no kernel for is an error: the plan's tables are laid out for it.
#define RSW_COL_E16(R, L, C) (e == 16 ? col_impl<R, L, C, 16, DET, BT>(a, s) : cudaErrorInvalidValue)
#define RSW_COL_E8(R, L, C8, C16) \
    case L: return e == 8 ? col_impl<R, L, C8, 8, DET, BT>(a, s) : RSW_COL_E16(R, L, C16);
#define RSW_COL_CASE16(R, L) \
    case L: return RSW_COL_E16(R, L, col_c(L));
// 8 or 16 samples per thread (C8 / C16 columns per CTA), 32 on request
#define RSW_COL_CASE_E(R, L, C8, C16)                                                       \
    case L: return e == 8 ? col_impl<R, L, C8, 8, DET, BT>(a, s)                           \
                          : e == 32 ? col_impl<R, L, col_c32<R>(L), 32, DET, BT>(a, s) : RSW_COL_E16(R, L, C16);
#define RSW_COL_CASE(R, L) \
    case L: return e == 32 ? col_impl<R, L, col_c32<R>(L), 32, DET, BT>(a, s) : RSW_COL_E16(R, L, col_c(L));

// Columns per CTA: col_c(L) (16-byte samples: 64- to 512-byte row
// segments); complex64 doubles them where the threads allow (col_c64).
// BT: the batched kernels (per-instance transmission factors, PassArgs::btr).
template <bool DET, bool BT = false> cudaError_t col_dispatch(const PassArgs &a, bool dbl, int e, cudaStream_t s) {
    if (dbl) {
        switch (a.log_n1) {
            RSW_COL_CASE16(double, 4) RSW_COL_CASE16(double, 5) RSW_COL_CASE16(double, 6)
            RSW_COL_CASE16(double, 7)
            RSW_COL_E8(double, 8, 16, 16)
            RSW_COL_CASE_E(double, 9, 8, 8) RSW_COL_CASE_E(double, 10, 4, 4) RSW_COL_CASE_E(double, 11, 4, 4)
            // 2^12 (the default at 2^24 and 2^25): two columns per CTA, 32-byte row segments
            RSW_COL_E8(double, 12, 2, 2)
        default: return cudaErrorInvalidValue;
        }
    }
    switch (a.log_n1) {
        RSW_COL_CASE16(float, 4) RSW_COL_CASE16(float, 5) RSW_COL_CASE16(float, 6)
        RSW_COL_CASE16(float, 7)
        RSW_COL_E8(float, 8, 32, 16)
        RSW_COL_CASE_E(float, 9, 16, 8) RSW_COL_CASE_E(float, 10, 4, col_c64(10))
        RSW_COL_CASE_E(float, 11, 4, col_c64(11)) RSW_COL_CASE(float, 12)
    default: return cudaErrorInvalidValue;
    }
}
#undef RSW_COL_E16
#undef RSW_COL_E8
#undef RSW_COL_CASE16
#undef RSW_COL_CASE_E
#undef RSW_COL_CASE
}  // namespace rsw
