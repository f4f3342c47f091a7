// Row-pass kernels of convolution plans (both precisions): the spectrum times a
// table (PropArgs::table).
#include "rsw_row_dispatch.h"

namespace rsw {
cudaError_t launch_row_pass_table(const PassArgs &a, bool dbl, cudaStream_t s) {
    return dbl ? row_table_dispatch<double>(a, s) : row_table_dispatch<float>(a, s);
}
}  // namespace rsw
