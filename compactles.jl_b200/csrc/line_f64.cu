// k_line (line_body.cuh) for double fields.
#include "line_body.cuh"

namespace cles {
bool launch_line_f64(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, int mode,
                     cudaStream_t st, const RkEpilogue& rk, bool rk_first, int num_sms) {
    return launch_line_dtype<double>(plan, in, out, count, mode, st, rk, rk_first, num_sms);
}
}  // namespace cles
