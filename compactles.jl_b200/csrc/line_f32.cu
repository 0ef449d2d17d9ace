// k_line (line_body.cuh) for float fields.
#include "line_body.cuh"

namespace cles {
bool launch_line_f32(const CompactPlan& plan, const FieldView& in, const FieldView& out, int count, int mode,
                     cudaStream_t st, const RkEpilogue& rk, bool rk_first, const void* in2, void* out2, int count2,
                     int num_sms) {
    return launch_line_dtype<float>(plan, in, out, count, mode, st, rk, rk_first, in2, out2, count2,
                                     num_sms);
}
}  // namespace cles
