// st_kernels_cyc_f32.cu - FP32-field instantiations of the periodic-line
// operators.
#include "st_linekern.cuh"

namespace st {

int launch_rec_cyc_f32(st_ctx *c, RecId id, LineArgsF &a, const float *const *in, float *const *out) {
    return launch_rec_t<true, float>(c, id, a, in, out);
}

}  // namespace st
