// st_kernels_f32.cu - FP32-field instantiations of the bounded-line
// operators (the FP32 mode's derivative inputs, outputs and arithmetic are
// float, two lines per thread).
#include "st_linekern.cuh"

namespace st {

int launch_rec_f32(st_ctx *c, RecId id, LineArgsF &a, const float *const *in, float *const *out) {
    return launch_rec_t<false, float>(c, id, a, in, out);
}

}  // namespace st
