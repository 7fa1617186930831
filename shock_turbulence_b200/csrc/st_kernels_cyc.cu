// st_kernels_cyc.cu - periodic-line instantiations of the line operators
// (src/derivCDopt6_periodic.f, src/filters_periodic.f).
#include "st_linekern.cuh"

namespace st {

int launch_rec_cyc(st_ctx *c, RecId id, LineArgs &a, const double *const *in, double *const *out) {
    return launch_rec_t<true, double>(c, id, a, in, out);
}

}  // namespace st
