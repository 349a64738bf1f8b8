// The forward slab pass for the lengths of two radices.
#include "ns_any_slab.cuh"

namespace sfl {

void launch_any_slab_fwd(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag) {
    launch_any_slab<0>(P, a, st, tag);
}

bool any_slab_fits(const NSPlan& P) {
    return any_len(P.dims[0]) && any_len(P.dims[1]) && any_smem(P.dims[0], P.dims[1], P.P1) <= kSlabSmemOneCta;
}

}  // namespace sfl
