// The denoiser's slab pass for the lengths of two radices.
#include "ns_any_slab.cuh"

namespace sfl {

void launch_any_slab_shrink(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag) {
    launch_any_slab<2>(P, a, st, tag);
}

}  // namespace sfl
