// The denoiser's slab pass for any axis lengths.
#include "ns_mix_slab.cuh"

namespace sfl {

void launch_mix_slab_shrink(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag) {
    launch_mix_slab_kind<kMixShrink>(P, a, st, tag);
    launch_mix_slab_kind<kMixUnshrink>(P, a, st, tag);
}

}  // namespace sfl
