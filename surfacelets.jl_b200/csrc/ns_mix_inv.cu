// The inverse slab pass for any axis lengths.
#include "ns_mix_slab.cuh"

namespace sfl {

void launch_mix_slab_inv(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag) {
    launch_mix_slab_kind<kMixInv>(P, a, st, tag);
}

}  // namespace sfl
