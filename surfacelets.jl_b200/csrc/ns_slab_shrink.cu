// The denoiser's slab pass of every compile-time slab size.
#include "ns_slab_pass.cuh"

namespace sfl {

void launch_slab_shrink(int na, int nb, const SlabArgs& a, int sms, size_t smem, cudaStream_t st, const char* tag) {
    launch_slab_kind<2>(na, nb, a, sms, smem, st, tag);
}

}  // namespace sfl
