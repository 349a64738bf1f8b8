// The forward slab pass for any axis lengths.
#include "ns_mix_slab.cuh"

namespace sfl {

void launch_mix_slab_fwd(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag) {
    launch_mix_slab_kind<kMixFwd>(P, a, st, tag);
}

// The slab and three tiles: larger slabs would run few lines a tile on one CTA
// an SM, and take the line pipeline.
bool mix_slab_fits(const NSPlan& P) {
    MixSlabGeom g;
    return mix_slab_geom(mix_args(*P.ffts.at(P.dims[0])), mix_args(*P.ffts.at(P.dims[1])), P.P1, true, g, 1);
}

}  // namespace sfl
