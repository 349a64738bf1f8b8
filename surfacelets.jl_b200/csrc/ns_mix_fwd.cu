// The forward slab pass for any axis lengths.
#include "ns_mix_slab.cuh"

namespace sfl {

void launch_mix_slab_fwd(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag) {
    launch_mix_slab_kind<0>(P, a, st, tag);
}

bool mix_slab_fits(const NSPlan& P) {
    MixSlabGeom g;
    for (int kind = 0; kind < 3; ++kind)
        if (!mix_slab_geom(mix_args(*P.ffts.at(P.dims[0])), mix_args(*P.ffts.at(P.dims[1])), P.P1, kind, g)) return false;
    return true;
}

}  // namespace sfl
