// What the axis-3 passes of the slab pipeline share: box lines, the mask of a
// chunk's item on a line, and the tiles of the analysis pass.
#pragma once

#include "ns_mask.cuh"
#include "slab_core.cuh"

namespace sfl {

// Line l = (k1, j) with k1 fastest; column j maps to k2 = j for j <= b2 and
// to the negative frequencies n2 - (nk2 - j) above.
struct BoxMap {
    int nk1, nk2, b2, n2;
    __device__ __forceinline__ void k12(int l, int& k1, int& k2) const {
        const int j = l / nk1;
        k1 = l - j * nk1;
        k2 = j <= b2 ? j : j + (n2 - nk2);
    }
};

// The mask context of a chunk's item on the line (k1, k2): NSMaskLine from the
// launch's own copy of the item.
__device__ __forceinline__ NSMaskLine chunk_mask_line(const NSMaskTables& tb, const ChunkSeg& sg, const ChunkItem& it,
                                                      int k1, int k2, bool synth) {
    NSMaskLine c;
    c.low = sg.low;
    c.plain = 0;
    c.m = nullptr;
    c.wa = c.wb = nullptr;
    c.was = c.wbs = 0;
    c.lowc = 0.f;
    c.lowv = nullptr;
    if (c.low) {
        c.lowc = tb.vec[tb.low_off[0] + k1] * tb.vec[tb.low_off[1] + k2];
        c.lowv = tb.vec + tb.low_off[2];
        return c;
    }
    const int l = k1 + tb.h1 * k2;
    if (synth && !tb.tight) {
        c.plain = 1;
        c.m = tb.Bl + (long long)sg.lv * tb.H + l;
        return c;
    }
    c.m = tb.G + (long long)sg.g * tb.H + l;
    // a plane over (lo, hi): index off + k_lo + dlo * k_hi; axis 3 can only be hi
    c.wa = tb.planes + it.wa_off + (it.wa_lo == 0 ? k1 : k2) + (it.wa_hi == 2 ? 0 : it.wa_dlo * k2);
    c.was = it.wa_hi == 2 ? it.wa_dlo : 0;
    c.wb = tb.planes + it.wb_off + (it.wb_lo == 0 ? k1 : k2) + (it.wb_hi == 2 ? 0 : it.wb_dlo * k2);
    c.wbs = it.wb_hi == 2 ? it.wb_dlo : 0;
    return c;
}

// The group factor of a segment at (k1, k2, k3): group table, bandpass table or
// the lowpass factors.
__device__ __forceinline__ float chunk_group_factor(const NSMaskTables& tb, const ChunkSeg& sg, int k1, int k2, int k3,
                                                    bool synth) {
    if (sg.low) return tb.vec[tb.low_off[0] + k1] * tb.vec[tb.low_off[1] + k2] * tb.vec[tb.low_off[2] + k3];
    const long long q = k1 + tb.h1 * (k2 + (long long)tb.n2 * k3);
    return synth && !tb.tight ? tb.Bl[(long long)sg.lv * tb.H + q] : tb.G[(long long)sg.g * tb.H + q];
}

// Plane a of an item at (k1, k2), for a plane constant along axis 3.
__device__ __forceinline__ float chunk_plane_a(const NSMaskTables& tb, const ChunkItem& it, int k1, int k2) {
    return __ldg(tb.planes + it.wa_off + (it.wa_lo == 0 ? k1 : k2) + it.wa_dlo * k2);
}

// Lines of a box.
struct AxisLines {
    BoxMap b;
    __device__ __forceinline__ void k12(int l, int& k1, int& k2) const { b.k12(l, k1, k2); }
};

// The CTAs of the analysis line pass: tile t takes the line blocks of its
// segment's box, CTAs [first[t], first[t + 1]), for cnt items from k0.
struct MaskTiles {
    int n;
    int first[kChunkItems + 1];
    signed char seg[kChunkItems], k0[kChunkItems], cnt[kChunkItems];
};

__device__ __forceinline__ int mask_tile_of(const MaskTiles& tl, int cta) {
    int t = 0;
    while (t + 1 < tl.n && cta >= tl.first[t + 1]) ++t;
    return t;
}

// The axis-3 passes with the length known at compile time (ns_axis3_mask.cu,
// ns_axis3_accum.cu), and the slab passes of the same lengths
// (ns_any_slab.cuh).
bool axis3_len(int n);
int axis3_lines(int n);   // lines a CTA of the analysis pass takes
void launch_axis3_mask(const NSPlan& P, const float2* X, const Chunk& ck, const MaskTiles& tl, int synth, float2* Y,
                       int nch, long long xchs, long long ychs, cudaStream_t st);
void launch_axis3_accum(const NSPlan& P, const Chunk& ck, const BoxMap& un, int synth, const float2* Y, float2* acc,
                        float2* comp, int nch, int ngrp, long long ychs, cudaStream_t st);
bool any_slab_fits(const NSPlan& P);
void launch_any_slab_fwd(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag);
void launch_any_slab_inv(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag);
void launch_any_slab_shrink(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag);

// The passes for any axis lengths (ns_mix_slab.cuh, ns_mix_axis3.cu).
bool mix_slab_fits(const NSPlan& P);
void launch_mix_slab_fwd(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag);
void launch_mix_slab_inv(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag);
void launch_mix_slab_shrink(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag);
int mix_axis3_lines(const NSPlan& P);
void launch_mix_mask(const NSPlan& P, const float2* X, const Chunk& ck, const MaskTiles& tl, int synth, float2* Y,
                     int nch, long long xchs, long long ychs, cudaStream_t st);
void launch_mix_accum(const NSPlan& P, const Chunk& ck, const BoxMap& un, int synth, const float2* Y, float2* acc,
                      float2* comp, int nch, int ngrp, long long ychs, cudaStream_t st);

}  // namespace sfl
