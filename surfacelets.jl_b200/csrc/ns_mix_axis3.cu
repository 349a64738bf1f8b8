// The axis-3 passes of the slab pipeline for any length, on the mixed-radix
// line FFT of mixpass.cuh: the arithmetic and the tiles of the compile-time
// passes (ns_axis3_mask.cu, ns_axis3_accum.cu), with the line's X (analysis) and
// the segment's sums (synthesis) in shared memory.
#include <algorithm>

#include "mixpass.cuh"
#include "ns_axis3.cuh"
#include "plan.h"
#include "slab_core.cuh"

namespace sfl {

namespace {

constexpr int kShare = 4;   // items that share one FFT in a step of the axis-3 passes

// A line's X times the group factor (in a tile), times the wedge planes of an
// item.
struct Axis3LoadMask {
    const float2* xg;
    int pitch, l0;
    AxisLines ln;
    NSMaskTables tb;
    const ChunkSeg* sg;
    const ChunkItem* it;
    bool synth;
    struct Ctx {
        const float2* x;
        const float* wa;
        const float* wb;
        int was, wbs, mode;   // 0: no wedges, 1: plane b, 2: plane a (times b's constant), 3: both
        float c;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool valid) const {
        int k1, k2;
        ln.k12(valid ? l : 0, k1, k2);
        const NSMaskLine m = chunk_mask_line(tb, *sg, *it, k1, k2, synth);
        Ctx c{xg + (valid ? l - l0 : 0) * pitch, m.wa, m.wb, m.was, m.wbs, 0, 1.f};
        if (!(m.low || m.plain)) {
            c.mode = m.was == 0 ? 1 : (m.wbs == 0 ? 2 : 3);
            if (c.mode == 2) c.c = m.wb[0];
        }
        return c;
    }
    __device__ __forceinline__ float2 get(const Ctx& c, int i) const {
        const float2 x = c.x[i];
        if (c.mode == 0) return x;
        if (c.mode == 1) return c_scale(x, __ldg(c.wb + i * c.wbs));
        if (c.mode == 2) return c_scale(x, __ldg(c.wa + i * c.was) * c.c);
        return c_scale(x, __ldg(c.wa + i * c.was) * __ldg(c.wb + i * c.wbs));
    }
};

// A transformed line out to np items that share it, each times its plane a's
// value at the line (after), or to one item as it is.
struct Axis3StoreItems {
    static constexpr bool kStaged = false;
    float2* Y;
    long long ystride;
    int P1, s3;
    AxisLines ln;
    NSMaskTables tb;
    const ChunkItem* it;   // the first item; the others follow zstep apart
    int np, zstep;
    bool after;
    struct Ctx {
        float2* y;
        float a[kShare];
    };
    __device__ __forceinline__ Ctx line(int, int l, bool) const {
        int k1, k2;
        ln.k12(l, k1, k2);
        Ctx c;
        c.y = Y + k1 + P1 * k2;
#pragma unroll
        for (int q = 0; q < kShare; ++q) c.a[q] = q < np && after ? chunk_plane_a(tb, it[q * zstep], k1, k2) : 1.f;
        return c;
    }
    __device__ __forceinline__ void put(const Ctx& c, int k, float2 v) const {
        float2* y = c.y + k * s3;
#pragma unroll
        for (int q = 0; q < kShare; ++q)
            if (q < np) y[q * zstep * ystride] = after ? c_scale(v, c.a[q]) : v;
    }
};

struct MixAxis3 {
    MixArgs a;
    int lg, P1, s3;
};

// Analysis axis-3 pass; tiles as in ns_slab_mask_group_kernel.
template <bool BIG>
__global__ void __launch_bounds__(256, 2)
    ns_mix_mask_kernel(const float2* __restrict__ X, const __grid_constant__ MixAxis3 g,
                       const __grid_constant__ NSMaskTables tb, const __grid_constant__ Chunk ck,
                       const __grid_constant__ MaskTiles tl, int synth, float2* Y, long long ystride, long long xchs,
                       long long ychs) {
    extern __shared__ float2 sm[];
    X += blockIdx.y * xchs;   // channel
    Y += blockIdx.y * ychs;
    const int t = mask_tile_of(tl, blockIdx.x);
    const ChunkSeg& sg = ck.seg[tl.seg[t]];
    const int n = g.a.sc.n, LP = 1 << g.lg, tsz = g.a.pitch << g.lg;
    const int l0 = ((int)blockIdx.x - tl.first[t]) << g.lg, nlines = sg.nk1 * sg.nk2;
    const AxisLines ln{BoxMap{sg.nk1, sg.nk2, sg.b2, tb.n2}};
    float2* xg = sm;
    float2* tile = sm + tsz;
    // X times the group factor
    for (int it = threadIdx.x; it < n << g.lg; it += blockDim.x) {
        const int tt = it & (LP - 1), i = it >> g.lg, l = l0 + tt;
        float2 v = make_float2(0.f, 0.f);
        if (l < nlines) {
            int k1, k2;
            ln.k12(l, k1, k2);
            v = c_scale(X[k1 + g.P1 * k2 + (long long)i * g.s3], chunk_group_factor(tb, sg, k1, k2, i, synth != 0));
        }
        xg[tt * g.a.pitch + i] = v;
    }
    const int k0 = tl.k0[t], kend = k0 + tl.cnt[t];
    const int nbq = sg.nbq, rows = nbq > 0 ? sg.nz / nbq : 0;
    const bool wedges = !(sg.low || (synth && !tb.tight));
    const bool after = wedges && ck.item[sg.i0].wa_hi != 2;   // plane a constant along the line
    for (int k = k0; k < kend;) {
        // items k .. k + np - 1 (q-major) of one plane-b wedge share an FFT
        int np = 1;
        if (after && nbq > 0) np = min(min(rows - k % rows, kend - k), kShare);
        const ChunkItem* it = ck.item + sg.i0 + (nbq > 0 ? (k % rows) * nbq + k / rows : k);
        __syncthreads();   // xg is complete; the tile was read
        mix_pass<true, BIG>(Axis3LoadMask{xg, g.a.pitch, l0, ln, tb, &sg, it, synth != 0},
                            Axis3StoreItems{Y + (it - ck.item) * ystride, ystride, g.P1, g.s3, ln, tb, it, np,
                                            nbq > 0 ? nbq : 1, after},
                            g.a, MixTile{l0, nlines, g.lg, 1}, tile, tile + tsz, tile + 2 * tsz, 0);
        k += np;
    }
}

// The sum of a term's items, plane a's value at the line times each (before),
// or one item as it is.
struct Axis3LoadTerm {
    const float2* Y;
    long long ystride;
    int P1, s3;
    AxisLines ln;
    NSMaskTables tb;
    const ChunkItem* it;
    int np, zstep;
    bool before;
    short nk1, b2, n2;   // the segment's box: lines outside read as zero
    struct Ctx {
        const float2* y;
        float a[kShare];
        bool in;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool valid) const {
        int k1, k2;
        ln.k12(valid ? l : 0, k1, k2);
        Ctx c;
        c.in = valid && k1 < nk1 && (k2 <= b2 || k2 >= n2 - b2);
        c.y = Y + k1 + P1 * k2;
#pragma unroll
        for (int q = 0; q < kShare; ++q) c.a[q] = q < np && before ? chunk_plane_a(tb, it[q * zstep], k1, k2) : 1.f;
        return c;
    }
    __device__ __forceinline__ float2 get(const Ctx& c, int i) const {
        if (!c.in) return make_float2(0.f, 0.f);
        const float2* y = c.y + i * s3;
        float2 v = c_scale(__ldg(y), c.a[0]);
#pragma unroll
        for (int q = 1; q < kShare; ++q)
            if (q < np) v = c_fma(__ldg(y + q * zstep * ystride), c.a[q], v);
        return v;
    }
};

// A transformed term times its wedge planes, added to the segment's sums with
// one Kahan step (their compensations lie `rest` behind them).
struct Axis3StoreSum {
    static constexpr bool kStaged = false;
    float2* sums;
    int rest, pitch, l0;
    AxisLines ln;
    NSMaskTables tb;
    const ChunkSeg* sg;
    const ChunkItem* it;
    bool synth, before, first;
    struct Ctx {
        float2* s;
        const float* wa;
        const float* wb;
        int was, wbs;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool) const {
        int k1, k2;
        ln.k12(l, k1, k2);
        const NSMaskLine m = chunk_mask_line(tb, *sg, *it, k1, k2, synth);
        return Ctx{sums + (l - l0) * pitch, m.wa, m.low || m.plain ? nullptr : m.wb, m.was, m.wbs};
    }
    __device__ __forceinline__ void put(const Ctx& c, int k, float2 v) const {
        float w = 1.f;
        if (c.wb) w = before ? __ldg(c.wb + k * c.wbs) : __ldg(c.wa + k * c.was) * __ldg(c.wb + k * c.wbs);
        float2 s = make_float2(0.f, 0.f), e = s;
        if (!first) {
            s = c.s[k];
            e = c.s[k + rest];
        }
        kahan_fma(s, e, v, w);
        c.s[k] = s;
        c.s[k + rest] = e;
    }
};

// Synthesis axis-3 pass; segments, terms and Kahan steps as in
// ns_slab_accum_kernel (STEPS), the group factor applied to a segment's sum.
template <bool BIG>
__global__ void __launch_bounds__(256, 2)
    ns_mix_accum_kernel(const float2* __restrict__ Y, long long ystride, const __grid_constant__ MixAxis3 g, BoxMap un,
                        const __grid_constant__ NSMaskTables tb, const __grid_constant__ Chunk ck, int synth, float2* acc,
                        float2* comp, long long ychs, long long achs, long long agrp) {
    extern __shared__ float2 sm[];
    Y += blockIdx.y * ychs;   // channel
    acc += blockIdx.y * achs + blockIdx.z * agrp;
    comp += blockIdx.y * achs + blockIdx.z * agrp;
    const int n = g.a.sc.n, LP = 1 << g.lg, tsz = g.a.pitch << g.lg;
    const int l0 = (int)blockIdx.x << g.lg, nlines = un.nk1 * un.nk2;
    const AxisLines ln{un};
    float2* sums = sm;   // and their compensations
    float2* tile = sm + 2 * tsz;
    const bool wedge_masks = !(synth && !tb.tight);
    // this thread's line in the Kahan steps, and its bins
    const int tt = threadIdx.x & (LP - 1);
    int k1 = 0, k2 = 0;
    const bool inl = l0 + tt < nlines;
    if (inl) ln.k12(l0 + tt, k1, k2);
    for (int s = 0; s < ck.nseg; ++s) {
        const ChunkSeg& sg = ck.seg[s];
        if (sg.ord % (int)gridDim.z != (int)blockIdx.z) continue;
        const bool in = inl && k1 < sg.nk1 && (k2 <= sg.b2 || k2 >= tb.n2 - sg.b2);
        if (!__syncthreads_or(in)) continue;
        const int nbq = sg.nbq, rows = nbq > 0 ? sg.nz / nbq : 1;
        const bool before = wedge_masks && !sg.low && ck.item[sg.i0].wa_hi != 2;
        const int nt = before ? rows : 1, nterms = nbq > 0 ? nbq : sg.nz;
        for (int t = 0; t < nterms; ++t)
            for (int p = 0; p < nt; p += kShare) {
                const ChunkItem* it = ck.item + sg.i0 + t + p * nbq;
                mix_pass<false, BIG>(Axis3LoadTerm{Y + (it - ck.item) * ystride, ystride, g.P1, g.s3, ln, tb, it,
                                                   min(nt - p, kShare), nbq > 0 ? nbq : 1, before, sg.nk1, sg.b2,
                                                   (short)tb.n2},
                                     Axis3StoreSum{sums, tsz, g.a.pitch, l0, ln, tb, &sg, it, synth != 0, before,
                                                   t == 0 && p == 0},
                                     g.a, MixTile{l0, nlines, g.lg, 1}, tile, tile + tsz, tile + 2 * tsz, 0);
                __syncthreads();
            }
        if (in)
            for (int i = threadIdx.x >> g.lg; i < n; i += blockDim.x >> g.lg) {
                const long long o = k1 + g.P1 * k2 + (long long)i * g.s3;
                const float f = chunk_group_factor(tb, sg, k1, k2, i, synth != 0);
                float2 sv = acc[o], cv = c_fma(sums[tsz + tt * g.a.pitch + i], f, comp[o]);
                kahan_fma(sv, cv, sums[tt * g.a.pitch + i], f);
                acc[o] = sv;
                comp[o] = cv;
            }
        __syncthreads();   // the sums are rewritten by the next segment
    }
}

// `beside`: tiles kept beside the FFT's own (analysis: the line's X; synthesis:
// the sums and their compensations).
MixAxis3 mix_axis3(const NSPlan& P, int beside, size_t& smem) {
    MixAxis3 g;
    g.a = mix_args(*P.ffts.at(P.dims[2]));
    g.P1 = P.P1;
    g.s3 = P.P1 * P.dims[1];
    g.lg = mix_lines_lg(g.a, false, beside * sizeof(float2) * g.a.pitch);
    smem = mix_smem_bytes(g.a.sc, g.lg, g.a.pitch, false) + beside * sizeof(float2) * ((size_t)g.a.pitch << g.lg);
    return g;
}

int axis3_threads(const MixAxis3& g) {
    // a whole number of threads a line
    return std::max(1 << g.lg, mix_threads(g.a, g.lg) >> g.lg << g.lg);
}

}  // namespace

bool ns_mix_slab_supported(const NSPlan& P) {
    size_t smem;
    mix_axis3(P, 2, smem);
    // 32-bit offsets within a spectrum
    return (any_slab_fits(P) || mix_slab_fits(P)) && smem <= kSlabSmemOneCta && P.SP < (1LL << 31) && P.dims[2] <= 4096;
}

int mix_axis3_lines(const NSPlan& P) {
    size_t smem;
    return 1 << mix_axis3(P, 1, smem).lg;
}

void launch_mix_mask(const NSPlan& P, const float2* X, const Chunk& ck, const MaskTiles& tl, int synth, float2* Y,
                     int nch, long long xchs, long long ychs, cudaStream_t st) {
    size_t smem;
    const MixAxis3 g = mix_axis3(P, 1, smem);
    const bool big = mix_big(g.a.sc);
    auto kern = big ? ns_mix_mask_kernel<true> : ns_mix_mask_kernel<false>;
    static DeviceOnce once[2];
    allow_smem(once[big], kern, kSlabSmemOneCta);
    kern<<<dim3(tl.first[tl.n], nch), axis3_threads(g), smem, st>>>(X, g, P.tb, ck, tl, synth, Y, P.SP, xchs, ychs);
    cuda_check(cudaGetLastError(), "ns_mix_mask_kernel launch");
}

void launch_mix_accum(const NSPlan& P, const Chunk& ck, const BoxMap& un, int synth, const float2* Y, float2* acc,
                      float2* comp, int nch, int ngrp, long long ychs, cudaStream_t st) {
    size_t smem;
    const MixAxis3 g = mix_axis3(P, 2, smem);
    const bool big = mix_big(g.a.sc);
    auto kern = big ? ns_mix_accum_kernel<true> : ns_mix_accum_kernel<false>;
    static DeviceOnce once[2];
    allow_smem(once[big], kern, kSlabSmemOneCta);
    const int lines = un.nk1 * un.nk2;
    kern<<<dim3((lines + (1 << g.lg) - 1) >> g.lg, nch, ngrp), axis3_threads(g), smem, st>>>(
        Y, P.SP, g, un, P.tb, ck, synth, acc, comp, ychs, P.SP, (long long)P.nch * P.SP);
    cuda_check(cudaGetLastError(), "ns_mix_accum_kernel launch");
}

}  // namespace sfl
