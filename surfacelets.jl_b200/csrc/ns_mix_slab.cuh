// The slab passes of the NSSurfacelet for any axis lengths, on the mixed-radix
// line FFT of mixpass.cuh (its axis-3 passes: ns_mix_axis3.cu).  Same data flow, spectra
// layout, support boxes and launch chunks as the compile-time passes
// (ns_slab_pass.cuh, ns_slab.cu): per subband one pass along axis 3 and one
// over the axis-3 slabs, where the three line passes of the line pipeline
// (ns.cu) read and write the whole half grid each and know no box.
//
// A slab CTA holds its slab (pitch P1) in shared memory beside one tile of
// lines that the FFTs of both axes exchange through.  The rows' first step
// reads the box straight from global memory and their last one writes the
// slab; the column pairs' first step reads the slab and their last one writes
// the volume (the forward pass the other way round).
#pragma once

#include <algorithm>

#include "mixpass.cuh"
#include "plan.h"
#include "slab_core.cuh"

namespace sfl {

namespace {

constexpr int kMixSlabThreads = 384;
constexpr size_t kMixSlabTwo = 112 * 1024;   // shared memory that lets two CTAs share an SM

// ── line ops ─────────────────────────────────────────────────────────────────

// Rows k1 of a slab in global memory; columns outside the box read as zero.
struct RowLoadBox {
    const float2* src;
    int P1, b2, k2hi;
    struct Ctx {
        const float2* p;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool valid) const { return Ctx{src + (valid ? l : 0)}; }
    __device__ __forceinline__ float2 get(const Ctx& c, int i) const {
        return i <= b2 || i >= k2hi ? __ldcs(c.p + P1 * i) : make_float2(0.f, 0.f);
    }
};

// Rows of the slab in shared memory.
struct RowLoadS {
    const float2* S;
    int P1;
    struct Ctx {
        const float2* p;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool valid) const { return Ctx{S + (valid ? l : 0)}; }
    __device__ __forceinline__ float2 get(const Ctx& c, int i) const { return c.p[P1 * i]; }
};
struct RowStoreS {
    static constexpr bool kStaged = false;
    float2* S;
    int P1;
    struct Ctx {
        float2* p;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool) const { return Ctx{S + l}; }
    __device__ __forceinline__ void put(const Ctx& c, int k, float2 v) const { c.p[P1 * k] = v; }
};
struct RowStoreBox {
    static constexpr bool kStaged = false;
    float2* dst;
    int P1, b2, k2hi;
    struct Ctx {
        float2* p;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool) const { return Ctx{dst + l}; }
    __device__ __forceinline__ void put(const Ctx& c, int k, float2 v) const {
        if (k <= b2 || k >= k2hi) c.p[P1 * k] = v;
    }
};

// Columns 2l and 2l + 1 of the slab as one complex line (C2R of both; the
// imaginary parts of self-conjugate bins are dropped); rows past the box are
// zero, and the missing column of an odd count.
struct ColLoadPair {
    const float2* S;
    int P1, nk1, n1, n2;
    struct Ctx {
        const float2* a;
        bool two;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool valid) const {
        return Ctx{S + P1 * (valid ? 2 * l : 0), valid && 2 * l + 1 < n2};
    }
    __device__ __forceinline__ float2 get(const Ctx& c, int i) const {
        const bool up = 2 * i <= n1;
        const int k = up ? i : n1 - i;
        float2 A = make_float2(0.f, 0.f), B = A;
        if (k < nk1) {
            A = c.a[k];
            if (c.two) B = c.a[P1 + k];
        }
        if (k == 0 || 2 * k == n1) A.y = B.y = 0.f;
        return up ? make_float2(A.x - B.y, A.y + B.x) : make_float2(A.x + B.y, B.x - A.y);
    }
};
struct ColStoreReal {
    static constexpr bool kStaged = false;
    float* out;
    int n1, n2, es;
    float scale;
    struct Ctx {
        float* a;
        float* b;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool) const {
        float* a = out + (long long)(2 * l) * n1 * es;
        return Ctx{a, 2 * l + 1 < n2 ? a + (long long)n1 * es : nullptr};
    }
    __device__ __forceinline__ void put(const Ctx& c, int k, float2 v) const {
        const float2 w = c_scale(v, scale);
        c.a[k * es] = w.x;
        if (c.b) c.b[k * es] = w.y;
    }
};
// The same two real lines, soft-thresholded (the denoiser).
struct ColStoreShrink {
    static constexpr bool kStaged = false;
    float* out;
    int n1, n2;
    float scale, tau;
    struct Ctx {
        float* a;
        float* b;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool) const {
        float* a = out + 2 * l * n1;
        return Ctx{a, 2 * l + 1 < n2 ? a + n1 : nullptr};
    }
    __device__ __forceinline__ void put(const Ctx& c, int k, float2 v) const {
        const float2 x = c_scale(v, scale);
        c.a[k] = copysignf(fmaxf(fabsf(x.x) - tau, 0.f), x.x);
        if (c.b) c.b[k] = copysignf(fmaxf(fabsf(x.y) - tau, 0.f), x.y);
    }
};
// Two real columns of a volume as one complex line, and its spectrum unpacked
// into the slab's columns (rows of the box).
struct ColLoadReal {
    const float* in;
    int n1, n2, es;
    struct Ctx {
        const float* a;
        const float* b;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool valid) const {
        const float* a = in + (long long)(valid ? 2 * l : 0) * n1 * es;
        return Ctx{a, valid && 2 * l + 1 < n2 ? a + (long long)n1 * es : nullptr};
    }
    __device__ __forceinline__ float2 get(const Ctx& c, int i) const {
        return make_float2(c.a[i * es], c.b ? c.b[i * es] : 0.f);
    }
};
struct ColStoreHalf {
    static constexpr bool kStaged = true;
    float2* S;
    int P1, nk1, n1, n2;
    struct Ctx {
        float2* a;
        bool two;
    };
    __device__ __forceinline__ Ctx line(int, int l, bool) const { return Ctx{S + P1 * 2 * l, 2 * l + 1 < n2}; }
    __device__ __forceinline__ void staged(const Ctx& c, const float2* Z, int p, int nth) const {
        for (int k = p; k < nk1; k += nth) {
            const float2 zk = Z[k], zn = Z[k == 0 ? 0 : n1 - k];
            c.a[k] = half_spec_a(zk, zn);
            if (c.two) c.a[P1 + k] = half_spec_b(zk, zn);
        }
    }
};

// ── slab passes ──────────────────────────────────────────────────────────────

struct MixSlabGeom {
    MixArgs a1, a2;
    int n1, n2;
    int lg;      // lines a tile
    int tsz;     // values of one tile (the larger pitch)
    int big;     // a large prime factor on either axis
};

// One pass of an axis over the lines [0, nlines) in tiles; ends with the tiles
// and the outputs settled.
template <bool INV, bool BIG, class Load, class Store>
__device__ __forceinline__ void mix_lines(const Load& ld, const Store& st, const MixArgs& a, int nlines, int lg, int tfast,
                                          float2* tile, int tsz) {
    for (int l0 = 0; l0 < nlines; l0 += 1 << lg) {
        mix_pass<INV, BIG>(ld, st, a, MixTile{l0, nlines, lg, tfast}, tile, tile + tsz, tile + 2 * tsz, 0);
        __syncthreads();
    }
}

// The slab passes of the run-time radices.  The denoiser runs two: the inverse
// one with thresholded stores into the slab's own block of the spectrum (its
// reals take at most half the block, and its CTA has read the block by then),
// and the forward one from there.  As one pass with three tiles a CTA it was
// slower than the two apart: 64 x 200 x 64 denoised 515 -> 411 us, 127 x 127 x 64
// 1889 -> 1082.
enum MixSlabKind { kMixFwd, kMixInv, kMixShrink, kMixUnshrink };

// One CTA a unit (channel, item, n3), striding over the launch's units.
template <int KIND, bool BIG>
__global__ void __launch_bounds__(kMixSlabThreads, 2)
    ns_mix_slab_kernel(const __grid_constant__ SlabArgs a, const __grid_constant__ MixSlabGeom g) {
    extern __shared__ float2 sm[];
    const int P1 = a.P1, n1 = g.n1, n2 = g.n2, npairs = (n2 + 1) / 2;
    float2* S = sm;
    float2* tile = sm + P1 * n2;
    const long long SL = (long long)P1 * n2, PLANE = (long long)n1 * n2;
    const int per = a.ck.nz * a.n3;
    for (int u = blockIdx.x; u < a.units; u += gridDim.x) {
        const int ch = u / per, ur = u - ch * per;
        const int z = ur / a.n3, s3 = ur - z * a.n3;
        const ChunkItem& it = a.ck.item[z];
        const int nk1 = it.nk1, b2 = it.b2, k2hi = n2 - (it.nk2 - b2 - 1);
        float2* slab = a.spec + ch * a.spec_chstride + z * a.spec_zstride + s3 * SL;
        // narrow boxes take half tiles, so that fewer lanes hold no row
        const int lgr = g.lg > 4 && nk1 <= 16 ? 4 : g.lg;
        constexpr bool kFwd = KIND == kMixFwd || KIND == kMixUnshrink;
        if constexpr (kFwd) {
            const float* in = a.vol + ch + a.vol_off(z) + (long long)s3 * PLANE * a.es;
            const int es = KIND == kMixUnshrink ? 1 : a.es;
            if constexpr (KIND == kMixUnshrink) in = reinterpret_cast<const float*>(slab);
            mix_lines<false, BIG>(ColLoadReal{in, n1, n2, es}, ColStoreHalf{S, P1, nk1, n1, n2}, g.a1, npairs, g.lg, 0, tile,
                                  g.tsz);
            mix_lines<false, BIG>(RowLoadS{S, P1}, RowStoreBox{slab, P1, b2, k2hi}, g.a2, nk1, lgr, 1, tile, g.tsz);
        } else {
            mix_lines<true, BIG>(RowLoadBox{slab, P1, b2, k2hi}, RowStoreS{S, P1}, g.a2, nk1, lgr, 1, tile, g.tsz);
            const ColLoadPair ld{S, P1, nk1, n1, n2};
            if constexpr (KIND == kMixInv) {
                float* out = a.vol + ch + a.vol_off(z) + (long long)s3 * PLANE * a.es;
                mix_lines<true, BIG>(ld, ColStoreReal{out, n1, n2, a.es, a.scale}, g.a1, npairs, g.lg, 0, tile, g.tsz);
            } else {
                mix_lines<true, BIG>(ld, ColStoreShrink{reinterpret_cast<float*>(slab), n1, n2, a.scale, a.tau[it.s - 1]},
                                     g.a1, npairs, g.lg, 0, tile, g.tsz);
            }
        }
    }
}

// Tiles of a pass: a forward one stages whole lines in a second tile.
int mix_slab_tiles(const MixSlabGeom& g, bool fwd) { return fwd || g.big ? 2 : 1; }

size_t mix_slab_smem(const MixSlabGeom& g, int P1, int tiles) {
    return sizeof(float2) * ((size_t)P1 * g.n2 + (size_t)tiles * g.tsz + (g.big ? std::max(g.n1, g.n2) : 0));
}

// Tiles of 32 or 16 lines where two CTAs then share an SM, else of as many as
// one CTA holds (two CTAs of 8 lines each were the slower: 160 x 124 x 96
// analysis 764 us, one CTA of 32 lines 493).
bool mix_slab_geom(const MixArgs& a1, const MixArgs& a2, int P1, bool fwd, MixSlabGeom& g, int more = 0) {
    g.a1 = a1;
    g.a2 = a2;
    g.n1 = a1.sc.n;
    g.n2 = a2.sc.n;
    g.big = mix_big(a1.sc) || mix_big(a2.sc);
    const int pitch = std::max(a1.pitch, a2.pitch);
    for (const bool two : {true, false})
        for (g.lg = 5; g.lg >= (two ? 4 : 3); --g.lg) {
            g.tsz = pitch << g.lg;
            if (mix_slab_smem(g, P1, mix_slab_tiles(g, fwd) + more) <= (two ? kMixSlabTwo : kSlabSmemOneCta)) return true;
        }
    return false;
}

template <int KIND, bool BIG>
void launch_mix_slab_b(const SlabArgs& a, const MixSlabGeom& g, int sms, cudaStream_t st, const char* tag) {
    auto kern = ns_mix_slab_kernel<KIND, BIG>;
    static DeviceOnce once;
    allow_smem(once, kern, kSlabSmemOneCta);
    const size_t smem = mix_slab_smem(g, a.P1, mix_slab_tiles(g, KIND == kMixFwd || KIND == kMixUnshrink));
    const int items = std::max(mix_items(g.a1.sc), mix_items(g.a2.sc)) << g.lg;
    const int threads = std::min(kMixSlabThreads, std::max(64, (items + 31) / 32 * 32));
    // the last geometry's answer: the query costs as much as a launch
    thread_local int resident = 0, asked_threads = -1;
    thread_local size_t asked_smem = 0;
    if (asked_threads != threads || asked_smem != smem) {
        cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, threads, smem),
                   "cudaOccupancyMaxActiveBlocksPerMultiprocessor(mix slab)");
        asked_threads = threads;
        asked_smem = smem;
    }
    const int grid = std::max(1, std::min(a.units, std::max(resident, 1) * sms));
    int tok = prof_begin(tag, st);
    kern<<<grid, threads, smem, st>>>(a, g);
    prof_end(tok, st);
    cuda_check(cudaGetLastError(), "ns_mix_slab_kernel launch");
}

template <int KIND>
void launch_mix_slab_kind(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag) {
    MixSlabGeom g;
    if (!mix_slab_geom(mix_args(*P.ffts.at(P.dims[0])), mix_args(*P.ffts.at(P.dims[1])), P.P1,
                       KIND == kMixFwd || KIND == kMixUnshrink, g))
        throw ArgError("no slab kernel for this size");
    if (g.big)
        launch_mix_slab_b<KIND, true>(a, g, P.sms, st, tag);
    else
        launch_mix_slab_b<KIND, false>(a, g, P.sms, st, tag);
}

}  // namespace

}  // namespace sfl
