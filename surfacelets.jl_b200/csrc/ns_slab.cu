// NSSurfacelet slab pipeline for sm_100a: per subband one line pass along
// axis 3 and one pass over the axis-3 slabs, with the zero rows and columns of
// band-limited masks skipped.
//
// Spectra (the input spectrum X, the per-subband intermediates Y and the
// synthesis accumulator) live on the rfft grid (h1, n2, n3) with the axis-1
// pitch padded to P1 (P1 >= h1, P1 = 2 mod 4): bin (k1, k2, k3) sits at
// k1 + P1 (k2 + n2 k3), so one slab (fixed k3 or n3) is a contiguous block of
// P1 n2 bins that a CTA holds in shared memory.
//
//   analysis of subband s, c_s = irfft(X M_s):
//     line pass  Y_s(k1, k2, n3) = IFFT_3(X M_s)(k1, k2, .) for the lines of
//                the mask's support box (mask applied on load);
//     slab pass  per n3: IFFT_2 of the rows k1 < nk1, then the C2R along
//                axis 1 of two columns at a time, written straight into c_s.
//   synthesis, x = irfft(sum_s M_s rfft(c_s)):
//     slab pass  per n3: R2C along axis 1 (two columns at a time), FFT_2 of
//                the rows in the box -> Y_s;
//     line pass  FFT_3 of Y_s times M_s, summed over the subbands of one mask
//                group on chip (with a Kahan step a term on mixed plans), then
//                one Kahan step into the accumulator (a round trip of it and its
//                compensation per group);
//     then the irfft of the accumulator (line pass and slab pass, no mask).
//
// Support boxes: the group factor B_j of scale j is a product of per-axis
// raised-cosine lowpass profiles of the finer levels
// (src/pyramid/fourier_pyramid.jl:143-150, src/transforms/ns_surfacelet.jl:
// 271-272), so it vanishes outside |k_d| <= b_d.  The plan scans each
// float64-designed group table for its box; lines and rows outside it are
// neither loaded nor transformed, and read as zeros downstream.
//
// Inside the slab pass the N2 lanes of a line sit in one warp, and the
// exchange between the two in-register DFT steps goes through the line's own
// slots of the slab (a row, or the two columns of a pair) with an XOR
// swizzle, so it needs only __syncwarp; CTA-wide barriers separate the
// phases.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "ns_axis3.cuh"
#include "plan.h"
#include "prof.h"
#include "regpass.cuh"
#include "slab_core.cuh"

namespace sfl {

namespace {

// ── lines along axis 3 of a padded spectrum, restricted to a box ───────────

struct L3LoadC {
    const float2* src;
    long long zstride;
    int P1, s3;
    BoxMap bx;
    struct Ctx {
        const float2* p;
    };
    __device__ __forceinline__ Ctx line(int z, int l, bool valid) const {
        int k1 = 0, k2 = 0;
        if (valid) bx.k12(l, k1, k2);
        return Ctx{src + z * zstride + k1 + P1 * k2};
    }
    __device__ __forceinline__ float2 get(const Ctx& c, int i) const { return c.p[i * s3]; }
};

// The plan's NG accumulators less their compensations, summed in the
// accumulators' order.  The first pass of the inverse FFT stores to the
// accumulators it reads: plain loads there, the read-only path for the
// compensations only.
template <int NG>
struct GroupSum {
    const float2* acc;
    const float2* comp;
    long long gstride;
    __device__ __forceinline__ float2 at(long long o) const {
        float2 s[NG], e[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            s[g] = acc[g * gstride + o];
            e[g] = __ldg(comp + g * gstride + o);
        }
        float2 v = c_sub(s[0], e[0]);
#pragma unroll
        for (int g = 1; g < NG; ++g) v = c_add(v, c_sub(s[g], e[g]));
        return v;
    }
};

template <int NG>
struct L3LoadSum {
    GroupSum<NG> gs;
    long long zstride;
    int P1, s3;
    BoxMap bx;
    struct Ctx {
        long long o;
    };
    __device__ __forceinline__ Ctx line(int z, int l, bool valid) const {
        int k1 = 0, k2 = 0;
        if (valid) bx.k12(l, k1, k2);
        return Ctx{z * zstride + k1 + P1 * k2};
    }
    __device__ __forceinline__ float2 get(const Ctx& c, int i) const { return gs.at(c.o + i * s3); }
};

// The accumulators summed into the first one, two bins a thread and step (the
// pitch is even and every accumulator starts 16-byte aligned).
template <int NG>
__global__ void __launch_bounds__(256) sum_groups_kernel(float4* acc, const float4* comp, long long gstride, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float4 s[NG], e[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            s[g] = acc[g * gstride + i];
            e[g] = __ldg(comp + g * gstride + i);
        }
        float2 a = c_sub(make_float2(s[0].x, s[0].y), make_float2(e[0].x, e[0].y));
        float2 b = c_sub(make_float2(s[0].z, s[0].w), make_float2(e[0].z, e[0].w));
#pragma unroll
        for (int g = 1; g < NG; ++g) {
            a = c_add(a, c_sub(make_float2(s[g].x, s[g].y), make_float2(e[g].x, e[g].y)));
            b = c_add(b, c_sub(make_float2(s[g].z, s[g].w), make_float2(e[g].z, e[g].w)));
        }
        acc[i] = make_float4(a.x, a.y, b.x, b.y);
    }
}

// A channel's accumulators added into a caller's spectrum and its compensation
// (on a cleared one, GroupSum's values exactly).
template <int NG>
__global__ void merge_groups_kernel(GroupSum<NG> gs, float2* A, float2* C, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float2 s = A[i], e = C[i];
        kahan_add(s, e, gs.at(i));
        A[i] = s;
        C[i] = e;
    }
}

struct L3StoreC {
    static constexpr bool kStaged = false;
    float2* dst;
    long long zstride;
    int P1, s3;
    BoxMap bx;
    struct Ctx {
        float2* p;
    };
    __device__ __forceinline__ Ctx line(int z, int l, bool valid) const {
        int k1 = 0, k2 = 0;
        if (valid) bx.k12(l, k1, k2);
        return Ctx{dst + z * zstride + k1 + P1 * k2};
    }
    __device__ __forceinline__ void put(const Ctx& c, int k, float2 v) const { c.p[k * s3] = v; }
};

bool slab_len(int n) { return n == 64 || n == 96 || n == 128 || n == 160 || n == 256; }

int slab_pitch(int h1) { return slab_pitch_c(h1); }

size_t slab_smem(int n1, int n2) {
    return sizeof(float2) * ((size_t)n1 + n2 + (size_t)slab_pitch(n1 / 2 + 1) * n2) + 16;   // + the mbarrier
}

// ── drivers ──────────────────────────────────────────────────────────────────

BoxMap box_map(const NSPlan& P, const NSBox& b) { return BoxMap{b.nk1, b.nk2, b.b2, P.dims[1]}; }

const NSBox& item_box(const NSPlan& P, int item) {
    const NSItem& it = P.items_host[item];
    return P.boxes[it.kind == 1 ? (int)P.boxes.size() - 1 : it.g];
}

// Items [i0, i0 + nz) as nbq plane-b wedges times whole rows of plane-a
// wedges constant along axis 3 (item t = p nbq + q, one mask group): nbq,
// else 0.  Only then do the axis-3 passes share FFTs between items.
int chunk_nbq(const NSPlan& P, int i0, int nz, bool synth_masks) {
    if (nz < 2 || (synth_masks && !P.p.tight)) return 0;
    const NSItem& f = P.items_host[i0];
    if (f.kind != 0 || f.wa_hi == 2) return 0;
    int nb = 1;
    while (nb < nz && P.items_host[i0 + nb].wb_off != f.wb_off) ++nb;
    if (nz % nb != 0) return 0;
    for (int t = 0; t < nz; ++t) {
        const NSItem& it = P.items_host[i0 + t];
        if (it.kind != 0 || it.g != f.g || it.wa_hi == 2 || it.wb_off != P.items_host[i0 + t % nb].wb_off ||
            it.wa_off != P.items_host[i0 + (t / nb) * nb].wa_off)
            return 0;
    }
    return nb;
}

// End of the segment that starts at item i0: consecutive items of one mask
// group, at most P.group of them.
int seg_end(const NSPlan& P, int i0, int i1) {
    auto key = [&](int i) { return P.items_host[i].kind == 1 ? -1 : P.items_host[i].g; };
    int e = i0 + 1;
    while (e < i1 && e - i0 < P.group && e - i0 < kChunkItems && key(e) == key(i0)) ++e;
    return e;
}

// Algorithmic bytes of one box of a spectrum (complex float32 bins).
double box_bytes(const NSPlan& P, const NSBox& b) { return 8.0 * b.nk1 * b.nk2 * P.dims[2]; }

// End of the chunk that starts at item i0: whole segments, as many as fit the
// work slots, one launch's tables and about the L2 (their intermediate
// spectra pass through it: 126 MB, of which the volumes' streams take their
// share).  A launch a mask group left the coarse scales' launches short: at
// 64^3 [2,2,3] 24 launches an analysis of 2 to 5 us each.
constexpr double kChunkBytes = 80e6;
int chunk_end(const NSPlan& P, int i0) {
    int i1 = i0, segs = 0;
    double bytes = 0;
    while (i1 < P.S && segs < kChunkSegs) {
        const int e = seg_end(P, i1, P.S);
        const double add = (e - i1) * box_bytes(P, item_box(P, i1)) * P.nch;
        if (i1 > i0 && (e - i0 > std::min(P.slots, kChunkItems) || bytes + add > kChunkBytes)) break;
        bytes += add;
        i1 = e;
        ++segs;
    }
    return i1;
}

// The launch tables of items [i0, i0 + nz).
Chunk make_chunk(const NSPlan& P, int i0, int nz, bool synth_masks) {
    if (nz < 1 || nz > kChunkItems) throw ArgError("too many subbands in one launch");
    Chunk c{};
    c.nz = nz;
    for (int a = i0; a < i0 + nz;) {
        const int e = seg_end(P, a, i0 + nz);
        if (c.nseg == kChunkSegs) throw ArgError("too many mask groups in one launch");
        const NSItem& f = P.items_host[a];
        const NSBox& b = item_box(P, a);
        ChunkSeg& sg = c.seg[c.nseg];
        sg.g = f.g;
        sg.lv = f.lv;
        sg.i0 = (short)(a - i0);
        sg.nz = (short)(e - a);
        sg.nbq = (short)chunk_nbq(P, a, e - a, synth_masks);
        sg.low = f.kind == 1;
        sg.ord = (short)(f.kind == 1 ? (int)P.boxes.size() - 1 : f.g);
        sg.nk1 = (short)b.nk1;
        sg.nk2 = (short)b.nk2;
        sg.b2 = (short)b.b2;
        for (int i = a; i < e; ++i) {
            const NSItem& it = P.items_host[i];
            ChunkItem& ci = c.item[i - i0];
            ci.s = it.s;
            ci.wa_off = it.wa_off;
            ci.wb_off = it.wb_off;
            ci.wa_dlo = (short)it.wa_dlo;
            ci.wb_dlo = (short)it.wb_dlo;
            ci.wa_lo = (signed char)it.wa_lo;
            ci.wa_hi = (signed char)it.wa_hi;
            ci.wb_lo = (signed char)it.wb_lo;
            ci.wb_hi = (signed char)it.wb_hi;
            ci.nk1 = sg.nk1;
            ci.nk2 = sg.nk2;
            ci.b2 = sg.b2;
        }
        ++c.nseg;
        a = e;
    }
    return c;
}

// The one full box of a volume's own spectrum.
Chunk full_chunk(const NSPlan& P) {
    Chunk c{};
    c.nz = 1;
    c.item[0].s = 1;
    c.item[0].nk1 = (short)P.boxes_full.nk1;
    c.item[0].nk2 = (short)P.boxes_full.nk2;
    c.item[0].b2 = (short)P.boxes_full.b2;
    return c;
}

// The union of the boxes of a chunk.
NSBox union_box(const Chunk& c) {
    NSBox u;
    for (int i = 0; i < c.nseg; ++i) {
        u.nk1 = std::max(u.nk1, (int)c.seg[i].nk1);
        u.nk2 = std::max(u.nk2, (int)c.seg[i].nk2);
        u.b2 = std::max(u.b2, (int)c.seg[i].b2);
    }
    return u;
}

// Sum of box_bytes over the items of a chunk, and over its segments.
double items_bytes(const NSPlan& P, const Chunk& c) {
    double b = 0;
    for (int i = 0; i < c.nz; ++i) b += 8.0 * c.item[i].nk1 * c.item[i].nk2 * P.dims[2];
    return b;
}
double segs_bytes(const NSPlan& P, const Chunk& c) {
    double b = 0;
    for (int i = 0; i < c.nseg; ++i) b += 8.0 * c.seg[i].nk1 * c.seg[i].nk2 * P.dims[2];
    return b;
}

SlabArgs slab_args(const NSPlan& P, const Chunk& ck, int nch) {
    SlabArgs a{};
    a.ck = ck;
    a.P1 = P.P1;
    a.n3 = P.dims[2];
    a.units = nch * ck.nz * P.dims[2];
    a.twa = P.ffts.at(P.dims[0])->sh.tw;
    a.twb = P.ffts.at(P.dims[1])->sh.tw;
    a.es = 1;
    a.scale = 1.f;
    a.status = P.status.dev;
    return a;
}

void set_volumes(SlabArgs& a, const float* vol, ZMap vz, int es) {
    a.vol = const_cast<float*>(vol);
    a.vol_zstride = vz.zstride;
    a.vol_sub_stride = vz.items ? vz.sub_stride : 0;
    a.es = es;
}

// Accumulators of a spectrum acc: the plan's own are P.ngrp (mask group g adds
// into number g mod ngrp, nch SP apart), a caller's is one.
int acc_groups(const NSPlan& P, const float2* acc) {
    const float2* a = P.acc.as<float2>();
    return acc >= a && acc < a + P.nch * P.SP ? P.ngrp : 1;
}

// KIND: 0 the forward slab pass, 1 the inverse, 2 the denoiser's shrink pass.
template <int KIND>
void launch_slab(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag) {
    const int na = P.dims[0], nb = P.dims[1];
    if (P.mixed) {
        if (any_slab_fits(P))
            return (KIND == 0 ? launch_any_slab_fwd : KIND == 1 ? launch_any_slab_inv : launch_any_slab_shrink)(P, a, st,
                                                                                                              tag);
        return (KIND == 0 ? launch_mix_slab_fwd : KIND == 1 ? launch_mix_slab_inv : launch_mix_slab_shrink)(P, a, st, tag);
    }
    if (slab_cluster_supported(na, nb)) {
        if (!launch_slab_cluster(KIND, na, nb, a, P.sms, st, tag)) throw ArgError("no slab kernel for this size");
        return;
    }
    (KIND == 0 ? launch_slab_fwd : KIND == 1 ? launch_slab_inv : launch_slab_shrink)(na, nb, a, P.sms, slab_smem(na, nb),
                                                                                    st, tag);
}

template <bool INV, class Load, class Store>
void line3(const NSPlan& P, const Load& ld, const Store& so, int nlines, int nz, cudaStream_t st, const char* tag) {
    launch_line<INV>(*P.ffts.at(P.dims[2]), ld, so, nlines, nz, true, st, tag);
}

thread_local bool t_concurrent = false;

// Subbands a CTA of the analysis axis-3 pass (the line's X and group factor
// are loaded once for all of them).  An explicit choice is taken as given:
// the plan's (the autotuner's tile), else SFL_MASK_IPC (1, 2, 4 or 8) from
// the environment, read once.  By default up to 8 (a finest-scale group of
// [2,2,3] in one CTA: 2027 vs 2013 Mvox/s for 4 on the bench workload),
// and for launches that run alone halved while the launch would hold fewer
// CTAs than the GPU has SMs.  In a batch graph the other branches fill the GPU
// and the split CTAs only reload X.
int mask_ipc_cap(const NSPlan& P) {
    static const int env_cap = [] {
        const char* e = std::getenv("SFL_MASK_IPC");
        if (!e) return 0;
        const int v = std::atoi(e);
        return v >= 8 ? 8 : (v >= 4 ? 4 : (v >= 2 ? 2 : 1));
    }();
    return P.ipc > 0 ? P.ipc : env_cap;
}

// The tiles of a chunk's analysis line pass with at most ipc subbands a CTA,
// the largest boxes first; returns the number of CTAs.
int mask_tiles(const Chunk& ck, int lp, int ipc, MaskTiles& t) {
    int order[kChunkSegs];
    for (int i = 0; i < ck.nseg; ++i) order[i] = i;
    std::stable_sort(order, order + ck.nseg, [&](int a, int b) {
        return ck.seg[a].nk1 * ck.seg[a].nk2 > ck.seg[b].nk1 * ck.seg[b].nk2;
    });
    t.n = 0;
    int first = 0;
    for (int i = 0; i < ck.nseg; ++i) {
        const ChunkSeg& sg = ck.seg[order[i]];
        const int blocks = (sg.nk1 * sg.nk2 + lp - 1) / lp;
        for (int k = 0; k < sg.nz; k += ipc) {
            t.first[t.n] = first;
            t.seg[t.n] = (signed char)order[i];
            t.k0[t.n] = (signed char)k;
            t.cnt[t.n] = (signed char)std::min(ipc, sg.nz - k);
            ++t.n;
            first += blocks;
        }
    }
    t.first[t.n] = first;
    return first;
}

int choose_mask_tiles(const NSPlan& P, const Chunk& ck, int lp, int nch, MaskTiles& tl) {
    const int cap = mask_ipc_cap(P);
    int ipc = cap > 0 ? cap : 8;
    int ctas = mask_tiles(ck, lp, ipc, tl);
    if (cap == 0 && !t_concurrent)
        while (ipc > 1 && ctas * nch < P.sms) ctas = mask_tiles(ck, lp, ipc /= 2, tl);
    return ctas;
}

// Channels: complex volumes run their two real channels in the same launches
// (spectra and intermediates one block per channel, the volume's channels
// interleaved floats), with each channel's arithmetic that of a real volume.
// Y blocks: channel ch of item z at work + ch * (slots SP) + z * SP.
long long ych_stride(const NSPlan& P) { return (long long)P.slots * P.SP; }

// rfft3 of nch interleaved real channels (element stride es) into the padded
// spectra X + ch SP.
void slab_rfft3(NSPlan& P, const float* x, int es, float2* X, int nch, cudaStream_t st) {
    const NSBox& full = P.boxes_full;
    prof_bytes("ns_slab_r2c", nch * (4.0 * P.N + box_bytes(P, full)));
    prof_bytes("ns_slab_line3", nch * 2 * box_bytes(P, full));
    SlabArgs a = slab_args(P, full_chunk(P), nch);
    a.spec_chstride = P.SP;
    a.spec = X;
    set_volumes(a, x, ZMap{}, es);
    launch_slab<0>(P, a, st, "ns_slab_r2c");
    const BoxMap bx = box_map(P, full);
    const int s3 = P.P1 * P.dims[1];
    line3<false>(P, L3LoadC{X, P.SP, P.P1, s3, bx}, L3StoreC{X, P.SP, P.P1, s3, bx}, full.nk1 * full.nk2, nch, st,
                 "ns_slab_line3");
}

void sum_groups(NSPlan& P, float2* A, const float2* K, int ng, int nch, cudaStream_t st) {
    const long long n = nch * P.SP / 2, blocks = std::min<long long>((n + 255) / 256, 16LL * P.sms);
    float4* a = reinterpret_cast<float4*>(A);
    const float4* k = reinterpret_cast<const float4*>(K);
    const long long gs = (long long)P.nch * P.SP / 2;
    int tok = prof_begin("ns_slab_line3", st);
    if (ng == 4)
        sum_groups_kernel<4><<<(unsigned)blocks, 256, 0, st>>>(a, k, gs, n);
    else
        sum_groups_kernel<2><<<(unsigned)blocks, 256, 0, st>>>(a, k, gs, n);
    prof_end(tok, st);
    cuda_check(cudaGetLastError(), "sum_groups_kernel launch");
}

// irfft3 of the padded spectra A + ch SP (overwritten) into nch channels.
void slab_irfft3(NSPlan& P, float2* A, float* x, int es, int nch, cudaStream_t st) {
    const NSBox& full = P.boxes_full;
    prof_bytes("ns_slab_line3", nch * 2 * box_bytes(P, full));
    prof_bytes("ns_slab_c2r", nch * (box_bytes(P, full) + 4.0 * P.N));
    const BoxMap bx = box_map(P, full);
    const int s3 = P.P1 * P.dims[1];
    const int ng = acc_groups(P, A), nl = full.nk1 * full.nk2;
    const L3StoreC so{A, P.SP, P.P1, s3, bx};
    const float2* K = P.comp.as<float2>() + (ng > 1 ? A - P.acc.as<float2>() : 0);
    const long long gs = (long long)P.nch * P.SP;
    // the register pass holds 24 or 40 values a thread at 96 and 160 points, too many beside their sums' loads: the
    // accumulators are summed ahead of it there (64 x 64 x 160: 29 -> 12 us, 96 cubed 14 -> 10; one launch more
    // elsewhere gains nothing)
    if (ng > 1 && (P.dims[2] == 96 || P.dims[2] == 160)) {
        sum_groups(P, A, K, ng, nch, st);
        line3<true>(P, L3LoadC{A, P.SP, P.P1, s3, bx}, so, nl, nch, st, "ns_slab_line3");
    } else if (ng == 4)
        line3<true>(P, L3LoadSum<4>{{A, K, gs}, P.SP, P.P1, s3, bx}, so, nl, nch, st, "ns_slab_line3");
    else if (ng == 2)
        line3<true>(P, L3LoadSum<2>{{A, K, gs}, P.SP, P.P1, s3, bx}, so, nl, nch, st, "ns_slab_line3");
    else
        line3<true>(P, L3LoadC{A, P.SP, P.P1, s3, bx}, so, nl, nch, st, "ns_slab_line3");
    SlabArgs a = slab_args(P, full_chunk(P), nch);
    a.spec_chstride = P.SP;
    a.spec = A;
    set_volumes(a, x, ZMap{}, es);
    a.scale = 1.0f / (float)P.N;
    launch_slab<1>(P, a, st, "ns_slab_c2r");
}

// The analysis axis-3 pass of a chunk: X times each mask, inverse FFT along
// axis 3, into Y (the plan's work spectra).
void slab_mask_pass(NSPlan& P, const float2* X, const Chunk& ck, bool synth_masks, int nch, cudaStream_t st) {
    prof_bytes("ns_slab_mask_axis3", nch * (1.5 * segs_bytes(P, ck) + items_bytes(P, ck)));
    const int sy = synth_masks ? 1 : 0;
    const long long xc = P.SP, yc = ych_stride(P);
    MaskTiles tl;
    const bool any = axis3_len(P.dims[2]);
    choose_mask_tiles(P, ck, any ? axis3_lines(P.dims[2]) : mix_axis3_lines(P), nch, tl);
    int tok = prof_begin("ns_slab_mask_axis3", st);
    (any ? launch_axis3_mask : launch_mix_mask)(P, X, ck, tl, sy, P.work.as<float2>(), nch, xc, yc, st);
    prof_end(tok, st);
}

// The synthesis axis-3 pass of a chunk from Y into acc + ch SP,
// Kahan-compensated through comp + ch SP.
void slab_accum_pass(NSPlan& P, const Chunk& ck, bool analysis_masks, float2* acc, float2* comp, int nch,
                     cudaStream_t st) {
    // Y once per item, the group table (4 B a bin), the accumulator and its compensation in and out
    prof_bytes("ns_slab_accum_axis3", nch * (items_bytes(P, ck) + 4.5 * segs_bytes(P, ck)));
    const int sy = analysis_masks ? 0 : 1;
    const long long yc = ych_stride(P);
    int tok = prof_begin("ns_slab_accum_axis3", st);
    (axis3_len(P.dims[2]) ? launch_axis3_accum : launch_mix_accum)(P, ck, box_map(P, union_box(ck)), sy,
                                                                   P.work.as<float2>(), acc, comp, nch,
                                                                   acc_groups(P, acc), yc, st);
    prof_end(tok, st);
}

// Analysis of items [i0, i0 + nz) (one chunk) from X (+ ch SP) into volumes at
// vol + vz.off(z) (+ ch, element stride es).
void slab_analyze_items(NSPlan& P, const float2* X, float* vol, ZMap vz, int es, int i0, int nz, bool synth_masks,
                        int nch, cudaStream_t st) {
    const Chunk ck = make_chunk(P, i0, nz, synth_masks);
    slab_mask_pass(P, X, ck, synth_masks, nch, st);
    prof_bytes("ns_slab_c2r", nch * (items_bytes(P, ck) + nz * 4.0 * P.N));
    SlabArgs a = slab_args(P, ck, nch);
    a.spec_chstride = ych_stride(P);
    a.spec = P.work.as<float2>();
    a.spec_zstride = P.SP;
    set_volumes(a, vol, vz, es);
    a.scale = 1.0f / (float)P.N;
    launch_slab<1>(P, a, st, "ns_slab_c2r");
}

// Synthesis staging of items [i0, i0 + nz) (within one chunk) read from
// vol + vz.off(z) (+ ch): slab R2C into work slots slot0.. (+ ch slots SP).
void slab_stage_items(NSPlan& P, const float* vol, ZMap vz, int es, int i0, int nz, int slot0, int nch,
                      cudaStream_t st) {
    const Chunk ck = make_chunk(P, i0, nz, false);
    prof_bytes("ns_slab_r2c", nch * (nz * 4.0 * P.N + items_bytes(P, ck)));
    SlabArgs a = slab_args(P, ck, nch);
    a.spec_chstride = ych_stride(P);
    a.spec = P.work.as<float2>() + (long long)slot0 * P.SP;
    a.spec_zstride = P.SP;
    set_volumes(a, vol, vz, es);
    launch_slab<0>(P, a, st, "ns_slab_r2c");
}

// The accumulation of items [i0, i0 + nz) (one chunk) from work slots 0.. into
// acc + ch SP.
void slab_accum_items(NSPlan& P, int i0, int nz, bool analysis_masks, float2* acc, float2* comp, int nch,
                      cudaStream_t st) {
    slab_accum_pass(P, make_chunk(P, i0, nz, !analysis_masks), analysis_masks, acc, comp, nch, st);
}

// Synthesis of items [i0, i0 + nz) (one chunk) read from vol + vz.off(z)
// (+ ch) into acc + ch SP.
void slab_synth_items(NSPlan& P, const float* vol, ZMap vz, int es, int i0, int nz, bool analysis_masks,
                      float2* acc, float2* comp, int nch, cudaStream_t st) {
    slab_stage_items(P, vol, vz, es, i0, nz, 0, nch, st);
    slab_accum_items(P, i0, nz, analysis_masks, acc, comp, nch, st);
}

// The denoiser on items [i0, i0 + nz) (one chunk; real data): the analysis
// axis-3 pass into Y, the shrink slab pass in place, the synthesis
// accumulation.
void slab_denoise_items(NSPlan& P, const float2* X, int i0, int nz, const float* tau, float2* acc, float2* comp,
                        cudaStream_t st) {
    const Chunk ck = make_chunk(P, i0, nz, false);
    slab_mask_pass(P, X, ck, false, 1, st);
    prof_bytes("ns_slab_shrink", 2 * items_bytes(P, ck));
    SlabArgs a = slab_args(P, ck, 1);
    a.spec = P.work.as<float2>();
    a.spec_zstride = P.SP;
    a.scale = 1.0f / (float)P.N;
    a.tau = tau;
    launch_slab<2>(P, a, st, "ns_slab_shrink");
    slab_accum_items(P, i0, nz, false, acc, comp, 1, st);
}

}  // namespace

void ns_set_concurrent(bool on) { t_concurrent = on; }

bool ns_slab_supported(int n1, int n2, int n3) {
    if (!reg_fft_supported(n3)) return false;
    // one CTA a slab where the slab fits its shared memory (two CTAs an SM up to 112 KB, one above),
    // else two-CTA clusters
    return (slab_len(n1) && slab_len(n2) && slab_smem(n1, n2) <= kSlabSmemOneCta) || slab_cluster_resident(n1, n2);
}

// Support box of a table on the rfft grid (h1, n2, n3), k1 fastest.
NSBox ns_table_box(const std::vector<double>& g, int h1, int n2, int n3) {
    int m1 = -1, m2 = -1;
    for (int k3 = 0; k3 < n3; ++k3)
        for (int k2 = 0; k2 < n2; ++k2) {
            const double* row = g.data() + (size_t)h1 * (k2 + (size_t)n2 * k3);
            for (int k1 = 0; k1 < h1; ++k1)
                if (row[k1] != 0.0) {
                    m1 = std::max(m1, k1);
                    m2 = std::max(m2, std::min(k2, n2 - k2));
                }
        }
    return ns_make_box(m1 + 1, m2, n2);
}

// Work slots of the slab pipeline: the group when one was chosen, else as many
// spectra as 256 MB hold (complex volumes: two channels each), so that a chunk
// spans the mask groups of small boxes; no more than the transforms' own
// chunks use.
void ns_slab_slots(NSPlan& P) {
    P.slots = P.group;
    if (P.chosen) return;
    const long long fit = (256LL << 20) / (8 * P.SP * P.nch);
    P.slots = (int)std::max<long long>(P.group, std::min<long long>({fit, (long long)kChunkItems, (long long)P.S}));
    int used = P.group;
    for (int i0 = 0, i1; i0 < P.S; i0 = i1) {
        i1 = chunk_end(P, i0);
        used = std::max(used, i1 - i0);
    }
    P.slots = used;
}

NSBox ns_make_box(int nk1, int b2, int n2) {
    NSBox b;
    b.nk1 = std::max(nk1, 1);
    if (b2 < 0) b2 = 0;
    if (2 * b2 + 1 >= n2) {
        b.nk2 = n2;
        b.b2 = n2;
    } else {
        b.nk2 = 2 * b2 + 1;
        b.b2 = b2;
    }
    return b;
}

void ns_slab_acc_clear(NSPlan& P, float2* acc, float2* comp, cudaStream_t st) {
    const int ng = acc_groups(P, acc);
    for (int g = 0; g < ng; ++g) {
        const long long o = (long long)g * P.nch * P.SP;
        cuda_check(cudaMemsetAsync(acc + o, 0, sizeof(float2) * P.SP, st), "cudaMemsetAsync(acc)");
        cuda_check(cudaMemsetAsync(comp + o, 0, sizeof(float2) * P.SP, st), "cudaMemsetAsync(comp)");
    }
}

void ns_slab_clear(NSPlan& P, cudaStream_t st) {
    const size_t bytes = sizeof(float2) * P.SP * P.nch * P.ngrp;
    cuda_check(cudaMemsetAsync(P.acc.p, 0, bytes, st), "cudaMemsetAsync(acc)");
    cuda_check(cudaMemsetAsync(P.comp.p, 0, bytes, st), "cudaMemsetAsync(comp)");
}

void ns_merge_groups(NSPlan& P, int ch, float2* A, float2* C, cudaStream_t st) {
    const long long blocks = std::min<long long>((P.SP + 255) / 256, 8LL * P.sms);
    const float2 *a = P.acc.as<float2>() + ch * P.SP, *k = P.comp.as<float2>() + ch * P.SP;
    const long long gs = (long long)P.nch * P.SP;
    if (P.ngrp == 4)
        merge_groups_kernel<4><<<(unsigned)blocks, 256, 0, st>>>(GroupSum<4>{a, k, gs}, A, C, P.SP);
    else
        merge_groups_kernel<2><<<(unsigned)blocks, 256, 0, st>>>(GroupSum<2>{a, k, gs}, A, C, P.SP);
    cuda_check(cudaGetLastError(), "merge_groups_kernel launch");
}

// Accumulators of the synthesis.  A CTA of the axis-3 pass walks the terms of
// its lines one after the other, and a small spectrum has too few lines to
// fill the GPU (66 CTAs at 64^3, 3.5 us a term): its mask groups then go to
// several accumulators, summed by the inverse FFT's first pass.
int ns_slab_groups(const NSPlan& P) {
    const long long lines = (long long)P.h1 * P.dims[1];
    return lines <= 3000 ? 4 : (lines <= 10000 ? 2 : 1);
}

void ns_use_mixed(NSPlan& P) {
    if (!ns_mix_slab_supported(P))
        throw ArgError("the mixed-radix slab pipeline does not support size " + std::to_string(P.dims[0]) + "x" +
                       std::to_string(P.dims[1]) + "x" + std::to_string(P.dims[2]));
    P.slab = P.mixed = true;
    ns_alloc_scratch(P);
}

void ns_use_slabs(NSPlan& P) {
    if (!ns_slab_supported(P.dims[0], P.dims[1], P.dims[2]))
        throw ArgError("the slab pipeline does not support size " + std::to_string(P.dims[0]) + "x" +
                       std::to_string(P.dims[1]) + "x" + std::to_string(P.dims[2]));
    P.slab = true;
    P.mixed = false;
    ns_alloc_scratch(P);
}

void ns_slab_rfft3(NSPlan& P, const float* x, int es, float2* X, cudaStream_t st) { slab_rfft3(P, x, es, X, 1, st); }

void ns_slab_irfft3(NSPlan& P, float2* A, float* x, int es, cudaStream_t st) { slab_irfft3(P, A, x, es, 1, st); }

// Whole transforms, both channels of complex data in every launch.
void ns_slab_analyze(NSPlan& P, const void* x, void* c, cudaStream_t st, bool synth_masks) {
    const int nch = P.nch;
    float2* X = P.X.as<float2>();
    slab_rfft3(P, static_cast<const float*>(x), nch, X, nch, st);
    for (int i0 = 0, i1; i0 < P.S; i0 = i1) {
        i1 = chunk_end(P, i0);
        slab_analyze_items(P, X, static_cast<float*>(c), ns_subband_map(P, i0, nch), nch, i0, i1 - i0, synth_masks,
                           nch, st);
    }
}

void ns_slab_synthesize(NSPlan& P, const void* c, void* x, cudaStream_t st, bool analysis_masks) {
    const int nch = P.nch;
    float2* A = P.acc.as<float2>();
    float2* K = P.comp.as<float2>();
    ns_slab_clear(P, st);
    for (int i0 = 0, i1; i0 < P.S; i0 = i1) {
        i1 = chunk_end(P, i0);
        slab_synth_items(P, static_cast<const float*>(c), ns_subband_map(P, i0, nch), nch, i0, i1 - i0,
                         analysis_masks, A, K, nch, st);
    }
    slab_irfft3(P, A, static_cast<float*>(x), nch, nch, st);
}

int ns_slab_chunk_end(const NSPlan& P, int i0) { return chunk_end(P, i0); }

void ns_slab_analyze_items(NSPlan& P, const float2* X, float* vol, ZMap vz, int es, int i0, int nz, bool synth_masks,
                           cudaStream_t st) {
    slab_analyze_items(P, X, vol, vz, es, i0, nz, synth_masks, 1, st);
}

void ns_slab_synth_items(NSPlan& P, const float* vol, ZMap vz, int es, int i0, int nz, bool analysis_masks,
                         float2* acc, float2* comp, cudaStream_t st) {
    slab_synth_items(P, vol, vz, es, i0, nz, analysis_masks, acc, comp, 1, st);
}

void ns_slab_denoise_items(NSPlan& P, const float2* X, int i0, int nz, const float* tau, float2* acc, float2* comp,
                           cudaStream_t st) {
    slab_denoise_items(P, X, i0, nz, tau, acc, comp, st);
}

void ns_slab_stage_items(NSPlan& P, const float* vol, ZMap vz, int es, int i0, int nz, int slot0, int nch,
                         cudaStream_t st) {
    slab_stage_items(P, vol, vz, es, i0, nz, slot0, nch, st);
}

void ns_slab_accum_items(NSPlan& P, int i0, int nz, bool analysis_masks, float2* acc, float2* comp, int nch,
                         cudaStream_t st) {
    slab_accum_items(P, i0, nz, analysis_masks, acc, comp, nch, st);
}

}  // namespace sfl
