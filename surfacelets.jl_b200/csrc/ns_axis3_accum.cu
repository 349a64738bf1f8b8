// The synthesis axis-3 pass of the slab pipeline, lengths of SFL_ANY_LENGTHS.
#include "anyfft.cuh"
#include "ns_axis3.cuh"
#include "prof.h"

namespace sfl {

namespace {

// Resident CTAs an SM the register budget aims at: three (85 registers a
// thread) where a thread holds at most ten values and its sums lie in shared
// memory, two (128) else.  The pass waits on L2 and gains from more warps (120 x
// 100 x 90 synthesis 300 -> 257 us), and loses far more to spilled registers
// (three CTAs at 128 points: 489 -> 534 us).
template <int N, bool STEPS>
constexpr int accum_minb() {
    return AnyLine<N>::N1 <= 10 && AnyLine<N>::E > (STEPS ? 6 : 8) && AnyLine<N>::E <= 10 ? 3 : 2;
}
// Lengths whose sums go to shared memory: where their register form spills, and
// with compensations from seven values on (at 64 points, sums and compensations
// in registers at two CTAs an SM: 224 x 224 x 64 synthesis 630 us; in shared
// memory at three: 546 us).
template <int N, bool STEPS>
constexpr bool accum_sums_shared() { return AnyLine<N>::E > (STEPS ? 6 : 8); }
template <int N, bool STEPS>
constexpr size_t accum_smem() {
    constexpr size_t value = STEPS ? 2 * sizeof(float2) : sizeof(float2) + sizeof(float);
    return AnyGeom<N>::SMEM + (accum_sums_shared<N, STEPS>() ? value * AnyLine<N>::E * AnyGeom<N>::THREADS : 0);
}

// Synthesis line pass over a chunk's segments: per segment FFT_3 of every item
// times its mask, summed in float32 over the segment's terms, then added into
// the accumulator with one Kahan step against the compensation grid comp: the
// compensation carries across segments and launches, so the sum over the mask
// groups of the whole synthesis is compensated
// (src/transforms/ns_surfacelet.jl:292, 355, 383 accumulate every subband into
// one spectrum).  STEPS, the mixed pipeline: the terms of a segment are added
// with compensation too, one Kahan step each, and the group factor multiplies
// their sum (holding it beside the sums and compensations would leave one CTA an
// SM at 120 points).  The compile-time slabs' sizes add them plainly.  CTAs take line blocks of the union box (un) and skip the
// segments whose box none of their lines meets.  With several accumulators
// (P.ngrp, blockIdx.z) mask group g goes to accumulator g mod ngrp.
//
// A wedge plane constant along axis 3 commutes with the axis-3 FFT, so the
// items that share plane b (and the group factor) are combined first,
// sum_p wa_p(k1, k2) Y_pq, and transformed once: with nbq > 0 the segment is
// nbq plane-b wedges q times whole rows p (item t = p nbq + q); otherwise
// every item is its own term.  Terms are added in q order.
template <int N, bool STEPS>
__global__ void __launch_bounds__(256, accum_minb<N, STEPS>())
    ns_slab_accum_kernel(const float2* __restrict__ Y, long long ystride, int P1, int s3, BoxMap un,
                         const __grid_constant__ NSMaskTables tb, const __grid_constant__ Chunk ck, int synth,
                         float2* acc, float2* comp, const float2* __restrict__ tw, long long ychs, long long achs,
                         long long agrp) {
    using Ge = AnyGeom<N>;
    constexpr int N1 = Ge::N1, N2 = Ge::N2, LP = Ge::LP, E = Ge::E;
    extern __shared__ float2 a3_sm[];
    float2* const tws = a3_sm;
    float2* const xch = a3_sm + N;
    any_load_twiddles<N>(tws, tw);
    __syncthreads();
    Y += blockIdx.y * ychs;   // channel
    acc += blockIdx.y * achs + blockIdx.z * agrp;
    comp += blockIdx.y * achs + blockIdx.z * agrp;
    const int tid = threadIdx.x;
    const int lp = tid % LP, p = tid / LP;
    const int l = blockIdx.x * LP + lp;
    const bool inl = l < un.nk1 * un.nk2;
    int k1 = 0, k2 = 0;
    if (inl) un.k12(l, k1, k2);
    float2* xl = xch + lp * Ge::XLINE;
    // a segment's sums: in registers, or (lengths whose registers would spill) in shared memory after the
    // exchange rows, value q of thread t at [q * THREADS + t]
    constexpr bool kSumsShared = accum_sums_shared<N, STEPS>();
    float2 sr[kSumsShared ? 1 : E];
    float2* ss = xch + LP * Ge::XLINE + tid;
    auto sum = [&](int q) -> float2& {
        if constexpr (kSumsShared)
            return ss[q * Ge::THREADS];
        else
            return sr[q];
    };
    // their compensations (STEPS), behind them
    float2 cr[kSumsShared || !STEPS ? 1 : E];
    auto rest = [&](int q) -> float2& {
        if constexpr (kSumsShared)
            return ss[(E + q) * Ge::THREADS];
        else
            return cr[q];
    };
    // the line's group factors, in registers or beside the sums
    float gr[kSumsShared || STEPS ? 1 : E];
    float* gs = reinterpret_cast<float*>(xch + LP * Ge::XLINE + (kSumsShared ? E * Ge::THREADS : 0)) + tid;
    auto gf = [&](int q) -> float& {
        if constexpr (kSumsShared)
            return gs[q * Ge::THREADS];
        else
            return gr[q];
    };
    const int si = tb.h1 * tb.n2;
    const bool wedge_masks = !(synth && !tb.tight);
    const float2* yl = Y + k1 + P1 * k2;
#pragma unroll 1
    for (int sgi = 0; sgi < ck.nseg; ++sgi) {
        const ChunkSeg& sg = ck.seg[sgi];
        if (sg.ord % (int)gridDim.z != (int)blockIdx.z) continue;   // another accumulator's
        const bool valid = inl && k1 < sg.nk1 && (k2 <= sg.b2 || k2 >= tb.n2 - sg.b2);
        // (the barrier also keeps the previous segment's exchange reads ahead of this one's writes)
        if (ck.nseg > 1 && !__syncthreads_or(valid)) continue;
#pragma unroll
        for (int q = 0; q < E; ++q) {
            sum(q) = make_float2(0.f, 0.f);
            if constexpr (STEPS) rest(q) = make_float2(0.f, 0.f);
        }
        // the group factor of the line (group table, bandpass table or the lowpass factors), once for all items
        if constexpr (!STEPS) {
            const NSMaskLine m0 = chunk_mask_line(tb, sg, ck.item[sg.i0], k1, k2, synth != 0);
#pragma unroll
            for (int j = 0; j < Ge::M; ++j)
#pragma unroll
                for (int k = 0; k < N2; ++k) {
                    const int k3 = Ge::has(p, j) ? (p + N2 * j) + N1 * k : 0;
                    gf(j * N2 + k) = m0.low ? m0.lowc * m0.lowv[k3] : m0.m[k3 * si];
                }
        }
        const int nbq = sg.nbq;
        const int rows = nbq > 0 ? sg.nz / nbq : 1;
        const int nterms = nbq > 0 ? nbq : sg.nz;
#pragma unroll 1
        for (int t = 0; t < nterms; ++t) {
            const ChunkItem& it0 = ck.item[sg.i0 + t];
            const bool before = wedge_masks && !sg.low && it0.wa_hi != 2;   // plane a applied before the FFT
            // the term: sum_p wa_p Y_pq (one item with weight 1 when plane a varies along the line; x 1 is
            // exact).
            const int nt = before ? rows : 1;
            auto weight = [&](int z) {
                const ChunkItem& it = ck.item[z];
                return before ? __ldg(tb.planes + it.wa_off + (it.wa_lo == 0 ? k1 : k2) + it.wa_dlo * k2) : 1.f;
            };
            // opaque to the compiler, which would otherwise keep the lines' offsets of all loops in registers and
            // spill others for them (176 bytes a thread at 128 points)
            int s3t = s3, wst = 1;
            asm volatile("" : "+r"(s3t), "+r"(wst));
            float2 v[N1], yb[N1];
            const int z0 = sg.i0 + t;
            float wz = weight(z0);
            {
                const float2* yz = yl + z0 * ystride;
#pragma unroll
                for (int r = 0; r < N1; ++r) yb[r] = valid ? yz[(p + N2 * r) * s3t] : make_float2(0.f, 0.f);
            }
#pragma unroll 1
            for (int pp = 0; pp < nt; ++pp) {
                const float az = wz;
#pragma unroll
                for (int r = 0; r < N1; ++r) v[r] = pp == 0 ? c_scale(yb[r], az) : c_fma(yb[r], az, v[r]);
                if (pp + 1 < nt) {
                    const int z = z0 + (pp + 1) * nbq;
                    const float2* yz = yl + z * ystride;
                    wz = weight(z);
#pragma unroll
                    for (int r = 0; r < N1; ++r)
                        yb[r] = valid ? yz[(p + N2 * r) * s3t] : make_float2(0.f, 0.f);
                }
            }
            float2 u[E];
            if (t > 0) __syncthreads();   // the exchange rows were read for the previous term
            any_block_fft<N, false>(v, p, xl, tws, u);
            // the term's first item carries plane b and the group factor
            const NSMaskLine mk = chunk_mask_line(tb, sg, it0, k1, k2, synth != 0);
            const bool wedges = !(mk.low || mk.plain);
            const int was = mk.was * wst, wbs = mk.wbs * wst;
#pragma unroll
            for (int j = 0; j < Ge::M; ++j)
#pragma unroll
                for (int k = 0; k < N2; ++k) {
                    const int k3 = Ge::has(p, j) ? (p + N2 * j) + N1 * k : 0;
                    float2& tsum = sum(j * N2 + k);
                    if constexpr (STEPS) {
                        const float m = !wedges ? 1.f : (before ? mk.wb[k3 * wbs] : mk.wa[k3 * was] * mk.wb[k3 * wbs]);
                        kahan_fma(tsum, rest(j * N2 + k), u[j * N2 + k], m);
                    } else {
                        const float g = gf(j * N2 + k);
                        const float m = !wedges ? g : (before ? g * mk.wb[k3 * wbs] : g * (mk.wa[k3 * was] * mk.wb[k3 * wbs]));
                        tsum = make_float2(fmaf(u[j * N2 + k].x, m, tsum.x), fmaf(u[j * N2 + k].y, m, tsum.y));
                    }
                }
        }
        if (valid) {
            float2* a = acc + k1 + P1 * k2;
            float2* ca = comp + k1 + P1 * k2;
            // a few bins at a time: all of them at once spill
            if constexpr (STEPS) {
                // the loads of a few bins ahead of their stores, which the compiler takes to alias
                constexpr int B = accum_minb<N, STEPS>() == 3 ? 2 : 4;
#pragma unroll(kSumsShared ? 1 : E)
                for (int q0 = 0; q0 < E; q0 += B) {
                    float2 sv[B], cv[B];
                    float g[B];
#pragma unroll
                    for (int b = 0; b < B; ++b) {
                        const int j = (q0 + b) / N2, k3 = (p + N2 * j) + N1 * (q0 + b - j * N2);
                        if (q0 + b < E && Ge::has(p, j)) {
                            sv[b] = a[k3 * s3];
                            cv[b] = ca[k3 * s3];
                            g[b] = chunk_group_factor(tb, sg, k1, k2, k3, synth != 0);
                        }
                    }
#pragma unroll
                    for (int b = 0; b < B; ++b) {
                        const int j = (q0 + b) / N2, k3 = (p + N2 * j) + N1 * (q0 + b - j * N2);
                        if (q0 + b < E && Ge::has(p, j)) {
                            cv[b] = c_fma(rest(q0 + b), g[b], cv[b]);
                            kahan_fma(sv[b], cv[b], sum(q0 + b), g[b]);
                            a[k3 * s3] = sv[b];
                            ca[k3 * s3] = cv[b];
                        }
                    }
                }
                continue;
            }
#pragma unroll(kSumsShared ? 1 : Ge::M)
            for (int j = 0; j < Ge::M; ++j)
                if (Ge::has(p, j)) {
#pragma unroll(kSumsShared ? 4 : N2)
                    for (int k = 0; k < N2; ++k) {
                        const int o = ((p + N2 * j) + N1 * k) * s3;
                        float2 sv = a[o], cv = ca[o];
                        kahan_add(sv, cv, sum(j * N2 + k));
                        a[o] = sv;
                        ca[o] = cv;
                    }
                }
        }
    }
}

template <int N, bool STEPS>
void launch_n(const NSPlan& P, const Chunk& ck, const BoxMap& un, int synth, const float2* Y, float2* acc, float2* comp,
              int nch, int ngrp, long long ychs, cudaStream_t st) {
    using Ge = AnyGeom<N>;
    static DeviceOnce once;
    allow_smem(once, ns_slab_accum_kernel<N, STEPS>, accum_smem<N, STEPS>());
    const dim3 grid((un.nk1 * un.nk2 + Ge::LP - 1) / Ge::LP, nch, ngrp);
    ns_slab_accum_kernel<N, STEPS><<<grid, Ge::THREADS, accum_smem<N, STEPS>(), st>>>(
        Y, P.SP, P.P1, P.P1 * P.dims[1], un, P.tb, ck, synth, acc, comp, P.ffts.at(N)->sh.tw, ychs, P.SP,
        (long long)P.nch * P.SP);
    cuda_check(cudaGetLastError(), "ns_slab_accum_kernel launch");
}

}  // namespace

void launch_axis3_accum(const NSPlan& P, const Chunk& ck, const BoxMap& un, int synth, const float2* Y, float2* acc,
                        float2* comp, int nch, int ngrp, long long ychs, cudaStream_t st) {
    if (P.mixed) {
        switch (P.dims[2]) {
#define SFL_AXIS3_CASE(N_) \
    case N_: launch_n<N_, true>(P, ck, un, synth, Y, acc, comp, nch, ngrp, ychs, st); return;
            SFL_ANY_LENGTHS(SFL_AXIS3_CASE)
#undef SFL_AXIS3_CASE
        }
    } else {
        switch (P.dims[2]) {   // the axis-3 lengths of the compile-time slabs (reg_fft_supported)
#define SFL_AXIS3_CASE(N_) \
    case N_: launch_n<N_, false>(P, ck, un, synth, Y, acc, comp, nch, ngrp, ychs, st); return;
            SFL_AXIS3_CASE(16) SFL_AXIS3_CASE(32) SFL_AXIS3_CASE(64) SFL_AXIS3_CASE(96) SFL_AXIS3_CASE(128)
            SFL_AXIS3_CASE(160) SFL_AXIS3_CASE(256)
#undef SFL_AXIS3_CASE
        }
    }
    throw ArgError("no axis-3 pass of this length");
}

}  // namespace sfl
