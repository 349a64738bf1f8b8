// The slab passes of the NSSurfacelet (see ns_slab.cu): one CTA holds an
// axis-3 slab of a spectrum in shared memory and runs both transforms of its
// plane.  Each kind of pass is instantiated in a translation unit of its own.
#pragma once

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "plan.h"
#include "prof.h"
#include "regfft.cuh"
#include "slab_core.cuh"
#include "tma.cuh"

namespace sfl {

namespace {

// ── slab passes ─────────────────────────────────────────────────────────────

// ── box rows between HBM and shared memory by bulk copies ──────────────────
//
// One cp.async.bulk a box column: the rows k1 < nk1 rounded up to an even
// count (16-byte multiples; the slab pitch P1 = 2 mod 4 is even, so every
// column starts 16-byte aligned).  The extra bin of an odd nk1 lies outside
// the box and is read by no one.  Loads complete on an mbarrier whose wait
// is bounded; stores are waited on for their shared-memory reads only.

// The slab pass's mbarrier, after the slab in shared memory.
template <int NA, int NB>
__device__ __forceinline__ uint64_t* slab_bar(float2* sm) {
    constexpr int P1 = slab_pitch_c(NA / 2 + 1);
    return reinterpret_cast<uint64_t*>(sm + NA + NB + P1 * NB);
}

__device__ __forceinline__ void slab_bar_init(uint64_t* bar) {
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
    }
    __syncthreads();
}

template <int NB, int P1>
__device__ __forceinline__ void slab_bulk_load(float2* S, const float2* src, int nk1, int nk2, int b2,
                                               uint64_t* bar, uint32_t& phase, int* status) {
    const uint32_t bytes = (uint32_t)(((nk1 + 1) & ~1) * sizeof(float2));
    fence_proxy_async();   // this thread's earlier accesses to S ahead of the copies' writes
    if (threadIdx.x == 0) mbar_arrive_expect_tx(bar, bytes * (uint32_t)nk2);
    __syncthreads();
    if ((int)threadIdx.x < nk2) {
        const int j = threadIdx.x;
        const int k2 = j <= b2 ? j : j + (NB - nk2);
        bulk_load(S + P1 * k2, src + P1 * k2, bytes, bar);
    }
    mbar_wait_bounded(bar, phase, status);
    phase ^= 1;
}

template <int NB, int P1>
__device__ __forceinline__ void slab_bulk_store(float2* dst, const float2* S, int nk1, int nk2, int b2) {
    const uint32_t bytes = (uint32_t)(((nk1 + 1) & ~1) * sizeof(float2));
    fence_proxy_async();   // this thread's writes of S visible to the copies
    __syncthreads();
    if ((int)threadIdx.x < nk2) {
        const int j = threadIdx.x;
        const int k2 = j <= b2 ? j : j + (NB - nk2);
        bulk_store(dst + P1 * k2, S + P1 * k2, bytes);
        bulk_commit();
        bulk_wait_read();   // S is rewritten by the next unit
    }
    __syncthreads();
}

// Analysis slab pass (inverse): spectra -> real volumes (element stride ES).
// The exchange slots of a column pair are the pair's two columns read as one
// run of 2 P1 >= NA values.
// A unit whose box spans every row and column (nk1 = NA/2 + 1, nk2 = NB; the
// finest scale) takes a body of its own, in which the box predicates fold away.
template <int NA, int NB, int ES, int MINB>
__global__ void __launch_bounds__(kSlabThreads, MINB) ns_slab_inv_kernel(const __grid_constant__ SlabArgs a) {
    using LA = SlabLine<NA>;
    using LB = SlabLine<NB>;
    constexpr int P1 = slab_pitch_c(NA / 2 + 1);
    constexpr int SL = P1 * NB;
    constexpr long long PLANE = (long long)NA * NB;
    extern __shared__ float2 sm[];
    float2* twA = sm;
    float2* twB = sm + NA;
    float2* S = sm + NA + NB;
    load_slab_twiddles<NA>(twA, a.twa);
    load_slab_twiddles<NB>(twB, a.twb);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t* bar = slab_bar<NA, NB>(sm);
    uint32_t phase = 0;
    slab_bar_init(bar);
    const int per = a.ck.nz * a.n3;
    auto slab_src = [&](int unit) {
        const int ch = unit / per, ur = unit - ch * per;
        const int z = ur / a.n3, s3 = ur - z * a.n3;
        return a.spec + ch * a.spec_chstride + z * a.spec_zstride + (long long)s3 * SL;
    };
    bool requested = false;   // the unit's box was requested during the previous unit's C2R
    auto run = [&](auto full, const int u) {
        constexpr bool FULL = decltype(full)::value;
        const int ch = u / per, ur = u - ch * per;
        const int z = ur / a.n3, s3 = ur - z * a.n3;
        const int nk1 = FULL ? NA / 2 + 1 : a.ck.item[z].nk1;
        const int nk2 = FULL ? NB : a.ck.item[z].nk2, b2 = FULL ? NB : a.ck.item[z].b2;
        const int k2hi = NB - (nk2 - b2 - 1);   // first negative-frequency column in the box
        float* out = a.vol + ch + a.vol_off(z) + (long long)s3 * PLANE * ES;
        // 1. the box of the slab into shared memory
        if (!requested) {
            slab_bulk_load<NB, P1>(S, slab_src(u), nk1, nk2, b2, bar, phase, a.status);
        } else {
            mbar_wait_bounded(bar, phase, a.status);
            phase ^= 1;
        }
        // the next unit of this CTA, whose box columns are requested as soon as their pair is transformed
        const int un = u + gridDim.x;
        requested = un < a.units;
        const float2* srcn = requested ? slab_src(un) : nullptr;
        // its box
        const int zn = requested ? un % per / a.n3 : z;
        const int nb2 = a.ck.item[zn].b2, nk2hi = NB - (a.ck.item[zn].nk2 - nb2 - 1);
        const uint32_t colbytes = (uint32_t)(((a.ck.item[zn].nk1 + 1) & ~1) * sizeof(float2));
        // 2. inverse FFT along axis 2 of the rows k1 < nk1; columns outside the box are zero
        {
            const int p = lane & (LB::N2 - 1), s = lane / LB::N2;
            for (int base = 0; base < nk1; base += LB::LPR) {
                if (base + warp * LB::LPW >= nk1) continue;   // warp-uniform
                const int k1 = base + warp * LB::LPW + s;
                const bool valid = k1 < nk1;
                float2* row = S + (valid ? k1 : 0);
                float2 v[LB::N1];
#pragma unroll
                for (int r = 0; r < LB::N1; ++r) {
                    const int k2 = p + LB::N2 * r;
                    const bool in = valid && (k2 <= b2 || k2 >= k2hi);
                    v[r] = in ? row[P1 * k2] : make_float2(0.f, 0.f);
                }
                warp_line_fft<NB, true, P1>(v, p, valid, twB, row);
                if (valid) {
#pragma unroll
                    for (int j = 0; j < LB::M; ++j)
#pragma unroll
                        for (int k = 0; k < LB::N2; ++k) row[P1 * ((p + LB::N2 * j) + LB::N1 * k)] = v[j * LB::N2 + k];
                }
            }
        }
        // the row phase's accesses to every column ahead of the next unit's copies into them
        if (requested) fence_proxy_async();
        __syncthreads();
        // 3. C2R along axis 1, columns 2l and 2l+1 as one complex line; rows k1 >= nk1 are zero
        {
            const int p = lane & (LA::N2 - 1), s = pair_subline<NA>(lane / LA::N2);
            constexpr int npairs = NB / 2;
            for (int base = 0; base < npairs; base += LA::LPR) {
                if (base + warp * LA::LPW >= npairs) continue;   // warp-uniform
                const int l = base + warp * LA::LPW + s;
                const bool valid = l < npairs;
                float2* ca = S + P1 * (2 * (valid ? l : 0));
                float2* cb = ca + P1;
                float2 v[LA::N1];
#pragma unroll
                for (int r = 0; r < LA::N1; ++r) {
                    const int i = p + LA::N2 * r;
                    const int k = 2 * i <= NA ? i : NA - i;
                    float2 A = make_float2(0.f, 0.f), B = make_float2(0.f, 0.f);
                    if (valid && k < nk1) {
                        A = ca[k];
                        B = cb[k];
                    }
                    if (k == 0 || 2 * k == NA) {
                        A.y = 0.f;
                        B.y = 0.f;
                    }
                    v[r] = 2 * i <= NA ? make_float2(A.x - B.y, A.y + B.x) : make_float2(A.x + B.y, B.x - A.y);
                }
                warp_line_fft<NA, true, 1>(v, p, valid, twA, ca);
                if (requested) {
                    // the warp's columns are free (the exchange ended with a warp barrier): lane c of the
                    // first 2 LPW requests column 2 (base + warp LPW) + c of the next unit, if in its box
                    fence_proxy_async();
                    __syncwarp();
                    const int k2 = 2 * (base + warp * LA::LPW) + lane;
                    if (lane < 2 * LA::LPW && k2 < NB && (k2 <= nb2 || k2 >= nk2hi)) {
                        mbar_expect_tx(bar, colbytes);
                        bulk_load(S + P1 * k2, srcn + P1 * k2, colbytes, bar);
                    }
                }
                if (valid) {
                    float* oa = out + (long long)(2 * l) * NA * ES;
                    float* ob = oa + (long long)NA * ES;
                    const float sc = a.scale;
#pragma unroll
                    for (int j = 0; j < LA::M; ++j)
#pragma unroll
                        for (int k = 0; k < LA::N2; ++k) {
                            const int i1 = (p + LA::N2 * j) + LA::N1 * k;
                            const float2 w = c_scale(v[j * LA::N2 + k], sc);
                            oa[i1 * ES] = w.x;
                            ob[i1 * ES] = w.y;
                        }
                }
            }
        }
        __syncthreads();   // the slab buffer is reused by the next unit
        // every copy of the next unit is issued and announced: the one arrival of the barrier's phase
        if (requested && threadIdx.x == 0) mbar_arrive(bar);
    };
    for (int u = blockIdx.x; u < a.units; u += gridDim.x) {
        const ChunkItem& it = a.ck.item[u % per / a.n3];
        if (it.nk1 == NA / 2 + 1 && it.nk2 == NB)
            run(std::true_type{}, u);
        else
            run(std::false_type{}, u);
    }
}

// Synthesis / rfft slab pass (forward): real volumes (element stride ES) ->
// spectra (the box rows).
template <int NA, int NB, int ES, int MINB>
__global__ void __launch_bounds__(kSlabThreads, MINB) ns_slab_fwd_kernel(const __grid_constant__ SlabArgs a) {
    using LA = SlabLine<NA>;
    using LB = SlabLine<NB>;
    constexpr int P1 = slab_pitch_c(NA / 2 + 1);
    constexpr int SL = P1 * NB;
    constexpr long long PLANE = (long long)NA * NB;
    constexpr int H1 = NA / 2 + 1;
    constexpr int QA = (H1 + LA::N2 - 1) / LA::N2;   // output bins a lane unpacks
    extern __shared__ float2 sm[];
    float2* twA = sm;
    float2* twB = sm + NA;
    float2* S = sm + NA + NB;
    load_slab_twiddles<NA>(twA, a.twa);
    load_slab_twiddles<NB>(twB, a.twb);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = a.ck.nz * a.n3;
    auto run = [&](auto full, const int u) {   // full: the box spans every row and column, as in the inverse pass
        constexpr bool FULL = decltype(full)::value;
        const int ch = u / per, ur = u - ch * per;
        const int z = ur / a.n3, s3 = ur - z * a.n3;
        const int nk1 = FULL ? NA / 2 + 1 : a.ck.item[z].nk1;
        const int nk2 = FULL ? NB : a.ck.item[z].nk2, b2 = FULL ? NB : a.ck.item[z].b2;
        // 1. R2C along axis 1 of columns 2l, 2l+1 (as the real and imaginary parts of one line)
        {
            const int p = lane & (LA::N2 - 1), s = pair_subline<NA>(lane / LA::N2);
            constexpr int npairs = NB / 2;
            const float* in = a.vol + ch + a.vol_off(z) + (long long)s3 * PLANE * ES;
            for (int base = 0; base < npairs; base += LA::LPR) {
                if (base + warp * LA::LPW >= npairs) continue;   // warp-uniform
                const int l = base + warp * LA::LPW + s;
                const bool valid = l < npairs;
                const float* ia = in + (long long)(2 * (valid ? l : 0)) * NA * ES;
                const float* ib = ia + (long long)NA * ES;
                float2 v[LA::N1];
#pragma unroll
                for (int r = 0; r < LA::N1; ++r) {
                    const int i = p + LA::N2 * r;
                    v[r] = valid ? make_float2(ia[i * ES], ib[i * ES]) : make_float2(0.f, 0.f);
                }
                float2* ca = S + P1 * (2 * (valid ? l : 0));
                float2* cb = ca + P1;
                warp_line_fft<NA, false, 1>(v, p, valid, twA, ca);
                // Z in natural order through the pair's slots, then the two half spectra
                if (valid) {
#pragma unroll
                    for (int j = 0; j < LA::M; ++j)
#pragma unroll
                        for (int k = 0; k < LA::N2; ++k) ca[(p + LA::N2 * j) + LA::N1 * k] = v[j * LA::N2 + k];
                }
                __syncwarp();
                float2 ha[QA], hb[QA];
#pragma unroll
                for (int q = 0; q < QA; ++q) {
                    const int k = p + LA::N2 * q;
                    ha[q] = hb[q] = make_float2(0.f, 0.f);
                    if (valid && k < nk1) {
                        const float2 zk = ca[k];
                        const float2 zn = ca[k == 0 ? 0 : NA - k];
                        ha[q] = half_spec_a(zk, zn);
                        hb[q] = half_spec_b(zk, zn);
                    }
                }
                __syncwarp();
                if (valid) {
#pragma unroll
                    for (int q = 0; q < QA; ++q) {
                        const int k = p + LA::N2 * q;
                        if (k < nk1) {
                            ca[k] = ha[q];
                            cb[k] = hb[q];
                        }
                    }
                }
            }
        }
        __syncthreads();
        // 2. forward FFT along axis 2 of the rows k1 < nk1
        {
            const int p = lane & (LB::N2 - 1), s = lane / LB::N2;
            for (int base = 0; base < nk1; base += LB::LPR) {
                if (base + warp * LB::LPW >= nk1) continue;   // warp-uniform
                const int k1 = base + warp * LB::LPW + s;
                const bool valid = k1 < nk1;
                float2* row = S + (valid ? k1 : 0);
                float2 v[LB::N1];
#pragma unroll
                for (int r = 0; r < LB::N1; ++r) v[r] = valid ? row[P1 * (p + LB::N2 * r)] : make_float2(0.f, 0.f);
                warp_line_fft<NB, false, P1>(v, p, valid, twB, row);
                if (valid) {
#pragma unroll
                    for (int j = 0; j < LB::M; ++j)
#pragma unroll
                        for (int k = 0; k < LB::N2; ++k) row[P1 * ((p + LB::N2 * j) + LB::N1 * k)] = v[j * LB::N2 + k];
                }
            }
        }
        __syncthreads();
        // 3. the box of the slab out to the spectrum
        float2* dst = a.spec + ch * a.spec_chstride + z * a.spec_zstride + (long long)s3 * SL;
        slab_bulk_store<NB, P1>(dst, S, nk1, nk2, b2);   // ends with the barrier before S is reused
    };
    for (int u = blockIdx.x; u < a.units; u += gridDim.x) {
        const ChunkItem& it = a.ck.item[u % per / a.n3];
        if (it.nk1 == NA / 2 + 1 && it.nk2 == NB)
            run(std::true_type{}, u);
        else
            run(std::false_type{}, u);
    }
}

// The denoiser's slab pass (real data): per slab of Y_s, the analysis half
// (inverse FFT along axis 2, C2R along axis 1, 1/N) gives the subband's slab
// in registers; it is soft-thresholded, c' = sign(c) max(|c| - tau_s, 0), and
// the synthesis half (R2C along axis 1, FFT along axis 2 of the box rows)
// writes the box back into the same slab of Y_s.  The subband itself never
// leaves the chip.  Same arithmetic, in the same order, as analyze ->
// threshold -> synthesize through the two slab passes.
template <int NA, int NB, int MINB>
__global__ void __launch_bounds__(kSlabThreads, MINB) ns_slab_shrink_kernel(const __grid_constant__ SlabArgs a) {
    using LA = SlabLine<NA>;
    using LB = SlabLine<NB>;
    constexpr int P1 = slab_pitch_c(NA / 2 + 1);
    constexpr int SL = P1 * NB;
    constexpr int H1 = NA / 2 + 1;
    constexpr int QA = (H1 + LA::N2 - 1) / LA::N2;
    extern __shared__ float2 sm[];
    float2* twA = sm;
    float2* twB = sm + NA;
    float2* S = sm + NA + NB;
    load_slab_twiddles<NA>(twA, a.twa);
    load_slab_twiddles<NB>(twB, a.twb);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t* bar = slab_bar<NA, NB>(sm);
    uint32_t phase = 0;
    slab_bar_init(bar);
    for (int u = blockIdx.x; u < a.units; u += gridDim.x) {
        const int per = a.ck.nz * a.n3;
        const int ch = u / per, ur = u - ch * per;
        const int z = ur / a.n3, s3 = ur - z * a.n3;
        const int nk1 = a.ck.item[z].nk1, nk2 = a.ck.item[z].nk2, b2 = a.ck.item[z].b2;
        const int k2hi = NB - (nk2 - b2 - 1);
        float2* slab = a.spec + ch * a.spec_chstride + z * a.spec_zstride + (long long)s3 * SL;
        const float tau = a.tau[a.ck.item[z].s - 1];
        slab_bulk_load<NB, P1>(S, slab, nk1, nk2, b2, bar, phase, a.status);
        {   // inverse FFT along axis 2 of the box rows
            const int p = lane & (LB::N2 - 1), s = lane / LB::N2;
            for (int base = 0; base < nk1; base += LB::LPR) {
                if (base + warp * LB::LPW >= nk1) continue;   // warp-uniform
                const int k1 = base + warp * LB::LPW + s;
                const bool valid = k1 < nk1;
                float2* row = S + (valid ? k1 : 0);
                float2 v[LB::N1];
#pragma unroll
                for (int r = 0; r < LB::N1; ++r) {
                    const int k2 = p + LB::N2 * r;
                    const bool in = valid && (k2 <= b2 || k2 >= k2hi);
                    v[r] = in ? row[P1 * k2] : make_float2(0.f, 0.f);
                }
                warp_line_fft<NB, true, P1>(v, p, valid, twB, row);
                if (valid) {
#pragma unroll
                    for (int j = 0; j < LB::M; ++j)
#pragma unroll
                        for (int k = 0; k < LB::N2; ++k) row[P1 * ((p + LB::N2 * j) + LB::N1 * k)] = v[j * LB::N2 + k];
                }
            }
        }
        __syncthreads();
        {   // per column pair: C2R, threshold, R2C
            const int p = lane & (LA::N2 - 1), s = pair_subline<NA>(lane / LA::N2);
            constexpr int npairs = NB / 2;
            for (int base = 0; base < npairs; base += LA::LPR) {
                if (base + warp * LA::LPW >= npairs) continue;   // warp-uniform
                const int l = base + warp * LA::LPW + s;
                const bool valid = l < npairs;
                float2* ca = S + P1 * (2 * (valid ? l : 0));
                float2* cb = ca + P1;
                float2 v[LA::N1];
#pragma unroll
                for (int r = 0; r < LA::N1; ++r) {
                    const int i = p + LA::N2 * r;
                    const int k = 2 * i <= NA ? i : NA - i;
                    float2 A = make_float2(0.f, 0.f), B = make_float2(0.f, 0.f);
                    if (valid && k < nk1) {
                        A = ca[k];
                        B = cb[k];
                    }
                    if (k == 0 || 2 * k == NA) {
                        A.y = 0.f;
                        B.y = 0.f;
                    }
                    v[r] = 2 * i <= NA ? make_float2(A.x - B.y, A.y + B.x) : make_float2(A.x + B.y, B.x - A.y);
                }
                warp_line_fft<NA, true, 1>(v, p, valid, twA, ca);
                // the two subband columns, thresholded, in natural order through the pair's slots
                if (valid) {
#pragma unroll
                    for (int j = 0; j < LA::M; ++j)
#pragma unroll
                        for (int k = 0; k < LA::N2; ++k) {
                            const float2 c = v[j * LA::N2 + k];
                            const float xa = c.x * a.scale, xb = c.y * a.scale;
                            ca[(p + LA::N2 * j) + LA::N1 * k] =
                                make_float2(copysignf(fmaxf(fabsf(xa) - tau, 0.f), xa),
                                            copysignf(fmaxf(fabsf(xb) - tau, 0.f), xb));
                        }
                }
                __syncwarp();
#pragma unroll
                for (int r = 0; r < LA::N1; ++r) v[r] = valid ? ca[p + LA::N2 * r] : make_float2(0.f, 0.f);
                warp_line_fft<NA, false, 1>(v, p, valid, twA, ca);
                if (valid) {
#pragma unroll
                    for (int j = 0; j < LA::M; ++j)
#pragma unroll
                        for (int k = 0; k < LA::N2; ++k) ca[(p + LA::N2 * j) + LA::N1 * k] = v[j * LA::N2 + k];
                }
                __syncwarp();
                float2 ha[QA], hb[QA];
#pragma unroll
                for (int q = 0; q < QA; ++q) {
                    const int k = p + LA::N2 * q;
                    ha[q] = hb[q] = make_float2(0.f, 0.f);
                    if (valid && k < nk1) {
                        const float2 zk = ca[k];
                        const float2 zn = ca[k == 0 ? 0 : NA - k];
                        ha[q] = half_spec_a(zk, zn);
                        hb[q] = half_spec_b(zk, zn);
                    }
                }
                __syncwarp();
                if (valid) {
#pragma unroll
                    for (int q = 0; q < QA; ++q) {
                        const int k = p + LA::N2 * q;
                        if (k < nk1) {
                            ca[k] = ha[q];
                            cb[k] = hb[q];
                        }
                    }
                }
            }
        }
        __syncthreads();
        {   // forward FFT along axis 2 of the box rows
            const int p = lane & (LB::N2 - 1), s = lane / LB::N2;
            for (int base = 0; base < nk1; base += LB::LPR) {
                if (base + warp * LB::LPW >= nk1) continue;   // warp-uniform
                const int k1 = base + warp * LB::LPW + s;
                const bool valid = k1 < nk1;
                float2* row = S + (valid ? k1 : 0);
                float2 v[LB::N1];
#pragma unroll
                for (int r = 0; r < LB::N1; ++r) v[r] = valid ? row[P1 * (p + LB::N2 * r)] : make_float2(0.f, 0.f);
                warp_line_fft<NB, false, P1>(v, p, valid, twB, row);
                if (valid) {
#pragma unroll
                    for (int j = 0; j < LB::M; ++j)
#pragma unroll
                        for (int k = 0; k < LB::N2; ++k) row[P1 * ((p + LB::N2 * j) + LB::N1 * k)] = v[j * LB::N2 + k];
                }
            }
        }
        __syncthreads();
        slab_bulk_store<NB, P1>(slab, S, nk1, nk2, b2);   // ends with the barrier before S is reused
    }
}

// ── launch tables ────────────────────────────────────────────────────────────

template <int N>
constexpr int slab_minb() {
    return LinePlan<N>::N1 <= 16 ? 2 : 1;
}

// One CTA a unit up to the resident capacity; CTAs stride over the rest.
// KIND: 0 the forward slab pass, 1 the inverse, 2 the denoiser's shrink pass.
template <int KIND, int NA, int NB, int ES>
void launch_slab_es(const SlabArgs& a, int sms, size_t smem, cudaStream_t st, const char* tag) {
    constexpr int MINB = (slab_minb<NA>() == 2 && slab_minb<NB>() == 2) ? 2 : 1;
    auto kern = KIND == 1 ? ns_slab_inv_kernel<NA, NB, ES, MINB>
                          : (KIND == 0 ? ns_slab_fwd_kernel<NA, NB, ES, MINB> : ns_slab_shrink_kernel<NA, NB, MINB>);
    static DeviceOnce once;
    static std::atomic<int> resident{1};   // the same on every device of sm_100a
    once_a_device(once, [&] {
        cuda_check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                   "cudaFuncSetAttribute(slab)");
        int r = 0;
        cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, kern, kSlabThreads, smem),
                   "cudaOccupancyMaxActiveBlocksPerMultiprocessor(slab)");
        resident = std::max(r, 1);
    });
    const int grid = std::max(1, std::min(a.units, resident * sms));
    int tok = prof_begin(tag, st);
    kern<<<grid, kSlabThreads, smem, st>>>(a);
    prof_end(tok, st);
    cuda_check(cudaGetLastError(), "slab kernel launch");
}

template <int KIND, int NA, int NB>
void launch_slab_nn(const SlabArgs& a, int sms, size_t smem, cudaStream_t st, const char* tag) {
    if (a.P1 != slab_pitch_c(NA / 2 + 1)) throw ArgError("slab pitch mismatch");
    if (KIND == 2 || a.es == 1)
        launch_slab_es<KIND, NA, NB, 1>(a, sms, smem, st, tag);
    else
        launch_slab_es<KIND, NA, NB, 2>(a, sms, smem, st, tag);
}

template <int KIND, int NA>
bool launch_slab_n(int nb, const SlabArgs& a, int sms, size_t smem, cudaStream_t st, const char* tag) {
    switch (nb) {
        case 64: launch_slab_nn<KIND, NA, 64>(a, sms, smem, st, tag); return true;
        case 96: launch_slab_nn<KIND, NA, 96>(a, sms, smem, st, tag); return true;
        case 128: launch_slab_nn<KIND, NA, 128>(a, sms, smem, st, tag); return true;
        case 160: launch_slab_nn<KIND, NA, 160>(a, sms, smem, st, tag); return true;
        case 256:
            if constexpr (NA != 256) {   // 256 x 256 slabs run on clusters (ns_slab_cluster.cu)
                launch_slab_nn<KIND, NA, 256>(a, sms, smem, st, tag);
                return true;
            }
            return false;
    }
    return false;
}

template <int KIND>
void launch_slab_kind(int na, int nb, const SlabArgs& a, int sms, size_t smem, cudaStream_t st, const char* tag) {
    bool ok = false;
    switch (na) {
        case 64: ok = launch_slab_n<KIND, 64>(nb, a, sms, smem, st, tag); break;
        case 96: ok = launch_slab_n<KIND, 96>(nb, a, sms, smem, st, tag); break;
        case 128: ok = launch_slab_n<KIND, 128>(nb, a, sms, smem, st, tag); break;
        case 160: ok = launch_slab_n<KIND, 160>(nb, a, sms, smem, st, tag); break;
        case 256: ok = launch_slab_n<KIND, 256>(nb, a, sms, smem, st, tag); break;
    }
    if (!ok) throw ArgError("no slab kernel for this size");
}

}  // namespace

}  // namespace sfl
