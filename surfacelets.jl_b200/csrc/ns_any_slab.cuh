// The slab passes of the NSSurfacelet for every pair of lengths in
// SFL_ANY_LENGTHS.  The row phase (axis 2) and the column phase (axis 1) of a
// slab are functions of their own per length, picked by two switches that are
// uniform over the grid, so that one kernel a kind covers every n1 x n2 (a
// kernel a pair would be 6724); between them the slab lies in shared memory at
// the run-time pitch P1.  They take shared memory by offset, so that its
// address space stays known across the call.  Box columns move by bulk copies, and the exchange of a line runs through
// its own slots with warp barriers only, as in ns_slab_pass.cuh.
#pragma once

#include <algorithm>

#include "anyfft.cuh"
#include "plan.h"
#include "prof.h"
#include "slab_core.cuh"
#include "tma.cuh"

namespace sfl {

namespace {

// ── phases ───────────────────────────────────────────────────────────────────

// FFT along axis 2 of the rows k1 < rows, in place; on the inverse the columns
// outside the box read as zero.
extern __shared__ __align__(16) float2 any_sm[];

template <int N, bool INV>
__device__ __noinline__ void any_rows(int so, int P1, int rows, int b2, int k2hi, int to) {
    float2* const S = any_sm + so;
    const float2* const tw2 = any_sm + to;
    using L = AnyLine<N>;
    constexpr int N1 = L::N1, N2 = L::N2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, step = (blockDim.x >> 5) * L::LPW;
    const int s = lane / N2, p = lane - s * N2;
#pragma unroll 1
    for (int l0 = warp * L::LPW; l0 < rows; l0 += step) {
        const auto [k1, valid] = any_lane_line<N>(l0, s, rows);
        float2* row = S + k1;
        float2 v[N1], u[L::E];
        if (!INV || b2 >= N) {
#pragma unroll
            for (int r = 0; r < N1; ++r) v[r] = row[P1 * (p + N2 * r)];
        } else {
#pragma unroll
            for (int r = 0; r < N1; ++r) {
                const int k2 = p + N2 * r;
                v[r] = k2 <= b2 || k2 >= k2hi ? row[P1 * k2] : make_float2(0.f, 0.f);
            }
        }
        any_warp_fft<N, INV>(v, p, valid, tw2, row, P1, u);
#pragma unroll
        for (int j = 0; j < L::M; ++j)
            if (valid && L::has(p, j)) {
#pragma unroll
                for (int k = 0; k < N2; ++k) row[P1 * ((p + N2 * j) + N1 * k)] = u[j * N2 + k];
            }
    }
}

// The column of zeros, behind the slab's spare column.
__device__ __forceinline__ const float2* any_zero(int so, int P1, int n2) { return any_sm + so + P1 * (n2 + 1); }

// The next unit's box columns, requested as soon as their pairs are transformed.
struct AnyNext {
    const float2* src;   // null: no next unit
    int b2, k2hi;
    uint32_t bytes;
    int bar;             // offset of the mbarrier
};

// The full spectrum of (column ca) + i (column cb) at v[r] = Z[p + N2 r]: rows
// k1 >= nk1 are zero; cb is a column of zeros where an odd count's last column
// has no partner.
template <int N>
__device__ __forceinline__ void any_load_pair(float2 (&v)[AnyLine<N>::N1], const float2* ca, const float2* cb, int nk1,
                                              int p) {
    auto fold = [&](float2& z, int i, int k, float2 A, float2 B) {
        if (k == 0 || 2 * k == N) {
            A.y = 0.f;
            B.y = 0.f;
        }
        z = 2 * i <= N ? make_float2(A.x - B.y, A.y + B.x) : make_float2(A.x + B.y, B.x - A.y);
    };
    if (nk1 == N / 2 + 1) {
#pragma unroll
        for (int r = 0; r < AnyLine<N>::N1; ++r) {
            const int i = p + AnyLine<N>::N2 * r, k = 2 * i <= N ? i : N - i;
            fold(v[r], i, k, ca[k], cb[k]);
        }
    } else {
#pragma unroll
        for (int r = 0; r < AnyLine<N>::N1; ++r) {
            const int i = p + AnyLine<N>::N2 * r, k = 2 * i <= N ? i : N - i;
            const bool in = k < nk1;
            fold(v[r], i, k, in ? ca[k] : make_float2(0.f, 0.f), in ? cb[k] : make_float2(0.f, 0.f));
        }
    }
}

// A transformed line into its slots in natural order.
template <int N>
__device__ __forceinline__ void any_put_natural(const float2 (&u)[AnyLine<N>::E], float2* slots, int p, bool valid) {
    using L = AnyLine<N>;
#pragma unroll
    for (int j = 0; j < L::M; ++j)
        if (valid && L::has(p, j)) {
#pragma unroll
            for (int k = 0; k < L::N2; ++k) slots[(p + L::N2 * j) + L::N1 * k] = u[j * L::N2 + k];
        }
}

// C2R along axis 1 of columns 2l and 2l + 1 as one complex line, scaled, into
// two columns of a real slab (element stride ES); rows k1 >= nk1 are zero, and
// the missing column of an odd count.
template <int N, int ES>
__device__ __noinline__ void any_cols_inv(int so, int P1, int nk1, int n2, int to, float* out, float scale,
                                          const AnyNext& nx) {
    float2* const S = any_sm + so;
    const float2* const tw2 = any_sm + to;
    using L = AnyLine<N>;
    constexpr int N1 = L::N1, N2 = L::N2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, step = (blockDim.x >> 5) * L::LPW;
    const int s = lane / N2, p = lane - s * N2, npairs = (n2 + 1) / 2;
#pragma unroll 1
    for (int l0 = warp * L::LPW; l0 < npairs; l0 += step) {
        const auto [l, valid] = any_lane_pair<N>(l0, s, npairs);
        const bool two = valid && 2 * l + 1 < n2;
        float2* ca = S + P1 * (2 * l);
        float2 v[N1], u[L::E];
        any_load_pair<N>(v, ca, two ? ca + P1 : any_zero(so, P1, n2), nk1, p);
        any_warp_fft<N, true>(v, p, valid, tw2, ca, 1, u);
        if (nx.src) {
            fence_proxy_async();
            __syncwarp();
            const int k2 = 2 * l0 + lane;
            if (lane < 2 * L::LPW && k2 < n2 && (k2 <= nx.b2 || k2 >= nx.k2hi)) {
                uint64_t* bar = reinterpret_cast<uint64_t*>(any_sm + nx.bar);
                mbar_expect_tx(bar, nx.bytes);
                bulk_load(S + P1 * k2, nx.src + P1 * k2, nx.bytes, bar);
            }
        }
        float* oa = out + (2 * l * N + p) * ES;
        float* ob = oa + N * ES;
#pragma unroll
        for (int j = 0; j < L::M; ++j)
            if (valid && L::has(p, j)) {
#pragma unroll
                for (int k = 0; k < N2; ++k) {
                    const float2 x = c_scale(u[j * N2 + k], scale);
                    oa[(N2 * j + N1 * k) * ES] = x.x;
                    if (two) ob[(N2 * j + N1 * k) * ES] = x.y;
                }
            }
    }
}

// Z of a column pair in its slots, natural order -> the two half spectra, bins
// k < nk1, in the columns.  Warp-uniform.
template <int N>
__device__ __forceinline__ void any_unpack(float2* ca, int P1, int nk1, int p, bool valid, bool two) {
    constexpr int N2 = AnyLine<N>::N2, Q = (N / 2 + 1 + N2 - 1) / N2;
    float2 ha[Q], hb[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int k = p + N2 * q;
        ha[q] = hb[q] = make_float2(0.f, 0.f);
        if (valid && k < nk1) {
            const float2 zk = ca[k], zn = ca[k == 0 ? 0 : N - k];
            ha[q] = half_spec_a(zk, zn);
            hb[q] = half_spec_b(zk, zn);
        }
    }
    __syncwarp();
    if (valid) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int k = p + N2 * q;
            if (k < nk1) {
                ca[k] = ha[q];
                if (two) ca[P1 + k] = hb[q];
            }
        }
    }
}

// R2C along axis 1 of columns 2l and 2l + 1 of a real slab (element stride ES).
template <int N, int ES>
__device__ __noinline__ void any_cols_fwd(int so, int P1, int nk1, int n2, int to, const float* in) {
    float2* const S = any_sm + so;
    const float2* const tw2 = any_sm + to;
    using L = AnyLine<N>;
    constexpr int N1 = L::N1, N2 = L::N2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, step = (blockDim.x >> 5) * L::LPW;
    const int s = lane / N2, p = lane - s * N2, npairs = (n2 + 1) / 2;
#pragma unroll 1
    for (int l0 = warp * L::LPW; l0 < npairs; l0 += step) {
        const auto [l, valid] = any_lane_pair<N>(l0, s, npairs);
        const bool two = valid && 2 * l + 1 < n2;
        const float* ia = in + (2 * l * N + p) * ES;
        const float* ib = ia + (two ? N * ES : 0);
        float2 v[N1], u[L::E];
#pragma unroll
        for (int r = 0; r < N1; ++r) v[r] = make_float2(ia[N2 * r * ES], ib[N2 * r * ES]);
        if (!two) {   // an odd count's last column has no partner
#pragma unroll
            for (int r = 0; r < N1; ++r) v[r].y = 0.f;
        }
        float2* ca = S + P1 * (2 * l);
        any_warp_fft<N, false>(v, p, valid, tw2, ca, 1, u);
        any_put_natural<N>(u, ca, p, valid);
        __syncwarp();
        any_unpack<N>(ca, P1, nk1, p, valid, two);
    }
}

// The denoiser's column phase: C2R of a pair, scaled by 1/N and thresholded,
// c' = sign(c) max(|c| - tau, 0), and its R2C back into the columns.
template <int N>
__device__ __noinline__ void any_cols_shrink(int so, int P1, int nk1, int n2, int to, float scale, float tau) {
    float2* const S = any_sm + so;
    const float2* const tw2 = any_sm + to;
    using L = AnyLine<N>;
    constexpr int N1 = L::N1, N2 = L::N2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, step = (blockDim.x >> 5) * L::LPW;
    const int s = lane / N2, p = lane - s * N2, npairs = (n2 + 1) / 2;
#pragma unroll 1
    for (int l0 = warp * L::LPW; l0 < npairs; l0 += step) {
        const auto [l, valid] = any_lane_pair<N>(l0, s, npairs);
        const bool two = valid && 2 * l + 1 < n2;
        float2* ca = S + P1 * (2 * l);
        float2 v[N1], u[L::E];
        any_load_pair<N>(v, ca, two ? ca + P1 : any_zero(so, P1, n2), nk1, p);
        any_warp_fft<N, true>(v, p, valid, tw2, ca, 1, u);
#pragma unroll
        for (int j = 0; j < L::M; ++j)
            if (valid && L::has(p, j)) {
#pragma unroll
                for (int k = 0; k < N2; ++k) {
                    const float2 x = c_scale(u[j * N2 + k], scale);
                    ca[(p + N2 * j) + N1 * k] = make_float2(copysignf(fmaxf(fabsf(x.x) - tau, 0.f), x.x),
                                                            two ? copysignf(fmaxf(fabsf(x.y) - tau, 0.f), x.y) : 0.f);
                }
            }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < N1; ++r) v[r] = ca[p + N2 * r];
        any_warp_fft<N, false>(v, p, valid, tw2, ca, 1, u);
        any_put_natural<N>(u, ca, p, valid);
        __syncwarp();
        any_unpack<N>(ca, P1, nk1, p, valid, two);
    }
}

// ── box columns by bulk copies (16-byte aligned: P1 is even) ────────────────

__device__ __forceinline__ uint32_t any_col_bytes(int nk1) { return (uint32_t)(((nk1 + 1) & ~1) * sizeof(float2)); }

__device__ __forceinline__ void any_bulk_load(float2* S, const float2* src, int P1, int n2, const ChunkItem& it,
                                              uint64_t* bar, uint32_t& phase, int* status) {
    const uint32_t bytes = any_col_bytes(it.nk1);
    fence_proxy_async();   // this thread's earlier accesses to S ahead of the copies' writes
    if (threadIdx.x == 0) mbar_arrive_expect_tx(bar, bytes * (uint32_t)it.nk2);
    __syncthreads();
    for (int j = threadIdx.x; j < it.nk2; j += blockDim.x) {
        const int k2 = j <= it.b2 ? j : j + (n2 - it.nk2);
        bulk_load(S + P1 * k2, src + P1 * k2, bytes, bar);
    }
    mbar_wait_bounded(bar, phase, status);
    phase ^= 1;
}

__device__ __forceinline__ void any_bulk_store(float2* dst, const float2* S, int P1, int n2, const ChunkItem& it) {
    fence_proxy_async();   // this thread's writes of S visible to the copies
    __syncthreads();
    bool mine = false;
    for (int j = threadIdx.x; j < it.nk2; j += blockDim.x) {
        const int k2 = j <= it.b2 ? j : j + (n2 - it.nk2);
        bulk_store(dst + P1 * k2, S + P1 * k2, any_col_bytes(it.nk1));
        mine = true;
    }
    if (mine) {
        bulk_commit();
        bulk_wait_read();   // S is rewritten by the next unit
    }
    __syncthreads();
}

// ── the passes ───────────────────────────────────────────────────────────────

constexpr int kAnyThreads = 512;

// Values before the slab: both axes' twiddles, rounded up so that the slab
// starts 16-byte aligned.
__host__ __device__ inline int any_tw_values(int n1, int n2) { return (n1 + n2 + 1) & ~1; }
// The slab, a spare column (the exchange slots of an odd count's last column)
// and a column of zeros, then the mbarrier.
inline size_t any_smem(int n1, int n2, int P1) {
    return sizeof(float2) * ((size_t)any_tw_values(n1, n2) + (size_t)P1 * (n2 + 2)) + 16;
}

// KIND: 0 the forward slab pass, 1 the inverse, 2 the denoiser's shrink pass.
// One CTA a unit (channel, item, n3), striding over the launch's units.
template <int KIND, int ES>
__global__ void __launch_bounds__(kAnyThreads, 2)
    ns_any_slab_kernel(const __grid_constant__ SlabArgs a, const int n1, const int n2) {
    const int P1 = a.P1, so = any_tw_values(n1, n2), bo = so + P1 * (n2 + 2);
    float2* S = any_sm + so;
    uint64_t* bar = reinterpret_cast<uint64_t*>(any_sm + bo);
    uint32_t phase = 0;
    switch (n1) {
#define SFL_ANY_CASE(N_) \
    case N_: any_load_twiddles<N_>(any_sm, a.twa); break;
        SFL_ANY_LENGTHS(SFL_ANY_CASE)
#undef SFL_ANY_CASE
    }
    switch (n2) {
#define SFL_ANY_CASE(N_) \
    case N_: any_load_twiddles<N_>(any_sm + n1, a.twb); break;
        SFL_ANY_LENGTHS(SFL_ANY_CASE)
#undef SFL_ANY_CASE
    }
    for (int i = threadIdx.x; i < P1; i += blockDim.x) S[P1 * (n2 + 1) + i] = make_float2(0.f, 0.f);
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
    }
    __syncthreads();
    const long long SL = (long long)P1 * n2, PLANE = (long long)n1 * n2;
    const int per = a.ck.nz * a.n3;
    auto slab_of = [&](int unit) {
        const int ch = unit / per, ur = unit - ch * per;
        const int z = ur / a.n3, s3 = ur - z * a.n3;
        return a.spec + ch * a.spec_chstride + z * a.spec_zstride + s3 * SL;
    };
    bool requested = false;   // the unit's box was requested during the previous unit's column phase
#pragma unroll 1
    for (int u = blockIdx.x; u < a.units; u += gridDim.x) {
        const int ch = u / per, ur = u - ch * per;
        const int z = ur / a.n3, s3 = ur - z * a.n3;
        const ChunkItem& it = a.ck.item[z];
        const int nk1 = it.nk1, b2 = it.b2, k2hi = n2 - (it.nk2 - b2 - 1);
        float* vol = a.vol + ch + a.vol_off(z) + (long long)s3 * PLANE * ES;
        if constexpr (KIND == 0) {
            switch (n1) {
#define SFL_ANY_CASE(N_) \
    case N_: any_cols_fwd<N_, ES>(so, P1, nk1, n2, 0, vol); break;
                SFL_ANY_LENGTHS(SFL_ANY_CASE)
#undef SFL_ANY_CASE
            }
            __syncthreads();
            switch (n2) {
#define SFL_ANY_CASE(N_) \
    case N_: any_rows<N_, false>(so, P1, nk1, b2, k2hi, n1); break;
                SFL_ANY_LENGTHS(SFL_ANY_CASE)
#undef SFL_ANY_CASE
            }
            __syncthreads();
            any_bulk_store(slab_of(u), S, P1, n2, it);   // ends with the barrier before S is reused
        } else {
            if (!requested) {
                any_bulk_load(S, slab_of(u), P1, n2, it, bar, phase, a.status);
            } else {
                mbar_wait_bounded(bar, phase, a.status);
                phase ^= 1;
            }
            switch (n2) {
#define SFL_ANY_CASE(N_) \
    case N_: any_rows<N_, true>(so, P1, nk1, b2, k2hi, n1); break;
                SFL_ANY_LENGTHS(SFL_ANY_CASE)
#undef SFL_ANY_CASE
            }
            if constexpr (KIND == 2) {
                __syncthreads();
                const float tau = a.tau[it.s - 1];
                switch (n1) {
#define SFL_ANY_CASE(N_) \
    case N_: any_cols_shrink<N_>(so, P1, nk1, n2, 0, a.scale, tau); break;
                    SFL_ANY_LENGTHS(SFL_ANY_CASE)
#undef SFL_ANY_CASE
                }
                __syncthreads();
                switch (n2) {
#define SFL_ANY_CASE(N_) \
    case N_: any_rows<N_, false>(so, P1, nk1, b2, k2hi, n1); break;
                    SFL_ANY_LENGTHS(SFL_ANY_CASE)
#undef SFL_ANY_CASE
                }
                __syncthreads();
                any_bulk_store(slab_of(u), S, P1, n2, it);
                continue;
            }
            // the next unit of this CTA (ns_slab_inv_kernel says how the barrier's phase closes)
            const int un = u + gridDim.x;
            requested = un < a.units;
            const ChunkItem& itn = a.ck.item[requested ? un % per / a.n3 : z];
            const AnyNext nx{requested ? slab_of(un) : nullptr, itn.b2, n2 - (itn.nk2 - itn.b2 - 1),
                             any_col_bytes(itn.nk1), bo};
            if (requested) fence_proxy_async();   // the row phase's accesses ahead of the next unit's copies
            __syncthreads();
            switch (n1) {
#define SFL_ANY_CASE(N_) \
    case N_: any_cols_inv<N_, ES>(so, P1, nk1, n2, 0, vol, a.scale, nx); break;
                SFL_ANY_LENGTHS(SFL_ANY_CASE)
#undef SFL_ANY_CASE
            }
            __syncthreads();   // the slab buffer is reused by the next unit
            // every copy of the next unit is issued and announced: the one arrival of the barrier's phase
            if (requested && threadIdx.x == 0) mbar_arrive(bar);
        }
    }
}

// Lines a warp holds.
inline int any_lpw(int n) {
    switch (n) {
#define SFL_ANY_CASE(N_) \
    case N_: return AnyLine<N_>::LPW;
        SFL_ANY_LENGTHS(SFL_ANY_CASE)
#undef SFL_ANY_CASE
    }
    return 1;
}

// Warps a CTA: as many CTAs as shared memory holds share the SM's 32 warps of
// 64 registers a thread, each then with the fewest warps that need no more
// rounds over its rows and column pairs.
inline int any_warps(int n1, int n2, size_t smem) {
    const int fit = std::max(1, (int)(kSlabSmemOneCta / (smem + 1024)));
    const int tr = (n1 / 2 + any_lpw(n2)) / any_lpw(n2), tc = ((n2 + 1) / 2 + any_lpw(n1) - 1) / any_lpw(n1);
    const int most = std::min(kAnyThreads / 32, std::max(4, 32 / fit));
    auto rounds = [&](int w) { return (tr + w - 1) / w + (tc + w - 1) / w; };
    int w = most;
    while (w > 4 && rounds(w - 1) == rounds(most)) --w;
    return w;
}

template <int KIND, int ES>
void launch_any_slab_es(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag) {
    auto kern = ns_any_slab_kernel<KIND, ES>;
    static DeviceOnce once;
    allow_smem(once, kern, kSlabSmemOneCta);
    const int n1 = P.dims[0], n2 = P.dims[1];
    const size_t smem = any_smem(n1, n2, a.P1);
    const int threads = 32 * any_warps(n1, n2, smem);
    // the last geometry's answer: the query costs as much as a launch
    thread_local int resident = 0, asked_threads = -1;
    thread_local size_t asked_smem = 0;
    if (asked_threads != threads || asked_smem != smem) {
        cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, threads, smem),
                   "cudaOccupancyMaxActiveBlocksPerMultiprocessor(any slab)");
        asked_threads = threads;
        asked_smem = smem;
    }
    const int grid = std::max(1, std::min(a.units, std::max(resident, 1) * P.sms));
    int tok = prof_begin(tag, st);
    kern<<<grid, threads, smem, st>>>(a, n1, n2);
    prof_end(tok, st);
    cuda_check(cudaGetLastError(), "ns_any_slab_kernel launch");
}

template <int KIND>
void launch_any_slab(const NSPlan& P, const SlabArgs& a, cudaStream_t st, const char* tag) {
    if (KIND == 2 || a.es == 1)
        launch_any_slab_es<KIND, 1>(P, a, st, tag);
    else
        launch_any_slab_es<KIND, 2>(P, a, st, tag);
}

}  // namespace

}  // namespace sfl
