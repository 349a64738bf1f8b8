// The analysis axis-3 pass of the slab pipeline, lengths of SFL_ANY_LENGTHS.
#include "anyfft.cuh"
#include "ns_axis3.cuh"
#include "prof.h"

namespace sfl {

namespace {

// Analysis line pass over up to 8 subbands of one mask group per CTA: a line's
// X times the group factor is loaded once, then per subband scaled by its
// wedge planes, transformed along axis 3 and stored.  The tiles of all the
// chunk's mask groups share the launch.
//
// Wedge planes constant along axis 3 (plane a of hourglasses 1 and 2, over
// (k1, k2)) are a per-line scalar and commute with the axis-3 FFT, so they
// are applied after it: Y_s = wa_p(k1, k2) IFFT_3(X G wb_q).  With nbq > 0
// the segment is nbq plane-b wedges q times whole rows of plane-a wedges p
// (item t = p nbq + q); the CTA takes the items q-major, and consecutive
// items of one q share a single FFT.  Every such item uses this order of
// operations whether or not it shares, so the values do not depend on the
// chunking.
template <int N>
__global__ void __launch_bounds__(256, 2)
    ns_slab_mask_group_kernel(const float2* __restrict__ X, int P1, int s3, const __grid_constant__ NSMaskTables tb,
                              const __grid_constant__ Chunk ck, const __grid_constant__ MaskTiles tl, int synth,
                              float2* Y, long long ystride, const float2* __restrict__ tw, long long xchs,
                              long long ychs) {
    using Ge = AnyGeom<N>;
    constexpr int N1 = Ge::N1, N2 = Ge::N2, LP = Ge::LP, E = Ge::E;
    extern __shared__ float2 a3_sm[];
    float2* const tws = a3_sm;
    float2* const xch = a3_sm + N;
    any_load_twiddles<N>(tws, tw);
    __syncthreads();
    X += blockIdx.y * xchs;   // channel
    Y += blockIdx.y * ychs;
    const int t = mask_tile_of(tl, blockIdx.x);
    const ChunkSeg& sg = ck.seg[tl.seg[t]];
    const int tid = threadIdx.x;
    const int lp = tid % LP, p = tid / LP;
    const int l = ((int)blockIdx.x - tl.first[t]) * LP + lp;
    const bool valid = l < sg.nk1 * sg.nk2;
    int k1 = 0, k2 = 0;
    if (valid) BoxMap{sg.nk1, sg.nk2, sg.b2, tb.n2}.k12(l, k1, k2);
    float2* xl = xch + lp * Ge::XLINE;
    const int k0 = tl.k0[t], kend = k0 + tl.cnt[t];
    const int nbq = sg.nbq, rows = nbq > 0 ? sg.nz / nbq : 0;
    auto zof = [&](int k) { return sg.i0 + (nbq > 0 ? (k % rows) * nbq + k / rows : k); };
    // the group factor of the line (group table, bandpass table or the lowpass factors)
    float2 xg[N1];
    {
        const NSMaskLine m0 = chunk_mask_line(tb, sg, ck.item[sg.i0], k1, k2, synth != 0);
        const float2* xp = X + k1 + P1 * k2;
        const int si = tb.h1 * tb.n2;
#pragma unroll
        for (int r = 0; r < N1; ++r) {
            const int i = p + N2 * r;
            const float g = m0.low ? m0.lowc * m0.lowv[i] : m0.m[i * si];
            xg[r] = valid ? c_scale(xp[i * s3], g) : make_float2(0.f, 0.f);
        }
    }
    float2 u[E];
#pragma unroll 1
    for (int k = k0; k < kend; ++k) {
        const int z = zof(k);
        const NSMaskLine mk = chunk_mask_line(tb, sg, ck.item[z], k1, k2, synth != 0);
        const bool wedges = !(mk.low || mk.plain);
        // plane a constant along the line: applied after the FFT
        const bool after = wedges && mk.was == 0;
        const bool reuse = after && nbq > 0 && k > k0 && (k - 1) / rows == k / rows;   // same q: uniform
        if (!reuse) {
            float2 v[N1];
            if (!wedges) {
#pragma unroll
                for (int r = 0; r < N1; ++r) v[r] = xg[r];
            } else if (after) {
#pragma unroll
                for (int r = 0; r < N1; ++r) v[r] = c_scale(xg[r], mk.wb[(p + N2 * r) * mk.wbs]);
            } else if (mk.wbs == 0) {
                const float b0 = mk.wb[0];
#pragma unroll
                for (int r = 0; r < N1; ++r) v[r] = c_scale(xg[r], mk.wa[(p + N2 * r) * mk.was] * b0);
            } else {
#pragma unroll
                for (int r = 0; r < N1; ++r) {
                    const int i = p + N2 * r;
                    v[r] = c_scale(xg[r], mk.wa[i * mk.was] * mk.wb[i * mk.wbs]);
                }
            }
            if (k > k0) __syncthreads();   // the exchange rows were read for the previous FFT
            any_block_fft<N, true>(v, p, xl, tws, u);
        }
        if (valid) {
            const float a0 = after ? mk.wa[0] : 1.f;
            float2* y = Y + z * ystride + k1 + P1 * k2;
#pragma unroll
            for (int j = 0; j < Ge::M; ++j)
                if (Ge::has(p, j)) {
#pragma unroll
                    for (int kk = 0; kk < N2; ++kk) {
                        const float2 w = u[j * N2 + kk];
                        y[((p + N2 * j) + N1 * kk) * s3] = after ? c_scale(w, a0) : w;
                    }
                }
        }
    }
}

template <int N>
void launch_n(const NSPlan& P, const float2* X, const Chunk& ck, const MaskTiles& tl, int synth, float2* Y, int nch,
              long long xchs, long long ychs, cudaStream_t st) {
    using Ge = AnyGeom<N>;
    static DeviceOnce once;
    allow_smem(once, ns_slab_mask_group_kernel<N>, Ge::SMEM);
    ns_slab_mask_group_kernel<N><<<dim3(tl.first[tl.n], nch), Ge::THREADS, Ge::SMEM, st>>>(
        X, P.P1, P.P1 * P.dims[1], P.tb, ck, tl, synth, Y, P.SP, P.ffts.at(N)->sh.tw, xchs, ychs);
    cuda_check(cudaGetLastError(), "ns_slab_mask_group_kernel launch");
}

}  // namespace

bool axis3_len(int n) { return any_len(n); }

int axis3_lines(int n) {
    switch (n) {
#define SFL_AXIS3_CASE(N_) \
    case N_: return AnyGeom<N_>::LP;
        SFL_ANY_LENGTHS(SFL_AXIS3_CASE)
#undef SFL_AXIS3_CASE
    }
    return 0;
}

void launch_axis3_mask(const NSPlan& P, const float2* X, const Chunk& ck, const MaskTiles& tl, int synth, float2* Y,
                       int nch, long long xchs, long long ychs, cudaStream_t st) {
    switch (P.dims[2]) {
#define SFL_AXIS3_CASE(N_) \
    case N_: launch_n<N_>(P, X, ck, tl, synth, Y, nch, xchs, ychs, st); return;
        SFL_ANY_LENGTHS(SFL_AXIS3_CASE)
#undef SFL_AXIS3_CASE
    }
    throw ArgError("no axis-3 pass of this length");
}

}  // namespace sfl
