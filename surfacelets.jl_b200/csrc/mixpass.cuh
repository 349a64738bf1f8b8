// Line passes of any length: a mixed-radix FFT whose radices are chosen at
// run time, for the lengths that have no compile-time register pass
// (regpass.cuh).
//
// A length n = R_1 R_2 ... R_s is transformed in s steps.  Step i runs DFTs of
// size R_i in registers (one compile-time body per radix up to 16, picked by a
// switch that is uniform over the grid), multiplies by the
// twiddles of the remaining length and puts every value back into the slot it
// came from, so one tile of shared memory serves all steps: with y the block
// of length L = R M that a step works on,
//
//   y'[m M + p] = w_L^{p m} sum_r y[p + M r] w_R^{r m},   p < M,
//
// and the blocks y'[m M ...] of length M are the next step's.  The first step
// reads its values through the load op (global memory), the last one hands
// them to the store op, so a length of two radices (nearly every length up to
// 256 without a prime factor above 13) makes one shared-memory exchange.
//
// Prime factors above 13 come first, in shared memory: the pairs x_r +- x_{q-r}
// are folded in place and the real and odd sums of q / 2 terms give the bins m
// and q - m together (half the products of the direct sum).
#pragma once

#include <type_traits>
#include <utility>

#include "passes.cuh"
#include "plan.h"
#include "prof.h"
#include "regfft.cuh"
#include "regpass.cuh"

namespace sfl {

// Division by an invariant d through a multiplication (Granlund and
// Montgomery, 1994): exact for n d < 2^32; the item indices divided here stay
// below 2^17 and the divisors below 2^13.
struct MixDiv {
    unsigned d = 1, m = 0;
    MixDiv() = default;
    __host__ __device__ explicit MixDiv(unsigned dv) : d(dv), m(dv > 1 ? 0xFFFFFFFFu / dv + 1u : 0u) {}
    __device__ __forceinline__ int div(int n) const { return d > 1 ? (int)__umulhi((unsigned)n, m) : n; }
};

// A length as the passes take it.
struct MixArgs {
    MixSchedule sc;
    const float2* tw;          // w_n^k, k < n (float64-designed)
    const unsigned short* rev; // output index of each last-step block (n / R_last entries)
    int pitch;                 // tile pitch of a line (odd)
    int m1p;                   // tile pitch of the first step's output blocks (odd: n / R_1 rounded up)
    MixDiv d_first, d_last, d_m1r, d_p1;   // divisors of the item indices
};

// The tile of one call: the 1 << lg lines from l0 of nlines; consecutive lanes
// take consecutive lines (tfast) or consecutive positions.
struct MixTile {
    int l0, nlines, lg, tfast;
};

// Radices of the first and the last step, and of the steps between.
#define SFL_MIX_RADICES(X) \
    X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)
#define SFL_MIX_MIDDLE(X) X(2) X(3) X(4) X(5) X(7) X(8) X(11) X(13)

// Item index -> (line of the tile, position).
__device__ __forceinline__ void mix_item(const MixTile& g, const MixDiv& d, int it, int& t, int& e) {
    if (g.tfast) {
        t = it & ((1 << g.lg) - 1);
        e = it >> g.lg;
    } else {
        t = d.div(it);
        e = it - t * (int)d.d;
    }
}

// First step: global memory -> registers -> tile.
template <int R, bool INV, class Load>
__device__ __forceinline__ void mix_first(const Load& ld, const MixArgs& a, const MixTile& g, float2* tile, int z) {
    const int M = (int)a.d_first.d;
    const int items = M << g.lg;
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
        int t, p;
        mix_item(g, a.d_first, it, t, p);
        const int l = g.l0 + t;
        const bool valid = l < g.nlines;
        const typename Load::Ctx c = ld.line(z, l, valid);
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = valid ? ld.get(c, p + M * r) : make_float2(0.f, 0.f);
        RegDft<R, INV>::run(v);
        float2* y = tile + t * a.pitch + p;
        y[0] = v[0];
#pragma unroll
        for (int m = 1; m < R; ++m) {
            float2 w = __ldg(a.tw + p * m);
            if (INV) w.y = -w.y;
            y[m * a.m1p] = c_mul(v[m], w);
        }
    }
}

// A step between the first and the last: blocks of length L in place.
template <int R, bool INV>
__device__ __forceinline__ void mix_middle(const MixArgs& a, const MixTile& g, float2* tile, int L) {
    const int n = a.sc.n, M = L / R, M1 = n / a.sc.R[0];
    const MixDiv dl((unsigned)(n / R)), d1((unsigned)(M1 / R)), dm((unsigned)M);
    const int items = (n / R) << g.lg, tstep = n / L;
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
        int t, e;
        mix_item(g, dl, it, t, e);
        const int m1 = d1.div(e), rem = e - m1 * (int)d1.d;
        const int j = dm.div(rem), p = rem - j * M;
        float2* y = tile + t * a.pitch + m1 * a.m1p + j * L + p;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = y[M * r];
        RegDft<R, INV>::run(v);
        y[0] = v[0];
#pragma unroll
        for (int m = 1; m < R; ++m) {
            float2 w = __ldg(a.tw + tstep * p * m);
            if (INV) w.y = -w.y;
            y[M * m] = c_mul(v[m], w);
        }
    }
}

// Last step: tile -> registers -> the store op, or in natural order into
// `out` (pitch outp) for ops that need the whole line.
template <int R, bool INV, class Store>
__device__ __forceinline__ void mix_last(const Store& st, const MixArgs& a, const MixTile& g, const float2* tile, float2* out, int outp,
                                         int z) {
    const int nb = (int)a.d_last.d;   // n / R blocks
    const int items = nb << g.lg;
    for (int it = threadIdx.x; it < items; it += blockDim.x) {
        int t, e;
        mix_item(g, a.d_last, it, t, e);
        const int l = g.l0 + t;
        const int m1 = a.d_m1r.div(e), rem = e - m1 * (int)a.d_m1r.d;
        const float2* y = tile + t * a.pitch + m1 * a.m1p + rem * R;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = y[r];
        RegDft<R, INV>::run(v);
        const int k0 = a.rev ? (int)__ldg(a.rev + e) : e;
        if constexpr (Store::kStaged) {
            float2* o = out + t * outp + k0;
#pragma unroll
            for (int m = 0; m < R; ++m) o[m * nb] = v[m];
        } else if (l < g.nlines) {
            const typename Store::Ctx c = st.line(z, l, true);
#pragma unroll
            for (int m = 0; m < R; ++m) st.put(c, k0 + nb * m, v[m]);
        }
    }
}

// ── lengths with a large prime factor ───────────────────────────────────────

constexpr int kMixPer = 8;   // elements a thread moves per line context in the plain copies

// Lines into the tile in natural order.
template <class Load>
__device__ __forceinline__ void mix_copy_in(const Load& ld, const MixArgs& a, const MixTile& g, float2* tile, int z) {
    const int ng = (int)a.d_p1.d, n = a.sc.n;   // d_p1: ceil(n / kMixPer)
    for (int it = threadIdx.x; it < (ng << g.lg); it += blockDim.x) {
        int t, c8;
        mix_item(g, a.d_p1, it, t, c8);
        const int l = g.l0 + t;
        const bool valid = l < g.nlines;
        const typename Load::Ctx c = ld.line(z, l, valid);
        float2 v[kMixPer];
#pragma unroll
        for (int u = 0; u < kMixPer; ++u) {
            const int i = c8 + ng * u;
            v[u] = valid && i < n ? ld.get(c, i) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kMixPer; ++u) {
            const int i = c8 + ng * u;
            if (i < n) tile[t * a.pitch + i] = v[u];
        }
    }
}

// Lines in natural order out of the tile.
template <class Store>
__device__ __forceinline__ void mix_copy_out(const Store& st, const MixArgs& a, const MixTile& g, const float2* tile, int z) {
    const int ng = (int)a.d_p1.d, n = a.sc.n;
    for (int it = threadIdx.x; it < (ng << g.lg); it += blockDim.x) {
        int t, c8;
        mix_item(g, a.d_p1, it, t, c8);
        const int l = g.l0 + t;
        if (l >= g.nlines) continue;
        const typename Store::Ctx c = st.line(z, l, true);
#pragma unroll
        for (int u = 0; u < kMixPer; ++u) {
            const int i = c8 + ng * u;
            if (i < n) st.put(c, i, tile[t * a.pitch + i]);
        }
    }
}

// A step of prime radix q on blocks of length L = q M, from `in` to `out`
// (both with the line pitch; `in` in natural order when first, else in the
// first step's padded blocks, as `out` always is).  The weights w_q^j are in
// shared memory; a thread forms kMixBins pairs of bins of two lines, so that
// a weight read serves two lines and a folded pair kMixBins bins.
constexpr int kMixBins = 4;
template <bool INV>
__device__ void mix_prime(const MixArgs& a, const MixTile& g, float2* in, float2* out, const float2* wq, int q, int L, bool first) {
    const int n = a.sc.n, M = L / q, h = (q - 1) / 2, LP = 1 << g.lg;
    const int M1 = n / a.sc.R[0];
    const int nbk = n / q;   // (block, p) pairs of a line
    const MixDiv dh((unsigned)h), dm((unsigned)M), d1((unsigned)(first ? M : M1 / q));
    // offsets of pair bp: input base, output base
    auto bases = [&](int bp, int& bi, int& bo, int& p) {
        if (first) {
            bi = bo = p = bp;
        } else {
            const int m1 = d1.div(bp), rem = bp - m1 * (int)d1.d;
            const int j = dm.div(rem);
            p = rem - j * M;
            bi = bo = m1 * a.m1p + j * L + p;
        }
    };
    // fold x_r, x_{q-r} -> x_r + x_{q-r}, x_r - x_{q-r}
    for (int it = threadIdx.x; it < ((nbk * h) << g.lg); it += blockDim.x) {
        const int t = it & (LP - 1), e = it >> g.lg;
        const int bp = dh.div(e), r = e - bp * h + 1;
        int bi, bo, p;
        bases(bp, bi, bo, p);
        float2* x = in + t * a.pitch + bi;
        const float2 u = x[M * r], v = x[M * (q - r)];
        x[M * r] = c_add(u, v);
        x[M * (q - r)] = c_sub(u, v);
    }
    __syncthreads();
    const int os = first ? a.m1p : M;   // step between the output blocks
    const int tstep = n / L;
    const int lp2 = LP > 1 ? LP / 2 : 1, lg2 = LP > 1 ? g.lg - 1 : 0;
    const int ngrp = (h + kMixBins - 1) / kMixBins;
    const MixDiv dg((unsigned)ngrp);
    for (int it = threadIdx.x; it < ((nbk * ngrp) << lg2); it += blockDim.x) {
        const int t = it & (lp2 - 1), e = it >> lg2;
        const int bp = dg.div(e), m0 = (e - bp * ngrp) * kMixBins + 1;
        int bi, bo, p;
        bases(bp, bi, bo, p);
        const int o2 = LP > 1 ? lp2 * a.pitch : 0;
        const float2* xa = in + t * a.pitch + bi;
        const float2* xb = xa + o2;
        float2 ca[kMixBins], da[kMixBins], cb[kMixBins], db[kMixBins];
        int idx[kMixBins], stp[kMixBins];
        const float2 x0a = xa[0], x0b = xb[0];
#pragma unroll
        for (int b = 0; b < kMixBins; ++b) {
            ca[b] = x0a;
            cb[b] = x0b;
            da[b] = db[b] = make_float2(0.f, 0.f);
            stp[b] = m0 + b <= h ? m0 + b : 0;   // bins past h repeat bin 0 and are dropped
            idx[b] = 0;
        }
        float2 za = x0a, zb = x0b;   // bin 0
        for (int r = 1; r <= h; ++r) {
            const float2 sa = xa[M * r], ta = xa[M * (q - r)];
            const float2 sb = xb[M * r], tb = xb[M * (q - r)];
            za = c_add(za, sa);
            zb = c_add(zb, sb);
#pragma unroll
            for (int b = 0; b < kMixBins; ++b) {
                idx[b] += stp[b];
                if (idx[b] >= q) idx[b] -= q;
                const float2 w = wq[idx[b]];
                ca[b] = c_fma(sa, w.x, ca[b]);
                da[b] = c_fma(ta, w.y, da[b]);
                cb[b] = c_fma(sb, w.x, cb[b]);
                db[b] = c_fma(tb, w.y, db[b]);
            }
        }
        float2* ya = out + t * a.pitch + bo;
        float2* yb = ya + o2;
        if (m0 == 1) {
            ya[0] = za;
            yb[0] = zb;
        }
#pragma unroll
        for (int b = 0; b < kMixBins; ++b) {
            const int m = m0 + b;
            if (m > h) continue;
            // C +- i D: bins m and q - m (exchanged for the inverse transform)
            const int mu = INV ? q - m : m, ml = q - mu;
            float2 wu = __ldg(a.tw + tstep * p * mu), wl = __ldg(a.tw + tstep * p * ml);
            if (INV) {
                wu.y = -wu.y;
                wl.y = -wl.y;
            }
            const float2 ua = make_float2(ca[b].x - da[b].y, ca[b].y + da[b].x);
            const float2 la = make_float2(ca[b].x + da[b].y, ca[b].y - da[b].x);
            const float2 ub = make_float2(cb[b].x - db[b].y, cb[b].y + db[b].x);
            const float2 lb = make_float2(cb[b].x + db[b].y, cb[b].y - db[b].x);
            ya[os * mu] = M > 1 ? c_mul(ua, wu) : ua;
            ya[os * ml] = M > 1 ? c_mul(la, wl) : la;
            yb[os * mu] = M > 1 ? c_mul(ub, wu) : ub;
            yb[os * ml] = M > 1 ? c_mul(lb, wl) : lb;
        }
    }
    __syncthreads();
}

// The steps before the last on a tile whose lines are loaded; returns the
// number of the next step.  Radices above 16 are the large primes, which come
// first.
template <bool INV>
__device__ __forceinline__ int mix_primes(const MixArgs& a, const MixTile& g, float2*& tile, float2*& other, float2* wq) {
    int s = 0, L = a.sc.n;
    for (; s < a.sc.ns && a.sc.R[s] > 16; ++s) {
        const int q = a.sc.R[s];
        for (int i = threadIdx.x; i < q; i += blockDim.x) wq[i] = __ldg(a.tw + (long long)(a.sc.n / q) * i);
        __syncthreads();
        mix_prime<INV>(a, g, tile, other, wq, q, L, s == 0);
        float2* x = tile;
        tile = other;
        other = x;
        L /= q;
    }
    return s;
}

template <bool INV>
__device__ __forceinline__ void mix_middles(const MixArgs& a, const MixTile& g, float2* tile, int s0) {
    int L = a.sc.n;
    for (int s = 0; s < s0; ++s) L /= a.sc.R[s];
    for (int s = s0; s + 1 < a.sc.ns; ++s) {
        switch (a.sc.R[s]) {
#define SFL_MIX_CASE(R_) \
    case R_: mix_middle<R_, INV>(a, g, tile, L); break;
            SFL_MIX_MIDDLE(SFL_MIX_CASE)
#undef SFL_MIX_CASE
        }
        L /= a.sc.R[s];
        __syncthreads();
    }
}

// One pass over a tile.  BIG: also lengths with a prime factor above 13.
// `other` is a second tile (BIG, and store ops that need whole lines), `wq`
// the weights of a large prime.
template <bool INV, bool BIG, class Load, class Store>
__device__ __forceinline__ void mix_pass(const Load& ld, const Store& st, const MixArgs& a, const MixTile& g, float2* tile, float2* other,
                                         float2* wq, int z) {
    int s = 1;
    bool big = false;
    if constexpr (BIG) {
        big = a.sc.R[0] > 16;
        if (big) {
            mix_copy_in(ld, a, g, tile, z);
            __syncthreads();
            s = mix_primes<INV>(a, g, tile, other, wq);
        }
    }
    if (!big) {
        switch (a.sc.R[0]) {
#define SFL_MIX_CASE(R_) \
    case R_: mix_first<R_, INV>(ld, a, g, tile, z); break;
            SFL_MIX_RADICES(SFL_MIX_CASE)
#undef SFL_MIX_CASE
        }
        __syncthreads();
    }
    mix_middles<INV>(a, g, tile, s);
    const float2* nat = tile;   // the finished lines in natural order, where they are needed
    if (s < a.sc.ns) {
        switch (a.sc.R[a.sc.ns - 1]) {
#define SFL_MIX_CASE(R_) \
    case R_: mix_last<R_, INV>(st, a, g, tile, other, a.pitch, z); break;
            SFL_MIX_RADICES(SFL_MIX_CASE)
#undef SFL_MIX_CASE
        }
        if constexpr (!Store::kStaged) return;
        __syncthreads();
        nat = other;
    }
    if constexpr (Store::kStaged) {
        const int nth = blockDim.x >> g.lg;   // threads a line
        int t, p;
        if (g.tfast) {
            t = threadIdx.x & ((1 << g.lg) - 1);
            p = threadIdx.x >> g.lg;
        } else {
            t = threadIdx.x / nth;
            p = threadIdx.x - t * nth;
        }
        const int l = g.l0 + t;
        if (t < (1 << g.lg) && p < nth && l < g.nlines) st.staged(st.line(z, l, true), nat + t * a.pitch, p, nth);
    } else {
        mix_copy_out(st, a, g, nat, z);
    }
}

template <bool INV, bool BIG, class Load, class Store>
__global__ void __launch_bounds__(256, 2) mix_pass_kernel(Load ld, Store st, const __grid_constant__ MixArgs a, int nlines,
                                                          int lg, int tfast) {
    extern __shared__ float2 mix_smem[];
    const int tsz = a.pitch << lg;
    const MixTile g{(int)blockIdx.x << lg, nlines, lg, tfast};
    mix_pass<INV, BIG>(ld, st, a, g, mix_smem, mix_smem + tsz, mix_smem + 2 * tsz, blockIdx.y);
}

inline bool mix_big(const MixSchedule& sc) { return sc.R[0] > 16; }

// Shared memory of a pass over tiles of 1 << lg lines.
inline size_t mix_smem_bytes(const MixSchedule& sc, int lg, int pitch, bool staged) {
    const bool big = mix_big(sc);
    return sizeof(float2) * (((size_t)pitch << lg) * (big || staged ? 2 : 1) + (big ? sc.R[0] : 0));
}

// small_first: the smaller of two radices first, so that the first step's loads
// spread over more threads.
inline MixArgs mix_args(const FFTLen& f, bool small_first = false) {
    MixArgs a;
    MixSchedule sc = f.mix;
    if (small_first && sc.ns == 2 && sc.R[0] <= 16 && sc.R[0] > sc.R[1]) std::swap(sc.R[0], sc.R[1]);
    a.sc = sc;
    a.tw = f.sh.tw;
    a.rev = sc.ns > 2 ? f.rev.as<unsigned short>() : nullptr;
    const int M1 = sc.n / sc.R[0];
    a.m1p = sc.ns == 1 ? 1 : (M1 | 1);
    a.pitch = std::max(sc.n, a.m1p * sc.R[0]) | 1;
    const int rl = sc.R[sc.ns - 1];
    a.d_first = MixDiv((unsigned)M1);
    a.d_last = MixDiv((unsigned)(sc.n / rl));
    a.d_m1r = MixDiv((unsigned)std::max(1, M1 / rl));
    a.d_p1 = MixDiv((unsigned)((sc.n + kMixPer - 1) / kMixPer));
    return a;
}

// Lines a tile: 32 (16 above 64 points) as shared memory allows; strided lines
// then read and write runs of at least 128 bytes.
inline int mix_lines_lg(const MixArgs& a, bool staged, size_t extra_per_line = 0) {
    int lg = a.sc.n <= 64 ? 5 : 4;
    while (lg > 0 && mix_smem_bytes(a.sc, lg, a.pitch, staged) + (extra_per_line << lg) > 100 * 1024) --lg;
    return lg;
}

// Items a line gives to the widest step.
inline int mix_items(const MixSchedule& sc) {
    int per = 1;
    for (int s = 0; s < sc.ns; ++s)
        if (sc.R[s] <= 16) per = std::max(per, sc.n / sc.R[s]);
    if (mix_big(sc)) per = std::max(per, sc.n / 4);
    return per;
}

// Threads a CTA: one item of the widest step each, at most 256.
inline int mix_threads(const MixArgs& a, int lg) {
    const int t = (((mix_items(a.sc) << lg) + 31) / 32) * 32;
    const int least = std::max(64, 1 << lg);
    return std::min(256, std::max(t, least));
}

// Load ops with several reads and products a value (Load::kHeavy: the masked
// axis-3 load).  The first step is where they run, so it takes the smaller radix
// of two (256 x 256 x 75 analysis, 5 x 15 for 15 x 5: 1825 -> 1083 us; 27
// points: 622 -> 505) and tiles of one round of items (505 -> 408).
template <class Load, class = void>
struct HeavyLoad : std::false_type {};
template <class Load>
struct HeavyLoad<Load, std::void_t<decltype(Load::kHeavy)>> : std::bool_constant<Load::kHeavy> {};

template <bool INV, bool BIG, class Load, class Store>
void launch_mix_b(const FFTLen& f, const Load& ld, const Store& st, int nlines, int nz, bool tfast,
                  cudaStream_t stream, const char* tag) {
    const MixArgs a = mix_args(f, HeavyLoad<Load>::value);
    int lg = mix_lines_lg(a, Store::kStaged);
    // heavy loads: one round of the widest step rather than a second one for a few items
    if (HeavyLoad<Load>::value)
        while (lg > 4 && (mix_items(a.sc) << lg) > 256) --lg;
    // Tiles of long lines are large, and a small volume has few: fewer lines a tile (strided ones keep 32-byte
    // runs) until every SM has two CTAs.  C2R of 1000 x 16 x 16, 8 subbands: 26 us a launch in 128 tiles of 8 lines.
    if (a.sc.n > 256)
        while (lg > (tfast ? 2 : 0) && (long long)((nlines + (1 << lg) - 1) >> lg) * nz < 2 * 148) --lg;
    const size_t smem = mix_smem_bytes(a.sc, lg, a.pitch, Store::kStaged);
    auto kern = mix_pass_kernel<INV, BIG, Load, Store>;
    static DeviceOnce once;
    allow_smem(once, kern, 227 * 1024);
    const dim3 grid((unsigned)((nlines + (1 << lg) - 1) >> lg), (unsigned)nz);
    int tok = prof_begin(tag, stream);
    kern<<<grid, mix_threads(a, lg), smem, stream>>>(ld, st, a, nlines, lg, tfast ? 1 : 0);
    prof_end(tok, stream);
    cuda_check(cudaGetLastError(), "mix_pass_kernel launch");
}

// A line pass of any length: the compile-time register pass where there is
// one, else the mixed-radix pass.
template <bool INV, class Load, class Store>
void launch_line(const FFTLen& f, const Load& ld, const Store& st, int nlines, int nz, bool tfast, cudaStream_t stream,
                 const char* tag) {
    if (launch_reg<INV>(f.sh.n, ld, st, f.sh.tw, nlines, nz, tfast, stream, tag)) return;
    if (mix_big(f.mix))
        launch_mix_b<INV, true>(f, ld, st, nlines, nz, tfast, stream, tag);
    else
        launch_mix_b<INV, false>(f, ld, st, nlines, nz, tfast, stream, tag);
}

}  // namespace sfl
