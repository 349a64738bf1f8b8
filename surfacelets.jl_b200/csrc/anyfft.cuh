// Line FFTs of the lengths from 16 to 256 that are products of two radices up
// to 16, known at compile time: N = N1 N2, N2 lanes a line, each with N1 values
// in registers (regfft.cuh's split without its conditions that N2 divide N1
// and be a power of two).  The second step's N1 DFTs of N2 points go round
// the N2 lanes, ceil(N1 / N2) times.
#pragma once

#include "regfft.cuh"

namespace sfl {

// The split of N: of those with both radices up to 16, the one that keeps most
// lanes busy (the lanes of a warp that hold a line, and those of the second
// step's last round), the smaller N1 among equals; 0 when N has none.
constexpr int any_n1(int N) {
    int best = 0;
    double cost = 0;
    for (int n1 = 2; n1 <= 16; ++n1) {
        if (N % n1 != 0) continue;
        const int n2 = N / n1;
        if (n2 < 2 || n2 > 16) continue;
        const int rounds = (n1 + n2 - 1) / n2;
        const double e1 = (32 / n2) * n2 / 32.0;
        const double c = 1 / e1 + rounds * n2 / (e1 * n1);
        if (best == 0 || c < cost - 1e-9) {
            best = n1;
            cost = c;
        }
    }
    return best;
}

#define SFL_ANY_LENGTHS(X) \
    X(16) X(18) X(20) X(21) X(22) X(24) X(25) X(26) X(27) X(28) X(30) X(32) X(33) X(35) \
    X(36) X(39) X(40) X(42) X(44) X(45) X(48) X(49) X(50) X(52) X(54) X(55) X(56) X(60) \
    X(63) X(64) X(65) X(66) X(70) X(72) X(75) X(77) X(78) X(80) X(81) X(84) X(88) X(90) \
    X(91) X(96) X(98) X(99) X(100) X(104) X(105) X(108) X(110) X(112) X(117) X(120) X(121) X(126) \
    X(128) X(130) X(132) X(135) X(140) X(143) X(144) X(150) X(154) X(156) X(160) X(165) X(168) X(169) \
    X(176) X(180) X(182) X(192) X(195) X(196) X(208) X(210) X(224) X(225) X(240) X(256)

inline bool any_len(int n) {
    switch (n) {
#define SFL_ANY_CASE(N_) case N_:
        SFL_ANY_LENGTHS(SFL_ANY_CASE)
#undef SFL_ANY_CASE
        return true;
    }
    return false;
}

template <int N>
struct AnyLine {
    static constexpr int N1 = any_n1(N);
    static constexpr int N2 = N / N1;
    static constexpr int M = (N1 + N2 - 1) / N2;   // rounds of the second step
    static constexpr int E = M * N2;               // outputs a lane: X[(p + N2 j) + N1 k] at [j N2 + k]
    static constexpr int LPW = 32 / N2;            // lines a warp
    static constexpr bool kWhole = N1 % N2 == 0;   // every lane works in every round
    // whether lane p has outputs in round j
    __device__ __forceinline__ static bool has(int p, int j) { return kWhole || p + N2 * j < N1; }
};

// Thread geometry of a block pass with lanes on consecutive lines: LP lines
// (a multiple of 8) times N2 threads.
template <int N>
struct AnyGeom : AnyLine<N> {
    static constexpr int LP = 256 / AnyLine<N>::N2 / 8 * 8;
    static constexpr int THREADS = LP * AnyLine<N>::N2;
    static constexpr int XROW = AnyLine<N>::N2 + 1;              // exchange row pitch (float2)
    static constexpr int XLINE = (AnyLine<N>::N1 * XROW) | 1;    // exchange line pitch, odd
    static constexpr size_t SMEM = sizeof(float2) * ((size_t)N + (size_t)LP * XLINE);   // twiddles, exchange rows
};

// Twiddles of a line FFT rearranged as tw2[m N2 + p] = w_N^{p m}.
template <int N>
__device__ __forceinline__ void any_load_twiddles(float2* tw2, const float2* __restrict__ tw) {
    using L = AnyLine<N>;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const int m = i / L::N2, p = i - m * L::N2;
        tw2[i] = tw[p * m];
    }
}

// The FFT of one line of a block pass from values in registers: v[r] =
// x[p + N2 r]; u as AnyLine says.  One barrier; the exchange rows may be
// rewritten after the next one.  The twiddles tw2 lie in shared memory: read from
// global memory they are loop constants to the compiler, which then holds them
// in registers across the terms and spills.
template <int N, bool INV>
__device__ __forceinline__ void any_block_fft(float2 (&v)[AnyLine<N>::N1], int p, float2* xl, const float2* tw2,
                                              float2 (&u)[AnyLine<N>::E]) {
    using G = AnyGeom<N>;
    constexpr int N1 = G::N1, N2 = G::N2;
    RegDft<N1, INV>::run(v);
#pragma unroll
    for (int m = 1; m < N1; ++m) {
        float2 w = tw2[m * N2 + p];
        if (INV) w.y = -w.y;
        v[m] = c_mul(v[m], w);
    }
#pragma unroll
    for (int m = 0; m < N1; ++m) xl[m * G::XROW + p] = v[m];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < G::M; ++j) {
        const int m = p + N2 * j;
        float2 w[N2];
        const float2* xm = xl + (G::has(p, j) ? m * G::XROW : 0);
#pragma unroll
        for (int q = 0; q < N2; ++q) w[q] = xm[q];
        RegDft<N2, INV>::run(w);
#pragma unroll
        for (int k = 0; k < N2; ++k) u[j * N2 + k] = w[k];
    }
}

// The line that a lane works on.  Lanes without one repeat the warp's first
// line and drop the values: they read its slots with the lanes it belongs to,
// between the same warp barriers, and never those of another warp's line,
// which may be rewritten meanwhile.
struct LaneLine {
    int l;
    bool valid;
};

// Lane group s = lane / N2 of the warp whose lines start at l0 < nlines.
template <int N>
__host__ __device__ __forceinline__ LaneLine any_lane_line(int l0, int s, int nlines) {
    const bool valid = s < AnyLine<N>::LPW && l0 + s < nlines;
    return LaneLine{valid ? l0 + s : l0, valid};
}

// The same for column pairs (lines 2 P1 slots apart, P1 = 2 mod 4): with four
// lines a warp the two lines of a half warp are two apart, so that their slots
// fall on disjoint banks.
template <int N>
__host__ __device__ __forceinline__ LaneLine any_lane_pair(int l0, int s, int npairs) {
    return any_lane_line<N>(l0, AnyLine<N>::N2 == 8 && (s == 1 || s == 2) ? 3 - s : s, npairs);
}

// FFT of one line by the N2 lanes p of a warp, exchanged through N slots of
// the line's own, base[stride t]: sender q's value m sits at t = N2 m + (q
// turned by m within N2), which spreads both sides over the banks.  Lanes
// without a line (valid false) have the slots of one of the warp's lines: they
// write none and keep to the warp barriers.
template <int N, bool INV>
__device__ __forceinline__ void any_warp_fft(float2 (&v)[AnyLine<N>::N1], int p, bool valid,
                                             const float2* __restrict__ tw2, float2* base, int stride,
                                             float2 (&u)[AnyLine<N>::E]) {
    using L = AnyLine<N>;
    constexpr int N1 = L::N1, N2 = L::N2;
    constexpr bool kPow2 = (N2 & (N2 - 1)) == 0;
    RegDft<N1, INV>::run(v);
#pragma unroll
    for (int m = 1; m < N1; ++m) {
        float2 w = tw2[m * N2 + p];
        if (INV) w.y = -w.y;
        v[m] = c_mul(v[m], w);
    }
    int xo[N2];
#pragma unroll
    for (int c = 0; c < N2; ++c) xo[c] = stride * (kPow2 ? p ^ c : (p + c >= N2 ? p + c - N2 : p + c));
    __syncwarp();   // the line's inputs may have come from its own slots
    if (valid) {
#pragma unroll
        for (int m = 0; m < N1; ++m) base[xo[m % N2] + stride * N2 * m] = v[m];
    }
    __syncwarp();
    const float2* rb = base + stride * N2 * p;
#pragma unroll
    for (int j = 0; j < L::M; ++j) {
        float2 w[N2];
        // lanes without an output read the line's first slots and are dropped by the caller
        const float2* rj = L::has(p, j) ? rb + stride * N2 * N2 * j : base;
#pragma unroll
        for (int q = 0; q < N2; ++q) w[q] = rj[xo[q]];
        RegDft<N2, INV>::run(w);
#pragma unroll
        for (int k = 0; k < N2; ++k) u[j * N2 + k] = w[k];
    }
    __syncwarp();   // slots are free again
}

}  // namespace sfl
