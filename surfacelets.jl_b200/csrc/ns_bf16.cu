// NSSurfacelet coefficients stored in bfloat16 with one float32 scale per
// subband: subband s = scales[s-1] * c[..., s-1].  The scale is the smallest
// power of two at or above the subband's largest magnitude, so the stored
// values lie in [-1, 1] and the scaling itself is exact (bfloat16 keeps
// float32's exponent range; its 8-bit significand sets the accuracy).
//
// The transforms run in float32 through the item-range building blocks of
// the slab and line pipelines; a chunk of subbands passes through a float32
// scratch of chunk x n1 n2 n3 values (L2-resident at 128^3) on its way to or
// from bfloat16.
#include <cuda_bf16.h>

#include <cmath>

#include "plan.h"
#include "prof.h"

namespace sfl {

namespace {

unsigned grid_blocks(long long n) {   // n: steps of a thread
    long long g = (n + 255) / 256;
    return (unsigned)std::max(1LL, std::min(g, 148LL * 8));
}

// The three band kernels below move V values a thread and step: four where the
// volume and the caller's array allow 16- and 8-byte accesses, else one.  At one
// value they ran at a third of the memory rate (160 x 128 x 96: peak 92, pack
// 102, unpack 103 us of 204 MB each).
template <int V>
struct Vec;
template <>
struct Vec<1> {
    using F = float;
    using B = __nv_bfloat16;
};
template <>
struct Vec<4> {
    using F = float4;
    using B = uint2;
};

// Largest magnitude of each band of a chunk (float bits of non-negative
// values order like unsigned integers).
template <int V>
__global__ void band_maxabs_kernel(const float* __restrict__ band, long long n, unsigned* maxbits) {
    const float* b = band + blockIdx.y * n;
    float m = 0.f;
    for (long long i = V * (blockIdx.x * (long long)blockDim.x + threadIdx.x); i < n; i += V * (long long)gridDim.x * blockDim.x) {
        typename Vec<V>::F x = *reinterpret_cast<const typename Vec<V>::F*>(b + i);
        const float* f = reinterpret_cast<const float*>(&x);
#pragma unroll
        for (int k = 0; k < V; ++k) m = fmaxf(m, fabsf(f[k]));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float wm[32];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x + 31) / 32 ? wm[threadIdx.x] : 0.f;
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) atomicMax(maxbits + blockIdx.y, __float_as_uint(m));
    }
}

__device__ __forceinline__ float pow2_scale(unsigned bits) {
    const float m = __uint_as_float(bits);
    if (!(m > 0.f)) return 1.f;
    int e = 0;
    frexpf(m, &e);   // m = f 2^e, f in [0.5, 1)
    return ldexpf(1.f, e);
}

template <int V>
__global__ void band_to_bf16_kernel(const float* __restrict__ band, long long n, const unsigned* __restrict__ maxbits,
                                    const NSItem* __restrict__ items, int item0, __nv_bfloat16* out, float* scales) {
    const float* b = band + blockIdx.y * n;
    const int s = items[item0 + blockIdx.y].s;
    const float scale = pow2_scale(maxbits[blockIdx.y]);
    const float inv = 1.f / scale;   // exact: a power of two
    if (blockIdx.x == 0 && threadIdx.x == 0) scales[s - 1] = scale;
    __nv_bfloat16* o = out + (long long)(s - 1) * n;
    for (long long i = V * (blockIdx.x * (long long)blockDim.x + threadIdx.x); i < n; i += V * (long long)gridDim.x * blockDim.x) {
        typename Vec<V>::F x = *reinterpret_cast<const typename Vec<V>::F*>(b + i);
        const float* f = reinterpret_cast<const float*>(&x);
        typename Vec<V>::B y;
        __nv_bfloat16* h = reinterpret_cast<__nv_bfloat16*>(&y);
#pragma unroll
        for (int k = 0; k < V; ++k) h[k] = __float2bfloat16_rn(f[k] * inv);
        *reinterpret_cast<typename Vec<V>::B*>(o + i) = y;
    }
}

template <int V>
__global__ void bf16_to_band_kernel(const __nv_bfloat16* __restrict__ in, const float* __restrict__ scales,
                                    const NSItem* __restrict__ items, int item0, long long n, float* band) {
    float* b = band + blockIdx.y * n;
    const int s = items[item0 + blockIdx.y].s;
    const float scale = scales[s - 1];
    const __nv_bfloat16* c = in + (long long)(s - 1) * n;
    for (long long i = V * (blockIdx.x * (long long)blockDim.x + threadIdx.x); i < n; i += V * (long long)gridDim.x * blockDim.x) {
        typename Vec<V>::B x = *reinterpret_cast<const typename Vec<V>::B*>(c + i);
        const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&x);
        typename Vec<V>::F y;
        float* f = reinterpret_cast<float*>(&y);
#pragma unroll
        for (int k = 0; k < V; ++k) f[k] = __bfloat162float(h[k]) * scale;
        *reinterpret_cast<typename Vec<V>::F*>(b + i) = y;
    }
}

// Whether every band of the caller's array starts on an 8-byte boundary and
// holds a multiple of four values (the float bands are the plan's own).
bool four_wide(const NSPlan& P, const void* c) { return P.N % 4 == 0 && reinterpret_cast<uintptr_t>(c) % 8 == 0; }

void need_bf16_path(const NSPlan& P) {
    if (P.nch != 1) throw ArgError("bfloat16 coefficients are for Float32 volumes");
}

void ensure_band(NSPlan& P) {
    const size_t need = sizeof(float) * (size_t)P.N * P.slots;
    if (P.band.bytes < need) P.band.alloc(need);
    if (P.maxbits.bytes < sizeof(unsigned) * (size_t)P.slots) P.maxbits.alloc(sizeof(unsigned) * P.slots);
}

}  // namespace

void ns_analyze_bf16(NSPlan& P, const float* x, void* c, float* scales, cudaStream_t st) {
    need_bf16_path(P);
    ensure_band(P);
    float2* X = P.X.as<float2>();
    float* band = P.band.as<float>();
    ns_forward_spectrum(P, x, 1, X, st);
    ZMap vz;
    vz.zstride = P.N;
    for (int i0 = 0, i1; i0 < P.S; i0 = i1) {
        i1 = ns_next_chunk(P, i0);
        const int nz = i1 - i0;
        ns_analyze_range(P, X, band, vz, 1, i0, nz, false, st);
        cuda_check(cudaMemsetAsync(P.maxbits.p, 0, sizeof(unsigned) * nz, st), "cudaMemsetAsync(maxbits)");
        const bool v4 = four_wide(P, c);
        const dim3 grid(grid_blocks(v4 ? P.N / 4 : P.N), nz);
        int tok = prof_begin("ns_bf16_pack", st);
        unsigned* mb = P.maxbits.as<unsigned>();
        (v4 ? band_maxabs_kernel<4> : band_maxabs_kernel<1>)<<<grid, 256, 0, st>>>(band, P.N, mb);
        (v4 ? band_to_bf16_kernel<4> : band_to_bf16_kernel<1>)<<<grid, 256, 0, st>>>(
            band, P.N, mb, P.items.as<NSItem>(), i0, reinterpret_cast<__nv_bfloat16*>(c), scales);
        prof_end(tok, st);
        prof_bytes("ns_bf16_pack", (double)nz * P.N * (4 + 4 + 2));
        cuda_check(cudaGetLastError(), "bfloat16 packing");
    }
}

void ns_synthesize_bf16(NSPlan& P, const void* c, const float* scales, float* x, cudaStream_t st) {
    need_bf16_path(P);
    ensure_band(P);
    float2* A = P.acc.as<float2>();
    float2* K = P.comp.as<float2>();
    float* band = P.band.as<float>();
    ZMap vz;
    vz.zstride = P.N;
    ns_acc_clear(P, A, K, st);
    for (int i0 = 0, i1; i0 < P.S; i0 = i1) {
        i1 = ns_next_chunk(P, i0);
        const int nz = i1 - i0;
        const bool v4 = four_wide(P, c);
        const dim3 grid(grid_blocks(v4 ? P.N / 4 : P.N), nz);
        int tok = prof_begin("ns_bf16_unpack", st);
        (v4 ? bf16_to_band_kernel<4> : bf16_to_band_kernel<1>)<<<grid, 256, 0, st>>>(
            reinterpret_cast<const __nv_bfloat16*>(c), scales, P.items.as<NSItem>(), i0, P.N, band);
        prof_end(tok, st);
        prof_bytes("ns_bf16_unpack", (double)nz * P.N * (2 + 4));
        cuda_check(cudaGetLastError(), "bfloat16 unpacking");
        ns_accumulate_range(P, band, vz, 1, i0, nz, false, A, K, st);
    }
    ns_inverse_spectrum(P, A, x, 1, st);
}

}  // namespace sfl
