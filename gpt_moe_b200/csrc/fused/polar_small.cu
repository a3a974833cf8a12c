// Polar Express on matrices of few rows (a router: experts x hidden) in one launch: a block owns a matrix X [M, k], M <= 32, in shared memory and
// runs all steps on the M x M side in fp32 (see polar_express in bindings.cpp for the scheme; with fp32 Gram matrices one run of all steps is
// closer to 64 bits than bf16 steps on every spectrum tried): A = X X^T, per step Q = a I + b A + c A^2, A <- Q A Q, T <- Q T, at the end X <- T X.
// As batched products of the GEMM the same took 15 launches of two to nine us each for a handful of rows.  2 of 8 x 768 take
// 22 us by events instead of 131, 13.5 each where a captured graph holds them in a row: a chain of small products between barriers.
// Reference counterparts: optimizers/polar_express.py:60-121, :155-230.
#include "../common/ptx.cuh"
#include "../kernels_decl.h"

namespace gm {

constexpr int PS_THREADS = 512;

struct PolarCoefficients { float c[8][3]; };

// out = alpha * a b (+ beta * add) (+ diag I), M x M matrices of pitch M + 4; every thread forms four elements of a row
template <int M>
__device__ __forceinline__ void ps_product(const float* a, const float* b, float* out, float alpha = 1.f, const float* add = nullptr, float beta = 0.f, float diag = 0.f) {
    constexpr int P = M + 4;
    for (int t = threadIdx.x; t < M * M / 4; t += PS_THREADS) {
        const int i = t / (M / 4), j = t % (M / 4) * 4;
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int l = 0; l < M; ++l) {
            const float x = a[i * P + l];
            const float4 y = *reinterpret_cast<const float4*>(b + l * P + j);
            s[0] = fmaf(x, y.x, s[0]); s[1] = fmaf(x, y.y, s[1]); s[2] = fmaf(x, y.z, s[2]); s[3] = fmaf(x, y.w, s[3]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) out[i * P + j + e] = alpha * s[e] + (add ? beta * add[i * P + j + e] : 0.f) + (i == j + e ? diag : 0.f);
    }
}

template <int M>
__global__ void __launch_bounds__(PS_THREADS, 1)
polar_small_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ sumsq, int k, PolarCoefficients coeffs, int steps) {
    constexpr int P = M + 4, PARTS = 32 / M, WARPS = PS_THREADS / 32;      // lanes beyond M * PARTS have no row
    extern __shared__ float smem[];
    float *gram = smem, *poly = gram + M * P, *tmp = poly + M * P, *total = tmp + M * P, *other = total + M * P;
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(other + M * P);
    const int pitch = k + 2;                                                // an odd number of words: the rows of a column lie on different banks
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __nv_bfloat16* mine = x + static_cast<long long>(blockIdx.x) * M * k;
    for (int i = threadIdx.x; i < M * k / 8; i += PS_THREADS) {             // k is a multiple of 8
        const uint4 v = reinterpret_cast<const uint4*>(mine)[i];
        const int row = i / (k / 8), col = (i - row * (k / 8)) * 8;
        uint32_t* to = reinterpret_cast<uint32_t*>(xs + row * pitch + col);
        to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w;
    }
    const float inv = sumsq ? 1.f / (sqrtf(sumsq[blockIdx.x]) * 1.02f + 1e-6f) : 1.f;
    __syncthreads();
    // A: a warp takes rows i and i + WARPS, a lane one row j and a share of the columns
    {
        const int j = lane % M, part = lane / M;
        const bool live = lane < M * PARTS;
        const uint32_t* xj = reinterpret_cast<const uint32_t*>(xs + (live ? j : 0) * pitch);
        const int words = k / 2, from = live ? words * part / PARTS : 0, to = live ? words * (part + 1) / PARTS : 0;
        for (int i = warp; i < M; i += WARPS) {
            const uint32_t* xi = reinterpret_cast<const uint32_t*>(xs + i * pitch);
            float s0 = 0.f, s1 = 0.f;
#pragma unroll 4
            for (int w = from; w < to; ++w) {
                const uint32_t a = xi[w], b = xj[w];
                s0 = fmaf(__uint_as_float(a << 16), __uint_as_float(b << 16), s0);
                s1 = fmaf(__uint_as_float(a & 0xffff0000u), __uint_as_float(b & 0xffff0000u), s1);
            }
            float s = s0 + s1;
            if (PARTS == 4) s += __shfl_xor_sync(0xffffffffu, s, 16);
            if (PARTS >= 2) s += __shfl_xor_sync(0xffffffffu, s, M);
            if (lane < M) gram[i * P + j] = s * inv * inv;
        }
    }
    __syncthreads();
    for (int step = 0; step < steps; ++step) {
        const float a = coeffs.c[step][0], b = coeffs.c[step][1], c = coeffs.c[step][2];
        ps_product<M>(gram, gram, poly, c, gram, b, a);                     // Q
        __syncthreads();
        if (step + 1 < steps) ps_product<M>(gram, poly, tmp);
        if (step == 0) {
            for (int t = threadIdx.x; t < M * P; t += PS_THREADS) total[t] = poly[t];
        } else {
            ps_product<M>(poly, total, other);
            float* t = total; total = other; other = t;
        }
        __syncthreads();
        if (step + 1 < steps) {
            ps_product<M>(poly, tmp, gram);                                 // Q (A Q)
            __syncthreads();
        }
    }
    // X <- T X, two columns a thread
    for (int w = threadIdx.x; w < k / 2; w += PS_THREADS) {
        float lo[M], hi[M];
#pragma unroll
        for (int l = 0; l < M; ++l) {
            const uint32_t v = reinterpret_cast<const uint32_t*>(xs + l * pitch)[w];
            lo[l] = __uint_as_float(v << 16);
            hi[l] = __uint_as_float(v & 0xffff0000u);
        }
        for (int i = 0; i < M; ++i) {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int l = 0; l < M; l += 4) {
                const float4 q = *reinterpret_cast<const float4*>(total + i * P + l);
                s0 = fmaf(q.x, lo[l], s0); s1 = fmaf(q.x, hi[l], s1);
                s0 = fmaf(q.y, lo[l + 1], s0); s1 = fmaf(q.y, hi[l + 1], s1);
                s0 = fmaf(q.z, lo[l + 2], s0); s1 = fmaf(q.z, hi[l + 2], s1);
                s0 = fmaf(q.w, lo[l + 3], s0); s1 = fmaf(q.w, hi[l + 3], s1);
            }
            reinterpret_cast<uint32_t*>(mine)[static_cast<long long>(i) * (k / 2) + w] = pack_bf16x2(s0 * inv, s1 * inv);
        }
    }
}

template <int M>
static cudaError_t launch_polar_rows(void* x, const float* sumsq, int n, int k, const PolarCoefficients& c, int steps, cudaStream_t s) {
    const int smem = 5 * M * (M + 4) * 4 + M * (k + 2) * 2;
    static int configured = 0;
    if (smem > configured) {
        cudaError_t e = cudaFuncSetAttribute(polar_small_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
        if (e != cudaSuccess) return e;
        configured = 232448;
    }
    polar_small_kernel<M><<<n, PS_THREADS, smem, s>>>(static_cast<__nv_bfloat16*>(x), sumsq, k, c, steps);
    return cudaGetLastError();
}

bool polar_small_supported(long long m, long long k, int steps) {
    return (m == 8 || m == 16 || m == 24 || m == 32) && k % 8 == 0 && steps >= 1 && steps <= 8 && 5 * m * (m + 4) * 4 + m * (k + 2) * 2 <= 232448;
}

cudaError_t launch_polar_small(void* x, const float* sumsq, int n, int m, int k, const float* coeffs, int steps, cudaStream_t s) {
    PolarCoefficients c;
    for (int i = 0; i < steps; ++i)
        for (int j = 0; j < 3; ++j) c.c[i][j] = coeffs[3 * i + j];
    switch (m) {
        case 8: return launch_polar_rows<8>(x, sumsq, n, k, c, steps, s);
        case 16: return launch_polar_rows<16>(x, sumsq, n, k, c, steps, s);
        case 24: return launch_polar_rows<24>(x, sumsq, n, k, c, steps, s);
        case 32: return launch_polar_rows<32>(x, sumsq, n, k, c, steps, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gm
