// Streaming fp32 cross-entropy over bf16 logits (forward + in-place gradient), AdamW, and the element-wise
// parts of Muon (momentum / Nesterov / bf16 pack, and the scaled weight update).
//
// Reference counterparts: `model/cross_entropy.py:12-69` (online-softmax CE, fp32 statistics, int64 row
// offsets), `model/loss.py:11-60` (gradients computed during the forward pass),
// `optimizers/polar_prepare.py:8-35` (momentum + Nesterov + bf16 pack), `optimizers/polar_express.py:325-377`
// (final update into fp32 master weights), torch's fused AdamW (`model/gpt.py:284-293`).
#include "../common/ptx.cuh"
#include "../kernels_decl.h"
#include <algorithm>

namespace gm {

// 2^x on the special-function unit (the softmax needs no more than its 2-ulp accuracy)
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// One block per row.  loss[row] = logsumexp(logits) - logits[target]; logits are overwritten by
// (softmax - onehot) * (*grad_scale) in bf16, zeros for ignored rows.  64-bit row offsets.  A target that is neither a class nor
// `ignore_index` is no address: the row's loss becomes NaN, its gradient zero, and the status word says so.
__device__ __forceinline__ bool outside(long long tgt, int vocab, long long ignore_index) {
    return tgt != ignore_index && (tgt < 0 || tgt >= vocab);
}

__global__ void __launch_bounds__(512)
ce_fwd_bwd_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets, float* __restrict__ loss,
                  const float* __restrict__ grad_scale, int vocab, long long row_stride, long long ignore_index, int write_grad, int* status) {
    __shared__ float red_m[16], red_s[16];
    const long long row = blockIdx.x;
    __nv_bfloat16* p = logits + row * row_stride;
    long long tgt = targets[row];
    if (!GM_IN_BOUNDS(tgt == ignore_index || (tgt >= 0 && tgt < vocab), 905)) tgt = ignore_index;      // checked build: the row is ignored
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int vec = vocab / 8;
    const bool bad = outside(tgt, vocab, ignore_index);
    if (tgt == ignore_index || bad) {
        if (threadIdx.x == 0) {
            loss[row] = bad ? __int_as_float(0x7fc00000) : 0.f;
            if (bad) atomicExch(status, 701);
        }
        if (write_grad) {
            for (int i = threadIdx.x; i < vec; i += blockDim.x) reinterpret_cast<uint4*>(p)[i] = make_uint4(0, 0, 0, 0);
            for (int i = vec * 8 + threadIdx.x; i < vocab; i += blockDim.x) p[i] = __float2bfloat16(0.f);
        }
        return;
    }
    float m = -INFINITY, s = 0.f;
    auto push = [&](float v) {
        if (v > m) { s = s * __expf(m - v) + 1.f; m = v; } else if (v != -INFINITY) { s += __expf(v - m); }      // -inf adds nothing, also to nothing
    };
    for (int i = threadIdx.x; i < vec; i += blockDim.x) {
        const uint4 raw = reinterpret_cast<const uint4*>(p)[i];
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int e = 0; e < 4; ++e) { const float2 f = __bfloat1622float2(h[e]); push(f.x); push(f.y); }
    }
    for (int i = vec * 8 + threadIdx.x; i < vocab; i += blockDim.x) push(__bfloat162float(p[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
        const float mm = fmaxf(m, m2);
        s = (m == -INFINITY ? 0.f : s * __expf(m - mm)) + (m2 == -INFINITY ? 0.f : s2 * __expf(m2 - mm));
        m = mm;
    }
    if (lane == 0) { red_m[warp] = m; red_s[warp] = s; }
    __syncthreads();
    float gm_ = red_m[0], gs = red_s[0];
    for (int w = 1; w < nwarps; ++w) {
        const float mm = fmaxf(gm_, red_m[w]);
        gs = (gm_ == -INFINITY ? 0.f : gs * __expf(gm_ - mm)) + (red_m[w] == -INFINITY ? 0.f : red_s[w] * __expf(red_m[w] - mm));
        gm_ = mm;
    }
    const float lse = gm_ + __logf(gs);
    if (threadIdx.x == 0) loss[row] = lse - __bfloat162float(p[tgt]);
    if (!write_grad) return;
    __syncthreads();     // every thread has read what it needs of the row before it is overwritten
    const float scale = *grad_scale;
    for (int i = threadIdx.x; i < vec; i += blockDim.x) {
        uint4 raw = reinterpret_cast<const uint4*>(p)[i];
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
        uint32_t* w = reinterpret_cast<uint32_t*>(&raw);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(h[e]);
            const int c = i * 8 + 2 * e;
            const float g0 = (__expf(f.x - lse) - (c == tgt ? 1.f : 0.f)) * scale;
            const float g1 = (__expf(f.y - lse) - (c + 1 == tgt ? 1.f : 0.f)) * scale;
            w[e] = pack_bf16x2(g0, g1);
        }
        reinterpret_cast<uint4*>(p)[i] = raw;
    }
    for (int i = vec * 8 + threadIdx.x; i < vocab; i += blockDim.x)
        p[i] = __float2bfloat16((__expf(__bfloat162float(p[i]) - lse) - (i == tgt ? 1.f : 0.f)) * scale);
}

// Same computation for rows that fit in shared memory (vocab a multiple of 8, up to 56 960 columns): the row arrives by bulk copies in
// four pieces, is read twice where it lies (maximum; sum of exponentials), turned into its gradient in place and leaves by bulk
// copies, a piece as soon as it is done.  Nothing of the row lives in registers, so two CTAs share an SM and one's copies run under the
// other's arithmetic: 8192 rows of 50304 columns take 330 us (5.0 TB/s),
// 412 us with the row in registers and one CTA per SM.  What is left above the copy rate is the exponentials, two per element.
constexpr int CE_THREADS = 512, CE_PIECES = 4;
constexpr int CE_MAX_BYTES = 113920;                       // two rows and their barriers in an SM's 227 KB

__global__ void __launch_bounds__(CE_THREADS, 2)
ce_fwd_bwd_bulk_kernel(__nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets, float* __restrict__ loss,
                       const float* __restrict__ grad_scale, int vocab, long long row_stride, long long ignore_index, int write_grad, int* status) {
    extern __shared__ __align__(128) uint8_t ce_smem[];
    __shared__ __align__(8) uint64_t full[CE_PIECES];
    __shared__ float red[CE_THREADS / 32];
    __shared__ float bcast;
    const long long row = blockIdx.x;
    __nv_bfloat16* p = logits + row * row_stride;
    long long tgt = targets[row];
    if (!GM_IN_BOUNDS(tgt == ignore_index || (tgt >= 0 && tgt < vocab), 905)) tgt = ignore_index;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int vec = vocab / 8;
    const bool bad = outside(tgt, vocab, ignore_index);
    if (tgt == ignore_index || bad) {
        if (threadIdx.x == 0) {
            loss[row] = bad ? __int_as_float(0x7fc00000) : 0.f;
            if (bad) atomicExch(status, 701);
        }
        if (write_grad)
            for (int i = threadIdx.x; i < vec; i += CE_THREADS) reinterpret_cast<uint4*>(p)[i] = make_uint4(0, 0, 0, 0);
        return;
    }
    uint4* v = reinterpret_cast<uint4*>(ce_smem);
    const int per = (vec + CE_PIECES - 1) / CE_PIECES;      // 16-byte units of a piece
    if (threadIdx.x == 0) {
        for (int k = 0; k < CE_PIECES; ++k) mbar_init(&full[k], 1);
        fence_barrier_init();
        fence_proxy_async();
        for (int k = 0; k < CE_PIECES; ++k) {
            const int first = min(k * per, vec), bytes = (min(first + per, vec) - first) * 16;
            mbar_expect_tx(&full[k], bytes);
            if (bytes > 0)
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_u32(v + first)), "l"(reinterpret_cast<const uint4*>(p) + first), "r"(bytes), "r"(smem_u32(&full[k])) : "memory");
        }
    }
    __syncthreads();
    auto block_max_or_sum = [&](float x, bool sum) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float y = __shfl_xor_sync(0xffffffffu, x, o);
            x = sum ? x + y : fmaxf(x, y);
        }
        __syncthreads();                                    // red / bcast are reused
        if (lane == 0) red[warp] = x;
        __syncthreads();
        if (threadIdx.x == 0) {
            float t = red[0];
#pragma unroll
            for (int w = 1; w < CE_THREADS / 32; ++w) t = sum ? t + red[w] : fmaxf(t, red[w]);
            bcast = t;
        }
        __syncthreads();
        return bcast;
    };
    constexpr float LOG2E = 1.4426950408889634f;
    __nv_bfloat162 mx2 = __halves2bfloat162(__ushort_as_bfloat16(0xff80), __ushort_as_bfloat16(0xff80));
    bool landed = true;
    for (int k = 0; k < CE_PIECES; ++k) {
        landed = mbar_wait(&full[k], 0) && landed;
        const int end = min((k + 1) * per, vec);
        for (int i = k * per + threadIdx.x; i < end; i += CE_THREADS) {
            const uint4 raw = v[i];
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
            mx2 = __hmax2(mx2, __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
        }
    }
    if (!landed) {                                          // whichever thread gave up: the row is void, and a late copy lands before the CTA ends
        atomicExch(status, 702);
        const long long start = clock64();
        while (clock64() - start < 200000) {}
    }
    const float gmax = block_max_or_sum(fmaxf(__bfloat162float(mx2.x), __bfloat162float(mx2.y)), false);
    const float mb = gmax * LOG2E;
    float s0 = 0.f, s1 = 0.f;
    for (int i = threadIdx.x; i < vec; i += CE_THREADS) {
        const uint4 raw = v[i];
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(h[e]);
            s0 += ex2_approx(fmaf(f.x, LOG2E, -mb));
            s1 += ex2_approx(fmaf(f.y, LOG2E, -mb));
        }
    }
    const float lse = gmax + __logf(block_max_or_sum(s0 + s1, true));
    if (threadIdx.x == 0) loss[row] = lse - __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(ce_smem)[tgt]);
    if (!write_grad) return;
    __syncthreads();                                        // the target logit has been read before the row is overwritten
    const float scale = *grad_scale, lb = lse * LOG2E;
    const int tvec = static_cast<int>(tgt >> 3), tsub = static_cast<int>(tgt & 7);
    for (int k = 0; k < CE_PIECES; ++k) {
        const int first = min(k * per, vec), end = min(first + per, vec);
        for (int i = first + threadIdx.x; i < end; i += CE_THREADS) {
            const uint4 raw = v[i];
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
            float g[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __bfloat1622float2(h[e]);
                g[2 * e] = ex2_approx(fmaf(f.x, LOG2E, -lb));
                g[2 * e + 1] = ex2_approx(fmaf(f.y, LOG2E, -lb));
            }
            if (i == tvec) {
#pragma unroll
                for (int e = 0; e < 8; ++e) g[e] -= e == tsub ? 1.f : 0.f;
            }
            uint4 o;
            o.x = pack_bf16x2(g[0] * scale, g[1] * scale); o.y = pack_bf16x2(g[2] * scale, g[3] * scale);
            o.z = pack_bf16x2(g[4] * scale, g[5] * scale); o.w = pack_bf16x2(g[6] * scale, g[7] * scale);
            v[i] = o;
        }
        fence_proxy_async();
        __syncthreads();
        if (threadIdx.x == 0 && end > first) {
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                         ::"l"(reinterpret_cast<uint4*>(p) + first), "r"(smem_u32(v + first)), "r"((end - first) * 16) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    }
    if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // shared memory goes to the next CTA
}

void launch_ce_fwd_bwd(void* logits, const long long* targets, float* loss, const float* grad_scale, int rows, int vocab,
                       long long row_stride, long long ignore_index, int write_grad, int* status, cudaStream_t s) {
    if (rows <= 0) return;
    if (vocab >= 8 && vocab % 8 == 0 && vocab * 2 <= CE_MAX_BYTES && row_stride % 8 == 0 && reinterpret_cast<uintptr_t>(logits) % 16 == 0) {
        cudaFuncSetAttribute(ce_fwd_bwd_bulk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CE_MAX_BYTES);
        ce_fwd_bwd_bulk_kernel<<<rows, CE_THREADS, vocab * 2, s>>>(static_cast<__nv_bfloat16*>(logits), targets, loss, grad_scale, vocab, row_stride,
                                                                  ignore_index, write_grad, status);
        return;
    }
    ce_fwd_bwd_kernel<<<rows, 512, 0, s>>>(static_cast<__nv_bfloat16*>(logits), targets, loss, grad_scale, vocab, row_stride,
                                           ignore_index, write_grad, status);
}

// ---- log-probabilities of given tokens from logits that somebody else keeps ------------------------------------------------
// Read-only: the row is streamed once, 64 bytes of it per thread and step; the maximum of a step is found on packed bf16 pairs, the
// sum is only rescaled when that maximum grows.  Exponents are differences of two logits times log2(e) and the target's logit meets the
// maximum before the logarithm joins, so that no rounding grows with the size of the logits (the difference of two bf16 numbers is exact
// or nearly so).  Bound by reading the logits: 8192 x 50304 take 135 us (6.1 TB/s), 32768 x 50304 0.60 ms where
// a cast to fp32, a log-softmax and a gather took 7.5 ms; 64 x 184 rows of which one in eight is scored 0.04 ms against 2.6 ms.
constexpr int LP_THREADS = 256, LP_UNROLL = 4;

// (max, sum of exp(x - max)) of one row, the same in every thread
__device__ __forceinline__ void row_statistics(const __nv_bfloat16* __restrict__ p, int vocab, bool vec16, float& m_out, float& s_out) {
    __shared__ float red_m[LP_THREADS / 32], red_s[LP_THREADS / 32];
    constexpr float kLog2e = 1.4426950408889634f;
    float m = -INFINITY, s = 0.f;
    const int vec = vec16 ? vocab / 8 : 0;
    for (int base = threadIdx.x; base < vec; base += LP_THREADS * LP_UNROLL) {
        uint4 raw[LP_UNROLL];
#pragma unroll
        for (int u = 0; u < LP_UNROLL; ++u) {
            const int i = base + u * LP_THREADS;
            raw[u] = i < vec ? __ldcs(reinterpret_cast<const uint4*>(p) + i) : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);
        }
        __nv_bfloat162 mx2 = *reinterpret_cast<const __nv_bfloat162*>(&raw[0]);
#pragma unroll
        for (int u = 0; u < LP_UNROLL; ++u) {
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[u]);
#pragma unroll
            for (int e = 0; e < 4; ++e) mx2 = __hmax2(mx2, h[e]);
        }
        const float mx = fmaxf(__bfloat162float(mx2.x), __bfloat162float(mx2.y));
        if (mx > m) { s *= ex2_approx((m - mx) * kLog2e); m = mx; }
        const float top = m == -INFINITY ? 0.f : m;
        float part[2] = {0.f, 0.f};
#pragma unroll
        for (int u = 0; u < LP_UNROLL; ++u) {
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw[u]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __bfloat1622float2(h[e]);
                part[0] += ex2_approx((f.x - top) * kLog2e);
                part[1] += ex2_approx((f.y - top) * kLog2e);
            }
        }
        s += part[0] + part[1];
    }
    for (int i = vec * 8 + threadIdx.x; i < vocab; i += LP_THREADS) {
        const float v = __bfloat162float(p[i]);
        if (v > m) { s *= ex2_approx((m - v) * kLog2e); m = v; }
        s += ex2_approx((v - (m == -INFINITY ? 0.f : m)) * kLog2e);
    }
    auto merge = [&](float m2, float s2) {
        const float mm = fmaxf(m, m2);
        s = (m == -INFINITY ? s : s * __expf(m - mm)) + (m2 == -INFINITY ? s2 : s2 * __expf(m2 - mm));
        m = mm;
    };
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o); merge(m2, s2); }
    if ((threadIdx.x & 31) == 0) { red_m[threadIdx.x >> 5] = m; red_s[threadIdx.x >> 5] = s; }
    __syncthreads();
    m = red_m[0]; s = red_s[0];
    for (int w = 1; w < LP_THREADS / 32; ++w) merge(red_m[w], red_s[w]);
    m_out = m;
    s_out = s;
}

// loss[row] = logsumexp(logits[row]) - logits[row, target]; 0 for ignored rows.  A target outside the vocabulary is no address: its row
// becomes NaN and the status word says so.
__global__ void __launch_bounds__(LP_THREADS)
row_nll_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets, float* __restrict__ loss, int vocab,
               long long row_stride, int vec16, long long ignore_index, int* status) {
    const long long row = blockIdx.x;
    const long long tgt = targets[row];
    const bool bad = outside(tgt, vocab, ignore_index);
    if (tgt == ignore_index || bad) {
        if (threadIdx.x == 0) {
            loss[row] = bad ? __int_as_float(0x7fc00000) : 0.f;
            if (bad) atomicExch(status, 701);
        }
        return;
    }
    const __nv_bfloat16* p = logits + row * row_stride;
    float m, s;
    row_statistics(p, vocab, vec16 != 0, m, s);
    if (threadIdx.x == 0) loss[row] = logf(s) + (m - __bfloat162float(p[tgt]));
}

// lp[i, j] = log p(tokens[i, j + 1] | row i up to j) for prefix[i] <= j + 1 < end[i], 0 elsewhere (those rows of the logits are not read)
__global__ void __launch_bounds__(LP_THREADS)
continuation_logprob_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ tokens, const long long* __restrict__ prefix,
                            const long long* __restrict__ end, float* __restrict__ lp, int length, int vocab, long long batch_stride,
                            long long row_stride, long long token_stride, int vec16, int* status) {
    const int j = blockIdx.x, i = blockIdx.y;
    float* dst = lp + static_cast<long long>(i) * (length - 1) + j;
    if (j + 1 < prefix[i] || j + 1 >= end[i]) {
        if (threadIdx.x == 0) *dst = 0.f;
        return;
    }
    const long long tok = tokens[i * token_stride + j + 1];
    if (tok < 0 || tok >= vocab) {
        if (threadIdx.x == 0) { *dst = __int_as_float(0x7fc00000); atomicExch(status, 701); }
        return;
    }
    const __nv_bfloat16* p = logits + i * batch_stride + j * row_stride;
    float m, s;
    row_statistics(p, vocab, vec16 != 0, m, s);
    if (threadIdx.x == 0) *dst = (__bfloat162float(p[tok]) - m) - logf(s);
}

void launch_row_nll(const void* logits, const long long* targets, float* loss, int rows, int vocab, long long row_stride, long long ignore_index,
                    int* status, cudaStream_t s) {
    if (rows == 0) return;
    const int vec16 = reinterpret_cast<uintptr_t>(logits) % 16 == 0 && row_stride % 8 == 0;
    row_nll_kernel<<<rows, LP_THREADS, 0, s>>>(static_cast<const __nv_bfloat16*>(logits), targets, loss, vocab, row_stride, vec16, ignore_index, status);
}

void launch_continuation_logprob(const void* logits, const long long* tokens, const long long* prefix, const long long* end, float* lp, int n, int length,
                                 int vocab, long long batch_stride, long long row_stride, long long token_stride, int* status, cudaStream_t s) {
    const int vec16 = reinterpret_cast<uintptr_t>(logits) % 16 == 0 && row_stride % 8 == 0 && batch_stride % 8 == 0;
    continuation_logprob_kernel<<<dim3(length - 1, n), LP_THREADS, 0, s>>>(static_cast<const __nv_bfloat16*>(logits), tokens, prefix, end, lp, length, vocab,
                                                                          batch_stride, row_stride, token_stride, vec16, status);
}

// ---- embedding gradient, added into the optimizer's buffer -----------------------------------------------------------------
// The gradient of an embedding table touches as many rows as there are tokens.  Formed as a tensor of the table's size it was filled with
// zeros, scattered into and added to the gradient buffer: three passes over 154 MB at 50304 x 768, whatever the number of tokens.  Here
// the tokens come sorted by id (stable, so every sum has the order of the positions) and runs of one id are summed and added to
// their row of the buffer: a CTA takes EMB_WINDOW sorted tokens, adds the runs that lie inside its window, and leaves the pieces of a
// run that crosses windows (the first and the last run of a window) in `edge`; the second kernel adds those up in window order.
// 32768 tokens of a 50304 x 768 table: 54 us and 36 for the sort, where torch's scatter, its sort, the fill and the addition took 560.
constexpr int EMB_WINDOW = 32;

__global__ void __launch_bounds__(256)
embedding_grad_kernel(const float* __restrict__ dy, const int* __restrict__ ids, const long long* __restrict__ order, float* __restrict__ grad,
                      float* __restrict__ edge, int tokens, int d, int vocab) {
    const int w0 = blockIdx.x * EMB_WINDOW, w1 = min(w0 + EMB_WINDOW, tokens);
    __shared__ int id_s[EMB_WINDOW + 2];
    __shared__ long long row_s[EMB_WINDOW];
    for (int i = threadIdx.x; i < EMB_WINDOW + 2; i += blockDim.x) {
        const int at = w0 - 1 + i;                                     // one neighbour on each side
        id_s[i] = at >= 0 && at < tokens ? ids[at] : -1;
        if (i < EMB_WINDOW && w0 + i < tokens) row_s[i] = order[w0 + i];
    }
    __syncthreads();
    const bool from_before = id_s[0] == id_s[1], goes_on = w1 < tokens && id_s[w1 - w0] == id_s[w1 - w0 + 1];
    for (int c = threadIdx.x * 4; c < d; c += blockDim.x * 4) {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        bool first_run = true;
        for (int i0 = 0; i0 < w1 - w0; i0 += 8) {
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)                                 // eight rows in flight
                v[u] = i0 + u < w1 - w0 ? __ldcs(reinterpret_cast<const float4*>(dy + row_s[i0 + u] * d + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int i = i0 + u;
                if (i >= w1 - w0) break;
                sum.x += v[u].x; sum.y += v[u].y; sum.z += v[u].z; sum.w += v[u].w;
                if (i + 1 < w1 - w0 && id_s[i + 2] == id_s[i + 1]) continue;            // the run goes on inside the window
                const long long id = id_s[i + 1];
                const bool last = i + 1 == w1 - w0;
                if (first_run && from_before) *reinterpret_cast<float4*>(edge + (2LL * blockIdx.x) * d + c) = sum;       // belongs to a run of earlier windows
                else if (last && goes_on) *reinterpret_cast<float4*>(edge + (2LL * blockIdx.x + 1) * d + c) = sum;      // starts here, ends later
                else if (GM_IN_BOUNDS(id >= 0 && id < vocab, 907) && id >= 0 && id < vocab) {
                    float4* g = reinterpret_cast<float4*>(grad + id * d + c);
                    float4 old = *g;
                    old.x += sum.x; old.y += sum.y; old.z += sum.z; old.w += sum.w;
                    *g = old;
                }
                sum = make_float4(0.f, 0.f, 0.f, 0.f);
                first_run = false;
            }
        }
    }
}

// one CTA per window in which a run starts that later windows continue
__global__ void __launch_bounds__(256)
embedding_grad_edges_kernel(const int* __restrict__ ids, const float* __restrict__ edge, float* __restrict__ grad, int tokens, int d, int vocab) {
    const int w0 = blockIdx.x * EMB_WINDOW, w1 = w0 + EMB_WINDOW;
    if (w1 >= tokens) return;
    const long long id = ids[w1 - 1];
    if (ids[w1] != id || id < 0 || id >= vocab) return;                 // the window's last run ends with it
    if (w0 > 0 && ids[w0 - 1] == id && ids[w0] == id) return;           // the run starts in an earlier window (this one holds nothing else)
    for (int c = threadIdx.x * 4; c < d; c += blockDim.x * 4) {
        float4 sum = *reinterpret_cast<const float4*>(edge + (2LL * blockIdx.x + 1) * d + c);
        for (int w = blockIdx.x + 1; static_cast<long long>(w) * EMB_WINDOW < tokens && ids[w * EMB_WINDOW] == id; ++w) {
            const float4 v = *reinterpret_cast<const float4*>(edge + 2LL * w * d + c);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
            const long long end = static_cast<long long>(w + 1) * EMB_WINDOW;
            if (end >= tokens || ids[end - 1] != id) break;
        }
        float4* g = reinterpret_cast<float4*>(grad + id * d + c);
        float4 old = *g;
        old.x += sum.x; old.y += sum.y; old.z += sum.z; old.w += sum.w;
        *g = old;
    }
}

void launch_embedding_grad(const float* dy, const int* ids, const long long* order, float* grad, float* edge, int tokens, int d, int vocab, cudaStream_t s) {
    if (tokens == 0) return;
    const int windows = (tokens + EMB_WINDOW - 1) / EMB_WINDOW, threads = d / 4 < 256 ? (d / 4 + 31) / 32 * 32 : 256;
    embedding_grad_kernel<<<windows, threads, 0, s>>>(dy, ids, order, grad, edge, tokens, d, vocab);
    embedding_grad_edges_kernel<<<windows, threads, 0, s>>>(ids, edge, grad, tokens, d, vocab);
}
int embedding_grad_windows(int tokens) { return (tokens + EMB_WINDOW - 1) / EMB_WINDOW; }

// ---- AdamW ---------------------------------------------------------------------------------------------
// p, g fp32; moments fp32 or bf16.  Decoupled weight decay; bias corrections passed in.  Optionally refreshes a
// bf16 copy of the parameter (the GEMM operand) in the same pass.
template <typename TM>
__global__ void __launch_bounds__(256)
adamw_kernel(float* __restrict__ p, const float* __restrict__ g, TM* __restrict__ m, TM* __restrict__ v,
             __nv_bfloat16* __restrict__ p_bf16, long long n, float lr, float beta1, float beta2, float eps, float wd,
             float bc1, float bc2_sqrt, float grad_scale) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n; i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const float grad = g[i] * grad_scale;
        float mi, vi;
        if constexpr (sizeof(TM) == 4) { mi = m[i]; vi = v[i]; } else { mi = __bfloat162float(m[i]); vi = __bfloat162float(v[i]); }
        mi = beta1 * mi + (1.f - beta1) * grad;
        vi = beta2 * vi + (1.f - beta2) * grad * grad;
        if constexpr (sizeof(TM) == 4) { m[i] = mi; v[i] = vi; } else { m[i] = __float2bfloat16(mi); v[i] = __float2bfloat16(vi); }
        float w = p[i] * (1.f - lr * wd);
        w -= lr / bc1 * mi / (sqrtf(vi) / bc2_sqrt + eps);
        p[i] = w;
        if (p_bf16) p_bf16[i] = __float2bfloat16(w);
    }
}

void launch_adamw(float* p, const float* g, void* m, void* v, bool moments_bf16, void* p_bf16, long long n, float lr, float beta1,
                  float beta2, float eps, float wd, float bc1, float bc2_sqrt, float grad_scale, cudaStream_t s) {
    const int blocks = static_cast<int>(std::min<long long>((n + 255) / 256, 2368LL));
    if (moments_bf16)
        adamw_kernel<__nv_bfloat16><<<blocks, 256, 0, s>>>(p, g, static_cast<__nv_bfloat16*>(m), static_cast<__nv_bfloat16*>(v),
                                                           static_cast<__nv_bfloat16*>(p_bf16), n, lr, beta1, beta2, eps, wd, bc1, bc2_sqrt, grad_scale);
    else
        adamw_kernel<float><<<blocks, 256, 0, s>>>(p, g, static_cast<float*>(m), static_cast<float*>(v),
                                                   static_cast<__nv_bfloat16*>(p_bf16), n, lr, beta1, beta2, eps, wd, bc1, bc2_sqrt, grad_scale);
}

// ---- Muon element-wise stages -----------------------------------------------------------------------------
// For matrix i of a same-shape bucket (pointer tables on the device):
//   buf = momentum*buf + g ;  u = nesterov ? g + momentum*buf : buf ;  packed[i] = bf16(u), transposed if tall
// and per-matrix sum of squares of bf16(u) (for the Frobenius normalisation) accumulated into sumsq[i].
// 32x32 tiles through shared memory keep both the row-major reads and the (possibly transposed) writes coalesced.
__global__ void __launch_bounds__(256)
muon_prepare_kernel(const float* const* __restrict__ grads, float* const* __restrict__ bufs, __nv_bfloat16* __restrict__ packed,
                    float* __restrict__ sumsq, int rows, int cols, long long g_stride, long long b_stride, float momentum,
                    int nesterov, int transpose, float grad_scale) {
    __shared__ float tile[32][33];
    __shared__ float part[8];
    const int mat = blockIdx.z;
    const float* g = grads[mat];
    float* buf = bufs[mat];
    __nv_bfloat16* out = packed + static_cast<long long>(mat) * rows * cols;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    float local = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = r0 + ty + 8 * i, c = c0 + tx;
        float u = 0.f;
        if (r < rows && c < cols) {
            const float grad = g[r * g_stride + c] * grad_scale;
            float b = buf[r * b_stride + c] * momentum;
            b = b + grad;
            buf[r * b_stride + c] = b;
            u = __bfloat162float(__float2bfloat16(nesterov ? fmaf(momentum, b, grad) : b));
            if (!transpose) out[static_cast<long long>(r) * cols + c] = __float2bfloat16(u);
        }
        tile[ty + 8 * i][tx] = u;
        local += u * u;
    }
    if (transpose) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = c0 + ty + 8 * i, r = r0 + tx;          // out is [cols][rows]
            if (r < rows && c < cols) out[static_cast<long long>(c) * rows + r] = __float2bfloat16(tile[tx][ty + 8 * i]);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
    if (tx == 0) part[ty] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int w = 0; w < 8; ++w) t += part[w];
        atomicAdd(&sumsq[mat], t);
    }
}

// x[i] *= 1 / (sqrt(sumsq[mat]) * 1.02 + 1e-6)   (spectral norm <= 1 before the first iteration)
__global__ void __launch_bounds__(256)
muon_normalize_kernel(__nv_bfloat16* __restrict__ packed, const float* __restrict__ sumsq, long long per_matrix) {
    const int mat = blockIdx.y;
    const float inv = 1.f / (sqrtf(sumsq[mat]) * 1.02f + 1e-6f);
    uint4* x = reinterpret_cast<uint4*>(packed + mat * per_matrix);
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < per_matrix / 8; i += static_cast<long long>(gridDim.x) * blockDim.x) {
        uint4 raw = x[i];
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(h[e]);
            h[e] = __floats2bfloat162_rn(f.x * inv, f.y * inv);
        }
        x[i] = raw;
    }
}

// W[i] += alpha * O[i] (O bf16, stored transposed when the matrix is tall); optionally refresh the bf16 copy of W
__global__ void __launch_bounds__(256)
muon_apply_kernel(float* const* __restrict__ weights, __nv_bfloat16* const* __restrict__ weights_bf16,
                  const __nv_bfloat16* __restrict__ update, int rows, int cols, long long w_stride, float alpha, int transpose) {
    __shared__ float tile[32][33];
    const int mat = blockIdx.z;
    float* w = weights[mat];
    __nv_bfloat16* wb = weights_bf16 ? weights_bf16[mat] : nullptr;
    const __nv_bfloat16* o = update + static_cast<long long>(mat) * rows * cols;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    if (transpose) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int c = c0 + ty + 8 * i, r = r0 + tx;          // update is [cols][rows]
            tile[ty + 8 * i][tx] = (r < rows && c < cols) ? __bfloat162float(o[static_cast<long long>(c) * rows + r]) : 0.f;
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = r0 + ty + 8 * i, c = c0 + tx;
        if (r < rows && c < cols) {
            const float upd = transpose ? tile[tx][ty + 8 * i] : __bfloat162float(o[static_cast<long long>(r) * cols + c]);
            const float nw = w[r * w_stride + c] + alpha * upd;
            w[r * w_stride + c] = nw;
            if (wb) wb[r * w_stride + c] = __float2bfloat16(nw);
        }
    }
}

void launch_muon_prepare(const float* const* grads, float* const* bufs, void* packed, float* sumsq, int n_mats, int rows, int cols,
                         long long g_stride, long long b_stride, float momentum, int nesterov, int transpose, float grad_scale,
                         cudaStream_t s) {
    const long long n = static_cast<long long>(rows) * cols;
    dim3 grid((cols + 31) / 32, (rows + 31) / 32, n_mats);
    muon_prepare_kernel<<<grid, 256, 0, s>>>(grads, bufs, static_cast<__nv_bfloat16*>(packed), sumsq, rows, cols, g_stride, b_stride,
                                             momentum, nesterov, transpose, grad_scale);
    dim3 grid2(static_cast<unsigned>(std::min<long long>((n / 8 + 255) / 256, 592LL)), n_mats);
    muon_normalize_kernel<<<grid2, 256, 0, s>>>(static_cast<__nv_bfloat16*>(packed), sumsq, n);
}

void launch_muon_normalize(void* packed, const float* sumsq, int n_mats, long long per_matrix, cudaStream_t s) {
    dim3 grid(static_cast<unsigned>(std::min<long long>((per_matrix / 8 + 255) / 256, 592LL)), n_mats);
    muon_normalize_kernel<<<grid, 256, 0, s>>>(static_cast<__nv_bfloat16*>(packed), sumsq, per_matrix);
}

void launch_muon_apply(float* const* weights, void* const* weights_bf16, const void* update, int n_mats, int rows, int cols,
                       long long w_stride, float alpha, int transpose, cudaStream_t s) {
    dim3 grid((cols + 31) / 32, (rows + 31) / 32, n_mats);
    muon_apply_kernel<<<grid, 256, 0, s>>>(weights, reinterpret_cast<__nv_bfloat16* const*>(weights_bf16),
                                           static_cast<const __nv_bfloat16*>(update), rows, cols, w_stride, alpha, transpose);
}

// dst_bf16 = bf16(src_fp32)  (compute copies of weights; n elements)
__global__ void __launch_bounds__(256) cast_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n) {
    for (long long i = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) * 4; i < n; i += static_cast<long long>(gridDim.x) * blockDim.x * 4) {
        if (i + 4 <= n) {
            const float4 f = *reinterpret_cast<const float4*>(src + i);
            uint2 o;
            o.x = pack_bf16x2(f.x, f.y);
            o.y = pack_bf16x2(f.z, f.w);
            *reinterpret_cast<uint2*>(dst + i) = o;
        } else {
            for (long long j = i; j < n; ++j) dst[j] = __float2bfloat16(src[j]);
        }
    }
}
void launch_cast_bf16(const float* src, void* dst, long long n, cudaStream_t s) {
    const int blocks = static_cast<int>(std::min<long long>((n / 4 + 255) / 256 + 1, 2368LL));
    cast_bf16_kernel<<<blocks, 256, 0, s>>>(src, static_cast<__nv_bfloat16*>(dst), n);
}

GM_DEFINE_BOUNDS_READER(loss)

}  // namespace gm
