// Many new tokens against the latent cache (a chunk of a prompt): attention over EXPANDED keys and values.
//
// The absorbed form of mla_decode.cu scores a query head against the latent itself, 2 (2 rank + rope) operations per head, query and
// position.  That is right while few queries share a position; with many it is cheaper to expand each visible position once per call,
//   k_content[s, h] = W_k[h] latent[s],  v[s, h] = W_v[h] latent[s]          (2 x 64 columns per head),
// and attend with 64 + 64-wide keys and 64-wide values: at rank 512 an eighth of the operations, on 128-row tcgen05 tiles.
// The numbers that are fp32 in the absorbed form keep more than its precision: W as two bf16 terms (16 bits of mantissa) in the
// expansion, whose fp32 sums are split into two bf16 terms per key and value, queries (after rotation and gain) and probabilities as two
// terms; products of a high and a low part are kept, fp32 accumulation throughout.  The latent and the rotary key are bf16 in the cache.
// Launches: mla_prefill_prepare (latent norm, rotations, query gains, cache rows of the new tokens; W's two terms, formed in every call:
// nothing of a weight is kept), two GEMMs (gemm_bf16.cu: W's low and high term, the second accumulating), mla_prefill_split (key gains of
// the new tokens, terms of keys and values), mla_prefill_attention.
// Measured (16 heads, rank 512, 2 x 512 tokens after 1500), layer with its projections: 170 us, 160 of them kernels (GEMMs 73, attention 61, split
// 14, prepare with W's terms 13), against 1193 us for the absorbed kernels; error of the layer's output against 64 bits 4.1e-3 (the fp32
// formulation that both forms replaced, whose W products ran in TF32, 5.9e-3; with the queries as one term 4.5e-3 and 162 us).
// mla_prefill_wanted in bindings_ops.cpp says which calls come here.
#include "../common/ptx.cuh"
#include "../kernels_decl.h"
#include "attn.h"
#include "attn_math.cuh"

namespace gm {

namespace {

__device__ __forceinline__ float pf_warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct PrefillPrepareParams {
    const __nv_bfloat16 *query, *low;            // [tokens, H * 128], [tokens, r + 64]
    long long q_pitch, low_pitch;
    const float *norm_w, *cos, *sin, *q_scale;   // tables: row of the first new position
    __nv_bfloat16 *latent, *rope;                // cache rows of the first new position
    long long latent_bs, rope_bs;
    __nv_bfloat16* q_out;                        // [2 terms, tokens, H * 128]
    int tokens, T, H, r, rms;
    float norm_eps, qk_eps, smin, smax;
    const float* w;                              // W [Hk * 128, r]: its two bf16 terms are formed by the first blocks
    __nv_bfloat16 *w_hi, *w_lo;
    int w_pieces, w_blocks;                      // pieces of four values
};

// W = high + low term + (at most 2^-17 of it) in the first `w_blocks` CTAs; then one CTA per token: warp 0 also does the latent and the rotary
// key; every warp takes query heads, a lane four columns
__global__ void __launch_bounds__(256)
mla_prefill_prepare_kernel(const PrefillPrepareParams p) {
    if (static_cast<int>(blockIdx.x) < p.w_blocks) {
        for (int i = blockIdx.x * 256 + threadIdx.x; i < p.w_pieces; i += p.w_blocks * 256) {
            const float4 x = reinterpret_cast<const float4*>(p.w)[i];
            const uint32_t h0 = pack_bf16x2(x.x, x.y), h1 = pack_bf16x2(x.z, x.w);
            reinterpret_cast<uint2*>(p.w_hi)[i] = make_uint2(h0, h1);
            reinterpret_cast<uint2*>(p.w_lo)[i] = make_uint2(pack_bf16x2(x.x - __uint_as_float(h0 << 16), x.y - __uint_as_float(h0 & 0xffff0000u)),
                                                             pack_bf16x2(x.z - __uint_as_float(h1 << 16), x.w - __uint_as_float(h1 & 0xffff0000u)));
        }
        return;
    }
    const int tok = blockIdx.x - p.w_blocks, b = tok / p.T, t = tok - b * p.T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool rot = lane >= 16;                                     // columns 64 .. 127 of a head: pairs 2 (lane - 16), + 1
    float c0 = 1.f, s0 = 0.f, c1 = 1.f, s1 = 0.f;
    if (rot) {
        const int pair = t * 32 + (lane - 16) * 2;
        c0 = p.cos[pair]; s0 = p.sin[pair]; c1 = p.cos[pair + 1]; s1 = p.sin[pair + 1];
    }
    if (warp == 0) {
        const __nv_bfloat16* src = p.low + tok * p.low_pitch;
        float sq = 0.f;
        for (int i = lane; i < p.r; i += 32) { const float v = __bfloat162float(src[i]); sq += v * v; }
        const float rstd = rsqrtf(pf_warp_sum(sq) / p.r + p.norm_eps);
        __nv_bfloat16* dst = p.latent + b * p.latent_bs + static_cast<long long>(t) * p.r;
        for (int i = lane; i < p.r; i += 32) dst[i] = __float2bfloat16(__bfloat162float(src[i]) * rstd * (p.norm_w ? p.norm_w[i] : 1.f));
        if (rot) {
            const int col = (lane - 16) * 4;
            const __nv_bfloat16* k = src + p.r + col;
            const float x0 = __bfloat162float(k[0]), x1 = __bfloat162float(k[1]), x2 = __bfloat162float(k[2]), x3 = __bfloat162float(k[3]);
            __nv_bfloat16* dr = p.rope + b * p.rope_bs + static_cast<long long>(t) * 64 + col;
            dr[0] = __float2bfloat16(x0 * c0 - x1 * s0); dr[1] = __float2bfloat16(x0 * s0 + x1 * c0);
            dr[2] = __float2bfloat16(x2 * c1 - x3 * s1); dr[3] = __float2bfloat16(x2 * s1 + x3 * c1);
        }
    }
    for (int h = warp; h < p.H; h += 8) {
        const uint2 raw = *reinterpret_cast<const uint2*>(p.query + tok * p.q_pitch + h * 128 + lane * 4);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), d = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        float gain = 1.f;
        if (p.q_scale) {
            const float sq = pf_warp_sum(a.x * a.x + a.y * a.y + d.x * d.x + d.y * d.y);       // a rotation keeps the norm
            gain = rsqrtf((p.rms ? sq / 128.f : sq) + p.qk_eps) * fminf(fmaxf(p.q_scale[h], p.smin), p.smax);
        }
        const float x0 = (a.x * c0 - a.y * s0) * gain, x1 = (a.x * s0 + a.y * c0) * gain;
        const float x2 = (d.x * c1 - d.y * s1) * gain, x3 = (d.x * s1 + d.y * c1) * gain;
        const uint32_t hi0 = pack_bf16x2(x0, x1), hi1 = pack_bf16x2(x2, x3);
        __nv_bfloat16* out = p.q_out + static_cast<long long>(tok) * p.H * 128 + h * 128 + lane * 4;
        *reinterpret_cast<uint2*>(out) = make_uint2(hi0, hi1);
        *reinterpret_cast<uint2*>(out + static_cast<long long>(p.tokens) * p.H * 128) =
            make_uint2(pack_bf16x2(x0 - __uint_as_float(hi0 << 16), x1 - __uint_as_float(hi0 & 0xffff0000u)),
                       pack_bf16x2(x2 - __uint_as_float(hi1 << 16), x3 - __uint_as_float(hi1 & 0xffff0000u)));
    }
}

struct PrefillSplitParams {
    const float* kv;                             // [B, S, Hk, 128] content | value, positions base .. base + S - 1
    const __nv_bfloat16* rope;                   // cache rows of position base
    __nv_bfloat16* key_gain;                     // cache rows of position base
    long long rope_bs, gain_bs;
    const float* k_scale;
    __nv_bfloat16 *k_hi, *k_lo, *v_hi, *v_lo;    // [B, S, Hk * 64]
    float* gain;                                 // [B, Hk, S_pad]: key gain * softmax scale * log2(e); 0 past S
    int S, S_pad, Hk, new_from, rms;             // positions >= new_from (relative to base) have no gain in the cache yet
    float qk_eps, smin, smax, scale_log2e;
};

// one warp per (position, kv head), a lane four of the 128 columns; bound by its 8 + 8 bytes per column pair
__global__ void __launch_bounds__(256)
mla_prefill_split_kernel(const PrefillSplitParams p) {
    const int lane = threadIdx.x & 31, b = blockIdx.y;
    const long long unit = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    const int s = static_cast<int>(unit / p.Hk), h = static_cast<int>(unit - static_cast<long long>(s) * p.Hk);
    if (s >= p.S_pad) return;
    float* gain_out = p.gain + (static_cast<long long>(b) * p.Hk + h) * p.S_pad + s;
    if (s >= p.S) {
        if (lane == 0) *gain_out = 0.f;
        return;
    }
    const long long row = (static_cast<long long>(b) * p.S + s) * p.Hk + h;
    const float4 x = *reinterpret_cast<const float4*>(p.kv + row * 128 + lane * 4);
    const float v[4] = {x.x, x.y, x.z, x.w};
    uint32_t hi[2], lo[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float h0 = __bfloat162float(__float2bfloat16(v[2 * e])), h1 = __bfloat162float(__float2bfloat16(v[2 * e + 1]));
        hi[e] = pack_bf16x2(h0, h1);
        lo[e] = pack_bf16x2(v[2 * e] - h0, v[2 * e + 1] - h1);
    }
    const bool value = lane >= 16;
    const long long at = row * 64 + (lane & 15) * 4;
    *reinterpret_cast<uint2*>((value ? p.v_hi : p.k_hi) + at) = make_uint2(hi[0], hi[1]);
    *reinterpret_cast<uint2*>((value ? p.v_lo : p.k_lo) + at) = make_uint2(lo[0], lo[1]);
    __nv_bfloat16* cached = p.key_gain + b * p.gain_bs + static_cast<long long>(s) * p.Hk + h;
    __nv_bfloat16 g;
    if (s >= p.new_from) {                                           // uniform across the warp
        float sq = 0.f;
        if (!value) {
            const __nv_bfloat16* r = p.rope + b * p.rope_bs + static_cast<long long>(s) * 64 + lane * 4;
#pragma unroll
            for (int e = 0; e < 4; ++e) { const float y = __bfloat162float(r[e]); sq += v[e] * v[e] + y * y; }
        }
        sq = pf_warp_sum(sq);
        g = __float2bfloat16(p.k_scale ? rsqrtf((p.rms ? sq / 128.f : sq) + p.qk_eps) * fminf(fmaxf(p.k_scale[h], p.smin), p.smax) : 1.f);
        if (lane == 0) *cached = g;
    } else {
        g = *cached;
    }
    if (lane == 0) *gain_out = __bfloat162float(g) * p.scale_log2e;
}

constexpr int PF_M = 128, PF_N = 128, PF_THREADS = 288;
constexpr int PF_SLAB = 128 * 64 * 2;            // 128 rows x 64 bf16 columns
constexpr int PF_STAGES = 2;
constexpr int PF_Q_BYTES = 4 * PF_SLAB;          // content and rotary columns, high terms then low
constexpr int PF_K_BYTES = 3 * PF_SLAB, PF_V_BYTES = 2 * PF_SLAB;      // content high, low and rotary; value high, low
constexpr uint32_t PF_TMEM_COLS = 512;
constexpr int PF_SMEM = PF_Q_BYTES + PF_STAGES * (PF_K_BYTES + PF_V_BYTES) + 1024 + 128 + 2 * PF_M * 4;
static_assert(PF_SMEM <= 232448, "shared memory of the prefill attention");

struct PrefillAttnParams {
    int T, H, group, S, S_pad, start, window;    // positions relative to the first expanded one; window < 0: none
    const float* gain;                           // [B, Hk, S_pad]
    __nv_bfloat16* out;                          // [B, T, H * 64]
    int* status;
};

// The roles, barriers and the running softmax are those of attn_fwd_kernel (attn_fwd.cu): warp 8 loads and issues, warps 0-7 are the
// softmax warps, w and w + 4 sharing the rows of a TMEM quadrant.  Different here: a score is the sum of five products (query content with
// both terms of the key, the low term of the query with the high one, both terms of the query's rotary part with the shared rotary key)
// times the key's gain, which every thread reads as it goes (all rows read the same one: one cache line per 32 keys); probabilities leave as two terms; P V is lo*hi + hi*lo + hi*hi.
__global__ void __launch_bounds__(PF_THREADS, 1)
mla_prefill_attention_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kh,
                             const __grid_constant__ CUtensorMap tmap_kl, const __grid_constant__ CUtensorMap tmap_rope, const __grid_constant__ CUtensorMap tmap_vh,
                             const __grid_constant__ CUtensorMap tmap_vl, const PrefillAttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sq = smem;
    uint8_t* sk = sq + PF_Q_BYTES;
    uint8_t* sv = sk + PF_STAGES * PF_K_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sv + PF_STAGES * PF_V_BYTES);
    uint64_t *bar_q = bars, *bar_s = bars + 1, *bar_p = bars + 2, *bar_o = bars + 3, *bar_k = bars + 4, *bar_v = bar_k + PF_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_v + PF_STAGES);
    float* row_stat = reinterpret_cast<float*>(bars + 16);           // [2 halves][128 rows]

    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int head = blockIdx.x, batch = blockIdx.y, q0 = (gridDim.z - 1 - blockIdx.z) * PF_M;      // the rows that see most first
    const int kv_head = head / p.group;
    const int first_pos = p.start + q0;                              // position of the tile's first query
    const int window = p.window < 0 ? p.S : p.window;
    const int lo = max(0, first_pos - window) & ~(PF_N - 1);
    const int hi = min(first_pos + PF_M - 1, p.S - 1);
    const int n_tiles = (hi - lo) / PF_N + 1;

    if (threadIdx.x == 0) {
        mbar_init(bar_q, 1); mbar_init(bar_s, 1); mbar_init(bar_p, 256); mbar_init(bar_o, 1);
        for (int st = 0; st < PF_STAGES; ++st) { mbar_init(&bar_k[st], 1); mbar_init(&bar_v[st], 1); }
        fence_barrier_init();
    }
    if (warp == 8) { tmem_alloc(tmem_slot, PF_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = uniform(*tmem_slot);
    const uint32_t tmem_s = tmem_base, tmem_ph = tmem_base + 128, tmem_pl = tmem_base + 192, tmem_pv = tmem_base + 256;
    bool ok = true;

    if (warp == 8) {
        {
            const uint32_t on = elect_one();
            constexpr uint32_t idesc_s = make_idesc_bf16(PF_M, PF_N, false, false);
            constexpr uint32_t idesc_pv = make_idesc_bf16(PF_M, 64, false, true);
            const uint64_t q_desc = make_smem_desc(smem_u32(sq), 16, 1024), k_desc = make_smem_desc(smem_u32(sk), 16, 1024);
            const uint64_t v_desc = make_smem_desc(smem_u32(sv), PF_N * 128, 1024);
            auto issue_s = [&](int st) {
                const uint64_t kd = k_desc + st * (PF_K_BYTES >> 4);
#pragma unroll
                for (int part = 0; part < 5; ++part) {               // small ones first: Q K low, Q low K, Q low rotary; Q K, Q rotary
                    constexpr int q_slab[5] = {0, 2, 3, 0, 1}, k_slab[5] = {1, 0, 2, 0, 2};
#pragma unroll
                    for (int k4 = 0; k4 < 4; ++k4)
                        umma_f16(tmem_s, q_desc + q_slab[part] * (PF_SLAB >> 4) + k4 * 2, kd + k_slab[part] * (PF_SLAB >> 4) + k4 * 2, idesc_s, (part | k4) != 0, on);
                }
                umma_commit(bar_s, on);
            };
            auto load_k = [&](int tile) {
                const int st = tile % PF_STAGES;
                uint8_t* dst = sk + st * PF_K_BYTES;
                if (on) mbar_expect_tx(&bar_k[st], PF_K_BYTES);
                tma_load_3d(dst, &tmap_kh, &bar_k[st], kv_head * 64, lo + tile * PF_N, batch, on);
                tma_load_3d(dst + PF_SLAB, &tmap_kl, &bar_k[st], kv_head * 64, lo + tile * PF_N, batch, on);
                tma_load_3d(dst + 2 * PF_SLAB, &tmap_rope, &bar_k[st], 0, lo + tile * PF_N, batch, on);
            };
            auto load_v = [&](int tile) {
                const int st = tile % PF_STAGES;
                uint8_t* dst = sv + st * PF_V_BYTES;
                if (on) mbar_expect_tx(&bar_v[st], PF_V_BYTES);
                tma_load_3d(dst, &tmap_vh, &bar_v[st], kv_head * 64, lo + tile * PF_N, batch, on);
                tma_load_3d(dst + PF_SLAB, &tmap_vl, &bar_v[st], kv_head * 64, lo + tile * PF_N, batch, on);
            };
            if (on) mbar_expect_tx(bar_q, PF_Q_BYTES);
#pragma unroll
            for (int sl = 0; sl < 4; ++sl)
                tma_load_3d(sq + sl * PF_SLAB, &tmap_q, bar_q, head * 128 + (sl & 1) * 64, q0, batch + (sl >> 1) * gridDim.y, on);
            for (int t = 0; t < PF_STAGES && t < n_tiles; ++t) { load_k(t); load_v(t); }
            if (!warp_wait(bar_q, 0) || !warp_wait(&bar_k[0], 0)) { atomicExch(p.status, 231); ok = false; }
            if (ok) { tc_fence_after(); issue_s(0); }
            for (int j = 0; j < n_tiles && ok; ++j) {
                const uint32_t ph = j & 1;
                const int st = j % PF_STAGES;
                const uint32_t st_ph = (j / PF_STAGES) & 1;
                if (!warp_wait(bar_s, ph)) { atomicExch(p.status, 232); ok = false; break; }
                if (j + PF_STAGES < n_tiles) load_k(j + PF_STAGES);            // S_j has consumed its key tile: refill the stage
                if (!warp_wait(bar_p, ph) || !warp_wait(&bar_v[st], st_ph)) { atomicExch(p.status, 233); ok = false; break; }
                tc_fence_after();
                const uint64_t vd = v_desc + st * (PF_V_BYTES >> 4);
#pragma unroll
                for (int part = 0; part < 3; ++part)                 // P low x V high, P high x V low, P high x V high
#pragma unroll
                    for (int k8 = 0; k8 < PF_N / 16; ++k8)
                        umma_f16_ta(tmem_pv, (part == 0 ? tmem_pl : tmem_ph) + k8 * 8, vd + (part == 1 ? (PF_SLAB >> 4) : 0) + k8 * 128, idesc_pv, (part | k8) != 0, on);
                umma_commit(bar_o, on);
                if (j + 1 < n_tiles) {
                    const int nst = (j + 1) % PF_STAGES;
                    if (!warp_wait(&bar_k[nst], ((j + 1) / PF_STAGES) & 1)) { atomicExch(p.status, 234); ok = false; break; }
                    tc_fence_after();
                    issue_s(nst);
                }
                if (!warp_wait(bar_o, ph)) { atomicExch(p.status, 235); ok = false; break; }
                if (j + PF_STAGES < n_tiles) load_v(j + PF_STAGES);            // PV_j has consumed its value tile
            }
        }
    } else {
        const int quad = warp & 3, half = warp >> 2;
        const int r = quad * 32 + lane;
        const int qpos = first_pos + r;
        const bool live = q0 + r < p.T;
        const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
        const uint32_t s_addr = tmem_s + lane_off + half * 64, ph_addr = tmem_ph + lane_off + half * 32, pl_addr = tmem_pl + lane_off + half * 32;
        const int bar_id = 1 + quad;
        float m = -INFINITY, l = 0.f, o[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0.f;
        for (int j = 0; j < n_tiles; ++j) {
            const uint32_t ph = j & 1;
            const int tile0 = lo + j * PF_N, kv0 = tile0 + half * 64;
            const float* gain = p.gain + (static_cast<long long>(batch) * (p.H / p.group) + kv_head) * p.S_pad + kv0;
            if (ok && !mbar_wait(bar_s, ph)) { atomicExch(p.status, 236); ok = false; }
            tc_fence_after();
            const bool need_mask = tile0 + PF_N - 1 > first_pos || first_pos + PF_M - 1 - tile0 > window;
            float v[64];
            {
                uint32_t raw[32];
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) {
                    tmem_ld_32x32b_x32(s_addr + cc * 32, raw);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        const float4 g = __ldg(reinterpret_cast<const float4*>(gain + cc * 32 + i));
                        v[cc * 32 + i] = __uint_as_float(raw[i]) * g.x; v[cc * 32 + i + 1] = __uint_as_float(raw[i + 1]) * g.y;
                        v[cc * 32 + i + 2] = __uint_as_float(raw[i + 2]) * g.z; v[cc * 32 + i + 3] = __uint_as_float(raw[i + 3]) * g.w;
                    }
                }
            }
            if (need_mask) {
#pragma unroll
                for (int i = 0; i < 64; ++i) {
                    const int kpos = kv0 + i;
                    if (kpos > qpos || qpos - kpos > window) v[i] = -INFINITY;
                }
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < 64; ++i) mx[i & 3] = fmaxf(mx[i & 3], v[i]);
            float tile_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            row_stat[half * PF_M + r] = tile_max;
            asm volatile("bar.sync %0, 64;" ::"r"(bar_id) : "memory");
            tile_max = fmaxf(tile_max, row_stat[(half ^ 1) * PF_M + r]);
            const float m_new = fmaxf(m, tile_max);
            const float base = m_new == -INFINITY ? 0.f : m_new;                 // a row may have no visible key yet
            const float alpha = exp2f(m - base);
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                uint32_t high[16], low[16];
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float e0 = exp2f(v[cc * 32 + i] - base), e1 = exp2f(v[cc * 32 + i + 1] - base);
                    sum[i & 3] += e0;
                    sum[(i + 1) & 3] += e1;
                    const uint32_t hp = pack_bf16x2(e0, e1);
                    high[i >> 1] = hp;
                    low[i >> 1] = pack_bf16x2(e0 - __uint_as_float(hp << 16), e1 - __uint_as_float(hp & 0xffff0000u));
                }
                tmem_st_32x32b_x16(ph_addr + cc * 16, high);
                tmem_st_32x32b_x16(pl_addr + cc * 16, low);
            }
            tmem_st_wait();
            l = l * alpha + (sum[0] + sum[1]) + (sum[2] + sum[3]);
            m = m_new;
            tc_fence_before();
            mbar_arrive(bar_p);
            if (ok && !mbar_wait(bar_o, ph)) { atomicExch(p.status, 237); ok = false; }
            tc_fence_after();
            {
                uint32_t oreg[32];
                tmem_ld_32x32b_x32(tmem_pv + lane_off + half * 32, oreg);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = o[i] * alpha + __uint_as_float(oreg[i]);
            }
            tc_fence_before();
            asm volatile("bar.sync %0, 64;" ::"r"(bar_id) : "memory");         // partner has read this tile's maximum
        }
        row_stat[half * PF_M + r] = l;
        asm volatile("bar.sync %0, 64;" ::"r"(bar_id) : "memory");
        l += row_stat[(half ^ 1) * PF_M + r];
        if (ok && live) {
            const float inv = 1.f / l;
            __nv_bfloat16* out = p.out + (static_cast<long long>(batch) * p.T + q0 + r) * p.H * 64 + head * 64 + half * 32;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint4 w;
                w.x = pack_bf16x2(o[8 * q] * inv, o[8 * q + 1] * inv); w.y = pack_bf16x2(o[8 * q + 2] * inv, o[8 * q + 3] * inv);
                w.z = pack_bf16x2(o[8 * q + 4] * inv, o[8 * q + 5] * inv); w.w = pack_bf16x2(o[8 * q + 6] * inv, o[8 * q + 7] * inv);
                *reinterpret_cast<uint4*>(out + 8 * q) = w;
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        if (*reinterpret_cast<volatile int*>(p.status) != 0) {    // a wait gave up: let MMAs and copies in flight drain before the columns are freed
            const long long start = clock64();
            while (clock64() - start < 200000) {}
        }
        tc_fence_after();
        tmem_dealloc(tmem_base, PF_TMEM_COLS);
    }
}

}  // namespace

void launch_mla_prefill_prepare(const MlaCachedArgs& a, void* q_out, void* w_hi, void* w_lo, cudaStream_t s) {
    PrefillPrepareParams p;
    p.query = static_cast<const __nv_bfloat16*>(a.query); p.low = static_cast<const __nv_bfloat16*>(a.low);
    p.q_pitch = a.q_pitch; p.low_pitch = a.low_pitch;
    p.norm_w = a.norm_w; p.cos = a.cos; p.sin = a.sin; p.q_scale = a.q_scale;
    p.latent = static_cast<__nv_bfloat16*>(a.latent) + static_cast<long long>(a.start) * a.r;
    p.rope = static_cast<__nv_bfloat16*>(a.rope) + static_cast<long long>(a.start) * 64;
    p.latent_bs = a.latent_bs; p.rope_bs = a.rope_bs;
    p.q_out = static_cast<__nv_bfloat16*>(q_out);
    p.tokens = a.B * a.T; p.T = a.T; p.H = a.H; p.r = a.r; p.rms = a.rms; p.norm_eps = a.norm_eps; p.qk_eps = a.qk_eps; p.smin = a.smin; p.smax = a.smax;
    p.w = a.w_up; p.w_hi = static_cast<__nv_bfloat16*>(w_hi); p.w_lo = static_cast<__nv_bfloat16*>(w_lo);
    p.w_pieces = a.Hkv * 128 * a.r / 4;                                 // at most 32 heads and rank 1024
    p.w_blocks = (p.w_pieces + 255) / 256 < 592 ? (p.w_pieces + 255) / 256 : 592;
    mla_prefill_prepare_kernel<<<p.w_blocks + a.B * a.T, 256, 0, s>>>(p);
}

void launch_mla_prefill_split(const MlaCachedArgs& a, int base, const float* kv, void* const* terms, float* gain, int S, int S_pad, cudaStream_t s) {
    PrefillSplitParams p;
    p.kv = kv;
    p.rope = static_cast<const __nv_bfloat16*>(a.rope) + static_cast<long long>(base) * 64;
    p.key_gain = static_cast<__nv_bfloat16*>(a.key_gain) + static_cast<long long>(base) * a.Hkv;
    p.rope_bs = a.rope_bs; p.gain_bs = a.gain_bs; p.k_scale = a.k_scale;
    p.k_hi = static_cast<__nv_bfloat16*>(terms[0]); p.k_lo = static_cast<__nv_bfloat16*>(terms[1]);
    p.v_hi = static_cast<__nv_bfloat16*>(terms[2]); p.v_lo = static_cast<__nv_bfloat16*>(terms[3]);
    p.gain = gain; p.S = S; p.S_pad = S_pad; p.Hk = a.Hkv; p.new_from = a.start - base; p.rms = a.rms;
    p.qk_eps = a.qk_eps; p.smin = a.smin; p.smax = a.smax; p.scale_log2e = a.scale * 1.4426950408889634f;
    const long long units = static_cast<long long>(S_pad) * a.Hkv;
    mla_prefill_split_kernel<<<dim3(static_cast<unsigned>((units + 7) / 8), a.B), 256, 0, s>>>(p);
}

cudaError_t launch_mla_prefill_attention(const MlaCachedArgs& a, int base, const CUtensorMap& tq, const CUtensorMap& tkh, const CUtensorMap& tkl, const CUtensorMap& trope,
                                         const CUtensorMap& tvh, const CUtensorMap& tvl, const float* gain, int S, int S_pad, int* status, cudaStream_t s) {
    PrefillAttnParams p;
    p.T = a.T; p.H = a.H; p.group = a.H / a.Hkv; p.S = S; p.S_pad = S_pad; p.start = a.start - base; p.window = a.window;
    p.gain = gain; p.out = static_cast<__nv_bfloat16*>(a.out); p.status = status;
    cudaError_t e = cudaFuncSetAttribute(mla_prefill_attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SMEM);
    if (e != cudaSuccess) return e;
    mla_prefill_attention_kernel<<<dim3(a.H, a.B, (a.T + PF_M - 1) / PF_M), PF_THREADS, PF_SMEM, s>>>(tq, tkh, tkl, trope, tvh, tvl, p);
    return cudaGetLastError();
}

}  // namespace gm
