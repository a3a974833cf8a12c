// Causal sliding-window attention backward for sm_100a.  Value heads are 64 wide; query / key heads are 64 wide (DQK = 64)
// or 128 wide (DQK = 128, multi-head latent attention).  With DQK = 128 the dK accumulator takes 128 TMEM columns, so the
// dQ product is written over the S columns once the softmax warps have consumed S (the next S then waits for the dQ
// read-out), and the fp32 dQ staging tile reuses the P / dS shared-memory tiles once the products have read them.
//
// One CTA owns 128 keys of one (batch, kv head) and walks the query tiles that can see them
// (q tile i with  kv0 <= q  and  q - W <= kv0 + 127), for every query head of the kv head's group:
//   S  = Q_i K^T,  dP = dO_i V^T            two tcgen05.mma M128 N128 K64 into TMEM (128 + 128 columns)
//   P  = exp2(S*c - LSE),  dS = P * (dP - delta)   softmax warps (thread = query row), token-exact mask; P and dS are
//                                                  written to shared memory as bf16 in the 128B-swizzled layout
//   dV += P^T dO_i,  dK += dS^T Q_i          M128 N64 K128, A read MN-major from the P / dS tiles, B MN-major from the
//                                            dO / Q tiles; accumulators stay in TMEM for the whole CTA (64 + 64 columns)
//   dQ_i = dS K                              M128 N64 K128, A = the same dS tile read K-major, B = K read MN-major;
//                                            the 128x64 fp32 result is scaled, staged in shared memory and added into
//                                            a fp32 dQ buffer by TMA reduce-add (several key tiles contribute to one row)
// The K and V tiles stay resident; Q / dO tiles run through a two-deep TMA ring.  Warp 8 is the control warp (loads and MMA issue, a whole
// warp: see umma_f16 in ptx.cuh), warps 0-7 are the softmax warps (warps w and w+4 share TMEM quadrant w and split the key columns).
// delta = rowsum(dO * O) comes from a small pre-pass kernel in this file, which also clears the dQ buffer.
// Calls with 64-wide heads go to attn_bwd_pipe.cu (transposed score tiles, P and dS in TMEM); this kernel serves 128-wide heads and is
// the one that kernel is tested against.  The delta pre-pass and the launcher of both live here.
// Reference counterpart: the backward of FlexAttention (model/attention/self_attention.py:250-255) as generated by Inductor.
#include "../common/ptx.cuh"
#include "attn.h"

namespace gm {

constexpr int BW_THREADS = 288;
constexpr int TILE = 128, HD = 64;
constexpr int T_BYTES = TILE * HD * 2;            // one 128 x 64 bf16 tile
constexpr int PD_BYTES = TILE * TILE * 2;         // P or dS tile (two 128-byte-wide slabs)
constexpr int STG_BYTES = TILE * HD * 4;          // dQ staging (two slabs of 32 fp32 columns)
constexpr int QDO_STAGES = 2;
constexpr uint32_t BW_TMEM_COLS = 512;
constexpr uint32_t COL_S = 0, COL_DP = 128, COL_DV = 256, COL_DK = 320, COL_DQ64 = 384;   // DQK = 128: dK spans 320..447, dQ aliases S

// delta[b, h, t] = sum_d dO[t, h, d] * O[t, h, d]; eight lanes (16 bytes each) per (token, head), four heads per warp pass.  The same pass
// clears the row of dQ that the backward adds to (a fill of its own took 10 us of 16384 tokens' 16 heads, and a launch)
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ d_out, const __nv_bfloat16* __restrict__ out, float* __restrict__ delta,
                  long long tokens, int heads, int seq_len, long long do_stride, long long o_stride, float* __restrict__ dq, int qk_dim) {
    const int lane = threadIdx.x & 31;
    const int sub = lane >> 3, li = lane & 7;
    const int groups = (heads + 3) / 4;
    const long long total = tokens * groups;
    for (long long idx = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5); idx < total; idx += static_cast<long long>(gridDim.x) * 8) {
        const long long tok = idx / groups;
        const int h = static_cast<int>(idx - tok * groups) * 4 + sub;
        float s = 0.f;
        if (h < heads) {
            float4* clear = reinterpret_cast<float4*>(dq + (tok * heads + h) * qk_dim);
            for (int i = li; i < qk_dim / 4; i += 8) clear[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            const uint4 ra = *reinterpret_cast<const uint4*>(d_out + tok * do_stride + h * HD + li * 8);
            const uint4 rb = *reinterpret_cast<const uint4*>(out + tok * o_stride + h * HD + li * 8);
            const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&ra);
            const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&rb);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 a = __bfloat1622float2(pa[i]), b = __bfloat1622float2(pb[i]);
                s += a.x * b.x + a.y * b.y;
            }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (li == 0 && h < heads) delta[((tok / seq_len) * heads + h) * seq_len + tok % seq_len] = s;
    }
}

// dQ [tokens, width] fp32 as bf16 rows `pitch` values apart (a slice of a packed gradient row): 32 bytes in, 16 out a thread.  Torch's copy
// between these layouts took 41 us for 16384 x 1024, this 18.
__global__ void __launch_bounds__(256)
attn_dq_store_kernel(const float* __restrict__ dq, __nv_bfloat16* __restrict__ out, long long tokens, int width, long long pitch) {
    const int per_row = width / 8;
    const long long total = tokens * per_row;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
        const long long tok = i / per_row;
        const int col = static_cast<int>(i - tok * per_row) * 8;
        const float4 a = *reinterpret_cast<const float4*>(dq + i * 8), b = *reinterpret_cast<const float4*>(dq + i * 8 + 4);
        *reinterpret_cast<uint4*>(out + tok * pitch + col) = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
    }
}

cudaError_t launch_attn_dq_store(const float* dq, void* out, long long tokens, int width, long long pitch, cudaStream_t s) {
    const long long blocks = (tokens * (width / 8) + 255) / 256;
    attn_dq_store_kernel<<<static_cast<int>(blocks < 4736 ? blocks : 4736), 256, 0, s>>>(dq, static_cast<__nv_bfloat16*>(out), tokens, width, pitch);
    return cudaGetLastError();
}

__device__ __forceinline__ float tanh_approx_bwd(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// CAP: logit soft-capping (see the forward kernel): the score becomes cap_a * tanh(s * cap_b) and dS picks up the factor 1 - tanh^2.
template <bool MASK, bool CAP>
__device__ __forceinline__ void bwd_tile_math(uint32_t s_addr, uint32_t dp_addr, uint8_t* p_row, uint8_t* ds_row, int sw, int kv0,
                                              int qpos, int window, float c, float lse2, float delta, float cap_a, float cap_b) {
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
        uint32_t sreg[32], dreg[32];
        tmem_ld_32x32b_x32(s_addr + cc * 32, sreg);
        tmem_ld_32x32b_x32(dp_addr + cc * 32, dreg);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float pv[8], dv[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int col = 8 * q + i;
                float sv = __uint_as_float(sreg[col]);
                float chain = 1.f;
                if (CAP) {
                    const float th = tanh_approx_bwd(sv * cap_b);
                    sv = cap_a * th;
                    chain = 1.f - th * th;
                }
                float e = exp2f(fmaf(sv, c, -lse2));
                if (MASK) {
                    const int kpos = kv0 + cc * 32 + col;
                    e = (kpos > qpos || qpos - kpos > window) ? 0.f : e;
                }
                pv[i] = e;
                dv[i] = e * (__uint_as_float(dreg[col]) - delta) * chain;
            }
            uint4 wp, wd;
            wp.x = pack_bf16x2(pv[0], pv[1]); wp.y = pack_bf16x2(pv[2], pv[3]); wp.z = pack_bf16x2(pv[4], pv[5]); wp.w = pack_bf16x2(pv[6], pv[7]);
            wd.x = pack_bf16x2(dv[0], dv[1]); wd.y = pack_bf16x2(dv[2], dv[3]); wd.z = pack_bf16x2(dv[4], dv[5]); wd.w = pack_bf16x2(dv[6], dv[7]);
            const int piece = ((cc * 4 + q) ^ sw) << 4;
            *reinterpret_cast<uint4*>(p_row + piece) = wp;
            *reinterpret_cast<uint4*>(ds_row + piece) = wd;
        }
    }
}

template <int DQK, bool CAPPED>
__global__ void __launch_bounds__(BW_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                const __grid_constant__ CUtensorMap tmap_dq, const AttnParams p) {
    constexpr int QK_SLABS = DQK / 64;
    constexpr int QK_BYTES = QK_SLABS * T_BYTES;      // a 128-row query or key tile: one 128 x 64 slab per 64 columns
    constexpr bool WIDE = DQK == 128;
    constexpr uint32_t COL_DQ = WIDE ? COL_S : COL_DQ64;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sk = smem;
    uint8_t* sv = sk + QK_BYTES;
    uint8_t* sq = sv + T_BYTES;                       // QDO_STAGES tiles
    uint8_t* sdo = sq + QDO_STAGES * QK_BYTES;        // QDO_STAGES tiles
    uint8_t* sp = sdo + QDO_STAGES * T_BYTES;
    uint8_t* sds = sp + PD_BYTES;
    uint8_t* stg = WIDE ? sp : sds + PD_BYTES;        // fp32 dQ staging: its own tile, or (wide heads) the P + dS tiles
    uint64_t* bars = reinterpret_cast<uint64_t*>(sds + PD_BYTES + (WIDE ? 0 : STG_BYTES));
    uint64_t* bar_kv = bars + 0;
    uint64_t* bar_sdp = bars + 1;
    uint64_t* bar_pds = bars + 2;
    uint64_t* bar_mma = bars + 3;
    uint64_t* bar_dq = bars + 4;                      // wide heads: the dQ tile has been read out of the S columns
    uint64_t* bar_qdo = bars + 5;                     // [QDO_STAGES]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_qdo + QDO_STAGES);

    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int kv_tile = p.long_first ? blockIdx.z : blockIdx.x, kv_head = p.long_first ? blockIdx.x : blockIdx.y;
    const int batch = p.long_first ? blockIdx.y : blockIdx.z;
    const int kv0 = kv_tile * TILE;
    const int window = uniform(p.window_ptr ? min(max(*p.window_ptr, 0), p.seq_len) : p.window);
    const int q_tiles_total = (p.seq_len + TILE - 1) / TILE;
    int last_q_tile = (kv0 + TILE - 1 + window) / TILE;
    if (last_q_tile > q_tiles_total - 1) last_q_tile = q_tiles_total - 1;
    const int n_q = last_q_tile - kv_tile + 1;        // query tiles per head that see this key tile
    const int n_iter = n_q * p.group;                 // times the query heads sharing this kv head
    const int row0 = batch * p.seq_len;

    if (threadIdx.x == 0) {
        mbar_init(bar_kv, 1); mbar_init(bar_sdp, 1); mbar_init(bar_pds, 256); mbar_init(bar_mma, 1); mbar_init(bar_dq, 256);
        for (int st = 0; st < QDO_STAGES; ++st) mbar_init(&bar_qdo[st], 1);
        fence_barrier_init();
    }
    if (warp == 8) { tmem_alloc(tmem_slot, BW_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = uniform(*tmem_slot);
    bool ok = true;

    if (warp == 8) {
        {
            const uint32_t on = elect_one();
            constexpr uint32_t idesc_sdp = make_idesc_bf16(TILE, TILE, false, false);
            constexpr uint32_t idesc_dv = make_idesc_bf16(TILE, HD, true, true);
            constexpr uint32_t idesc_dk = make_idesc_bf16(TILE, DQK, true, true);
            constexpr uint32_t idesc_dq = make_idesc_bf16(TILE, DQK, false, true);
            // descriptors formed once (K-major and MN-major forms of the same tiles); the address field counts 16-byte units
            const uint64_t k_kmaj = make_smem_desc(smem_u32(sk), 16, 1024), v_kmaj = make_smem_desc(smem_u32(sv), 16, 1024);
            const uint64_t q_kmaj = make_smem_desc(smem_u32(sq), 16, 1024), do_kmaj = make_smem_desc(smem_u32(sdo), 16, 1024);
            const uint64_t q_mn = make_smem_desc(smem_u32(sq), TILE * 128, 1024), do_mn = make_smem_desc(smem_u32(sdo), TILE * 128, 1024);
            const uint64_t k_mn = make_smem_desc(smem_u32(sk), TILE * 128, 1024);
            const uint64_t p_mn = make_smem_desc(smem_u32(sp), TILE * 128, 1024), ds_mn = make_smem_desc(smem_u32(sds), TILE * 128, 1024);
            const uint64_t ds_kmaj = make_smem_desc(smem_u32(sds), 16, 1024);
            auto load_qdo = [&](int it) {
                const int st = it % QDO_STAGES;
                const int head = kv_head * p.group + it / n_q;
                const int q0 = (kv_tile + it % n_q) * TILE;
                if (on) mbar_expect_tx(&bar_qdo[st], QK_BYTES + T_BYTES);
#pragma unroll
                for (int sl = 0; sl < QK_SLABS; ++sl)
                    tma_load_3d(sq + st * QK_BYTES + sl * T_BYTES, &tmap_q, &bar_qdo[st], head * DQK + 64 * sl, q0, batch, on);
                tma_load_3d(sdo + st * T_BYTES, &tmap_do, &bar_qdo[st], head * HD, q0, batch, on);
            };
            if (on) mbar_expect_tx(bar_kv, QK_BYTES + T_BYTES);
#pragma unroll
            for (int sl = 0; sl < QK_SLABS; ++sl) tma_load_3d(sk + sl * T_BYTES, &tmap_k, bar_kv, kv_head * DQK + 64 * sl, kv0, batch, on);
            tma_load_3d(sv, &tmap_v, bar_kv, kv_head * p.v_head, kv0, batch, on);
            for (int it = 0; it < QDO_STAGES && it < n_iter; ++it) load_qdo(it);
            if (!warp_wait(bar_kv, 0)) { atomicExch(p.status, 301); ok = false; }
            auto issue_sdp = [&](int it) -> bool {               // S = Q K^T ; dP = dO V^T for iteration `it`
                const int st = it % QDO_STAGES;
                if (!warp_wait(&bar_qdo[st], (it / QDO_STAGES) & 1)) return false;
                tc_fence_after();
                const uint64_t qa = q_kmaj + st * (QK_BYTES >> 4), da = do_kmaj + st * (T_BYTES >> 4);
#pragma unroll
                for (int sl = 0; sl < QK_SLABS; ++sl)
#pragma unroll
                    for (int k4 = 0; k4 < 4; ++k4)
                        umma_f16(tmem_base + COL_S, qa + sl * (T_BYTES >> 4) + k4 * 2, k_kmaj + sl * (T_BYTES >> 4) + k4 * 2, idesc_sdp, (sl | k4) != 0, on);
#pragma unroll
                for (int k4 = 0; k4 < HD / 16; ++k4) umma_f16(tmem_base + COL_DP, da + k4 * 2, v_kmaj + k4 * 2, idesc_sdp, k4 != 0, on);
                umma_commit(bar_sdp, on);
                return true;
            };
            if (ok && n_iter > 0 && !issue_sdp(0)) { atomicExch(p.status, 302); ok = false; }
            for (int it = 0; it < n_iter && ok; ++it) {
                const uint32_t ph = it & 1;
                const int st = it % QDO_STAGES;
                const uint64_t qa = q_mn + st * (QK_BYTES >> 4), da = do_mn + st * (T_BYTES >> 4);
                if (!warp_wait(bar_pds, ph)) { atomicExch(p.status, 303); ok = false; break; }
                tc_fence_after();
#pragma unroll
                for (int k8 = 0; k8 < TILE / 16; ++k8)          // dV += P^T dO   (contraction over the 128 query rows)
                    umma_f16(tmem_base + COL_DV, p_mn + k8 * 128, da + k8 * 128, idesc_dv, (it | k8) != 0, on);
#pragma unroll
                for (int k8 = 0; k8 < TILE / 16; ++k8)          // dK += dS^T Q
                    umma_f16(tmem_base + COL_DK, ds_mn + k8 * 128, qa + k8 * 128, idesc_dk, (it | k8) != 0, on);
#pragma unroll
                for (int k8 = 0; k8 < TILE / 16; ++k8)          // dQ = dS K      (contraction over the 128 keys)
                    umma_f16(tmem_base + COL_DQ, ds_kmaj + (k8 >> 2) * (TILE * 128 >> 4) + (k8 & 3) * 2, k_mn + k8 * 128, idesc_dq, k8 != 0, on);
                umma_commit(bar_mma, on);
                // S / dP of this iteration were consumed before bar_pds: the next pair can queue behind the three products
                // (narrow heads; with wide heads dQ sits in the S columns until the softmax warps have read it out)
                if (!WIDE && it + 1 < n_iter && !issue_sdp(it + 1)) { atomicExch(p.status, 302); ok = false; break; }
                if (!warp_wait(bar_mma, ph)) { atomicExch(p.status, 304); ok = false; break; }
                if (it + QDO_STAGES < n_iter) load_qdo(it + QDO_STAGES);      // this stage's Q / dO tiles are consumed
                if (WIDE && it + 1 < n_iter) {
                    if (!warp_wait(bar_dq, ph)) { atomicExch(p.status, 307); ok = false; break; }
                    tc_fence_after();
                    if (!issue_sdp(it + 1)) { atomicExch(p.status, 302); ok = false; break; }
                }
            }
        }
    } else {
        const int quad = warp & 3, half = warp >> 2;
        const int r = quad * 32 + lane;
        const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
        const int sw = r & 7;
        const bool leader = threadIdx.x == 0;
        uint8_t* p_row = sp + half * (TILE * 128) + r * 128;
        uint8_t* ds_row = sds + half * (TILE * 128) + r * 128;
        // fp32 dQ staging: slabs of 32 columns; this thread fills DQK / 64 slabs of its row
        uint8_t* stg_row = stg + half * (DQK / 64) * (TILE * 128) + r * 128;
        const float c = p.scale_log2e;
        constexpr bool capped = CAPPED;
        const float cap_a = capped ? p.softcap / p.scale : 0.f, cap_b = capped ? p.scale / p.softcap : 0.f;
        for (int it = 0; it < n_iter; ++it) {
            const uint32_t ph = it & 1;
            const int head = kv_head * p.group + it / n_q;
            const int q0 = (kv_tile + it % n_q) * TILE;
            const int qpos = q0 + r;
            const long long stat = (static_cast<long long>(batch) * p.heads + head) * p.seq_len + qpos;
            // rows past the sequence end are zeros; an infinite log-sum-exp makes their probabilities 0
            const bool live = qpos < p.seq_len;
            const float lse2 = live ? p.lse[stat] * 1.4426950408889634f : INFINITY;
            const float delta = live ? p.delta[stat] : 0.f;
            int w_row = window, w_last = window;                        // document masking: see the forward kernel
            if (p.doc_start) {
                const int last = min(q0 + TILE, p.seq_len) - 1;
                if (live) w_row = min(window, qpos - p.doc_start[row0 + qpos]);
                w_last = min(window, last - p.doc_start[row0 + last]);
            }
            const bool need_mask = (q0 == kv0) || (q0 + TILE - 1 - kv0 > w_last);
            if (ok && !mbar_wait(bar_sdp, ph)) { atomicExch(p.status, 305); ok = false; }
            tc_fence_after();
            if (WIDE) {                      // the previous dQ reduce-add must have finished reading the P / dS tiles it was staged in
                if (leader) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                asm volatile("bar.sync 1, 256;" ::: "memory");
            }
            const uint32_t s_addr = tmem_base + COL_S + lane_off + half * 64, dp_addr = tmem_base + COL_DP + lane_off + half * 64;
            if (capped) {
                if (need_mask) bwd_tile_math<true, true>(s_addr, dp_addr, p_row, ds_row, sw, kv0 + half * 64, qpos, w_row, c, lse2, delta, cap_a, cap_b);
                else bwd_tile_math<false, true>(s_addr, dp_addr, p_row, ds_row, sw, kv0 + half * 64, qpos, w_row, c, lse2, delta, cap_a, cap_b);
            } else {
                if (need_mask) bwd_tile_math<true, false>(s_addr, dp_addr, p_row, ds_row, sw, kv0 + half * 64, qpos, w_row, c, lse2, delta, 0.f, 0.f);
                else bwd_tile_math<false, false>(s_addr, dp_addr, p_row, ds_row, sw, kv0 + half * 64, qpos, w_row, c, lse2, delta, 0.f, 0.f);
            }
            tc_fence_before();
            fence_proxy_async();
            mbar_arrive(bar_pds);
            if (ok && !mbar_wait(bar_mma, ph)) { atomicExch(p.status, 306); ok = false; }
            tc_fence_after();
            // dQ tile: this thread's row, half of the DQK columns; scaled, staged, then one TMA reduce-add per 32-column slab
            uint32_t qreg[DQK / 64][32];
#pragma unroll
            for (int j = 0; j < DQK / 64; ++j)
                tmem_ld_32x32b_x32(tmem_base + COL_DQ + lane_off + half * (DQK / 2) + j * 32, qreg[j]);
            tmem_ld_wait();
            tc_fence_before();
            if (WIDE) {
                mbar_arrive(bar_dq);                                      // the S columns may be overwritten by the next S
            } else {
                if (leader) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                asm volatile("bar.sync 1, 256;" ::: "memory");              // previous reduce has finished reading the staging tile
            }
#pragma unroll
            for (int j = 0; j < DQK / 64; ++j) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    *reinterpret_cast<float4*>(stg_row + j * (TILE * 128) + ((q ^ sw) << 4)) =
                        make_float4(__uint_as_float(qreg[j][4 * q]) * p.scale, __uint_as_float(qreg[j][4 * q + 1]) * p.scale,
                                    __uint_as_float(qreg[j][4 * q + 2]) * p.scale, __uint_as_float(qreg[j][4 * q + 3]) * p.scale);
                }
            }
            fence_proxy_async();
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (leader) {
#pragma unroll
                for (int sl = 0; sl < DQK / 32; ++sl) {
                    asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
                                 ::"l"(&tmap_dq), "r"(smem_u32(stg + sl * (TILE * 128))), "r"(head * DQK + sl * 32), "r"(q0), "r"(batch) : "memory");
                }
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        }
        if (ok && n_iter > 0) {
            // dK, dV: TMEM lanes are the 128 keys of this CTA; each thread writes half of the columns of its key row
            const bool live = kv0 + r < p.seq_len;
            const long long token = static_cast<long long>(row0) + kv0 + r;
            __nv_bfloat16* dk = reinterpret_cast<__nv_bfloat16*>(p.dk) + token * p.dkv_stride + kv_head * DQK + half * (DQK / 2);
            __nv_bfloat16* dv = reinterpret_cast<__nv_bfloat16*>(p.dv) + token * p.dv_stride + kv_head * p.dv_head + half * 32;
            uint32_t vreg[32];
            tmem_ld_32x32b_x32(tmem_base + COL_DV + lane_off + half * 32, vreg);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint4 wv;
                wv.x = pack_bf16x2(__uint_as_float(vreg[8 * q]), __uint_as_float(vreg[8 * q + 1]));
                wv.y = pack_bf16x2(__uint_as_float(vreg[8 * q + 2]), __uint_as_float(vreg[8 * q + 3]));
                wv.z = pack_bf16x2(__uint_as_float(vreg[8 * q + 4]), __uint_as_float(vreg[8 * q + 5]));
                wv.w = pack_bf16x2(__uint_as_float(vreg[8 * q + 6]), __uint_as_float(vreg[8 * q + 7]));
                if (live) *reinterpret_cast<uint4*>(dv + 8 * q) = wv;
            }
#pragma unroll
            for (int j = 0; j < DQK / 64; ++j) {
                uint32_t kreg[32];
                tmem_ld_32x32b_x32(tmem_base + COL_DK + lane_off + half * (DQK / 2) + j * 32, kreg);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint4 wk;
                    wk.x = pack_bf16x2(__uint_as_float(kreg[8 * q]) * p.scale, __uint_as_float(kreg[8 * q + 1]) * p.scale);
                    wk.y = pack_bf16x2(__uint_as_float(kreg[8 * q + 2]) * p.scale, __uint_as_float(kreg[8 * q + 3]) * p.scale);
                    wk.z = pack_bf16x2(__uint_as_float(kreg[8 * q + 4]) * p.scale, __uint_as_float(kreg[8 * q + 5]) * p.scale);
                    wk.w = pack_bf16x2(__uint_as_float(kreg[8 * q + 6]) * p.scale, __uint_as_float(kreg[8 * q + 7]) * p.scale);
                    if (live) *reinterpret_cast<uint4*>(dk + j * 32 + 8 * q) = wk;
                }
            }
        }
        if (leader) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        if (*reinterpret_cast<volatile int*>(p.status) != 0) {
            const long long start = clock64();
            while (clock64() - start < 200000) {}
        }
        tc_fence_after();
        tmem_dealloc(tmem_base, BW_TMEM_COLS);
    }
}

template <int DQK, bool CAPPED>
static cudaError_t launch_bwd_variant(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                      const CUtensorMap& tdq, const AttnParams& p, cudaStream_t stream) {
    constexpr int qk_bytes = (DQK / 64) * T_BYTES;
    constexpr int smem = qk_bytes + T_BYTES + QDO_STAGES * (qk_bytes + T_BYTES) + 2 * PD_BYTES + (DQK == 128 ? 0 : STG_BYTES) + 1024 + 128;
    auto kernel = attn_bwd_kernel<DQK, CAPPED>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    const int tiles = (p.seq_len + TILE - 1) / TILE, kv_heads = p.heads / p.group;
    const dim3 grid = p.long_first ? dim3(kv_heads, p.batch, tiles) : dim3(tiles, kv_heads, p.batch);
    kernel<<<grid, BW_THREADS, smem, stream>>>(tq, tk, tv, tdo, tdq, p);
    return cudaGetLastError();
}

cudaError_t launch_attn_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                            const CUtensorMap& tdq, const AttnParams& params, const void* d_out, const void* out, long long do_stride,
                            long long o_stride, float* delta, cudaStream_t stream) {
    // Without a window the first key tiles are seen by every query and the last by a few: in head-major order the last head's first tile
    // starts when most SMs are about to run dry (2 x 4096 tokens, 16 heads of 128: 644 us; longest first 573).  With a window all tiles
    // are alike, and neighbours share query tiles in L2 when they run together (16 x 2048, 12 heads, window 1024: 470 us against 478);
    // nor does the order matter while everything fits one wave.
    AttnParams p = params;
    const long long ctas = static_cast<long long>((p.seq_len + TILE - 1) / TILE) * (p.heads / p.group) * p.batch;
    p.long_first = p.window > p.seq_len / 2 && ctas > 148;
    const long long tokens = static_cast<long long>(p.batch) * p.seq_len;
    attn_delta_kernel<<<1184, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(d_out), static_cast<const __nv_bfloat16*>(out), delta,
                                                tokens, p.heads, p.seq_len, do_stride, o_stride, p.dq_accum, p.qk_dim);
    const bool capped = p.softcap > 0.f;
    if (p.qk_dim == 128)
        return capped ? launch_bwd_variant<128, true>(tq, tk, tv, tdo, tdq, p, stream) : launch_bwd_variant<128, false>(tq, tk, tv, tdo, tdq, p, stream);
    if (!p.single_tile) return launch_attn_bwd_pipe(tq, tk, tv, tdo, tdq, p, stream);
    return capped ? launch_bwd_variant<64, true>(tq, tk, tv, tdo, tdq, p, stream) : launch_bwd_variant<64, false>(tq, tk, tv, tdo, tdq, p, stream);
}

}  // namespace gm
