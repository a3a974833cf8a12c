// Causal sliding-window attention backward for sm_100a, 64-wide heads, with the score products of the next query tile issued
// ahead of the gradient products of the current one.
//
// Same tiling and products as attn_bwd.cu (sequences of any length: the tensor maps end at the sequence's last row; one CTA owns 128 keys
// of one (batch, kv head) and walks the query tiles that see them; S = Q K^T and dP = dO V^T into TMEM, P and dS to shared memory, dV += P^T dO, dK += dS^T Q, dQ = dS K reduced into a
// fp32 buffer by TMA).  What differs is the order.  In attn_bwd.cu one iteration is a chain: S/dP -> softmax warps -> three
// gradient products -> dQ read-out, and the S/dP of the next iteration queue behind the gradient products, so the tensor
// core idles while the softmax warps work and the other way round.  Here:
//   warp 8             issues S/dP of iteration i+1 as soon as the softmax warps have READ S/dP of iteration i from TMEM
//                    (bar_sread)
//   warp 10            waits for P/dS of iteration i in shared memory and issues the three gradient products (its own warp so
//                    that neither chain waits behind the other's barrier)
//   softmax warps    read S/dP of iteration i, form P and dS as packed bf16 in REGISTERS (64 per thread), release S/dP, and
//                    only then wait for the gradient products of iteration i-1 (which still read the P/dS tiles in shared
//                    memory), store P/dS of iteration i, and drain dQ of iteration i-1 while the products of iteration i
//                    write the other of two dQ tiles
//   loader warp      K, V once; Q / dO through a three-deep ring, a stage refilled when the gradient products that read it
//                    have completed
// so the exponentials of iteration i+1 run under the gradient products of iteration i.  Measured on 16 x 2048 tokens, 12 heads,
// window 1024 (delta pre-pass and dQ zero-fill included): 445 us against 516 us for attn_bwd.cu (476 and 545 with one issuing lane).  An iteration
// takes 4000 clocks: the softmax warps' arithmetic 1450, their stores of P and dS 680, the dQ read-out 760 to 1200; products wait for them.
// Reference counterpart: the backward of FlexAttention (model/attention/self_attention.py:250-255) as generated by Inductor.
#include "../common/ptx.cuh"
#include "attn.h"

namespace gm {

constexpr int BP_THREADS = 352;
constexpr int BP_TILE = 128, BP_HD = 64;
constexpr int BP_T_BYTES = BP_TILE * BP_HD * 2;          // one 128 x 64 bf16 tile
constexpr int BP_PD_BYTES = BP_TILE * BP_TILE * 2;       // P or dS tile (two 128-byte-wide slabs)
constexpr int BP_STG_BYTES = BP_TILE * BP_HD * 4;        // dQ staging (two slabs of 32 fp32 columns)
constexpr int BP_STAGES = 3;
constexpr uint32_t BP_TMEM_COLS = 512;
constexpr uint32_t BP_COL_S = 0, BP_COL_DP = 128, BP_COL_DV = 256, BP_COL_DK = 320, BP_COL_DQ = 384;       // two dQ tiles, in turn

__device__ __forceinline__ float bp_tanh_approx(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// P = exp2(S*c - LSE) and dS = P * (dP - delta) for this thread's 64 keys of its query row, packed to bf16 in registers:
// wp[4 * cc + q] / wd[4 * cc + q] hold keys 32 * cc + 8 * q .. + 7.
// CAP: logit soft-capping: the score becomes cap_a * tanh(s * cap_b) and dS picks up the factor 1 - tanh^2.
template <bool MASK, bool CAP>
__device__ __forceinline__ void bp_tile_math(uint32_t s_addr, uint32_t dp_addr, uint4 (&wp)[8], uint4 (&wd)[8], int kv0, int qpos, int window,
                                             float c, float lse2, float delta, float cap_a, float cap_b) {
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
                    const float th = bp_tanh_approx(sv * cap_b);
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
            uint4 a, b;
            a.x = pack_bf16x2(pv[0], pv[1]); a.y = pack_bf16x2(pv[2], pv[3]); a.z = pack_bf16x2(pv[4], pv[5]); a.w = pack_bf16x2(pv[6], pv[7]);
            b.x = pack_bf16x2(dv[0], dv[1]); b.y = pack_bf16x2(dv[2], dv[3]); b.z = pack_bf16x2(dv[4], dv[5]); b.w = pack_bf16x2(dv[6], dv[7]);
            wp[4 * cc + q] = a;
            wd[4 * cc + q] = b;
        }
    }
}

template <bool CAPPED>
__global__ void __launch_bounds__(BP_THREADS, 1)
attn_bwd_pipe_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                     const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                     const __grid_constant__ CUtensorMap tmap_dq, const AttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sk = smem;
    uint8_t* sv = sk + BP_T_BYTES;
    uint8_t* sq = sv + BP_T_BYTES;                       // BP_STAGES tiles
    uint8_t* sdo = sq + BP_STAGES * BP_T_BYTES;          // BP_STAGES tiles
    uint8_t* sp = sdo + BP_STAGES * BP_T_BYTES;
    uint8_t* sds = sp + BP_PD_BYTES;
    uint8_t* stg = sds + BP_PD_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(stg + BP_STG_BYTES);
    uint64_t* bar_kv = bars + 0;
    uint64_t* bar_sdp = bars + 1;                        // S and dP of an iteration complete
    uint64_t* bar_sread = bars + 2;                      // the softmax warps have read them out of TMEM (256 arrivals)
    uint64_t* bar_pds = bars + 3;                        // P and dS of an iteration are in shared memory (256 arrivals)
    uint64_t* bar_mma = bars + 4;                        // the three gradient products of an iteration complete
    uint64_t* bar_qdo = bars + 5;                        // [BP_STAGES] Q / dO tile landed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_qdo + BP_STAGES);

    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int kv_tile = p.long_first ? blockIdx.z : blockIdx.x, kv_head = p.long_first ? blockIdx.x : blockIdx.y;
    const int batch = p.long_first ? blockIdx.y : blockIdx.z;
    const int kv0 = kv_tile * BP_TILE;
    const int window = uniform(p.window_ptr ? min(max(*p.window_ptr, 0), p.seq_len) : p.window);
    const int q_tiles_total = (p.seq_len + BP_TILE - 1) / BP_TILE;
    int last_q_tile = (kv0 + BP_TILE - 1 + window) / BP_TILE;
    if (last_q_tile > q_tiles_total - 1) last_q_tile = q_tiles_total - 1;
    const int n_q = last_q_tile - kv_tile + 1;        // query tiles per head that see this key tile
    const int n_iter = n_q * p.group;                 // times the query heads sharing this kv head
    const int row0 = batch * p.seq_len;

    if (threadIdx.x == 0) {
        mbar_init(bar_kv, 1); mbar_init(bar_sdp, 1); mbar_init(bar_sread, 256); mbar_init(bar_pds, 256); mbar_init(bar_mma, 1);
        for (int st = 0; st < BP_STAGES; ++st) mbar_init(&bar_qdo[st], 1);
        fence_barrier_init();
    }
    if (warp == 8) { tmem_alloc(tmem_slot, BP_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = uniform(*tmem_slot);
    bool ok = true;

    if (warp == 9) {
        {
            const uint32_t on = elect_one();
            auto load_qdo = [&](int it) {
                const int st = it % BP_STAGES;
                const int head = kv_head * p.group + it / n_q;
                const int q0 = (kv_tile + it % n_q) * BP_TILE;
                if (on) mbar_expect_tx(&bar_qdo[st], 2 * BP_T_BYTES);
                tma_load_3d(sq + st * BP_T_BYTES, &tmap_q, &bar_qdo[st], head * BP_HD, q0, batch, on);
                tma_load_3d(sdo + st * BP_T_BYTES, &tmap_do, &bar_qdo[st], head * BP_HD, q0, batch, on);
            };
            if (on) mbar_expect_tx(bar_kv, 2 * BP_T_BYTES);
            tma_load_3d(sk, &tmap_k, bar_kv, kv_head * BP_HD, kv0, batch, on);
            tma_load_3d(sv, &tmap_v, bar_kv, kv_head * p.v_head, kv0, batch, on);
            for (int it = 0; it < BP_STAGES && it < n_iter; ++it) load_qdo(it);
            for (int it = BP_STAGES; it < n_iter; ++it) {
                // the stage was read by S/dP and by the gradient products of iteration it - BP_STAGES
                if (!warp_wait(bar_mma, (it - BP_STAGES) & 1)) { atomicExch(p.status, 311); break; }
                load_qdo(it);
            }
        }
    } else if (warp == 8 || warp == 10) {
        {
            const uint32_t on = elect_one();
            constexpr uint32_t idesc_sdp = make_idesc_bf16(BP_TILE, BP_TILE, false, false);
            constexpr uint32_t idesc_g = make_idesc_bf16(BP_TILE, BP_HD, true, true);         // dV, dK: A and B MN-major
            constexpr uint32_t idesc_dq = make_idesc_bf16(BP_TILE, BP_HD, false, true);       // dQ: A K-major, B MN-major
            // descriptors formed once; the address field counts 16-byte units: a 16-column slice of a K-major tile is 2 units on, a
            // 16-row slice of an MN-major tile 128 units, a ring stage 1024 units
            const uint64_t k_kmaj = make_smem_desc(smem_u32(sk), 16, 1024), v_kmaj = make_smem_desc(smem_u32(sv), 16, 1024);
            const uint64_t q_kmaj = make_smem_desc(smem_u32(sq), 16, 1024), do_kmaj = make_smem_desc(smem_u32(sdo), 16, 1024);
            const uint64_t q_mn = make_smem_desc(smem_u32(sq), BP_TILE * 128, 1024), do_mn = make_smem_desc(smem_u32(sdo), BP_TILE * 128, 1024);
            const uint64_t k_mn = make_smem_desc(smem_u32(sk), BP_TILE * 128, 1024);
            const uint64_t p_mn = make_smem_desc(smem_u32(sp), BP_TILE * 128, 1024), ds_mn = make_smem_desc(smem_u32(sds), BP_TILE * 128, 1024);
            const uint64_t ds_kmaj = make_smem_desc(smem_u32(sds), 16, 1024);
            auto issue_sdp = [&](int it) -> bool {               // S = Q K^T ; dP = dO V^T for iteration `it`
                const int st = it % BP_STAGES;
                if (!warp_wait(&bar_qdo[st], (it / BP_STAGES) & 1)) return false;
                tc_fence_after();
                const uint64_t qa = q_kmaj + st * (BP_T_BYTES >> 4), da = do_kmaj + st * (BP_T_BYTES >> 4);
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) umma_f16(tmem_base + BP_COL_S, qa + k4 * 2, k_kmaj + k4 * 2, idesc_sdp, k4 != 0, on);
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) umma_f16(tmem_base + BP_COL_DP, da + k4 * 2, v_kmaj + k4 * 2, idesc_sdp, k4 != 0, on);
                umma_commit(bar_sdp, on);
                return true;
            };
            if (!warp_wait(bar_kv, 0)) { atomicExch(p.status, 301); ok = false; }
            if (warp == 8) {
                if (ok && n_iter > 0 && !issue_sdp(0)) { atomicExch(p.status, 302); ok = false; }
                for (int it = 0; it + 1 < n_iter && ok; ++it) {
                    if (!warp_wait(bar_sread, it & 1)) { atomicExch(p.status, 308); ok = false; break; }      // S / dP columns are free again
                    tc_fence_after();
                    if (!issue_sdp(it + 1)) { atomicExch(p.status, 302); ok = false; break; }
                }
            } else {
                for (int it = 0; it < n_iter && ok; ++it) {
                    // P / dS of the iteration are in shared memory; its Q / dO stage landed before its S / dP were issued (the wait on
                    // the stage's barrier returns at once and orders this thread's products after the copy as well)
                    const int st = it % BP_STAGES;
                    if (!warp_wait(bar_pds, it & 1) || !warp_wait(&bar_qdo[st], (it / BP_STAGES) & 1)) { atomicExch(p.status, 303); ok = false; break; }
                    tc_fence_after();
                    const uint64_t qb = q_mn + st * (BP_T_BYTES >> 4), db = do_mn + st * (BP_T_BYTES >> 4);
#pragma unroll
                    for (int k8 = 0; k8 < BP_TILE / 16; ++k8)        // dV += P^T dO   (contraction over the 128 query rows)
                        umma_f16(tmem_base + BP_COL_DV, p_mn + k8 * 128, db + k8 * 128, idesc_g, (it | k8) != 0, on);
#pragma unroll
                    for (int k8 = 0; k8 < BP_TILE / 16; ++k8)        // dK += dS^T Q
                        umma_f16(tmem_base + BP_COL_DK, ds_mn + k8 * 128, qb + k8 * 128, idesc_g, (it | k8) != 0, on);
#pragma unroll
                    for (int k8 = 0; k8 < BP_TILE / 16; ++k8)        // dQ = dS K      (contraction over the 128 keys: two 64-key slabs of dS)
                        umma_f16(tmem_base + BP_COL_DQ + (it & 1) * BP_HD, ds_kmaj + (k8 >> 2) * (BP_TILE * 128 >> 4) + (k8 & 3) * 2, k_mn + k8 * 128, idesc_dq, k8 != 0, on);
                    umma_commit(bar_mma, on);
                }
            }
        }
    } else {
        const int quad = warp & 3, half = warp >> 2;
        const int r = quad * 32 + lane;
        const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
        const int sw = r & 7;
        const bool leader = threadIdx.x == 0;
        uint8_t* p_row = sp + half * (BP_TILE * 128) + r * 128;
        uint8_t* ds_row = sds + half * (BP_TILE * 128) + r * 128;
        uint8_t* stg_row = stg + half * (BP_TILE * 128) + r * 128;         // fp32 dQ staging: this thread fills one slab of 32 columns of its row
        const float c = p.scale_log2e;
        constexpr bool capped = CAPPED;
        const float cap_a = capped ? p.softcap / p.scale : 0.f, cap_b = capped ? p.scale / p.softcap : 0.f;
        const uint32_t s_addr = tmem_base + BP_COL_S + lane_off + half * 64, dp_addr = tmem_base + BP_COL_DP + lane_off + half * 64;
        // dQ of iteration `jt`: this thread's row, 32 of the 64 columns; scaled, staged, then one TMA reduce-add per 32-column slab
        auto drain_dq = [&](int jt) {
            uint32_t qreg[32];
            tmem_ld_32x32b_x32(tmem_base + BP_COL_DQ + (jt & 1) * BP_HD + lane_off + half * 32, qreg);
            tmem_ld_wait();
            tc_fence_before();
            if (leader) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            asm volatile("bar.sync 1, 256;" ::: "memory");                  // the previous reduce has finished reading the staging tile
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                *reinterpret_cast<float4*>(stg_row + ((q ^ sw) << 4)) =
                    make_float4(__uint_as_float(qreg[4 * q]) * p.scale, __uint_as_float(qreg[4 * q + 1]) * p.scale,
                                __uint_as_float(qreg[4 * q + 2]) * p.scale, __uint_as_float(qreg[4 * q + 3]) * p.scale);
            }
            fence_proxy_async();
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (leader) {
                const int head = kv_head * p.group + jt / n_q;
                const int q0 = (kv_tile + jt % n_q) * BP_TILE;
#pragma unroll
                for (int sl = 0; sl < 2; ++sl) {
                    asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
                                 ::"l"(&tmap_dq), "r"(smem_u32(stg + sl * (BP_TILE * 128))), "r"(head * BP_HD + sl * 32), "r"(q0), "r"(batch) : "memory");
                }
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        };
        // statistics of this thread's query row of iteration `jt`, [batch, head, seq].  Rows past the sequence end are zeros; an
        // infinite log-sum-exp makes their probabilities 0
        float lse_next = INFINITY, delta_next = 0.f;
        auto fetch_stats = [&](int jt) {
            const int head_j = kv_head * p.group + jt / n_q;
            const int qpos_j = (kv_tile + jt % n_q) * BP_TILE + r;
            const bool live = qpos_j < p.seq_len;
            const long long stat = (static_cast<long long>(batch) * p.heads + head_j) * p.seq_len + qpos_j;
            lse_next = live ? p.lse[stat] : INFINITY;
            delta_next = live ? p.delta[stat] : 0.f;
        };
        if (n_iter > 0) fetch_stats(0);
        for (int it = 0; it < n_iter; ++it) {
            const uint32_t ph = it & 1;
            const int head = kv_head * p.group + it / n_q;
            const int q0 = (kv_tile + it % n_q) * BP_TILE;
            const int qpos = q0 + r;
            // the row statistics were fetched during the previous iteration; fetch the next iteration's now, so that their global-memory
            // latency runs under this iteration's arithmetic instead of in front of it
            const float lse2 = lse_next * 1.4426950408889634f;
            const float delta = delta_next;
            if (it + 1 < n_iter) fetch_stats(it + 1);
            int w_row = window, w_last = window;                        // document masking: see the forward kernel
            if (p.doc_start) {
                const int last = min(q0 + BP_TILE, p.seq_len) - 1;
                if (qpos < p.seq_len) w_row = min(window, qpos - p.doc_start[row0 + qpos]);
                w_last = min(window, last - p.doc_start[row0 + last]);
            }
            const bool need_mask = (q0 == kv0) || (q0 + BP_TILE - 1 - kv0 > w_last);
            if (ok && !mbar_wait(bar_sdp, ph)) { atomicExch(p.status, 305); ok = false; }
            tc_fence_after();
            uint4 wp[8], wd[8];
            if (need_mask) bp_tile_math<true, capped>(s_addr, dp_addr, wp, wd, kv0 + half * 64, qpos, w_row, c, lse2, delta, cap_a, cap_b);
            else bp_tile_math<false, capped>(s_addr, dp_addr, wp, wd, kv0 + half * 64, qpos, w_row, c, lse2, delta, cap_a, cap_b);
            tc_fence_before();
            mbar_arrive(bar_sread);                                       // S / dP of the next iteration may be written
            // the gradient products of the previous iteration read the P / dS tiles
            if (it > 0) {
                if (ok && !mbar_wait(bar_mma, (it - 1) & 1)) { atomicExch(p.status, 306); ok = false; }
                tc_fence_after();
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int piece = (j ^ sw) << 4;
                *reinterpret_cast<uint4*>(p_row + piece) = wp[j];
                *reinterpret_cast<uint4*>(ds_row + piece) = wd[j];
            }
            fence_proxy_async();
            mbar_arrive(bar_pds);
            // the previous iteration's dQ leaves while the tensor core works on this one's products, whose dQ goes to the other columns
            // (those were read out before this thread's arrival above, so the issuing thread may overwrite them)
            if (it > 0) drain_dq(it - 1);
        }
        if (n_iter > 0) {
            if (ok && !mbar_wait(bar_mma, (n_iter - 1) & 1)) { atomicExch(p.status, 306); ok = false; }
            tc_fence_after();
            drain_dq(n_iter - 1);
        }
        if (ok && n_iter > 0) {
            // dK, dV: TMEM lanes are the 128 keys of this CTA; each thread writes half of the columns of its key row
            const bool live = kv0 + r < p.seq_len;
            const long long token = static_cast<long long>(row0) + kv0 + r;
            __nv_bfloat16* dk = reinterpret_cast<__nv_bfloat16*>(p.dk) + token * p.dkv_stride + kv_head * BP_HD + half * 32;
            __nv_bfloat16* dv = reinterpret_cast<__nv_bfloat16*>(p.dv) + token * p.dv_stride + kv_head * p.dv_head + half * 32;
            uint32_t vreg[32], kreg[32];
            tmem_ld_32x32b_x32(tmem_base + BP_COL_DV + lane_off + half * 32, vreg);
            tmem_ld_32x32b_x32(tmem_base + BP_COL_DK + lane_off + half * 32, kreg);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint4 wv, wk;
                wv.x = pack_bf16x2(__uint_as_float(vreg[8 * q]), __uint_as_float(vreg[8 * q + 1]));
                wv.y = pack_bf16x2(__uint_as_float(vreg[8 * q + 2]), __uint_as_float(vreg[8 * q + 3]));
                wv.z = pack_bf16x2(__uint_as_float(vreg[8 * q + 4]), __uint_as_float(vreg[8 * q + 5]));
                wv.w = pack_bf16x2(__uint_as_float(vreg[8 * q + 6]), __uint_as_float(vreg[8 * q + 7]));
                if (live) *reinterpret_cast<uint4*>(dv + 8 * q) = wv;
                wk.x = pack_bf16x2(__uint_as_float(kreg[8 * q]) * p.scale, __uint_as_float(kreg[8 * q + 1]) * p.scale);
                wk.y = pack_bf16x2(__uint_as_float(kreg[8 * q + 2]) * p.scale, __uint_as_float(kreg[8 * q + 3]) * p.scale);
                wk.z = pack_bf16x2(__uint_as_float(kreg[8 * q + 4]) * p.scale, __uint_as_float(kreg[8 * q + 5]) * p.scale);
                wk.w = pack_bf16x2(__uint_as_float(kreg[8 * q + 6]) * p.scale, __uint_as_float(kreg[8 * q + 7]) * p.scale);
                if (live) *reinterpret_cast<uint4*>(dk + 8 * q) = wk;
            }
        }
        if (leader) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        if (*reinterpret_cast<volatile int*>(p.status) != 0) {    // a wait gave up: let MMAs and copies in flight drain before the columns are freed
            const long long start = clock64();
            while (clock64() - start < 200000) {}
        }
        tc_fence_after();
        tmem_dealloc(tmem_base, BP_TMEM_COLS);
    }
}

template <bool CAPPED>
static cudaError_t launch_pipe_variant(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                       const CUtensorMap& tdq, const AttnParams& p, cudaStream_t stream) {
    constexpr int smem = 2 * BP_T_BYTES + 2 * BP_STAGES * BP_T_BYTES + 2 * BP_PD_BYTES + BP_STG_BYTES + 1024 + 256;
    static_assert(smem <= 232448, "shared memory of the pipelined attention backward");
    auto kernel = attn_bwd_pipe_kernel<CAPPED>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    const int tiles = (p.seq_len + BP_TILE - 1) / BP_TILE, kv_heads = p.heads / p.group;
    const dim3 grid = p.long_first ? dim3(kv_heads, p.batch, tiles) : dim3(tiles, kv_heads, p.batch);
    kernel<<<grid, BP_THREADS, smem, stream>>>(tq, tk, tv, tdo, tdq, p);
    return cudaGetLastError();
}

cudaError_t launch_attn_bwd_pipe(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                 const CUtensorMap& tdq, const AttnParams& p, cudaStream_t stream) {
    return p.softcap > 0.f ? launch_pipe_variant<true>(tq, tk, tv, tdo, tdq, p, stream) : launch_pipe_variant<false>(tq, tk, tv, tdo, tdq, p, stream);
}

}  // namespace gm
