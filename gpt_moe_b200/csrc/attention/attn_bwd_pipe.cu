// Causal sliding-window attention backward for sm_100a, 64-wide heads, on transposed score tiles.
//
// One CTA owns 128 keys of one (batch, kv head) and walks the query tiles that see them (sequences of any length: the tensor maps end at
// the sequence's last row).  Scores are formed as S^T = K Q^T and dP^T = V dO^T, a TMEM lane per key, so that P^T and dS^T go back to TMEM as
// bf16 and are the A operand of dV += P^T dO and dK += dS^T Q without touching shared memory; only dS^T is also stored there, for
// dQ = dS K, which leaves by TMA reduce-add into an fp32 buffer.  The row statistics, which are per COLUMN of these tiles, are taken off by
// the products themselves: 16 more columns of contraction hold ones beside the keys and -LSE / scale (for dP^T: -delta) beside the queries,
// as three bf16 terms each, which is all 24 bits.
//   warps 0-7    softmax: thread = key row and half of the 128 queries.  P = exp2(c S) while dP^T is still being formed, P^T to
//                TMEM, then dS = P dP to TMEM (in dP's own columns) and to shared memory (two tiles in turn)
//   warp  8      MMA issue (a whole warp, see umma_f16 in ptx.cuh), per iteration: S^T of the next query tile and dV once P is there, dK and dQ
//                once dS is there, then dP^T of the next tile (its columns hold dS^T until dK is complete)
//   warp  9      TMA loads: K, V once; Q / dO through a three-deep ring, a stage refilled when the products that read it are complete
//   warps 10-13  dQ read-out and reduction (a warp stages and sends its 32 rows by itself), and the statistics of the query tiles through a
//                three-deep ring, the first visible key of every query among them (read in tiles that need a mask)
// us, 16 x 2048 tokens, 12 heads, window 1024 / 16384 tokens, 16 heads of 4 (delta pre-pass and dQ zero-fill included): this kernel 380 / 1480;
// with P and dS stored to shared memory for three products and dQ drained by the softmax warps 444 / 1740 (368 KB through shared memory an
// iteration are 2900 clocks at 128 bytes a clock, here 272 KB); transposed, but with the statistics read as broadcasts 452 / 1776 (32 16-byte
// reads a thread return 128 KB more); attn_bwd.cu 516 / 2375.  An iteration takes 2950 clocks, 2000 of them products: P 1350 (its 64
// exponentials; a quarter or half of them as polynomials change nothing), dS 720, the rest waits.  Registers: 14 warps leave 128 each.
// Reference counterpart: the backward of FlexAttention (model/attention/self_attention.py:250-255) as generated by Inductor.
#include "../common/ptx.cuh"
#include "attn.h"
#include "attn_math.cuh"

namespace gm {

constexpr int BP_THREADS = 448;
constexpr int BP_TILE = 128, BP_HD = 64;
constexpr int BP_T_BYTES = BP_TILE * BP_HD * 2;          // one 128 x 64 bf16 tile
constexpr int BP_DS_BYTES = BP_TILE * BP_TILE * 2;       // dS^T tile (two 128-byte-wide slabs)
constexpr int BP_STG_BYTES = BP_TILE * 32 * 4;           // dQ staging: per drain warp a slab of 32 rows x 32 fp32 columns
constexpr int BP_STAGES = 3;
constexpr int BP_AUG_BYTES = BP_TILE * 16;               // eight more bf16 columns of 128 rows, unswizzled: 16 bytes a row
constexpr int BP_MASK_BYTES = BP_TILE * 4 + 16;          // first visible key of each query; whether the tile needs a mask
constexpr uint32_t BP_TMEM_COLS = 512;
constexpr uint32_t BP_COL_S = 0, BP_COL_DP = 128, BP_COL_DV = 256, BP_COL_DK = 320, BP_COL_DQ = 384, BP_COL_P = 448;

__device__ __forceinline__ float bp_tanh_approx(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// unswizzled K-major operand of 16 columns: 8-row groups of the first eight columns 128 bytes apart, the other eight `lbo` bytes on
__device__ __forceinline__ uint64_t bp_plain_desc(uint32_t addr, uint32_t lbo) {
    return static_cast<uint64_t>((addr & 0x3FFFF) >> 4) | static_cast<uint64_t>((lbo >> 4) & 0x3FFF) << 16 | static_cast<uint64_t>(128 >> 4) << 32 | 1ull << 46;
}
// an fp32 value as three bf16 terms (24 bits), the rest of the 16 bytes zeros
__device__ __forceinline__ uint4 bp_terms(float x) {
    const uint32_t a = pack_bf16x2(x, 0.f);
    const float r1 = x - __uint_as_float(a << 16);
    const uint32_t b = pack_bf16x2(r1, 0.f);
    const uint32_t c = pack_bf16x2(r1 - __uint_as_float(b << 16), 0.f);
    return make_uint4((a & 0xffffu) | (b << 16), c & 0xffffu, 0u, 0u);
}

// P of this thread's key and 32 queries from its S columns: packed to bf16 for TMEM, and (in place) the factor that dS takes: P, with soft-capping
// P (1 - tanh^2).  The scores arrive with the log-sum-exp of their queries taken off; soft-capped ones arrive as they are, and `lse2` (log2 units) is read.
template <bool MASK, bool CAP>
__device__ __forceinline__ void bp_probabilities(uint32_t (&s)[32], uint32_t (&packed)[16], const float* lse2, const int* first_key, int kpos, int qpos0,
                                                 float c, float cap_a, float cap_b) {
    const uint64_t c2 = pack2(c, c);
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        float e[2], chain[2] = {1.f, 1.f};
        if (CAP) {
            const float2 l = *reinterpret_cast<const float2*>(lse2 + i);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float th = bp_tanh_approx(__uint_as_float(s[i + j]) * cap_b);
                chain[j] = 1.f - th * th;
                e[j] = exp2f(fmaf(cap_a * th, c, j == 0 ? -l.x : -l.y));
            }
        } else {
            unpack2(mul2(pack2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), c2), e[0], e[1]);
            e[0] = exp2f(e[0]);
            e[1] = exp2f(e[1]);
        }
        if (MASK) {
            const int2 first = *reinterpret_cast<const int2*>(first_key + i);
            if (kpos > qpos0 + i || kpos < first.x) e[0] = 0.f;
            if (kpos > qpos0 + i + 1 || kpos < first.y) e[1] = 0.f;
        }
        s[i] = __float_as_uint(CAP ? e[0] * chain[0] : e[0]);
        s[i + 1] = __float_as_uint(CAP ? e[1] * chain[1] : e[1]);
        packed[i / 2] = pack_bf16x2(e[0], e[1]);
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
    uint8_t* sds = sdo + BP_STAGES * BP_T_BYTES;         // two tiles
    uint8_t* stg = sds + 2 * BP_DS_BYTES;
    uint8_t* aug_lse = stg + BP_STG_BYTES;               // BP_STAGES: -LSE / scale of the queries as bf16 terms (soft-capping: LSE in log2 units, fp32)
    uint8_t* aug_delta = aug_lse + BP_STAGES * BP_AUG_BYTES;         // BP_STAGES: -delta as bf16 terms
    uint8_t* aug_ones = aug_delta + BP_STAGES * BP_AUG_BYTES;        // ones in three columns, for the 128 keys
    uint8_t* aug_zero = aug_ones + BP_AUG_BYTES;                     // columns 8 .. 15 of all of these
    uint8_t* masks = aug_zero + BP_AUG_BYTES;            // BP_STAGES entries
    uint64_t* bars = reinterpret_cast<uint64_t*>(masks + BP_STAGES * BP_MASK_BYTES);
    uint64_t* bar_kv = bars + 0;
    uint64_t* bar_s = bars + 1;                          // S^T of an iteration complete
    uint64_t* bar_p = bars + 2;                          // S^T read and P^T in TMEM (256 arrivals)
    uint64_t* bar_dv = bars + 3;                         // dV product complete: P^T may be overwritten
    uint64_t* bar_dp = bars + 4;                         // dP^T complete
    uint64_t* bar_ds = bars + 5;                         // dS^T in TMEM and in shared memory (256 arrivals)
    uint64_t* bar_dk = bars + 6;                         // dK product complete: dS^T's columns may be overwritten
    uint64_t* bar_mma = bars + 7;                        // all products of an iteration complete: dQ may be read out
    uint64_t* bar_dq = bars + 8;                         // dQ read out of TMEM (one arrival per drain warp)
    uint64_t* bar_end = bars + 9;                        // all products of the last iteration complete
    uint64_t* bar_free = bars + 10;                      // [BP_STAGES] the products that read a Q / dO stage are complete
    uint64_t* bar_qdo = bar_free + BP_STAGES;            // [BP_STAGES] Q / dO tile landed
    uint64_t* bar_stat = bar_qdo + BP_STAGES;            // [BP_STAGES] statistics of a query tile are there (one arrival per drain warp)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_stat + BP_STAGES);

    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int kv_tile = p.long_first ? blockIdx.z : blockIdx.x, kv_head = p.long_first ? blockIdx.x : blockIdx.y;
    const int batch = p.long_first ? blockIdx.y : blockIdx.z;
    const int kv0 = kv_tile * BP_TILE;
    const int window = uniform(p.window_ptr ? min(max(*p.window_ptr, 0), p.seq_len) : p.window);
    const int q_tiles_total = (p.seq_len + BP_TILE - 1) / BP_TILE;
    int last_q_tile = (kv0 + BP_TILE - 1 + window) / BP_TILE;
    if (last_q_tile > q_tiles_total - 1) last_q_tile = q_tiles_total - 1;
    const int n_q = last_q_tile - kv_tile + 1;        // query tiles per head that see this key tile: at least its own
    const int n_iter = n_q * p.group;                 // times the query heads sharing this kv head
    const int row0 = batch * p.seq_len;

    if (threadIdx.x == 0) {
        mbar_init(bar_kv, 1); mbar_init(bar_s, 1); mbar_init(bar_p, 256); mbar_init(bar_dv, 1); mbar_init(bar_dp, 1); mbar_init(bar_ds, 256);
        mbar_init(bar_dk, 1); mbar_init(bar_mma, 1); mbar_init(bar_dq, 4); mbar_init(bar_end, 1);
        for (int st = 0; st < BP_STAGES; ++st) { mbar_init(&bar_free[st], 1); mbar_init(&bar_qdo[st], 1); mbar_init(&bar_stat[st], 4); }
        fence_barrier_init();
    }
    if (threadIdx.x < BP_TILE) {
        reinterpret_cast<uint4*>(aug_ones)[threadIdx.x] = make_uint4(0x3f803f80u, 0x00003f80u, 0u, 0u);
        reinterpret_cast<uint4*>(aug_zero)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async();
    }
    if (warp == 8) { tmem_alloc(tmem_slot, BP_TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = uniform(*tmem_slot);
    bool ok = true;

    if (warp == 9) {
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
            if (!warp_wait(&bar_free[it % BP_STAGES], (it / BP_STAGES - 1) & 1)) { atomicExch(p.status, 311); break; }
            load_qdo(it);
        }
    } else if (warp == 8) {
        const uint32_t on = elect_one();
        constexpr uint32_t idesc_sdp = make_idesc_bf16(BP_TILE, BP_TILE, false, false);
        constexpr uint32_t idesc_g = make_idesc_bf16(BP_TILE, BP_HD, false, true);        // dV, dK: A in TMEM, B MN-major
        constexpr uint32_t idesc_dq = make_idesc_bf16(BP_TILE, BP_HD, true, true);        // dQ: A and B MN-major
        // descriptors formed once; the address field counts 16-byte units: a 16-column slice of a K-major tile is 2 units on, a
        // 16-row slice of an MN-major tile 128 units, a ring stage 1024 units
        const uint64_t k_kmaj = make_smem_desc(smem_u32(sk), 16, 1024), v_kmaj = make_smem_desc(smem_u32(sv), 16, 1024);
        const uint64_t q_kmaj = make_smem_desc(smem_u32(sq), 16, 1024), do_kmaj = make_smem_desc(smem_u32(sdo), 16, 1024);
        const uint64_t q_mn = make_smem_desc(smem_u32(sq), BP_TILE * 128, 1024), do_mn = make_smem_desc(smem_u32(sdo), BP_TILE * 128, 1024);
        const uint64_t k_mn = make_smem_desc(smem_u32(sk), BP_TILE * 128, 1024), ds_mn = make_smem_desc(smem_u32(sds), BP_TILE * 128, 1024);
        const uint32_t zero = smem_u32(aug_zero);
        const uint64_t ones = bp_plain_desc(smem_u32(aug_ones), zero - smem_u32(aug_ones));
        auto terms = [&](const uint8_t* aug, int it) {
            const uint32_t at = smem_u32(aug) + (it % BP_STAGES) * BP_AUG_BYTES;
            return bp_plain_desc(at, zero - at);
        };
        auto issue_s = [&](int it) {                     // S^T = K Q^T - LSE / scale
            const uint64_t qb = q_kmaj + (it % BP_STAGES) * (BP_T_BYTES >> 4);
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4) umma_f16(tmem_base + BP_COL_S, k_kmaj + k4 * 2, qb + k4 * 2, idesc_sdp, k4 != 0, on);
            if (!CAPPED) umma_f16(tmem_base + BP_COL_S, ones, terms(aug_lse, it), idesc_sdp, 1, on);
            umma_commit(bar_s, on);
        };
        auto issue_dp = [&](int it) {                    // dP^T = V dO^T - delta
            const uint64_t db = do_kmaj + (it % BP_STAGES) * (BP_T_BYTES >> 4);
#pragma unroll
            for (int k4 = 0; k4 < 4; ++k4) umma_f16(tmem_base + BP_COL_DP, v_kmaj + k4 * 2, db + k4 * 2, idesc_sdp, k4 != 0, on);
            umma_f16(tmem_base + BP_COL_DP, ones, terms(aug_delta, it), idesc_sdp, 1, on);
            umma_commit(bar_dp, on);
        };
        if (!warp_wait(bar_kv, 0) || !warp_wait(&bar_qdo[0], 0) || !warp_wait(&bar_stat[0], 0)) { atomicExch(p.status, 301); ok = false; }
        if (ok) { tc_fence_after(); issue_s(0); issue_dp(0); }
        for (int it = 0; it < n_iter && ok; ++it) {
            const int st = it % BP_STAGES, next = (it + 1) % BP_STAGES;
            const bool more = it + 1 < n_iter;
            if (!warp_wait(bar_p, it & 1)) { atomicExch(p.status, 302); ok = false; break; }
            if (more && (!warp_wait(&bar_qdo[next], ((it + 1) / BP_STAGES) & 1) || !warp_wait(&bar_stat[next], ((it + 1) / BP_STAGES) & 1))) { atomicExch(p.status, 303); ok = false; break; }
            tc_fence_after();
            if (more) issue_s(it + 1);
            const uint64_t qb = q_mn + st * (BP_T_BYTES >> 4), db = do_mn + st * (BP_T_BYTES >> 4);
#pragma unroll
            for (int k8 = 0; k8 < BP_TILE / 16; ++k8)        // dV += P^T dO   (contraction over the 128 queries, 16 of them in 8 columns)
                umma_f16_ta(tmem_base + BP_COL_DV, tmem_base + BP_COL_P + k8 * 8, db + k8 * 128, idesc_g, (it | k8) != 0, on);
            umma_commit(bar_dv, on);
            if (!warp_wait(bar_ds, it & 1)) { atomicExch(p.status, 304); ok = false; break; }
            tc_fence_after();
#pragma unroll
            for (int k8 = 0; k8 < BP_TILE / 16; ++k8)        // dK += dS^T Q   (each half of the queries in the first half of its own dP^T columns)
                umma_f16_ta(tmem_base + BP_COL_DK, tmem_base + BP_COL_DP + (k8 >> 2) * 64 + (k8 & 3) * 8, qb + k8 * 128, idesc_g, (it | k8) != 0, on);
            umma_commit(bar_dk, on);
            if (it > 0) {
                if (!warp_wait(bar_dq, (it - 1) & 1)) { atomicExch(p.status, 307); ok = false; break; }
                tc_fence_after();
            }
            const uint64_t da = ds_mn + (it & 1) * (BP_DS_BYTES >> 4);
#pragma unroll
            for (int k8 = 0; k8 < BP_TILE / 16; ++k8)        // dQ = dS K      (contraction over the 128 keys)
                umma_f16(tmem_base + BP_COL_DQ, da + k8 * 128, k_mn + k8 * 128, idesc_dq, k8 != 0, on);
            umma_commit(&bar_free[st], on);
            umma_commit(bar_mma, on);
            if (more) {
                if (!warp_wait(bar_dk, it & 1)) { atomicExch(p.status, 308); ok = false; break; }
                issue_dp(it + 1);
            }
        }
        umma_commit(bar_end, on);
    } else if (warp >= 10) {
        const int quad = warp & 3;                       // TMEM lanes 32 quad .. + 31: query rows of the dQ tile
        const int r = quad * 32 + lane, sw = lane & 7;
        uint8_t* mine = stg + quad * (BP_STG_BYTES / 4);
        // statistics of query row r of iteration `jt`, [batch, head, seq].  Rows past the sequence end are zeros; a huge log-sum-exp makes
        // their probabilities 0 - over the scale a constant, as 1e30 over a scale of 1e-12 would be infinite and the second of its terms a NaN
        const float per_scale = 1.f / p.scale, never = copysignf(1e38f, -p.scale);
        float lse = 1e30f, delta = 0.f;
        bool live = false;
        int first_key = 0, need_mask = 0;
        auto fetch_stats = [&](int jt) {
            const int head = kv_head * p.group + jt / n_q, q0 = (kv_tile + jt % n_q) * BP_TILE, qpos = q0 + r;
            live = qpos < p.seq_len;
            const long long stat = (static_cast<long long>(batch) * p.heads + head) * p.seq_len + qpos;
            lse = live ? p.lse[stat] : 1e30f;
            delta = live ? p.delta[stat] : 0.f;
            const int last = min(q0 + BP_TILE, p.seq_len) - 1;
            int w_row = window, w_last = window;                        // document masking: see the forward kernel
            if (p.doc_start) {
                if (live) w_row = min(window, qpos - p.doc_start[row0 + qpos]);
                w_last = min(window, last - p.doc_start[row0 + last]);
            }
            first_key = qpos - w_row;
            need_mask = q0 == kv0 || q0 + BP_TILE - 1 - kv0 > w_last;
        };
        auto put_stats = [&](int jt) {
            const int st = jt % BP_STAGES;
            if (CAPPED) reinterpret_cast<float*>(aug_lse + st * BP_AUG_BYTES)[r] = lse * 1.4426950408889634f;
            else reinterpret_cast<uint4*>(aug_lse + st * BP_AUG_BYTES)[r] = bp_terms(live ? -lse * per_scale : never);
            reinterpret_cast<uint4*>(aug_delta + st * BP_AUG_BYTES)[r] = bp_terms(-delta);
            int* mask = reinterpret_cast<int*>(masks + st * BP_MASK_BYTES);
            mask[r] = first_key;
            if (r == 0) mask[BP_TILE] = need_mask;
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_stat[jt % BP_STAGES]);
        };
        for (int jt = 0; jt < BP_STAGES && jt < n_iter; ++jt) { fetch_stats(jt); put_stats(jt); }
        for (int jt = 0; jt < n_iter; ++jt) {
            if (jt + BP_STAGES < n_iter) fetch_stats(jt + BP_STAGES);       // in flight while dQ is awaited
            if (ok && !mbar_wait(bar_mma, jt & 1)) { atomicExch(p.status, 306); ok = false; }
            tc_fence_after();
            uint32_t q[2][32];
#pragma unroll
            for (int sl = 0; sl < 2; ++sl) tmem_ld_32x32b_x32(tmem_base + BP_COL_DQ + sl * 32 + (static_cast<uint32_t>(quad * 32) << 16), q[sl]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_dq);
            if (jt + BP_STAGES < n_iter) put_stats(jt + BP_STAGES);         // iteration jt is through: its entry is free
            const int head = kv_head * p.group + jt / n_q, q0 = (kv_tile + jt % n_q) * BP_TILE + quad * 32;
#pragma unroll
            for (int sl = 0; sl < 2; ++sl) {
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the previous reduction has read the slab
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    *reinterpret_cast<float4*>(mine + lane * 128 + ((k ^ sw) << 4)) =
                        make_float4(__uint_as_float(q[sl][4 * k]) * p.scale, __uint_as_float(q[sl][4 * k + 1]) * p.scale,
                                    __uint_as_float(q[sl][4 * k + 2]) * p.scale, __uint_as_float(q[sl][4 * k + 3]) * p.scale);
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    if (q0 < p.seq_len)
                        asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
                                     ::"l"(&tmap_dq), "r"(smem_u32(mine)), "r"(head * BP_HD + sl * 32), "r"(q0), "r"(batch) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else {
        const int quad = warp & 3, half = warp >> 2;
        const int r = quad * 32 + lane;                  // key row
        const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
        const int sw = r & 7;
        const float c = p.scale_log2e;
        constexpr bool capped = CAPPED;
        const float cap_a = capped ? p.softcap / p.scale : 0.f, cap_b = capped ? p.scale / p.softcap : 0.f;
        const uint32_t s_addr = tmem_base + BP_COL_S + lane_off + half * 64, dp_addr = tmem_base + BP_COL_DP + lane_off + half * 64;
        const uint32_t p_addr = tmem_base + BP_COL_P + lane_off + half * 32;
        uint8_t* ds_row = sds + half * (BP_TILE * 128) + r * 128;
        for (int it = 0; it < n_iter; ++it) {
            const int st = it % BP_STAGES;
            const float* lse2 = reinterpret_cast<const float*>(aug_lse + st * BP_AUG_BYTES) + half * 64;
            const int* mask = reinterpret_cast<const int*>(masks + st * BP_MASK_BYTES);
            const int q0 = (kv_tile + it % n_q) * BP_TILE + half * 64;
            if (ok && !mbar_wait(&bar_stat[st], (it / BP_STAGES) & 1)) { atomicExch(p.status, 309); ok = false; }
            if (ok && !mbar_wait(bar_s, it & 1)) { atomicExch(p.status, 305); ok = false; }
            tc_fence_after();
            uint32_t s[2][32];
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) tmem_ld_32x32b_x32(s_addr + cc * 32, s[cc]);
            tmem_ld_wait();
            const bool masked = mask[BP_TILE] != 0;
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                uint32_t packed[16];
                const int* first_key = mask + half * 64 + cc * 32;
                if (masked) bp_probabilities<true, capped>(s[cc], packed, lse2 + cc * 32, first_key, kv0 + r, q0 + cc * 32, c, cap_a, cap_b);
                else bp_probabilities<false, capped>(s[cc], packed, lse2 + cc * 32, first_key, kv0 + r, q0 + cc * 32, c, cap_a, cap_b);
                if (cc == 0) {
                    if (it > 0 && ok && !mbar_wait(bar_dv, (it - 1) & 1)) { atomicExch(p.status, 310); ok = false; }      // P^T of the tile before has been used
                    tc_fence_after();
                }
                tmem_st_32x32b_x16(p_addr + cc * 16, packed);
            }
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(bar_p);                                           // S^T of the next tile may be written
            if (ok && !mbar_wait(bar_dp, it & 1)) { atomicExch(p.status, 312); ok = false; }
            tc_fence_after();
            uint8_t* row = ds_row + (it & 1) * BP_DS_BYTES;               // last read by dQ of iteration it - 2, complete before dP^T of this one was issued
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                uint32_t d[32], packed[16];
                tmem_ld_32x32b_x32(dp_addr + cc * 32, d);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    float a, b;
                    unpack2(mul2(pack2(__uint_as_float(s[cc][i]), __uint_as_float(s[cc][i + 1])), pack2(__uint_as_float(d[i]), __uint_as_float(d[i + 1]))), a, b);
                    packed[i / 2] = pack_bf16x2(a, b);
                }
                tmem_st_32x32b_x16(dp_addr + cc * 16, packed);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    *reinterpret_cast<uint4*>(row + (((cc * 4 + k) ^ sw) << 4)) = make_uint4(packed[4 * k], packed[4 * k + 1], packed[4 * k + 2], packed[4 * k + 3]);
            }
            tmem_st_wait();
            fence_proxy_async();
            tc_fence_before();
            mbar_arrive(bar_ds);
        }
        if (ok && !mbar_wait(bar_end, 0)) { atomicExch(p.status, 313); ok = false; }
        tc_fence_after();
        // dK, dV: TMEM lanes are the 128 keys; a thread takes half of the columns of its key row to shared memory (dS^T has been used), and
        // the rows leave 128 bytes at a time
#pragma unroll
        for (int which = 0; which < 2; ++which) {
            uint32_t v[32];
            tmem_ld_32x32b_x32(tmem_base + (which == 0 ? BP_COL_DV : BP_COL_DK) + lane_off + half * 32, v);
            tmem_ld_wait();
            const float f = which == 0 ? 1.f : p.scale;
            uint8_t* to = sds + which * BP_T_BYTES + r * 128;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                uint4 w;
                w.x = pack_bf16x2(__uint_as_float(v[8 * k]) * f, __uint_as_float(v[8 * k + 1]) * f);
                w.y = pack_bf16x2(__uint_as_float(v[8 * k + 2]) * f, __uint_as_float(v[8 * k + 3]) * f);
                w.z = pack_bf16x2(__uint_as_float(v[8 * k + 4]) * f, __uint_as_float(v[8 * k + 5]) * f);
                w.w = pack_bf16x2(__uint_as_float(v[8 * k + 6]) * f, __uint_as_float(v[8 * k + 7]) * f);
                *reinterpret_cast<uint4*>(to + (((half * 4 + k) ^ sw) << 4)) = w;
            }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const int piece = lane & 7;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int key = warp * 16 + i * 4 + (lane >> 3);
            if (ok && kv0 + key < p.seq_len) {
                const long long token = static_cast<long long>(row0) + kv0 + key;
                const uint8_t* from = sds + key * 128 + ((piece ^ (key & 7)) << 4);
                *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.dv) + token * p.dv_stride + kv_head * p.dv_head + piece * 8) = *reinterpret_cast<const uint4*>(from);
                *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.dk) + token * p.dkv_stride + kv_head * BP_HD + piece * 8) = *reinterpret_cast<const uint4*>(from + BP_T_BYTES);
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
        tmem_dealloc(tmem_base, BP_TMEM_COLS);
    }
}

template <bool CAPPED>
static cudaError_t launch_pipe_variant(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                       const CUtensorMap& tdq, const AttnParams& p, cudaStream_t stream) {
    constexpr int smem = 2 * BP_T_BYTES + 2 * BP_STAGES * BP_T_BYTES + 2 * BP_DS_BYTES + BP_STG_BYTES + (2 * BP_STAGES + 2) * BP_AUG_BYTES +
                         BP_STAGES * BP_MASK_BYTES + 1024 + 192;
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
