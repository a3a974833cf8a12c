// Persistent, warp-specialised bf16 GEMM for sm_100a: D = alpha * A * B^T (+ beta * C) (+ D).
//
// CTAs run as pairs (a cluster of two on neighbouring SMs, tcgen05 cta_group::2).  A pair walks a list of
// 256 x 256 output tiles: each CTA owns 128 of the rows and stages only HALF of the B tile, the tensor cores of
// both SMs read both halves, so a CTA pulls 32 KB instead of 48 KB through L2 per 128 x 256 x 64 block of work -
// the main loop of a one-CTA kernel is bound by exactly that traffic.  Roles inside each CTA:
//   warp 0  : TMA producer   - fills a 5-stage ring of {A 128x64, B 128x64} bf16 tiles (128B swizzle; with
//                              128-column tiles six stages and B 64x64); the
//                              bytes of both CTAs are counted on the leader's (even CTA's) barrier
//   warp 1  : MMA issuer     - leader CTA only: the whole warp walks the loop, one lane's tcgen05.mma (M256 N256 K16) go into one of
//                              two TMEM accumulators (2 x 256 columns in each CTA), commits to both CTAs
//   warps 2-9: epilogue      - tcgen05.ld the finished accumulator (thread = row; two warps per TMEM lane
//                              quadrant split the columns), scale / add C, convert, stage 128-byte-swizzled
//                              slabs of its 32 rows by itself and hand them to TMA (store, or
//                              reduce-add for fp32 accumulation and split-K); overlaps the next tile's main
//                              loop.  TMA clips rows/columns outside the tensor.
// Operands may be K-major ([rows, K] with K contiguous) or MN-major ([K, rows] with rows
// contiguous); both are read straight from row-major tensors by TMA, so forward (X W^T), input
// gradient (dY W) and weight gradient (dY^T X) all run without a transposed copy.
//
// Three tile enumerations share the kernel:
//   DENSE     (optionally batched over z)                      - projections, LM head, Polar Express
//             symmetric results (X X^T, A A with A symmetric): only the tiles on or above the diagonal are computed, the
//             epilogue stores every off-diagonal tile a second time transposed (the reference's triangle-and-mirror
//             kernels, optimizers/polar_express.py:60-121 and :155-230)
//   GROUPED_M rows of A belong to experts; tile -> expert table on the device picks B's z slice
//             (expert segments are padded to 256 rows, so a pair's tile never straddles two experts)
//   GROUPED_K one output matrix per expert, contraction over that expert's (padded) row segment
//             - the expert weight gradient; empty experts get exact zeros
// Reference counterparts: Triton `_grouped_mm_kernel` (model/linear/default/grouped.py:12-70) and the
// cuBLAS calls behind every F.linear (model/linear/linear.py:23).
#include "../common/ptx.cuh"
#include "gemm.h"

#include <cuda.h>

namespace gm {

constexpr int BM = 128, BK = 64;
// columns of a pair's tile and the ring that goes with them: 256, or 128 where those leave half of the CTA pairs without a tile
template <int WIDTH>
struct Tiling {
    static constexpr int BN = WIDTH, BN_HALF = BN / 2, STAGES = WIDTH == 256 ? 5 : 6;
    static constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN_HALF * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
};
constexpr int GEMM_THREADS = 320;           // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
constexpr int GROUP_M = 4;               // in pair tiles (256 rows each)
constexpr uint32_t TMEM_COLS = 512;
constexpr int SLAB_BYTES = BM * 128;              // one slab of [128 rows][128 bytes]
constexpr int STAGING_BYTES = 2 * SLAB_BYTES;    // the staging area is twice this: two slabs of 4 KB for each epilogue warp, beside a C through TMA four slabs of all 128 rows

constexpr uint32_t kIdescBf16Operands = (1u << 7) | (1u << 10);      // operand formats of the instruction descriptor: 1 = bf16, 0 = fp16

// eight 16-bit values, bf16 or fp16 (uniform over the grid), to and from fp32
__device__ __forceinline__ void unpack_16bit(const uint4& raw, int f16, float* v) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 f = f16 ? __half22float2(*reinterpret_cast<const __half2*>(&w[e])) : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[e]));
        v[2 * e] = f.x;
        v[2 * e + 1] = f.y;
    }
}
__device__ __forceinline__ uint4 pack_16bit(const float* v, int f16) {
    uint4 o;
    if (f16) {
        o.x = pack_half2(v[0], v[1]); o.y = pack_half2(v[2], v[3]); o.z = pack_half2(v[4], v[5]); o.w = pack_half2(v[6], v[7]);
    } else {
        o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]); o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
    }
    return o;
}

struct TileCoord {
    int m0, n0;        // element offsets of the tile in the output
    int az, bz, dz;    // z (batch / expert) coordinates for A, B, D
    int k_begin, k_blocks;
    int m_limit, n_limit;
    bool store_zeros;  // no contraction work at all for this output tile: write zeros unless accumulating
};

// Work is enumerated in PAIR tiles (two vertically adjacent 128-row tiles, one per CTA of the pair); `m_tiles` counts
// the 128-row tiles rounded up to an even number.
template <int BN>
__device__ __forceinline__ int total_tiles(const GemmParams& p, int& m_tiles, int& n_tiles) {
    n_tiles = (p.N + BN - 1) / BN;
    if (p.mode == GEMM_GROUPED_M) {
        m_tiles = (*p.num_m_tiles + 1) & ~1;
        return m_tiles / 2 * n_tiles;
    }
    m_tiles = ((p.M + BM - 1) / BM + 1) & ~1;
    if (p.symmetric) return n_tiles * (n_tiles + 1) / 2 * p.batch;      // M == N: pair tiles (i, j) with i <= j
    return m_tiles / 2 * n_tiles * p.batch * p.split_k;
}

template <int BN>
__device__ __forceinline__ TileCoord tile_coord(const GemmParams& p, int tile, int cta_rank, int m_tiles, int n_tiles) {
    TileCoord t;
    int split = 0;
    if (p.mode != GEMM_GROUPED_M && p.split_k > 1) {
        split = tile % p.split_k;
        tile /= p.split_k;
    }
    const int m_pairs = m_tiles / 2;
    const int per_batch = p.symmetric ? n_tiles * (n_tiles + 1) / 2 : m_pairs * n_tiles;
    const int z = (p.mode == GEMM_GROUPED_M) ? 0 : tile / per_batch;
    int r = tile - z * per_batch;
    int mt, nt;
    if (p.symmetric) {
        // row i of the upper triangle holds n_tiles - i tiles
        int i = 0;
        while (r >= n_tiles - i) { r -= n_tiles - i; ++i; }
        mt = 2 * i + cta_rank;
        nt = i + r;
    } else {
        // grouped raster: GROUP_M pair-rows share their column sweep so A tiles stay in L2
        const int group = r / (GROUP_M * n_tiles);
        const int first_m = group * GROUP_M;
        const int rows_in_group = min(GROUP_M, m_pairs - first_m);
        r -= group * GROUP_M * n_tiles;
        mt = 2 * (first_m + r % rows_in_group) + cta_rank;
        nt = r / rows_in_group;
    }
    t.m0 = mt * BM;
    t.n0 = nt * BN;
    t.m_limit = p.M;
    t.n_limit = p.N;
    t.k_begin = 0;
    t.k_blocks = (p.K + BK - 1) / BK;
    t.az = t.dz = z;
    t.bz = p.b_shared ? 0 : z;
    if (p.mode == GEMM_GROUPED_M) {
        t.az = 0;
        t.dz = 0;
        t.bz = p.tile_expert[mt & ~1];          // both tiles of a pair belong to one expert (segments are padded to 256 rows)
        t.m_limit = *p.num_m_tiles * BM;
    } else if (p.mode == GEMM_GROUPED_K) {
        const int begin = z == 0 ? 0 : p.seg_ends[z - 1];
        t.az = t.bz = 0;
        t.k_begin = begin;
        t.k_blocks = (p.seg_ends[z] - begin) / BK;
    }
    t.store_zeros = t.k_blocks == 0;
    if (p.split_k > 1) {          // contiguous share of the K blocks; partial results meet in a TMA reduce-add
        const int per = (t.k_blocks + p.split_k - 1) / p.split_k;
        const int first = min(split * per, t.k_blocks);
        const int count = min(per, t.k_blocks - first);
        t.k_begin += first * BK;
        t.k_blocks = count;
        t.store_zeros = false;
        if (p.split_slabs) t.dz = split;
    }
    return t;
}

template <bool A_MN, bool B_MN, bool TMA_C, int WIDTH>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 const __grid_constant__ CUtensorMap tmap_d, const __grid_constant__ CUtensorMap tmap_c,
                 const __grid_constant__ CUtensorMap tmap_mirror, const GemmParams p) {
    using Tile = Tiling<WIDTH>;
    constexpr int BN = Tile::BN, BN_HALF = Tile::BN_HALF, STAGES = Tile::STAGES, A_BYTES = Tile::A_BYTES, STAGE_BYTES = Tile::STAGE_BYTES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* staging = smem + STAGES * STAGE_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(staging + 2 * STAGING_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* c_full = acc_empty + 2;                              // TMA_C: [2] slab of C landed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(c_full + 2);

    const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int cta_rank = static_cast<int>(cluster_ctarank());     // 0 = leader of the pair
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        // acc_empty of the leader collects one arrival per epilogue warp of each of the two CTAs (a remote arrival per thread
        // would put 256 messages per tile on the cluster's shared-memory network)
        for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 16); mbar_init(&c_full[a], 1); }
        fence_barrier_init();
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
        tma_prefetch_desc(&tmap_d);
        if (TMA_C) tma_prefetch_desc(&tmap_c);
    }
    if (warp == 1) { tmem_alloc_pair(tmem_slot, TMEM_COLS); tmem_relinquish_pair(); }
    tc_fence_before();
    cluster_sync_all();                                            // both CTAs' barriers exist before either signals the other
    tc_fence_after();
    const uint32_t tmem_base = uniform(*tmem_slot);
    grid_wait();                                                   // the above ran beside the end of the kernel before: sampling step 1.67 -> 1.52 ms, MLA prefill 151 -> 140 us

    int m_tiles, n_tiles;
    const int tiles = uniform(total_tiles<BN>(p, m_tiles, n_tiles));
    const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
    bool ok = true;

    if (warp == 0) {
        const uint32_t on = elect_one();
        int s = 0; uint32_t ph = 0;
        for (int tile = first_tile; tile < tiles && ok; tile += tile_step) {
            const TileCoord t = tile_coord<BN>(p, tile, cta_rank, m_tiles, n_tiles);
            const int k_blocks = uniform(t.k_blocks), k_begin = uniform(t.k_begin), bz = uniform(t.bz);
            for (int kb = 0; kb < k_blocks; ++kb) {
                if (!warp_wait(&empty[s], ph ^ 1)) { atomicExch(p.status, 101); ok = false; break; }
                if (cta_rank == 0 && on) mbar_expect_tx(&full[s], 2 * STAGE_BYTES);      // both CTAs' copies land on the leader's barrier
                uint8_t* a_dst = smem + s * STAGE_BYTES;
                uint8_t* b_dst = a_dst + A_BYTES;
                const int k = k_begin + kb * BK;
                const int bn0 = t.n0 + cta_rank * BN_HALF;                          // this CTA stages its half of the B tile
                if (A_MN) {
                    for (int i = 0; i < BM / 64; ++i) tma_load_3d_pair(a_dst + i * (64 * BK * 2), &tmap_a, &full[s], t.m0 + 64 * i, k, t.az, on);
                } else {
                    tma_load_3d_pair(a_dst, &tmap_a, &full[s], k, t.m0, t.az, on);
                }
                if (B_MN) {
                    for (int i = 0; i < BN_HALF / 64; ++i) tma_load_3d_pair(b_dst + i * (64 * BK * 2), &tmap_b, &full[s], bn0 + 64 * i, k, bz, on);
                } else {
                    tma_load_3d_pair(b_dst, &tmap_b, &full[s], k, bn0, bz, on);
                }
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        if (cta_rank == 0) {
            const uint32_t on = elect_one();
            const uint32_t idesc = make_idesc_bf16(2 * BM, BN, A_MN, B_MN) & ~(p.in_f16 ? kIdescBf16Operands : 0u);
            // K-major: 8-row groups are 1024 B apart, 16 K-elements = 32 B.  MN-major: 64-element column slabs are
            // BK*128 B apart (leading offset), 8-K-row groups 1024 B apart, 16 K-rows = 2048 B.
            constexpr uint32_t a_lbo = A_MN ? BK * 128 : 16, b_lbo = B_MN ? BK * 128 : 16;
            constexpr uint32_t a_kstep = A_MN ? 2048 : 32, b_kstep = B_MN ? 2048 : 32;
            int s = 0; uint32_t ph = 0; int acc = 0; uint32_t acc_ph = 0;
            for (int tile = first_tile; tile < tiles && ok; tile += tile_step) {
                const int k_blocks = uniform(tile_coord<BN>(p, tile, cta_rank, m_tiles, n_tiles).k_blocks);
                if (k_blocks == 0) continue;
                if (!warp_wait(&acc_empty[acc], acc_ph ^ 1)) { atomicExch(p.status, 102); ok = false; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * BN;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!warp_wait(&full[s], ph)) { atomicExch(p.status, 103); ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * STAGE_BYTES), b_addr = a_addr + A_BYTES;
                    const uint64_t adesc = make_smem_desc(a_addr, a_lbo, 1024), bdesc = make_smem_desc(b_addr, b_lbo, 1024);
#pragma unroll
                    for (int k4 = 0; k4 < BK / 16; ++k4)          // the address field counts 16-byte units
                        umma_f16_pair(d_tmem, adesc + k4 * (a_kstep >> 4), bdesc + k4 * (b_kstep >> 4), idesc, (kb | k4) != 0, on);
                    umma_commit_pair(&empty[s], on);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                if (!ok) break;
                umma_commit_pair(&acc_full[acc], on);
                if (++acc == 2) { acc = 0; acc_ph ^= 1; }
            }
        }
    } else if (TMA_C) {
        // Epilogue of D = alpha * acc + beta * C for dense 16-bit outputs.  C arrives by TMA in the slab the result is staged in: rounds of 64
        // columns walk a ring of four slabs [128 rows][128 bytes], the slab of the next round is requested while this one is worked
        // on, and every thread replaces the 16-byte pieces of its row in place.  (Read by the threads themselves, 64 bytes of a row
        // each, C cost 32 cache lines per load in the chain between accumulator and store: 128 symmetric products of 768^3 took 134 us, 103 now.)
        const int quad = warp & 3;
        const int half = (warp - 2) >> 2;                          // 32 of a round's 64 columns
        const int row_in_tile = quad * 32 + lane;
        const bool leader = threadIdx.x == 64;
        const int sw = row_in_tile & 7;
        // A thread whose wait gives up goes on through the loops without waiting (see mbar_wait in ptx.cuh): the 256 threads meet at named
        // barriers, and one that left would keep the others there for good
        int acc = 0; uint32_t acc_ph = 0;
        uint32_t use = 0, fetched = 0;                             // slabs handed to a store so far; slabs of C consumed so far
        auto fetch_c = [&](const TileCoord& t, int round, uint32_t slab, uint32_t k) {
            mbar_expect_tx(&c_full[k & 1], SLAB_BYTES);
            tma_load_3d(staging + (slab & 3) * SLAB_BYTES, &tmap_c, &c_full[k & 1], t.n0 + round * 64, t.m0, t.dz);
        };
        if (leader && first_tile < tiles) fetch_c(tile_coord<BN>(p, first_tile, cta_rank, m_tiles, n_tiles), 0, 0, 0);
        for (int tile = first_tile; tile < tiles; tile += tile_step) {
            const TileCoord t = tile_coord<BN>(p, tile, cta_rank, m_tiles, n_tiles);
            const int rounds = min(BN / 64, (t.n_limit - t.n0 + 63) / 64);
            float alpha = p.alpha, beta = p.beta;
            if (p.batch_sumsq != nullptr) {                   // an operand is an un-normalised Muon update: scale the result instead
                const float inv = 1.f / (sqrtf(p.batch_sumsq[t.dz]) * 1.02f + 1e-6f);
                if (p.scale_mode == 2) alpha *= inv * inv;
                else { alpha *= inv; beta *= inv; }
            }
            const bool mirror = p.symmetric && t.n0 != t.m0 - cta_rank * BM;
            if (ok && !mbar_wait(&acc_full[acc], acc_ph)) { atomicExch(p.status, 104); ok = false; }
            tc_fence_after();
            for (int round = 0; round < rounds; ++round) {
                if (leader && ok) {                                    // a barrier that was given up is not armed again
                    // at most the latest store still reads its slab: the one before it, whose slab comes next at the earliest, is done
                    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    const uint32_t next = use + (mirror ? 2 : 1);
                    if (round + 1 < rounds) fetch_c(t, round + 1, next, fetched + 1);
                    else if (tile + tile_step < tiles) fetch_c(tile_coord<BN>(p, tile + tile_step, cta_rank, m_tiles, n_tiles), 0, next, fetched + 1);
                }
                uint32_t r[32];
                tmem_ld_32x32b_x32(tmem_base + acc * BN + (round * 2 + half) * 32 + (static_cast<uint32_t>(quad * 32) << 16), r);
                tmem_ld_wait();
                if (round == rounds - 1) {                                    // accumulator fully read: release it early
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(&acc_empty[acc], 0);
                }
                if (ok && !mbar_wait(&c_full[fetched & 1], (fetched >> 1) & 1)) { atomicExch(p.status, 105); ok = false; }
                uint8_t* slab = staging + (use & 3) * SLAB_BYTES;
                uint8_t* slab_row = slab + row_in_tile * 128;
                // column of this chunk that lies on the diagonal in this thread's row (p.diag is added there; -1: none)
                const int on_diag = p.diag != 0.f ? t.m0 + row_in_tile - (t.n0 + round * 64 + half * 32) : -1;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint4* piece = reinterpret_cast<uint4*>(slab_row + (((half * 4 + q) ^ sw) << 4));
                    const uint4 cv = *piece;
                    float v[8];
                    unpack_16bit(cv, p.in_f16, v);
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[8 * q + e]) * alpha + beta * v[e];
                    if (on_diag >= 8 * q && on_diag < 8 * q + 8) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[e] += on_diag == 8 * q + e ? p.diag : 0.f;
                    }
                    const uint4 o = pack_16bit(v, p.out_f16);
                    *piece = o;
                    if (mirror) { r[4 * q] = o.x; r[4 * q + 1] = o.y; r[4 * q + 2] = o.z; r[4 * q + 3] = o.w; }      // kept packed for the transposed store
                }
                fence_proxy_async();
                asm volatile("bar.sync 1, 256;" ::: "memory");                 // slab complete and visible to the async proxy
                const int col = t.n0 + round * 64;
                if (leader) {
                    if (t.m0 < t.m_limit)
                        asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                                     ::"l"(&tmap_d), "r"(smem_u32(slab)), "r"(col), "r"(t.m0), "r"(t.dz) : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
                ++use; ++fetched;
                if (mirror) {
                    // the 128 x 64 block goes out transposed: 64 rows of two 128-byte slab rows (this CTA's rows [m0, m0 + 64) and the next 64).
                    // The slab was free before this round's first barrier (see above)
                    uint8_t* tbuf = staging + (use & 3) * SLAB_BYTES;
                    uint8_t* tcol = tbuf + (row_in_tile >> 6) * (SLAB_BYTES / 2) + (row_in_tile & 7) * 2;
                    const int piece = (row_in_tile & 63) >> 3;
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const uint16_t bits = static_cast<uint16_t>(r[(i >> 3) * 4 + ((i & 7) >> 1)] >> ((i & 1) * 16));
                        *reinterpret_cast<uint16_t*>(tcol + (half * 32 + i) * 128 + ((piece ^ (i & 7)) << 4)) = bits;
                    }
                    fence_proxy_async();
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                    if (leader) {
                        for (int sl = 0; sl < 2; ++sl) {
                            const int tc = t.m0 + sl * 64;
                            if (tc >= t.n_limit) break;
                            asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                                         ::"l"(&tmap_mirror), "r"(smem_u32(tbuf + sl * (SLAB_BYTES / 2))), "r"(tc), "r"(col), "r"(t.dz) : "memory");
                        }
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                    ++use;
                }
            }
            if (++acc == 2) { acc = 0; acc_ph ^= 1; }
        }
        if (leader) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else {
        // Every epilogue warp works by itself: it owns 32 rows (TMEM lanes 32 * quad ..) and half of the columns, stages 128 bytes of each row
        // at a time in one of two slabs of its own and sends the slab with its own TMA store (or reduce-add), so that no warp waits for another.
        // An off-diagonal tile of a symmetric result goes out a second time as 64 rows of 32 columns.  With slabs of all 128 rows, two CTA
        // barriers and a wait per store, 96 symmetric products of 768^3 took 67.6 us (63.2 now), 32768 x 2304 x 768 81.9 (78.8), 16 fp32 ones of
        // 6144 x 768 94 (85).
        const int quad = warp & 3;
        const int half = (warp - 2) >> 2;
        const int sw = lane & 7;
        uint8_t* slabs = staging + (warp - 2) * (2 * STAGING_BYTES / 8);
        constexpr int WARP_SLAB = STAGING_BYTES / 8;                // 32 rows of 128 bytes, or 64 of 64
        const bool reduce = p.accumulate || (p.split_k > 1 && !p.split_slabs);
        int acc = 0; uint32_t acc_ph = 0;
        uint32_t stores = 0;
        // the warp's next slab, once the store of two slabs ago has finished reading it; and its way out
        const auto next_slab = [&]() {
            uint8_t* slab = slabs + (stores++ & 1) * WARP_SLAB;
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            __syncwarp();
            return slab;
        };
        const auto send = [&](const CUtensorMap* map, const uint8_t* slab, int x, int y, int z, bool add) {
            fence_proxy_async();
            __syncwarp();
            if (lane != 0) return;
            if (add)
                asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
                             ::"l"(map), "r"(smem_u32(slab)), "r"(x), "r"(y), "r"(z) : "memory");
            else
                asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                             ::"l"(map), "r"(smem_u32(slab)), "r"(x), "r"(y), "r"(z) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        };
        for (int tile = first_tile; tile < tiles; tile += tile_step) {
            const TileCoord t = tile_coord<BN>(p, tile, cta_rank, m_tiles, n_tiles);
            const bool have_acc = t.k_blocks != 0;
            if (!have_acc && !(t.store_zeros && !p.accumulate)) continue;      // nothing to add, nothing to clear
            const int row0 = t.m0 + quad * 32;
            float alpha = p.alpha, beta = p.beta;
            if (p.batch_sumsq != nullptr) {                   // an operand is an un-normalised Muon update: scale the result instead
                const float inv = 1.f / (sqrtf(p.batch_sumsq[t.dz]) * 1.02f + 1e-6f);
                if (p.scale_mode == 2) alpha *= inv * inv;
                else { alpha *= inv; beta *= inv; }
            }
            const bool mirror = p.symmetric && t.n0 != t.m0 - cta_rank * BM;      // off-diagonal pair tile (uniform across the pair)
            if (have_acc) {
                if (ok && !mbar_wait(&acc_full[acc], acc_ph)) { atomicExch(p.status, 104); ok = false; }
                tc_fence_after();
            }
#pragma unroll
            for (int sl = 0; sl < BN / 128; ++sl) {
                const int col = t.n0 + half * BN_HALF + sl * 64;
                uint32_t r[2][32];
                if (have_acc) {
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        tmem_ld_32x32b_x32(tmem_base + acc * BN + half * BN_HALF + sl * 64 + j * 32 + (static_cast<uint32_t>(quad * 32) << 16), r[j]);
                    tmem_ld_wait();
                    if (sl == BN / 128 - 1) {                                   // accumulator fully read: release it early
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(&acc_empty[acc], 0);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 2; ++j)
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[j][i] = 0u;
                }
                if (col >= t.n_limit || row0 >= t.m_limit) continue;            // uniform across the warp
                uint32_t packed[32];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    float v[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[j][i]) * alpha;
                    const int col0 = col + j * 32, row = row0 + lane;
                    if (p.C != nullptr && row < t.m_limit && col0 < t.n_limit) {
                        const __nv_bfloat16* c = reinterpret_cast<const __nv_bfloat16*>(p.C) +
                            static_cast<long long>(t.dz) * p.c_batch_stride + static_cast<long long>(row) * p.ldc + col0;
                        if (col0 + 32 <= t.n_limit) {
#pragma unroll
                            for (int i = 0; i < 32; i += 8) {
                                float f[8];
                                unpack_16bit(*reinterpret_cast<const uint4*>(c + i), 0, f);
#pragma unroll
                                for (int e = 0; e < 8; ++e) v[i + e] += beta * f[e];
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < 32; ++i)
                                if (col0 + i < t.n_limit) v[i] += beta * __bfloat162float(c[i]);
                        }
                    }
                    if (p.out_fp32) {
                        if (col0 >= t.n_limit) continue;
                        uint8_t* slab = next_slab();
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            *reinterpret_cast<float4*>(slab + lane * 128 + ((q ^ sw) << 4)) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                        send(&tmap_d, slab, col0, row0, t.dz, reduce);
                        continue;
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint4 o = pack_16bit(v + 8 * q, p.out_f16);
                        packed[j * 16 + 4 * q] = o.x; packed[j * 16 + 4 * q + 1] = o.y; packed[j * 16 + 4 * q + 2] = o.z; packed[j * 16 + 4 * q + 3] = o.w;
                    }
                }
                if (p.out_fp32) continue;
                uint8_t* slab = next_slab();
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    *reinterpret_cast<uint4*>(slab + lane * 128 + ((q ^ sw) << 4)) = make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
                send(&tmap_d, slab, col, row0, t.dz, false);
                if (mirror) {
                    slab = next_slab();
#pragma unroll
                    for (int i = 0; i < 64; ++i)                                // row i of the transposed block: a warp writes its 64 bytes
                        *reinterpret_cast<uint16_t*>(slab + i * 64 + lane * 2) = static_cast<uint16_t>(packed[i >> 1] >> ((i & 1) * 16));
                    send(&tmap_mirror, slab, row0, col, t.dz, false);
                }
            }
            if (have_acc && ++acc == 2) { acc = 0; acc_ph ^= 1; }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }

    // common teardown: every path (including a timed-out wait) reaches it, so TMEM is always released
    tc_fence_before();
    cluster_sync_all();                       // the partner no longer reads this CTA's shared memory or signals its barriers
    if (warp == 1) {
        if (*reinterpret_cast<volatile int*>(p.status) != 0) {
            // a wait gave up: give any TMA copy still in flight time to land before the CTA's smem is recycled
            const long long start = clock64();
            while (clock64() - start < 200000) {}
        }
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
}

// The shares of a split contraction, summed in their order (the same bits every time) and rounded once.  A thread owns four columns; bound by
// the copy rate: six shares of 1024 x 768 take 6 us, four of 7680 x 768 21.
__global__ void __launch_bounds__(256)
split_sum_kernel(const float* __restrict__ parts, int splits, long long rows, int cols, int ldp, __nv_bfloat16* __restrict__ d, long long ldd) {
    const int quads = (cols + 3) >> 2;
    const long long slab = rows * ldp, total = rows * quads;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
        const long long row = i / quads;
        const int col = static_cast<int>(i - row * quads) * 4;
        const float* src = parts + row * ldp + col;
        float4 v = *reinterpret_cast<const float4*>(src);
#pragma unroll 4
        for (int s = 1; s < splits; ++s) {
            const float4 w = *reinterpret_cast<const float4*>(src + s * slab);
            v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
        __nv_bfloat16* dst = d + row * ldd + col;
        if (col + 4 <= cols) {
            *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
        } else {
            const float t[3] = {v.x, v.y, v.z};
#pragma unroll
            for (int e = 0; e < 3; ++e)
                if (col + e < cols) dst[e] = __float2bfloat16_rn(t[e]);
        }
    }
}

void launch_split_sum(const float* parts, int splits, long long rows, int cols, int ldp, void* d, long long ldd, cudaStream_t s) {
    const long long blocks = (rows * ((cols + 3) / 4) + 255) / 256;
    split_sum_kernel<<<static_cast<int>(blocks < 8192 ? blocks : 8192), 256, 0, s>>>(parts, splits, rows, cols, ldp, static_cast<__nv_bfloat16*>(d), ldd);
}

template <bool A_MN, bool B_MN, bool TMA_C, int WIDTH>
static cudaError_t launch_variant(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const CUtensorMap& tc, const CUtensorMap& tm,
                                  const GemmParams& p, int sms, cudaStream_t stream) {
    constexpr int GEMM_SMEM_BYTES = Tiling<WIDTH>::STAGES * Tiling<WIDTH>::STAGE_BYTES + 2 * STAGING_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
    auto kernel = gemm_bf16_kernel<A_MN, B_MN, TMA_C, WIDTH>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM_BYTES);
        if (e != cudaSuccess) return e;
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms & ~1);
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = GEMM_SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, ta, tb, td, tc, tm, p);
}

// Half the width where even so every tile has a CTA pair of its own: the chain of loads, products and read-out that such a launch consists of is
// then half as long.  us with cold caches, 256 / 128 columns: 360 x 2304 x 768 11.6 / 9.0, 1024 x 2048 x 1024 13.3 / 10.3, 1024 x 1024 x 1024 12.7 / 9.6,
// 2048 rows of eight experts x 768 x 3072 26.8 / 22.3.  Rows of a grouped product are the most there can be, p.M.
int gemm_bf16_tile_width(const GemmParams& p, bool a_mn, bool c_by_tma, int sms) {
    const long long halves = static_cast<long long>((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + 127) / 128) * (p.mode == GEMM_GROUPED_M ? 1 : p.batch);
    const bool plain = !a_mn && !c_by_tma && !p.symmetric && !p.out_fp32 && p.split_k == 1 && p.mode != GEMM_GROUPED_K;
    return plain && p.N > 128 && halves <= sms / 2 ? 128 : 256;
}

cudaError_t launch_gemm_bf16(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const CUtensorMap* tc, const CUtensorMap* tmirror,
                             const GemmParams& p, bool a_mn, bool b_mn, int sms, cudaStream_t stream) {
    const CUtensorMap& tm = tmirror != nullptr ? *tmirror : td;
    if (gemm_bf16_tile_width(p, a_mn, tc != nullptr, sms) == 128)
        return b_mn ? launch_variant<false, true, false, 128>(ta, tb, td, td, tm, p, sms, stream) : launch_variant<false, false, false, 128>(ta, tb, td, td, tm, p, sms, stream);
    if (tc != nullptr) return launch_variant<false, false, true, 256>(ta, tb, td, *tc, tm, p, sms, stream);
    if (a_mn) return b_mn ? launch_variant<true, true, false, 256>(ta, tb, td, td, tm, p, sms, stream) : launch_variant<true, false, false, 256>(ta, tb, td, td, tm, p, sms, stream);
    return b_mn ? launch_variant<false, true, false, 256>(ta, tb, td, td, tm, p, sms, stream) : launch_variant<false, false, false, 256>(ta, tb, td, td, tm, p, sms, stream);
}

}  // namespace gm
