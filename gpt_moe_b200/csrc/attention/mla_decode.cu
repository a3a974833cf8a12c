// Absorbed-weight decode for multi-head latent attention: new tokens attend over the LATENT cache directly.
//
//   score[b, h, t, s] = (q_latent[b,t,h,:] . latent[b,s,:] + q_rope[b,t,h,:] . rope[b,s,:]) * key_gain[b,s,kv(h)] * scale
//   (optional soft-capping cap * tanh(score / cap); causal: s <= start + t; optional window: start + t - s <= W)
//   context[b, t, h, :] = sum_s softmax_s(score) * latent[b, s, :]                        (latent space, fp32)
//
// Every head of a token reads the same latent rows (keys and values are both the latent cache), so one token's heads are the
// rows of a 16-row matrix product and the kernel should be bound by reading the cache once.  tcgen05 has no tile with fewer than
// 64 rows (48 of them would be padding), so the products are warp-level m16n8k16 instructions:
//   * a CTA per split of the cache (fastest), group of MT * 16 rows and sequence; a row is a (token, head) pair, token-major, so 16
//     heads make one token a tile of rows.  All grids of the file are one-dimensional: rows and sequences may number more than 65535;
//   * a CTA walks its share of the cache in tiles of 32 positions that arrive through a cp.async ring;
//   * warp w owns the latent dimensions [w r/8, (w+1) r/8) for both products: it multiplies its slice of the queries (held in
//     registers) with its slice of the 32 latent rows, the eight partial score tiles are summed through shared memory together
//     with the rotary part (one 16-wide slice each for the first warps), and the same slice of the tile is the value operand of
//     its slice of the context, which stays in registers;
//   * queries and probabilities are fp32 numbers: each enters as bf16 terms, one product each, accumulated in fp32; the cache is bf16 and
//     needs no splitting.  Three terms hold all bits, and a context that is returned in fp32 gets them (`mla_decode`).  The layer's own
//     call rounds the context's expansion to bf16: two terms (16 bits) leave its error as it is (3.9e-3 against 64 bits either way)
//     and shorten the chain of products of every tile.
// Measured (16 heads, rank 512): 8 sequences x 1 token over 4022 positions 18 us against 96 us for a kernel that formed the products
// with fp32 multiply-adds and warp reductions (38 MB of cache; its merge took another 48 us, now 9 with W_v); 32 x 1 over 8000 positions
// 97 us, 3.1 TB/s, the tensor pipe 37 % busy: a tile's chain of products, sums and softmax is the limit.  Error of the layer's output (of
// the output alone, without the cache entries) against 64 bits: 3.8e-3 against 5.7e-3 (queries and rotation stay fp32 between the
// projection and the scores, and the W products are fp32 instead of TF32).
// The first kernel of the file turns projections into what the split kernel reads (and appends the new tokens to the cache); the
// last one merges the splits by their log-sum-exp and, for the module's own use, expands the context with W_v.
// Reference: the Triton kernels `_mla_decode_kernel` / `_mla_decode_merge_kernel` (experiments/073-mla-current-kv768.patch:456-673)
// and the paired-head variant (experiments/051-paired-head-mla-decode.patch).
#include "../common/ptx.cuh"
#include "../kernels_decl.h"

namespace gm {

constexpr int MD_TILE = 32;          // cache positions per tile
constexpr int MD_WARPS = 8;
// One tile of rows of an up to 512-wide latent leaves room for two CTAs on an SM: every tile passes three barriers, and the other CTA's
// products run meanwhile.  Wider latents, two tiles of rows and three terms take the SM to themselves.  Ring depth: as many tiles as fit beside
// the scores.
constexpr int md_ctas(int ks, int mt, int terms) { return ks <= 4 && mt == 1 && terms == 2 ? 2 : 1; }
constexpr int md_stages(int ks, int mt, int terms) { return ks <= 2 ? 4 : md_ctas(ks, mt, terms) == 2 ? 2 : ks <= 4 ? 4 : ks <= 6 ? 3 : 2; }
constexpr int MD_ROPE_MAX = 64;
constexpr int MD_MAX_SPLITS = 64;
constexpr int MD_SP_PITCH = 40;      // floats per row of a partial score tile: two half-warps' rows fall on different banks
constexpr int MD_P_PITCH = 40;       // bf16 per row of a probability tile (80 bytes: ldmatrix rows on different banks)

struct MlaDecodeParams {
    const float* q_latent;           // [B, T, H, r]
    const float* q_rope;             // [B, T, H, dr]
    const __nv_bfloat16* latent;     // [B, S, r]   (row pitch r, batch stride given)
    const __nv_bfloat16* rope;       // [B, S, dr]
    const __nv_bfloat16* key_gain;   // [B, S, Hkv]
    long long latent_bs, rope_bs, gain_bs;      // batch strides in elements
    float* part_ctx;                 // [B, T, H, splits, r]  un-normalised partial contexts
    float* part_ml;                  // [B, T, H, splits, 2]  running max (of base-e scores) and sum
    int B, T, H, Hkv, r, dr, S, splits, start, window;
    int latent_vec, rope_vec;        // rows may be fetched in 16-byte pieces (alignment of base and strides)
    float scale, softcap;
};

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Two neighbouring column tiles: d += sum over the terms of a * b, smallest first.  The tensor core cuts a sum off instead of rounding it, which adds up over a long chain:
// three terms, which are there for the last bits, form each step's sum from zero and add it in fp32.
template <int TERMS>
__device__ __forceinline__ void mma_terms(float (&d0)[4], float (&d1)[4], const uint32_t (&a)[TERMS][4], const uint32_t (&b)[4]) {
    if constexpr (TERMS == 3) {
        float p0[4] = {0.f, 0.f, 0.f, 0.f}, p1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int t = TERMS - 1; t >= 0; --t) {
            mma16816(p0, a[t], b[0], b[1]);
            mma16816(p1, a[t], b[2], b[3]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) { d0[e] += p0[e]; d1[e] += p1[e]; }
    } else {
#pragma unroll
        for (int t = TERMS - 1; t >= 0; --t) {
            mma16816(d0, a[t], b[0], b[1]);
            mma16816(d1, a[t], b[2], b[3]);
        }
    }
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {      // zeros when not valid
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// x as a sum of bf16 terms, largest first (the remainder after each is exact): up to 2^-17 of x with two, all of it with three
template <int TERMS>
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&term)[TERMS]) {
#pragma unroll
    for (int i = 0; i < TERMS; ++i) {
        term[i] = pack_bf16x2(x, y);
        x -= __uint_as_float(term[i] << 16);
        y -= __uint_as_float(term[i] & 0xffff0000u);
    }
}

// KS = k-steps of 16 latent dimensions per warp (r = 128 * KS); MT = 16-row tiles per CTA; MD_TERMS = bf16 terms of a query or probability
template <int KS, int MT, int MD_TERMS>
__global__ void __launch_bounds__(MD_WARPS * 32, md_ctas(KS, MT, MD_TERMS))
mla_decode_split_kernel(const MlaDecodeParams p) {
    extern __shared__ __align__(16) uint8_t md_smem[];
    constexpr int r = KS * 128, MD_STAGES = md_stages(KS, MT, MD_TERMS);
    constexpr int LAT_PITCH = r * 2 + 16, ROPE_PITCH = MD_ROPE_MAX * 2 + 16;     // bytes; ldmatrix rows on different banks
    constexpr int STAGE = MD_TILE * (LAT_PITCH + ROPE_PITCH);
    constexpr int ROWS = MT * 16;
    float* sp = reinterpret_cast<float*>(md_smem + MD_STAGES * STAGE);                          // [8 warps][ROWS][MD_SP_PITCH]
    __nv_bfloat16* pr = reinterpret_cast<__nv_bfloat16*>(sp + MD_WARPS * ROWS * MD_SP_PITCH);   // [MD_TERMS][ROWS][MD_P_PITCH]
    float* alpha_s = reinterpret_cast<float*>(pr + MD_TERMS * ROWS * MD_P_PITCH);                      // [ROWS]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int total_rows = p.T * p.H, row_groups = (total_rows + ROWS - 1) / ROWS;
    const int split = blockIdx.x % p.splits, group_of_all = blockIdx.x / p.splits;
    const int b = group_of_all / row_groups, row_group = group_of_all - b * row_groups;
    const int row_base = row_group * ROWS;
    const int t_first = row_base / p.H, t_last = min(row_base + ROWS - 1, total_rows - 1) / p.H;
    const int hi_max = min(p.S - 1, p.start + t_last);                                          // last position any row sees
    const int lo_min = p.window >= 0 ? max(0, p.start + t_first - p.window) : 0;                // first one
    const int first_tile = lo_min / MD_TILE;
    const int tiles = hi_max >= lo_min ? hi_max / MD_TILE - first_tile + 1 : 0;
    const int per = (tiles + p.splits - 1) / p.splits;
    const int tile_begin = first_tile + split * per, tile_end = min(first_tile + tiles, tile_begin + per);
    const int n_tiles = tile_end - tile_begin;                                                  // may be <= 0

    const int g = lane >> 2, tq = lane & 3;
    const int rope_steps = (p.dr + 15) / 16;
    const bool has_rope = warp < rope_steps;

    // rotary columns past dr are multiplied by zero queries, so they only have to be finite: clear them once
    for (int i = tid; i < MD_STAGES * MD_TILE * MD_ROPE_MAX; i += blockDim.x) {
        const int row = i / MD_ROPE_MAX, c = i - row * MD_ROPE_MAX;
        if (c >= p.dr) {
            uint8_t* st = md_smem + (row / MD_TILE) * STAGE + MD_TILE * LAT_PITCH + (row % MD_TILE) * ROPE_PITCH;
            reinterpret_cast<__nv_bfloat16*>(st)[c] = __float2bfloat16(0.f);
        }
    }
    auto load_tile = [&](int i) {                          // i: tile of this CTA, into ring stage i % MD_STAGES
        if (i < n_tiles) {
            uint8_t* st = md_smem + (i % MD_STAGES) * STAGE;
            const int s0 = (tile_begin + i) * MD_TILE;
            if (p.latent_vec) {
                constexpr int vec = r / 8;
                for (int j = tid; j < MD_TILE * vec; j += MD_WARPS * 32) {
                    const int row = j / vec, v = j - row * vec;
                    const bool valid = s0 + row >= lo_min && s0 + row <= hi_max;      // what no row of the CTA sees does not get near its sums
                    cp_async16(smem_u32(st + row * LAT_PITCH + v * 16), p.latent + b * p.latent_bs + static_cast<long long>(valid ? s0 + row : 0) * r + v * 8, valid);
                }
            } else {
                for (int j = tid; j < MD_TILE * r; j += MD_WARPS * 32) {
                    const int row = j / r, c = j - row * r;
                    reinterpret_cast<__nv_bfloat16*>(st + row * LAT_PITCH)[c] =
                        s0 + row >= lo_min && s0 + row <= hi_max ? p.latent[b * p.latent_bs + static_cast<long long>(s0 + row) * r + c] : __float2bfloat16(0.f);
                }
            }
            uint8_t* sr = st + MD_TILE * LAT_PITCH;
            if (p.rope_vec) {
                const int vec = p.dr / 8;
                for (int j = tid; j < MD_TILE * vec; j += MD_WARPS * 32) {
                    const int row = j / vec, v = j - row * vec;
                    const bool valid = s0 + row >= lo_min && s0 + row <= hi_max;      // what no row of the CTA sees does not get near its sums
                    cp_async16(smem_u32(sr + row * ROPE_PITCH + v * 16), p.rope + b * p.rope_bs + static_cast<long long>(valid ? s0 + row : 0) * p.dr + v * 8, valid);
                }
            } else {
                for (int j = tid; j < MD_TILE * p.dr; j += MD_WARPS * 32) {
                    const int row = j / p.dr, c = j - row * p.dr;
                    reinterpret_cast<__nv_bfloat16*>(sr + row * ROPE_PITCH)[c] =
                        s0 + row >= lo_min && s0 + row <= hi_max ? p.rope[b * p.rope_bs + static_cast<long long>(s0 + row) * p.dr + c] : __float2bfloat16(0.f);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int i = 0; i < MD_STAGES - 1; ++i) load_tile(i);

    // this warp's slice of the queries as A fragments (all terms): rows g / g + 8, columns 2 tq, 2 tq + 1 and + 8
    uint32_t qa[MT][KS][MD_TERMS][4], qr[MT][MD_TERMS][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int row = row_base + mt * 16 + g + 8 * hf;
            const bool live = row < total_rows;
            const long long base = static_cast<long long>(b) * total_rows + (live ? row : 0);
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) {
                    float2 v = *reinterpret_cast<const float2*>(p.q_latent + base * r + (warp * KS + ks) * 16 + cc * 8 + tq * 2);
                    if (!live) v = make_float2(0.f, 0.f);
                    uint32_t term[MD_TERMS];
                    split_pair(v.x, v.y, term);
#pragma unroll
                    for (int i = 0; i < MD_TERMS; ++i) qa[mt][ks][i][cc * 2 + hf] = term[i];
                }
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                const int c0 = warp * 16 + cc * 8 + tq * 2;                       // dr is even: a pair is in or out as a whole
                float2 v = make_float2(0.f, 0.f);
                if (live && has_rope && c0 < p.dr) v = *reinterpret_cast<const float2*>(p.q_rope + base * p.dr + c0);
                uint32_t term[MD_TERMS];
                split_pair(v.x, v.y, term);
#pragma unroll
                for (int i = 0; i < MD_TERMS; ++i) qr[mt][i][cc * 2 + hf] = term[i];
            }
        }
    }
    float acc[MT][KS * 2][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int n = 0; n < KS * 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[mt][n][e] = 0.f;

    // softmax: thread owns row tid / 16 of each 16-row tile and positions 2 (tid % 16), + 1 of the key tile
    const int srow = tid >> 4, skey = (tid & 15) * 2;
    float m[MT], l[MT];
    int hi[MT], lo[MT], kvh[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        m[mt] = -INFINITY; l[mt] = 0.f;
        const int row = row_base + mt * 16 + srow;
        const int t = min(row, total_rows - 1) / p.H, h = min(row, total_rows - 1) % p.H;
        const int qpos = p.start + t;
        hi[mt] = row < total_rows ? min(p.S - 1, qpos) : -1;
        lo[mt] = p.window >= 0 ? max(0, qpos - p.window) : 0;
        kvh[mt] = h / (p.H / p.Hkv);
    }

    for (int i = 0; i < n_tiles; ++i) {
        const int s0 = (tile_begin + i) * MD_TILE;
        float gain[MT][2];                                   // fetched under the products
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int pos = s0 + skey + e;
                gain[mt][e] = pos < p.S ? __bfloat162float(p.key_gain[b * p.gain_bs + static_cast<long long>(pos) * p.Hkv + kvh[mt]]) : 0.f;
            }
        asm volatile("cp.async.wait_group %0;" ::"n"(MD_STAGES - 2) : "memory");
        __syncthreads();                                     // tile i has landed; everybody is done with tile i - 1
        load_tile(i + MD_STAGES - 1);
        uint8_t* st = md_smem + (i % MD_STAGES) * STAGE;
        const uint32_t lat_a = smem_u32(st) + warp * KS * 32, rope_a = smem_u32(st) + MD_TILE * LAT_PITCH + warp * 32;

        float sc[MT][4][4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) sc[mt][n][e] = 0.f;
        // B fragments of two neighbouring 8-position tiles for one k-step: lanes 0-7 / 8-15 address columns 0-7 / 8-15 of the first
        // eight positions, lanes 16-31 those of the next eight
        const int key_l = (lane & 7) + (lane >> 4) * 8, col_l = ((lane >> 3) & 1) * 16;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks)
#pragma unroll
            for (int np = 0; np < 2; ++np) {
                uint32_t bf[4];
                ldsm_x4(bf, lat_a + (np * 16 + key_l) * LAT_PITCH + ks * 32 + col_l);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) mma_terms(sc[mt][np * 2], sc[mt][np * 2 + 1], qa[mt][ks], bf);
            }
        if (has_rope) {
#pragma unroll
            for (int np = 0; np < 2; ++np) {
                uint32_t bf[4];
                ldsm_x4(bf, rope_a + (np * 16 + key_l) * ROPE_PITCH + col_l);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) mma_terms(sc[mt][np * 2], sc[mt][np * 2 + 1], qr[mt], bf);
            }
        }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                float* dst = sp + (warp * ROWS + mt * 16 + g) * MD_SP_PITCH + n * 8 + tq * 2;
                *reinterpret_cast<float2*>(dst) = make_float2(sc[mt][n][0], sc[mt][n][1]);
                *reinterpret_cast<float2*>(dst + 8 * MD_SP_PITCH) = make_float2(sc[mt][n][2], sc[mt][n][3]);
            }
        __syncthreads();
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            float s[2] = {0.f, 0.f};
#pragma unroll
            for (int w = 0; w < MD_WARPS; ++w) {
                const float2 v = *reinterpret_cast<const float2*>(sp + (w * ROWS + mt * 16 + srow) * MD_SP_PITCH + skey);
                s[0] += v.x; s[1] += v.y;
            }
            bool vis[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                s[e] = s[e] * gain[mt][e] * p.scale;
                if (p.softcap > 0.f) s[e] = p.softcap * tanhf(s[e] / p.softcap);
                vis[e] = s0 + skey + e >= lo[mt] && s0 + skey + e <= hi[mt];
                s[e] = vis[e] ? s[e] : -INFINITY;
            }
            float mx = fmaxf(s[0], s[1]);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));     // the 16 threads of a row
            const float m_new = fmaxf(m[mt], mx);
            const float corr = m_new == -INFINITY ? 1.f : expf(m[mt] - m_new);                       // nothing visible yet: 1
            const float p0 = vis[0] ? expf(s[0] - m_new) : 0.f, p1 = vis[1] ? expf(s[1] - m_new) : 0.f;
            l[mt] = l[mt] * corr + (p0 + p1);
            m[mt] = m_new;
            uint32_t prob[MD_TERMS];
            split_pair(p0, p1, prob);
            uint32_t* dst = reinterpret_cast<uint32_t*>(pr + (mt * 16 + srow) * MD_P_PITCH + skey);
            constexpr int term_words = ROWS * MD_P_PITCH / 2;
#pragma unroll
            for (int i = 0; i < MD_TERMS; ++i) dst[i * term_words] = prob[i];
            if ((tid & 15) == 0) alpha_s[mt * 16 + srow] = corr;
        }
        __syncthreads();
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
            const float a0 = alpha_s[mt * 16 + g], a1 = alpha_s[mt * 16 + g + 8];
            if (a0 != 1.f || a1 != 1.f) {
#pragma unroll
                for (int n = 0; n < KS * 2; ++n) { acc[mt][n][0] *= a0; acc[mt][n][1] *= a0; acc[mt][n][2] *= a1; acc[mt][n][3] *= a1; }
            }
        }
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {                     // 16 positions each
            uint32_t pa[MT][MD_TERMS][4];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int term = 0; term < MD_TERMS; ++term)
                    ldsm_x4(pa[mt][term], smem_u32(pr + (term * ROWS + mt * 16 + (lane & 15)) * MD_P_PITCH + ks * 16 + (lane >> 4) * 8));
#pragma unroll
            for (int np = 0; np < KS; ++np) {                // 16 dimensions: two column tiles
                uint32_t bf[4];
                ldsm_x4_t(bf, lat_a + (ks * 16 + (lane & 15)) * LAT_PITCH + np * 32 + (lane >> 4) * 16);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) mma_terms(acc[mt][np * 2], acc[mt][np * 2 + 1], pa[mt], bf);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int row = row_base + mt * 16 + g + 8 * hf;
            if (row < total_rows) {
                float* out = p.part_ctx + ((static_cast<long long>(b) * total_rows + row) * p.splits + split) * r + warp * KS * 16 + tq * 2;
#pragma unroll
                for (int n = 0; n < KS * 2; ++n) *reinterpret_cast<float2*>(out + n * 8) = make_float2(acc[mt][n][2 * hf], acc[mt][n][2 * hf + 1]);
            }
        }
        float sum = l[mt];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const int row = row_base + mt * 16 + srow;
        if ((tid & 15) == 0 && row < total_rows) {
            float* ml = p.part_ml + ((static_cast<long long>(b) * total_rows + row) * p.splits + split) * 2;
            ml[0] = m[mt];
            ml[1] = sum;
        }
    }
}

// factor[i] = exp(m_i - M) / sum_j l_j exp(m_j - M) of one row's splits (0 for a split that saw nothing); one warp
__device__ __forceinline__ void merge_factors(const float* ml, int splits, float* factor, int lane) {
    float big = -INFINITY;
    for (int i = lane; i < splits; i += 32) big = fmaxf(big, ml[2 * i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
    float denom = 0.f;
    for (int i = lane; i < splits; i += 32) denom += ml[2 * i] != -INFINITY ? ml[2 * i + 1] * expf(ml[2 * i] - big) : 0.f;
    denom = wsum(denom);
    const float inv = denom > 0.f ? 1.f / denom : 0.f;
    for (int i = lane; i < splits; i += 32) factor[i] = ml[2 * i] != -INFINITY ? expf(ml[2 * i] - big) * inv : 0.f;
}

// context[row, :] = sum_i part[row, i, :] * factor_i;  one CTA per (b, t, h) row
__global__ void __launch_bounds__(128)
mla_decode_merge_kernel(const float* __restrict__ part_ctx, const float* __restrict__ part_ml, float* __restrict__ context, int splits, int r) {
    __shared__ float factor[MD_MAX_SPLITS];
    const long long row = blockIdx.x;
    if (threadIdx.x < 32) merge_factors(part_ml + row * splits * 2, splits, factor, threadIdx.x);
    __syncthreads();
    for (int c = threadIdx.x * 4; c < r; c += 512) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int i = 0; i < splits; ++i) {
            const float f = factor[i];
            const float4 v = *reinterpret_cast<const float4*>(part_ctx + (row * splits + i) * r + c);
            // a split without a visible position has factor 0 and finite (zero) sums
            s.x = fmaf(v.x, f, s.x); s.y = fmaf(v.y, f, s.y); s.z = fmaf(v.z, f, s.z); s.w = fmaf(v.w, f, s.w);
        }
        *reinterpret_cast<float4*>(context + row * r + c) = s;
    }
}

// Merge, then expand: out[b, t, h, d] = sum_c context[b, t, h, c] * W_v[kv(h), d, c] in fp32, stored as bf16.  One CTA per head and
// TB tokens: the head's W_v rows (value_dim x r fp32) cross from L2 once per CTA, eight warps take a row each.
template <int NV, int TB>                  // r = 128 * NV
__global__ void __launch_bounds__(256)
mla_decode_values_kernel(const float* __restrict__ part_ctx, const float* __restrict__ part_ml, const float* __restrict__ w_up,
                         __nv_bfloat16* __restrict__ out, int tokens, int H, int group, int content, int value, int splits) {
    constexpr int r = NV * 128;
    __shared__ float factor[TB][MD_MAX_SPLITS];
    __shared__ __align__(16) float ctx_s[TB][r];
    const int h = blockIdx.x % H, tok0 = blockIdx.x / H * TB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int tb = warp; tb < TB; tb += 8)
        if (tok0 + tb < tokens) merge_factors(part_ml + (static_cast<long long>(tok0 + tb) * H + h) * splits * 2, splits, factor[tb], lane);
    __syncthreads();
    for (int j = threadIdx.x; j < TB * r / 4; j += 256) {
        const int tb = j / (r / 4), c = (j - tb * (r / 4)) * 4;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tok0 + tb < tokens) {
            const float* src = part_ctx + (static_cast<long long>(tok0 + tb) * H + h) * splits * r + c;
#pragma unroll 8
            for (int i = 0; i < splits; ++i) {
                const float f = factor[tb][i];
                const float4 v = *reinterpret_cast<const float4*>(src + static_cast<long long>(i) * r);
                s.x = fmaf(v.x, f, s.x); s.y = fmaf(v.y, f, s.y); s.z = fmaf(v.z, f, s.z); s.w = fmaf(v.w, f, s.w);
            }
        }
        *reinterpret_cast<float4*>(&ctx_s[tb][c]) = s;
    }
    __syncthreads();
    float4 cx[TB][NV];
#pragma unroll
    for (int tb = 0; tb < TB; ++tb)
#pragma unroll
        for (int i = 0; i < NV; ++i) cx[tb][i] = *reinterpret_cast<const float4*>(&ctx_s[tb][i * 128 + lane * 4]);
    const float* w = w_up + (static_cast<long long>(h / group) * (content + value) + content) * r;
#pragma unroll 2
    for (int d = warp; d < value; d += 8) {
        float s[TB];
#pragma unroll
        for (int tb = 0; tb < TB; ++tb) s[tb] = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const float4 wv = __ldg(reinterpret_cast<const float4*>(w + static_cast<long long>(d) * r + i * 128 + lane * 4));
#pragma unroll
            for (int tb = 0; tb < TB; ++tb) s[tb] += cx[tb][i].x * wv.x + cx[tb][i].y * wv.y + cx[tb][i].z * wv.z + cx[tb][i].w * wv.w;
        }
#pragma unroll
        for (int tb = 0; tb < TB; ++tb) {
            const float v = wsum(s[tb]);
            if (lane == 0 && tok0 + tb < tokens) out[(static_cast<long long>(tok0 + tb) * H + h) * value + d] = __float2bfloat16(v);
        }
    }
}

struct MlaPrepareParams {
    const __nv_bfloat16* query;      // [tokens, H * (content + dr)], row pitch q_pitch
    const __nv_bfloat16* low;        // [tokens, r + dr]: latent before its norm | rotary key, row pitch low_pitch
    long long q_pitch, low_pitch;
    const float* norm_w;             // [r] or null
    const float* cos;                // [T, dr / 2]: rows of the new positions
    const float* sin;
    const float* w_up;               // [Hkv, content + value, r]
    const float* q_scale;            // [H] or null (no QK-norm); k_scale [Hkv]
    const float* k_scale;
    __nv_bfloat16 *latent, *rope, *key_gain;     // cache, first new position of batch 0
    long long latent_bs, rope_bs, gain_bs;
    float* q_latent;                 // [tokens, H, r]
    float* q_rope;                   // [tokens, H, dr]
    int tokens, T, H, Hkv, content, value, dr;
    float norm_eps, qk_eps, smin, smax;
    int rms;
};

// What the split kernel needs from the projections of new tokens, and their entries in the cache.  One CTA per kv head and TB tokens:
//   latent <- RMSNorm(latent), rotary key and query <- rotation, QK-norm gains of query and key over [content | rotary];
//   k_content = W_k latent (only its norm is needed), q_latent = q_content^T W_k  (fp32, W_k as stored)
// Both products read the same W_k rows: a warp takes a row, a lane 4 NV of its columns; every row is read once per CTA.
template <int NV, int TB>
__global__ void __launch_bounds__(256)
mla_prepare_kernel(const MlaPrepareParams p) {
    constexpr int r = NV * 128;
    extern __shared__ __align__(16) float mp_smem[];
    float* lat_s = mp_smem;                                   // [TB][r]
    float* red_s = lat_s + TB * r;                            // [8 warps][TB][r]
    float* q_s = red_s + 8 * TB * r;                          // [TB][content]
    __shared__ float ksq_s[8][TB], rsq_s[TB];
    const int kvh = blockIdx.x % p.Hkv, tok0 = blockIdx.x / p.Hkv * TB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = p.H / p.Hkv, head_w = p.content + p.dr;

    if (warp < TB && tok0 + warp < p.tokens) {
        const int tok = tok0 + warp, b = tok / p.T, t = tok - b * p.T;
        const __nv_bfloat16* src = p.low + tok * p.low_pitch;
        float v[NV][4], sq = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) { v[i][e] = __bfloat162float(src[i * 128 + lane * 4 + e]); sq += v[i][e] * v[i][e]; }
        const float rstd = rsqrtf(wsum(sq) / r + p.norm_eps);
#pragma unroll
        for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int c = i * 128 + lane * 4 + e;
                const __nv_bfloat16 y = __float2bfloat16(v[i][e] * rstd * (p.norm_w ? p.norm_w[c] : 1.f));
                lat_s[warp * r + c] = __bfloat162float(y);
                if (kvh == 0) p.latent[b * p.latent_bs + static_cast<long long>(t) * r + c] = y;
            }
        float rsq = 0.f;
        for (int j = lane; j < p.dr / 2; j += 32) {
            const float x0 = __bfloat162float(src[r + 2 * j]), x1 = __bfloat162float(src[r + 2 * j + 1]);
            const float cs = p.cos[t * (p.dr / 2) + j], sn = p.sin[t * (p.dr / 2) + j];
            const __nv_bfloat16 y0 = __float2bfloat16(x0 * cs - x1 * sn), y1 = __float2bfloat16(x0 * sn + x1 * cs);
            rsq += __bfloat162float(y0) * __bfloat162float(y0) + __bfloat162float(y1) * __bfloat162float(y1);
            if (kvh == 0) {
                __nv_bfloat16* dst = p.rope + b * p.rope_bs + static_cast<long long>(t) * p.dr + 2 * j;
                dst[0] = y0; dst[1] = y1;
            }
        }
        rsq = wsum(rsq);
        if (lane == 0) rsq_s[warp] = rsq;
    }
    float4 lt[TB][NV];
    for (int gq = 0; gq < group; ++gq) {
        const int h = kvh * group + gq;
        if (warp < TB && tok0 + warp < p.tokens) {
            const int tok = tok0 + warp, t = tok % p.T;
            const __nv_bfloat16* src = p.query + tok * p.q_pitch + static_cast<long long>(h) * head_w;
            float gain = 1.f;
            if (p.q_scale) {
                float sq = 0.f;
                for (int j = lane; j < head_w; j += 32) { const float x = __bfloat162float(src[j]); sq += x * x; }    // a rotation keeps the norm
                sq = wsum(sq);
                gain = rsqrtf((p.rms ? sq / head_w : sq) + p.qk_eps) * fminf(fmaxf(p.q_scale[h], p.smin), p.smax);
            }
            for (int j = lane; j < p.content; j += 32) q_s[warp * p.content + j] = __bfloat162float(src[j]) * gain;
            for (int j = lane; j < p.dr / 2; j += 32) {
                const float x0 = __bfloat162float(src[p.content + 2 * j]) * gain, x1 = __bfloat162float(src[p.content + 2 * j + 1]) * gain;
                const float cs = p.cos[t * (p.dr / 2) + j], sn = p.sin[t * (p.dr / 2) + j];
                float* dst = p.q_rope + (static_cast<long long>(tok) * p.H + h) * p.dr + 2 * j;
                dst[0] = x0 * cs - x1 * sn;
                dst[1] = x0 * sn + x1 * cs;
            }
        }
        __syncthreads();
        if (gq == 0) {
#pragma unroll
            for (int tb = 0; tb < TB; ++tb)
#pragma unroll
                for (int i = 0; i < NV; ++i)
                    lt[tb][i] = tok0 + tb < p.tokens ? *reinterpret_cast<const float4*>(lat_s + tb * r + i * 128 + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float4 qa[TB][NV];
        float ksq[TB];
#pragma unroll
        for (int tb = 0; tb < TB; ++tb) {
            ksq[tb] = 0.f;
#pragma unroll
            for (int i = 0; i < NV; ++i) qa[tb][i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const float* w = p.w_up + static_cast<long long>(kvh) * (p.content + p.value) * r;
#pragma unroll 2
        for (int d = warp; d < p.content; d += 8) {
            float4 wv[NV];
#pragma unroll
            for (int i = 0; i < NV; ++i) wv[i] = __ldg(reinterpret_cast<const float4*>(w + static_cast<long long>(d) * r + i * 128 + lane * 4));
#pragma unroll
            for (int tb = 0; tb < TB; ++tb) {
                const float q = tok0 + tb < p.tokens ? q_s[tb * p.content + d] : 0.f;
                float kc = 0.f;
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    qa[tb][i].x = fmaf(q, wv[i].x, qa[tb][i].x); qa[tb][i].y = fmaf(q, wv[i].y, qa[tb][i].y);
                    qa[tb][i].z = fmaf(q, wv[i].z, qa[tb][i].z); qa[tb][i].w = fmaf(q, wv[i].w, qa[tb][i].w);
                    if (gq == 0) kc += lt[tb][i].x * wv[i].x + lt[tb][i].y * wv[i].y + lt[tb][i].z * wv[i].z + lt[tb][i].w * wv[i].w;
                }
                if (gq == 0) { kc = wsum(kc); ksq[tb] += kc * kc; }
            }
        }
#pragma unroll
        for (int tb = 0; tb < TB; ++tb) {
#pragma unroll
            for (int i = 0; i < NV; ++i) *reinterpret_cast<float4*>(red_s + (warp * TB + tb) * r + i * 128 + lane * 4) = qa[tb][i];
            if (gq == 0 && lane == 0) ksq_s[warp][tb] = ksq[tb];
        }
        __syncthreads();
        for (int j = threadIdx.x; j < TB * r; j += 256) {
            const int tb = j / r;
            if (tok0 + tb < p.tokens) {
                float s = 0.f;
#pragma unroll
                for (int wi = 0; wi < 8; ++wi) s += red_s[wi * TB * r + j];
                p.q_latent[(static_cast<long long>(tok0 + tb) * p.H + h) * r + (j - tb * r)] = s;
            }
        }
        if (gq == 0 && threadIdx.x < TB && tok0 + threadIdx.x < p.tokens) {
            const int tb = threadIdx.x, tok = tok0 + tb, b = tok / p.T, t = tok - b * p.T;
            float gain = 1.f;
            if (p.k_scale) {
                float sq = rsq_s[tb];
#pragma unroll
                for (int wi = 0; wi < 8; ++wi) sq += ksq_s[wi][tb];
                gain = rsqrtf((p.rms ? sq / head_w : sq) + p.qk_eps) * fminf(fmaxf(p.k_scale[kvh], p.smin), p.smax);
            }
            p.key_gain[b * p.gain_bs + static_cast<long long>(t) * p.Hkv + kvh] = __float2bfloat16(gain);
        }
        __syncthreads();                                       // q_s and red_s are rewritten for the group's next query head
    }
}

// y[m, n] = sum_k x[m, k] w[n, k] for few rows: every weight is read once, so the weights' bytes bound it.  A CTA owns 16 weight
// rows (the 16 rows of m16n8k16; 8 tokens are its columns), its eight warps split the contraction and add up in shared memory; a
// lane's fragment of two k-steps is one 16-byte piece of a row (k is dealt to the lanes the same way for both operands, its order
// inside the sum does not matter).  The 256 x 256 pair tiles of gemm_bf16.cu would occupy 2048 / 256 = 8 SM pairs here.
template <int NT>                          // 8 * NT tokens
__global__ void __launch_bounds__(256)
rows_linear_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y, int rows, int N, int K,
                   long long x_pitch, long long y_pitch) {
    __shared__ float red[8][16][8 * NT + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
    const int n0 = blockIdx.x * 16;
    const __nv_bfloat16* w0 = w + static_cast<long long>(min(n0 + g, N - 1)) * K + tq * 8;
    const __nv_bfloat16* w1 = w + static_cast<long long>(min(n0 + g + 8, N - 1)) * K + tq * 8;
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
#pragma unroll 4
    for (int c = warp; c < K / 32; c += 8) {
        const uint4 a0 = __ldg(reinterpret_cast<const uint4*>(w0 + c * 32)), a1 = __ldg(reinterpret_cast<const uint4*>(w1 + c * 32));
        const uint32_t f0[4] = {a0.x, a1.x, a0.y, a1.y}, f1[4] = {a0.z, a1.z, a0.w, a1.w};
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int row = i * 8 + g;
            uint4 b = make_uint4(0, 0, 0, 0);
            if (row < rows) b = *reinterpret_cast<const uint4*>(x + row * x_pitch + c * 32 + tq * 8);
            mma16816(acc[i], f0, b.x, b.y);
            mma16816(acc[i], f1, b.z, b.w);
        }
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
        red[warp][g][i * 8 + 2 * tq] = acc[i][0];
        red[warp][g][i * 8 + 2 * tq + 1] = acc[i][1];
        red[warp][g + 8][i * 8 + 2 * tq] = acc[i][2];
        red[warp][g + 8][i * 8 + 2 * tq + 1] = acc[i][3];
    }
    __syncthreads();
    for (int j = threadIdx.x; j < 16 * 8 * NT; j += 256) {
        const int n = j & 15, row = j >> 4;
        if (row < rows && n0 + n < N) {
            float s = 0.f;
#pragma unroll
            for (int wi = 0; wi < 8; ++wi) s += red[wi][n][row];
            y[row * y_pitch + n0 + n] = __float2bfloat16(s);
        }
    }
}

bool rows_linear_supported(int rows, int N, int K) { return rows >= 1 && rows <= 32 && N >= 1 && K >= 32 && K % 32 == 0; }

bool launch_rows_linear(const void* x, const void* w, void* y, int rows, int N, int K, long long x_pitch, long long y_pitch, cudaStream_t s) {
    if (!rows_linear_supported(rows, N, K)) return false;
    const auto* xb = static_cast<const __nv_bfloat16*>(x);
    const auto* wb = static_cast<const __nv_bfloat16*>(w);
    auto* yb = static_cast<__nv_bfloat16*>(y);
    const int grid = (N + 15) / 16;
    if (rows <= 8) rows_linear_kernel<1><<<grid, 256, 0, s>>>(xb, wb, yb, rows, N, K, x_pitch, y_pitch);
    else if (rows <= 16) rows_linear_kernel<2><<<grid, 256, 0, s>>>(xb, wb, yb, rows, N, K, x_pitch, y_pitch);
    else rows_linear_kernel<4><<<grid, 256, 0, s>>>(xb, wb, yb, rows, N, K, x_pitch, y_pitch);
    return true;
}

template <int KS, int MT, int TERMS>
static void launch_split(const MlaDecodeParams& p, cudaStream_t s) {
    constexpr int rows = MT * 16;
    constexpr int smem = md_stages(KS, MT, TERMS) * MD_TILE * (KS * 256 + 16 + MD_ROPE_MAX * 2 + 16) + MD_WARPS * rows * MD_SP_PITCH * 4 + TERMS * rows * MD_P_PITCH * 2 + rows * 4;
    static_assert((smem + 1024) * md_ctas(KS, MT, TERMS) <= 233472, "shared memory of the decode kernel");
    auto k = mla_decode_split_kernel<KS, MT, TERMS>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k<<<static_cast<unsigned>(p.splits) * ((p.T * p.H + rows - 1) / rows) * p.B, MD_WARPS * 32, smem, s>>>(p);
}

// 16-row tiles per CTA: two when there are tiles to share a pass over the cache (a CTA then does twice the products per byte), but
// the fragments of 1024-wide queries fill the registers
static int decode_row_tiles(int T, int H, int r) { return T * H > 16 && r <= 512 ? 2 : 1; }

int mla_decode_splits(int B, int T, int H, int r, int S, int terms) {
    const int rows = 16 * decode_row_tiles(T, H, r);
    const int ctas = B * ((T * H + rows - 1) / rows);
    const int tiles = (S + MD_TILE - 1) / MD_TILE;
    // one wave of CTAs, since a second would cost as much as the first: two CTAs an SM where they fit and have six tiles each, else one (8 x
    // 4022 positions: 18 splits of 7 tiles 18.1 + 8.7 us with the merge, 37 of 4 tiles 17.2 + 11.9; 32 x 8000: 4 splits 146 us, 9 splits 97)
    const int both = 148 * md_ctas(r / 128, rows / 16, terms) / ctas;
    int want = both > 0 && tiles / both >= 6 ? both : 148 / ctas;
    want = want < 1 ? 1 : (want > MD_MAX_SPLITS ? MD_MAX_SPLITS : want);
    return want < tiles ? want : (tiles < 1 ? 1 : tiles);
}

bool mla_decode_supported(int H, int Hkv, int r, int dr) {
    return (r == 256 || r == 512 || r == 768 || r == 1024) && H % 8 == 0 && H >= 8 && H <= 32 && H != 24 && r / 32 * (H / 8) <= 64 && Hkv >= 1 &&
           H % Hkv == 0 && dr % 2 == 0 && dr <= MD_ROPE_MAX && dr >= 2;
}

template <int TERMS>
static bool launch_decode_split(const float* q_latent, const float* q_rope, const void* latent, const void* rope, const void* key_gain,
                                long long latent_bs, long long rope_bs, long long gain_bs, float* part_ctx, float* part_ml, int B, int T, int H, int Hkv,
                                int r, int dr, int S, int splits, int start, int window, float scale, float softcap, cudaStream_t s) {
    if (!mla_decode_supported(H, Hkv, r, dr) || B <= 0 || T <= 0 || S <= 0 || splits < 1 || splits > MD_MAX_SPLITS) return false;
    if (static_cast<long long>(B) * T * H * splits >= (1LL << 31)) return false;            // an upper bound of every grid of a call
    MlaDecodeParams p;
    p.q_latent = q_latent; p.q_rope = q_rope;
    p.latent = static_cast<const __nv_bfloat16*>(latent); p.rope = static_cast<const __nv_bfloat16*>(rope);
    p.key_gain = static_cast<const __nv_bfloat16*>(key_gain);
    p.latent_bs = latent_bs; p.rope_bs = rope_bs; p.gain_bs = gain_bs;
    p.part_ctx = part_ctx; p.part_ml = part_ml;
    p.B = B; p.T = T; p.H = H; p.Hkv = Hkv; p.r = r; p.dr = dr; p.S = S; p.splits = splits; p.start = start; p.window = window;
    p.latent_vec = reinterpret_cast<uintptr_t>(latent) % 16 == 0 && latent_bs % 8 == 0;
    p.rope_vec = reinterpret_cast<uintptr_t>(rope) % 16 == 0 && rope_bs % 8 == 0 && dr % 8 == 0;
    p.scale = scale; p.softcap = softcap;
    const bool two = decode_row_tiles(T, H, r) == 2;
    if (r == 256) { if (two) launch_split<2, 2, TERMS>(p, s); else launch_split<2, 1, TERMS>(p, s); }
    else if (r == 512) { if (two) launch_split<4, 2, TERMS>(p, s); else launch_split<4, 1, TERMS>(p, s); }
    else if (r == 768) launch_split<6, 1, TERMS>(p, s);
    else launch_split<8, 1, TERMS>(p, s);
    return true;
}

bool launch_mla_decode(const float* q_latent, const float* q_rope, const void* latent, const void* rope, const void* key_gain,
                       long long latent_bs, long long rope_bs, long long gain_bs, float* part_ctx, float* part_ml, float* context, int B, int T,
                       int H, int Hkv, int r, int dr, int S, int splits, int start, int window, float scale, float softcap, cudaStream_t s) {
    if (!launch_decode_split<3>(q_latent, q_rope, latent, rope, key_gain, latent_bs, rope_bs, gain_bs, part_ctx, part_ml, B, T, H, Hkv, r, dr, S, splits,
                             start, window, scale, softcap, s))
        return false;
    mla_decode_merge_kernel<<<static_cast<unsigned>(B) * T * H, 128, 0, s>>>(part_ctx, part_ml, context, splits, r);
    return true;
}

template <int NV, int TB>
static void launch_prepare(const MlaPrepareParams& p, cudaStream_t s) {
    const size_t smem = (static_cast<size_t>(9) * TB * NV * 128 + static_cast<size_t>(TB) * p.content) * 4;
    auto k = mla_prepare_kernel<NV, TB>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    k<<<static_cast<unsigned>(p.Hkv) * ((p.tokens + TB - 1) / TB), 256, smem, s>>>(p);
}

template <int NV>
static void launch_cached(const MlaPrepareParams& p, bool many, const float* part_ctx, const float* part_ml, __nv_bfloat16* out, int splits, bool values,
                          cudaStream_t s) {
    constexpr int TB = NV <= 4 ? 4 : 2;       // tokens that share a pass over a head's weights; more of them do not fit the registers
    if (!values) {
        if (many) launch_prepare<NV, TB>(p, s); else launch_prepare<NV, 1>(p, s);
        return;
    }
    const int group = p.H / p.Hkv;
    if (many)
        mla_decode_values_kernel<NV, TB><<<static_cast<unsigned>(p.H) * ((p.tokens + TB - 1) / TB), 256, 0, s>>>(part_ctx, part_ml, p.w_up, out, p.tokens, p.H, group, p.content, p.value, splits);
    else
        mla_decode_values_kernel<NV, 1><<<static_cast<unsigned>(p.H) * p.tokens, 256, 0, s>>>(part_ctx, part_ml, p.w_up, out, p.tokens, p.H, group, p.content, p.value, splits);
}

bool launch_mla_cached(const MlaCachedArgs& a, cudaStream_t s) {
    if (!mla_decode_supported(a.H, a.Hkv, a.r, a.dr) || a.content < 1 || a.content > 256 || a.value < 1 || a.B <= 0 || a.T <= 0) return false;
    MlaPrepareParams p;
    p.query = static_cast<const __nv_bfloat16*>(a.query); p.low = static_cast<const __nv_bfloat16*>(a.low);
    p.q_pitch = a.q_pitch; p.low_pitch = a.low_pitch;
    p.norm_w = a.norm_w; p.cos = a.cos; p.sin = a.sin; p.w_up = a.w_up; p.q_scale = a.q_scale; p.k_scale = a.k_scale;
    auto* latent = static_cast<__nv_bfloat16*>(a.latent);
    auto* rope = static_cast<__nv_bfloat16*>(a.rope);
    auto* gain = static_cast<__nv_bfloat16*>(a.key_gain);
    p.latent = latent + static_cast<long long>(a.start) * a.r;
    p.rope = rope + static_cast<long long>(a.start) * a.dr;
    p.key_gain = gain + static_cast<long long>(a.start) * a.Hkv;
    p.latent_bs = a.latent_bs; p.rope_bs = a.rope_bs; p.gain_bs = a.gain_bs;
    p.q_latent = a.q_latent; p.q_rope = a.q_rope;
    p.tokens = a.B * a.T; p.T = a.T; p.H = a.H; p.Hkv = a.Hkv; p.content = a.content; p.value = a.value; p.dr = a.dr;
    p.norm_eps = a.norm_eps; p.qk_eps = a.qk_eps; p.smin = a.smin; p.smax = a.smax; p.rms = a.rms;
    // one token per CTA keeps every SM busy while there are few; from about 500 (head, token) pairs on, sharing the weights' reads pays
    const bool many = static_cast<long long>(p.tokens) * a.Hkv >= 512;
    auto* out = static_cast<__nv_bfloat16*>(a.out);
    auto stage = [&](bool values) {
        if (a.r == 256) launch_cached<2>(p, many, a.part_ctx, a.part_ml, out, a.splits, values, s);
        else if (a.r == 512) launch_cached<4>(p, many, a.part_ctx, a.part_ml, out, a.splits, values, s);
        else if (a.r == 768) launch_cached<6>(p, many, a.part_ctx, a.part_ml, out, a.splits, values, s);
        else launch_cached<8>(p, many, a.part_ctx, a.part_ml, out, a.splits, values, s);
    };
    stage(false);
    if (!launch_decode_split<2>(a.q_latent, a.q_rope, latent, rope, gain, a.latent_bs, a.rope_bs, a.gain_bs, a.part_ctx, a.part_ml, a.B, a.T, a.H, a.Hkv, a.r,
                             a.dr, a.start + a.T, a.splits, a.start, a.window, a.scale, a.softcap, s))
        return false;
    stage(true);
    return true;
}

}  // namespace gm
