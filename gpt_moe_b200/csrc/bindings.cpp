// Python bindings (pybind11 through torch's extension headers).  Kernels live in .cu files that do not
// include torch headers; this file converts tensors to raw pointers, builds TMA descriptors and launches.
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include <cstring>
#include <list>
#include <unordered_map>

#include "bindings_shared.h"
#include "guarded_alloc.h"
#include "gemm/gemm.h"
#include "attention/attn.h"
#include "kernels.h"
#include "kernels_decl.h"

namespace {

#define GM_CHECK(cond, msg) TORCH_CHECK(cond, "gpt_moe_b200: ", msg)

cudaStream_t current_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

int sm_count() {
    static int sms = 0;
    if (sms == 0) sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
    return sms;
}

// One status word per device: kernels write a non-zero code when a bounded wait gives up.
torch::Tensor& status_tensor(int device) {
    static std::unordered_map<int, torch::Tensor> words;
    auto it = words.find(device);
    if (it == words.end()) {
        it = words.emplace(device, torch::zeros({1}, torch::dtype(torch::kInt32).device(torch::kCUDA, device))).first;
    }
    return it->second;
}

int64_t read_status() {
    int device = at::cuda::current_device();
    return status_tensor(device).item<int32_t>();
}
void reset_status() { status_tensor(at::cuda::current_device()).zero_(); }
// the device word itself, for an asynchronous copy to pinned host memory
torch::Tensor status_word_tensor() { return status_tensor(at::cuda::current_device()); }

// ---- tensor map cache -----------------------------------------------------------------------------
struct MapKey {
    const void* ptr; uint64_t cols, rows, batch, rs, bs; uint32_t bc, br; int eb, sw;
    bool operator==(const MapKey& o) const { return std::memcmp(this, &o, sizeof(MapKey)) == 0; }
};
struct MapKeyHash {
    size_t operator()(const MapKey& k) const {
        const uint64_t* w = reinterpret_cast<const uint64_t*>(&k);
        size_t h = 1469598103934665603ull;
        for (size_t i = 0; i < sizeof(MapKey) / 8; ++i) h = (h ^ w[i]) * 1099511628211ull;
        return h;
    }
};
// Returned BY VALUE: the cache is emptied when it grows past its limit (runs whose shapes change every step, e.g. the NCCL
// expert-parallel path with its variable row counts, keep adding keys), and a reference handed out earlier in the same call
// would then dangle.
CUtensorMap cached_map(const void* ptr, int elem_bytes, uint64_t cols, uint64_t rows, uint64_t batch,
                       uint64_t row_stride_bytes, uint64_t batch_stride_bytes, uint32_t box_cols, uint32_t box_rows, int swizzle) {
    static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
    MapKey key;
    std::memset(&key, 0, sizeof(key));
    key.ptr = ptr; key.cols = cols; key.rows = rows; key.batch = batch; key.rs = row_stride_bytes; key.bs = batch_stride_bytes;
    key.bc = box_cols; key.br = box_rows; key.eb = elem_bytes; key.sw = swizzle;
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    if (cache.size() > 8192) cache.clear();
    // the encoder is a driver call and wants a current context, which a thread that has not launched anything yet (autograd's, on its first
    // node) does not have
    GM_CHECK(cudaSetDevice(at::cuda::current_device()) == cudaSuccess, "cudaSetDevice failed");
    CUtensorMap map;
    GM_CHECK(reinterpret_cast<uintptr_t>(ptr) % 16 == 0, "TMA base address must be 16-byte aligned");
    GM_CHECK(row_stride_bytes % 16 == 0 && (batch == 1 || batch_stride_bytes % 16 == 0), "TMA strides must be multiples of 16 bytes");
    GM_CHECK(gm::make_tensor_map(&map, ptr, elem_bytes, cols, rows, batch, row_stride_bytes, batch_stride_bytes, box_cols, box_rows, swizzle),
             "cuTensorMapEncodeTiled failed");
    return cache.emplace(key, map).first->second;
}

// operand map for the bf16 GEMM: `t` is [rows, cols] or [batch, rows, cols] with cols contiguous
CUtensorMap operand_map(const torch::Tensor& t, bool mn_major, int tile_rows_k_major, torch::ScalarType type = torch::kBFloat16) {
    GM_CHECK(t.is_cuda() && t.scalar_type() == type, "GEMM operands must be CUDA bf16 tensors");
    GM_CHECK(t.dim() == 2 || t.dim() == 3, "GEMM operands must be 2-D or 3-D");
    GM_CHECK(t.stride(-1) == 1, "GEMM operands must have a contiguous last dimension");
    const uint64_t batch = t.dim() == 3 ? t.size(0) : 1;
    const uint64_t rows = t.size(-2), cols = t.size(-1);
    const uint64_t rs = t.stride(-2) * 2, bs = t.dim() == 3 ? t.stride(0) * 2 : 0;
    return cached_map(t.data_ptr(), 2, cols, rows, batch, rs, bs, 64, mn_major ? 64 : tile_rows_k_major, 128);
}

// Shares of the contraction for a bf16 result whose output tiles fill the CTA pairs badly (the input gradient of the LM head contracts over
// the vocabulary into 12 to 128 tiles).  Estimates in us, fitted to 45 to 12544 rows of 768 to 2048 columns with contractions of 2048 to 50304 (cold caches,
// launches from a graph; 8 % off on average, the choice 2 % above the best of 1 to 8 shares): a launch takes 3.4; a block of 64 takes a pair 0.29,
// up to 0.38 when all pairs pull operands from L2, and a tile's read-out 1.8; tiles of 128 columns (`narrow`) 0.18 to 0.23 and 2.7; the sum costs a
// launch in a gap, 4.5, and its bytes at 14 TB/s, as the slabs still lie in L2.  us, whole / in shares: 1024 x 768 x 50304 159 / 64, 4096 rows 247 / 220,
// 9472 545 / 480; 360 x 768 x 8192 30 / 18; 360 x 1024 x 2048 12 / 15 and 2048 x 1024 x 4096 20 / 23 stay whole.
int bf16_splits(int64_t m, int64_t n, int64_t k, bool narrow, int sms) {
    const int64_t rows = (m + 255) / 256, tiles = rows * ((n + 255) / 256), blocks = (k + 63) / 64, pairs = std::max(1, sms / 2);
    const auto busy = [&](int64_t items) { return static_cast<double>(std::min(items, pairs)) / pairs; };
    const auto estimate = [&](int64_t s) {
        if (s == 1 && narrow) return 3.4 + blocks * (0.18 + 0.053 * busy(rows * ((n + 127) / 128))) + 2.7;
        const double sum = s > 1 ? 4.5 + static_cast<double>(m) * n * (8 * s + 2) / 14.0e6 : 0.0;
        return 3.4 + ((tiles * s + pairs - 1) / pairs) * (((blocks + s - 1) / s) * (0.287 + 0.097 * busy(tiles * s)) + 1.8) + sum;
    };
    int64_t best = 1;
    for (int64_t s = 2; s <= 8 && blocks / s >= 16; ++s)
        if (estimate(s) < estimate(best)) best = s;
    if (best == 1 || estimate(best) > 0.93 * estimate(1)) return 1;
    const int64_t per = (blocks + best - 1) / best;
    return static_cast<int>((blocks + per - 1) / per);                        // every share has work
}

// D[.., M, N] = alpha * op(A) op(B)^T + beta * C, optionally accumulated into an fp32 D.
//   a_mn = false: a is [.., M, K];  a_mn = true: a is [.., K, M]   (same for b with N)
//   mode 0 (dense): a, b and d with the same batch, or one 2-D b for a whole batch
//   mode 1 (grouped M): a [rows, K], b [E, N, K] or [E, K, N], d [rows, N]; tile_expert/num_m_tiles on device
//   mode 2 (grouped K): a [rows, M] (a_mn), b [rows, N] (b_mn), d [E, M, N]; seg_ends on device
//   may_split: a long contraction with few output tiles may be shared by several CTAs, whose partial results meet in the order of arrival
//   half_types: A, B and C may all be fp16 instead of bf16, and so may d (Polar Express; the calls from Python take bf16 and fp32)
//   diag: added to the diagonal of a symmetric result alpha * A B^T + beta * C
void gemm_run(const torch::Tensor& a, const torch::Tensor& b, torch::Tensor& d, bool a_mn, bool b_mn, double alpha,
              double beta, const c10::optional<torch::Tensor>& c, bool accumulate, int64_t mode,
              const c10::optional<torch::Tensor>& tile_expert, const c10::optional<torch::Tensor>& num_m_tiles,
              const c10::optional<torch::Tensor>& seg_ends, bool symmetric, const c10::optional<torch::Tensor>& batch_sumsq,
              int64_t scale_mode, bool may_split, bool half_types = false, double diag = 0.0) {
    c10::cuda::CUDAGuard guard(a.device());
    gm::GemmParams p;
    std::memset(&p, 0, sizeof(p));
    p.mode = static_cast<int>(mode);
    GM_CHECK(d.is_cuda() && d.stride(-1) == 1, "GEMM output must be a CUDA tensor with a contiguous last dimension");
    GM_CHECK(d.scalar_type() == torch::kBFloat16 || d.scalar_type() == torch::kFloat32 || (half_types && d.scalar_type() == torch::kHalf),
             "GEMM output must be bf16 or fp32");
    const torch::ScalarType in_type = half_types && a.scalar_type() == torch::kHalf ? torch::kHalf : torch::kBFloat16;
    p.in_f16 = in_type == torch::kHalf;
    p.out_f16 = d.scalar_type() == torch::kHalf;
    p.M = d.size(-2);
    p.N = d.size(-1);
    p.batch = d.dim() == 3 ? d.size(0) : 1;
    if (mode == gm::GEMM_GROUPED_K) {
        GM_CHECK(a_mn && b_mn, "grouped-K GEMM reads both operands MN-major");
        GM_CHECK(seg_ends.has_value() && seg_ends->scalar_type() == torch::kInt32, "grouped-K GEMM needs int32 seg_ends");
        GM_CHECK(a.size(-1) == p.M && b.size(-1) == p.N && a.size(0) == b.size(0), "grouped-K operand shapes");
        p.K = 0;
        p.seg_ends = seg_ends->data_ptr<int>();
    } else {
        p.K = a_mn ? a.size(-2) : a.size(-1);
        GM_CHECK((b_mn ? b.size(-2) : b.size(-1)) == p.K, "GEMM contraction sizes differ");
        GM_CHECK((b_mn ? b.size(-1) : b.size(-2)) == p.N, "GEMM: B does not match the output width");
        if (mode == gm::GEMM_GROUPED_M) {
            GM_CHECK(tile_expert.has_value() && num_m_tiles.has_value(), "grouped-M GEMM needs tile_expert and num_m_tiles");
            GM_CHECK(!a_mn && a.dim() == 2 && b.dim() == 3 && d.dim() == 2, "grouped-M operand ranks");
            p.tile_expert = tile_expert->data_ptr<int>();
            p.num_m_tiles = num_m_tiles->data_ptr<int>();
        } else {
            GM_CHECK((a_mn ? a.size(-1) : a.size(-2)) == p.M, "GEMM: A does not match the output height");
            GM_CHECK(p.batch == 1 || (a.dim() == 3 && a.size(0) == p.batch && (b.dim() == 2 || b.size(0) == p.batch)),
                     "GEMM: a batch of outputs takes as many A and as many B, or one B for all");
            p.b_shared = b.dim() == 2;
        }
    }
    p.D = d.data_ptr();
    p.ldd = d.stride(-2);
    p.d_batch_stride = d.dim() == 3 ? d.stride(0) : 0;
    p.out_fp32 = d.scalar_type() == torch::kFloat32;
    p.accumulate = accumulate;
    GM_CHECK(!accumulate || p.out_fp32, "accumulation needs an fp32 output");
    p.alpha = static_cast<float>(alpha);
    p.beta = static_cast<float>(beta);
    if (c.has_value()) {
        GM_CHECK(c->scalar_type() == in_type && c->stride(-1) == 1, "C must be bf16 with a contiguous last dimension");
        p.C = c->data_ptr();
        p.ldc = c->stride(-2);
        p.c_batch_stride = c->dim() == 3 ? c->stride(0) : 0;
        GM_CHECK(reinterpret_cast<uintptr_t>(p.C) % 16 == 0 && p.c_batch_stride % 8 == 0, "C must lie on 16-byte boundaries");      // read 16 bytes at a time
    }
    GM_CHECK(p.ldd % 8 == 0 && (p.C == nullptr || p.ldc % 8 == 0), "output row pitch must be a multiple of 8 elements");
    // here, not only in the tensor map: a shared contraction's map describes its slabs, and the sum stores to D by itself
    GM_CHECK(reinterpret_cast<uintptr_t>(p.D) % 16 == 0, "the GEMM output must lie on a 16-byte boundary");
    if (symmetric) {      // the caller vouches that alpha * A B^T + beta * C is symmetric; only the upper triangle of tiles is computed
        GM_CHECK(mode == gm::GEMM_DENSE && p.M == p.N && !p.out_fp32 && !accumulate, "symmetric GEMM: dense, square, bf16 output");
        p.symmetric = 1;
    }
    if (batch_sumsq.has_value()) {
        GM_CHECK(mode == gm::GEMM_DENSE && batch_sumsq->is_cuda() && batch_sumsq->scalar_type() == torch::kFloat32 &&
                 batch_sumsq->is_contiguous() && batch_sumsq->numel() == p.batch && (scale_mode == 1 || scale_mode == 2),
                 "batch_sumsq: one fp32 value per batched problem of a dense GEMM, scale_mode 1 or 2");
        p.batch_sumsq = batch_sumsq->data_ptr<float>();
        p.scale_mode = static_cast<int>(scale_mode);
    }
    p.status = status_tensor(a.device().index()).data_ptr<int>();
    // split-K: a long contraction with too few output tiles to fill the GPU (weight gradients) is shared by several CTAs per tile
    p.split_k = 1;
    // (not beside C, which every share would add)
    if (mode == gm::GEMM_DENSE && p.out_fp32 && may_split && p.C == nullptr) {
        const int64_t tiles = ((p.M + 255) / 256) * 2 * ((p.N + 255) / 256) * p.batch;      // CTA pairs own 256-row tiles
        const int64_t k_blocks = (p.K + 63) / 64;
        if (tiles * 2 <= sm_count() && k_blocks >= 16)
            p.split_k = static_cast<int>(std::min<int64_t>(sm_count() / tiles, k_blocks / 8));
        if (p.split_k > 1 && !accumulate) d.zero_();
    }
    // a bf16 result: the shares go to fp32 slabs of their own and are summed in order
    torch::Tensor parts;
    if (mode == gm::GEMM_DENSE && d.scalar_type() == torch::kBFloat16 && !half_types && p.batch == 1 && d.dim() == 2 && p.C == nullptr && !p.symmetric &&
        p.batch_sumsq == nullptr && p.M > 0 && p.N > 0) {
        const int splits = bf16_splits(p.M, p.N, p.K, gm::gemm_bf16_tile_width(p, a_mn, false, sm_count()) == 128, sm_count());
        if (splits > 1) {
            parts = gm::out_empty({splits, p.M, (p.N + 3) / 4 * 4}, d.options().dtype(torch::kFloat32));
            p.split_k = splits;
            p.split_slabs = 1;
            p.out_fp32 = 1;
            p.ldd = parts.stride(1);
            p.d_batch_stride = parts.stride(0);
        }
    }
    const CUtensorMap& ta = operand_map(a, a_mn, 128, in_type);
    const int eb = p.out_fp32 ? 4 : 2;
    // C of the output's shape comes through TMA; any other (broadcast over the batch or over rows, beside an fp32 output or an MN-major operand) is read by the threads
    CUtensorMap tc, tmirror;
    const bool tma_c = p.C != nullptr && mode == gm::GEMM_DENSE && !p.out_fp32 && !a_mn && !b_mn && p.K > 0 && c->dim() == d.dim() && c->sizes() == d.sizes() &&
                       p.ldc > 0 && (p.batch == 1 || p.c_batch_stride > 0);
    const CUtensorMap& tb = operand_map(b, b_mn, gm::gemm_bf16_tile_width(p, a_mn, tma_c, sm_count()) / 2, in_type);
    const bool slabs = parts.defined();
    const CUtensorMap& td = cached_map(slabs ? parts.data_ptr() : d.data_ptr(), eb, p.N, p.M, slabs ? p.split_k : d.dim() == 3 ? d.size(0) : 1, p.ldd * eb,
                                       slabs || d.dim() == 3 ? p.d_batch_stride * eb : 0, 128 / eb, tma_c ? 128 : 32, 128);        // a warp stores its 32 rows, beside a C through TMA the CTA its 128
    GM_CHECK((!p.in_f16 || p.C == nullptr || tma_c) && (diag == 0.0 || (tma_c && symmetric)), "GEMM: an fp16 C or a diagonal term needs C in the layout of the output");
    p.diag = static_cast<float>(diag);
    if (tma_c) {
        tc = cached_map(p.C, 2, p.N, p.M, p.batch, p.ldc * 2, d.dim() == 3 ? p.c_batch_stride * 2 : 0, 64, 128, 128);
    }
    // the transposed blocks of a symmetric result: 64 rows of 128 bytes beside a C through TMA, else 64 rows of a warp's 32 columns
    if (p.symmetric) tmirror = cached_map(p.D, 2, p.N, p.M, p.batch, p.ldd * 2, d.dim() == 3 ? p.d_batch_stride * 2 : 0, tma_c ? 64 : 32, 64, tma_c ? 128 : 0);
    cudaError_t e = gm::launch_gemm_bf16(ta, tb, td, tma_c ? &tc : nullptr, p.symmetric ? &tmirror : nullptr, p, a_mn, b_mn, sm_count(),
                                         current_stream());
    GM_CHECK(e == cudaSuccess, cudaGetErrorString(e));
    if (slabs) {
        gm::launch_split_sum(parts.data_ptr<float>(), p.split_k, p.M, p.N, static_cast<int>(p.ldd), d.data_ptr(), d.stride(-2), current_stream());
        e = cudaGetLastError();
        GM_CHECK(e == cudaSuccess, cudaGetErrorString(e));
    }
}
void gemm_bf16(const torch::Tensor& a, const torch::Tensor& b, torch::Tensor& d, bool a_mn, bool b_mn, double alpha, double beta,
               const c10::optional<torch::Tensor>& c, bool accumulate, int64_t mode, const c10::optional<torch::Tensor>& tile_expert,
               const c10::optional<torch::Tensor>& num_m_tiles, const c10::optional<torch::Tensor>& seg_ends, bool symmetric,
               const c10::optional<torch::Tensor>& batch_sumsq, int64_t scale_mode) {
    gemm_run(a, b, d, a_mn, b_mn, alpha, beta, c, accumulate, mode, tile_expert, num_m_tiles, seg_ends, symmetric, batch_sumsq, scale_mode, true);
}

// ---- Polar Express ------------------------------------------------------------------------------------
// Five steps X <- (a I + b A + c A^2) X, A = X X^T, on a batch of bf16 matrices x [n, m, k], wide ones (m <= k) as
// a rule; the result is bf16, and a contiguous x is scratch.
// The polynomials of consecutive steps commute, so a run of steps is carried out on the small m x m side: with Q = a I + b A + c A^2
// the next Gram matrix is Q A Q, and the product of the run's Q goes to X once.  A run costs one X X^T and one Q X whatever its length,
// where every step paid for both.  Runs of two and three steps are 18 products, 14 of them small, single steps 15 with 5 small ones.
// us, single steps with bf16 Gram matrices / here: 96 of 768 x 6144 5060 / 2870, 96 of 768 x 3072 3050 / 2060, 128 of 768 x 1536 2490 / 2310,
// 16 of 768 x 6144 990 / 657, 16 of 768 x 3072 607 / 505, in runs; where a run's fourteen small products are launches of a few waves they
// cost what the large ones save (24 of 1024 x 2048 1075 / 1113, 3 of 512 x 2048 286 / 308): runs are taken for X at least three times as wide
// as high with two tiles of Q X for every CTA pair, or twice as wide with six tiles of a small product.  A run holds four m x m matrices where
// single steps hold two (226 MB more for 96 of 768).
// Rounding noise of A grows by a^2 a step against the smallest singular values.  Error against 64 bits (2-norm; matrices 768 x 3072:
// Gaussian / rank 8 plus noise / singular values 1/i / exp(-12 i / m)): single steps in bf16 1.06e-2 / 5.8e-2 / 3.6e-2 / 9.3e-2, runs of two and
// three 0.48e-2 / 4.8e-2 / 3.4e-2 / 6.8e-2; one run of five reaches 0.1 to 20 and is not taken, nor are runs of matrices lower than 256.
// That takes fp16 for A and Q and the order Q (A Q), whose error in the directions
// that A hardly has is of second order; and the product of a run's Q is computed in full: mirrored, errors were three to five times as large,
// since rounded Q commute only nearly.  The first Q X stays bf16 x bf16, as x arrives with any scale; X is fp16 after it.
// fp16 has 2^-24 as its smallest step, so every fp16 matrix is held times a power of two that the next product's alpha takes off: singular values
// up to 1 (of x as it comes; the polynomials diverge from 1.03 on) give |A| <= 3.97, |Q| <= 8.16, a run's product <= 33.0 and |X| <= 1.99 in every step, and
// the powers leave a factor of two to 65504.  Without them rows of 1e-5 of the others lost a tenth to a quarter of their result (error of these
// rows 0.22; bf16 steps 0.010, with the powers 0.0040: 16 of 768 x 1536), rows of 1e-6 all of it, and so did matrices of norm 1e-11 (0.23, 0.005, 0.004).
// Rows of 1e-8 (0.007 to 0.009 in emulation) and norms of 1e-15 are farther than bf16 steps are: their results lie at 1e-5 of a row's usual size and less.
constexpr double kPolarGram = 8192.0, kPolarFactor = 4096.0, kPolarRun = 1024.0, kPolarX = 16384.0;
torch::Tensor polar_express(torch::Tensor x, const c10::optional<torch::Tensor>& sumsq, const std::vector<std::vector<double>>& coeffs) {
    GM_CHECK(x.is_cuda() && x.dim() == 3 && x.scalar_type() == torch::kBFloat16 && x.stride(2) == 1 && x.stride(1) % 8 == 0 && (x.size(0) <= 1 || x.stride(0) % 8 == 0) &&
             reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0, "polar_express wants bf16 matrices [n, m, k] of contiguous rows on 16-byte boundaries");
    if (!x.is_contiguous()) x = x.contiguous();                               // a batch or row pitch of its own
    for (const auto& c : coeffs) GM_CHECK(c.size() == 3, "polar_express: three coefficients a step");
    const int64_t n = x.size(0), m = x.size(1), k = x.size(2);
    GM_CHECK(!coeffs.empty(), "polar_express wants at least one step");
    c10::cuda::CUDAGuard guard(x.device());
    const int steps = static_cast<int>(coeffs.size());
    if (gm::polar_small_supported(m, k, steps) && n > 0) {
        GM_CHECK(!sumsq.has_value() || (sumsq->is_cuda() && sumsq->scalar_type() == torch::kFloat32 && sumsq->is_contiguous() && sumsq->numel() == n) ,
                 "polar_express: one fp32 sum of squares per matrix");
        std::vector<float> flat;
        for (const auto& c : coeffs) flat.insert(flat.end(), c.begin(), c.end());
        const cudaError_t e = gm::launch_polar_small(x.data_ptr(), sumsq.has_value() ? sumsq->data_ptr<float>() : nullptr, static_cast<int>(n), static_cast<int>(m),
                                                     static_cast<int>(k), flat.data(), steps, current_stream());
        GM_CHECK(e == cudaSuccess, cudaGetErrorString(e));
        return x;
    }
    const int64_t mt = (m + 255) / 256, kt = (k + 255) / 256;
    const bool runs = m >= 256 && ((k >= 3 * m && n * mt * kt >= sm_count()) || (k >= 2 * m && n * mt * (mt + 1) / 2 >= 3 * sm_count()));
    const auto half = x.options().dtype(torch::kHalf);
    torch::Tensor small[4];
    for (int i = 0; i < (runs ? 4 : 2); ++i) small[i] = gm::out_empty({n, m, m}, half);
    torch::Tensor y = gm::out_empty({n, m, k}, half);
    const auto product = [&](const torch::Tensor& a, const torch::Tensor& b, torch::Tensor d) {        // a and b symmetric: a b^T = a b; A times a Q
        gemm_run(a, b, d, false, false, 1.0 / kPolarFactor, 0.0, c10::nullopt, false, gm::GEMM_DENSE, c10::nullopt, c10::nullopt, c10::nullopt, true, c10::nullopt, 0, false, true);
    };
    torch::Tensor in = x;
    double in_scale = 1.0;                                                     // what X is held times
    for (int first = 0; first < steps;) {
        const int count = !runs ? 1 : first == 0 ? std::min(2, steps) : std::min(3, steps - first);
        const bool raw = first == 0 && sumsq.has_value();                      // not normalised yet: the epilogues do it
        const auto type = in.scalar_type();                                    // of the factor that meets X
        const torch::Tensor& gram = small[0];
        gemm_run(in, in, small[0], false, false, kPolarGram / (in_scale * in_scale), 0.0, c10::nullopt, false, gm::GEMM_DENSE, c10::nullopt, c10::nullopt, c10::nullopt, true,
                 raw ? sumsq : c10::nullopt, raw ? 2 : 0, false, true);
        int q = 1, total = 1, spare = 2;                                       // buffers of the step's Q, of the run's product, and a free one
        double total_scale = kPolarFactor;
        for (int j = 0; j < count; ++j) {
            if (j > 0) {
                product(gram, small[q], small[spare]);
                product(small[q], small[spare], gram);
            }
            const auto& c = coeffs[first + j];
            const int next = j == 0 ? q : spare;
            torch::Tensor poly = small[next];
            if (count == 1) poly = poly.view(type);
            gemm_run(gram, gram, poly, false, false, c[2] * kPolarFactor / (kPolarGram * kPolarGram), c[1] * kPolarFactor / kPolarGram, gram, false, gm::GEMM_DENSE, c10::nullopt, c10::nullopt, c10::nullopt, true, c10::nullopt, 0, false,
                     true, c[0] * kPolarFactor);
            if (j > 0) {
                const int to = q == total ? 3 : q;                             // the last Q is not needed any more
                torch::Tensor both = j == count - 1 ? small[to].view(type) : small[to];
                gemm_run(poly, small[total], both, false, true, kPolarRun / (kPolarFactor * total_scale), 0.0, c10::nullopt, false, gm::GEMM_DENSE, c10::nullopt, c10::nullopt, c10::nullopt, false,
                         c10::nullopt, 0, false, true);
                spare = total;
                total = to;
                total_scale = kPolarRun;
                q = next;
            }
        }
        const bool done = first + count == steps;
        torch::Tensor out = in.data_ptr() == y.data_ptr() ? x : y;
        out = out.view(done ? torch::kBFloat16 : torch::kHalf);
        const double out_scale = done ? 1.0 : kPolarX;
        gemm_run(small[total].view(type), in, out, false, true, out_scale / (total_scale * in_scale), 0.0, c10::nullopt, false, gm::GEMM_DENSE, c10::nullopt, c10::nullopt, c10::nullopt, false,
                 raw ? sumsq : c10::nullopt, raw ? 1 : 0, false, true);
        in = out;
        in_scale = out_scale;
        first += count;
    }
    return in;
}

// ---- MXFP8 ----------------------------------------------------------------------------------------
int64_t sf_records(int64_t rows, int64_t k) { return ((rows + 127) / 128) * ((k + 127) / 128); }

// x [.., rows, cols] bf16 (last dim contiguous, uniform row pitch) -> (q e4m3 as uint8 [.., rows, cols], scales uint8 [batch, records * 512])
std::vector<torch::Tensor> mxfp8_quantize(const torch::Tensor& x, const c10::optional<torch::Tensor>& rows_limit) {
    c10::cuda::CUDAGuard guard(x.device());
    GM_CHECK(x.is_cuda() && x.scalar_type() == torch::kBFloat16 && (x.dim() == 2 || x.dim() == 3), "mxfp8_quantize wants a 2-D or 3-D bf16 CUDA tensor");
    GM_CHECK(x.stride(-1) == 1 && x.size(-1) % 32 == 0 && x.stride(-2) % 8 == 0, "mxfp8_quantize: last dimension contiguous, multiple of 32");
    const int64_t batch = x.dim() == 3 ? x.size(0) : 1, rows = x.size(-2), cols = x.size(-1);
    GM_CHECK(batch == 1 || rows % 128 == 0 || x.is_contiguous(), "mxfp8_quantize: batched input must be contiguous");
    auto q = gm::out_empty(x.sizes(), x.options().dtype(torch::kUInt8));
    // not cleared: bytes of rows that exist are all written; the rest belongs to rows the GEMM clips
    auto sf = gm::out_empty({batch, sf_records(rows, cols) * 512}, x.options().dtype(torch::kUInt8));
    for (int64_t z = 0; z < batch; ++z) {
        const auto* src = static_cast<const at::BFloat16*>(x.data_ptr()) + (x.dim() == 3 ? z * x.stride(0) : 0);
        gm::launch_quantize_rows(src, q.data_ptr<uint8_t>() + z * rows * cols, sf.data_ptr<uint8_t>() + z * sf.stride(0), rows,
                                 static_cast<int>(cols), x.stride(-2), rows_limit.has_value() ? rows_limit->data_ptr<int>() : nullptr,
                                 current_stream());
    }
    return {q, sf};
}

// w [.., rows, cols] bf16 contiguous -> (q [.., rows, cols], scales along cols, qt [.., cols, rows], scales along the original rows)
std::vector<torch::Tensor> mxfp8_quantize_weight(const torch::Tensor& weight) {
    c10::cuda::CUDAGuard guard(weight.device());
    const torch::Tensor w = reinterpret_cast<uintptr_t>(weight.data_ptr()) % 16 == 0 ? weight : weight.clone();      // the kernel loads 16 bytes at a time
    GM_CHECK(w.is_cuda() && w.scalar_type() == torch::kBFloat16 && w.is_contiguous() && (w.dim() == 2 || w.dim() == 3), "mxfp8_quantize_weight wants a contiguous bf16 CUDA tensor");
    const int64_t batch = w.dim() == 3 ? w.size(0) : 1, rows = w.size(-2), cols = w.size(-1);
    GM_CHECK(rows % 32 == 0 && cols % 32 == 0, "mxfp8_quantize_weight: both dimensions must be multiples of 32");
    auto opt = w.options().dtype(torch::kUInt8);
    auto q = gm::out_empty(w.sizes(), opt);
    auto qt = w.dim() == 3 ? gm::out_empty({batch, cols, rows}, opt) : gm::out_empty({cols, rows}, opt);
    auto sf = gm::out_empty({batch, sf_records(rows, cols) * 512}, opt);
    auto sft = gm::out_empty({batch, sf_records(cols, rows) * 512}, opt);
    gm::launch_quantize_weight_dual(w.data_ptr(), q.data_ptr(), sf.data_ptr(), qt.data_ptr(), sft.data_ptr(), static_cast<int>(batch),
                                    static_cast<int>(rows), static_cast<int>(cols), sf.stride(0), sft.stride(0), current_stream());
    return {q, sf, qt, sft};
}

// d [.., M, N] bf16 = alpha * a [.., M, K] b [.., N, K]^T from e4m3 bytes and their scale records.
// grouped: a [rows, K] in padded expert-major order, b [E, N, K], tile_expert / num_m_tiles on the device.
void gemm_mxfp8(const torch::Tensor& a, const torch::Tensor& sfa, const torch::Tensor& b, const torch::Tensor& sfb, torch::Tensor& d, double alpha,
                const c10::optional<torch::Tensor>& tile_expert, const c10::optional<torch::Tensor>& num_m_tiles) {
    c10::cuda::CUDAGuard guard(a.device());
    GM_CHECK(a.is_cuda() && a.scalar_type() == torch::kUInt8 && b.scalar_type() == torch::kUInt8 && a.is_contiguous() && b.is_contiguous(), "mxfp8 operands are contiguous uint8 tensors");
    GM_CHECK(d.scalar_type() == torch::kBFloat16 && d.stride(-1) == 1 && d.stride(-2) % 8 == 0, "mxfp8 output is bf16 with a 16-byte aligned row pitch");
    gm::Mxfp8Params p;
    std::memset(&p, 0, sizeof(p));
    p.M = d.size(-2); p.N = d.size(-1); p.K = a.size(-1);
    GM_CHECK(b.size(-1) == p.K && b.size(-2) == p.N && p.K % 128 == 0, "mxfp8 GEMM shapes (K must be a multiple of 128)");
    p.grouped = tile_expert.has_value();
    if (p.grouped) {
        GM_CHECK(a.dim() == 2 && b.dim() == 3 && d.dim() == 2 && num_m_tiles.has_value() && a.size(0) % 256 == 0, "grouped mxfp8 operand ranks (rows padded to 256)");
        p.tile_expert = tile_expert->data_ptr<int>();
        p.num_m_tiles = num_m_tiles->data_ptr<int>();
        p.batch = 1;
    } else {
        GM_CHECK(a.size(-2) == p.M && a.dim() == d.dim() && b.dim() == d.dim(), "mxfp8 GEMM: operand ranks");
        p.batch = d.dim() == 3 ? d.size(0) : 1;
    }
    p.sfa_row_blocks = (a.size(-2) + 127) / 128;
    p.sfb_row_blocks = (p.N + 127) / 128;
    const int64_t kb = p.K / 128;
    GM_CHECK(sfa.numel() == (a.dim() == 3 ? a.size(0) : 1) * p.sfa_row_blocks * kb * 512, "mxfp8 GEMM: A scale tensor size");
    GM_CHECK(sfb.numel() == (b.dim() == 3 ? b.size(0) : 1) * p.sfb_row_blocks * kb * 512, "mxfp8 GEMM: B scale tensor size");
    p.sfa = sfa.data_ptr<uint8_t>();
    p.sfb = sfb.data_ptr<uint8_t>();
    p.alpha = static_cast<float>(alpha);
    p.status = status_tensor(a.device().index()).data_ptr<int>();
    const uint64_t ab = a.dim() == 3 ? a.size(0) : 1, bb = b.dim() == 3 ? b.size(0) : 1;
    const CUtensorMap& ta = cached_map(a.data_ptr(), 1, p.K, a.size(-2), ab, p.K, a.size(-2) * static_cast<uint64_t>(p.K), 128, 128, 128);
    const CUtensorMap& tb = cached_map(b.data_ptr(), 1, p.K, p.N, bb, p.K, static_cast<uint64_t>(p.N) * p.K, 128, gm::mxfp8_b_box_rows(p), 128);
    const CUtensorMap& td = cached_map(d.data_ptr(), 2, p.N, p.M, d.dim() == 3 ? d.size(0) : 1, d.stride(-2) * 2, d.dim() == 3 ? d.stride(0) * 2 : 0, 64, 32, 128);
    // scale arrays as [records, 128 words]: one TMA row per 512-byte record, no swizzle
    GM_CHECK(reinterpret_cast<uintptr_t>(sfa.data_ptr()) % 16 == 0 && reinterpret_cast<uintptr_t>(sfb.data_ptr()) % 16 == 0, "scale arrays must be 16-byte aligned");
    const CUtensorMap& tsfa = cached_map(sfa.data_ptr(), 4, 128, sfa.numel() / 512, 1, 512, 0, 128, 1, 0);
    const CUtensorMap& tsfb = cached_map(sfb.data_ptr(), 4, 128, sfb.numel() / 512, 1, 512, 0, 128, 1, 0);
    cudaError_t e = gm::launch_gemm_mxfp8(ta, tb, td, tsfa, tsfb, p, sm_count(), current_stream());
    GM_CHECK(e == cudaSuccess, cudaGetErrorString(e));
}

// map over a [B, T, H, 64] bf16 view whose tokens are rows of a wider matrix (e.g. the packed QKV projection output): [column, position,
// sequence], so that a tile past the end of a sequence reads zeros and a reduction into it is clipped
// Elements from one token to the next of a [B, T, H, D] view.  Torch leaves the stride of a dimension of size one open: with one token
// a sequence the sequence stride says it, with one token altogether there is nothing to say.
int64_t head_pitch(const torch::Tensor& t) { return t.size(2) != 1 ? t.stride(2) : t.size(3); }
int64_t token_pitch(const torch::Tensor& t) {
    if (t.size(1) != 1) return t.stride(1);
    return t.size(0) != 1 ? t.stride(0) : t.size(2) * head_pitch(t);
}

// `values`: value heads may lie further apart than they are wide (by whole 16-byte pieces), as in a projection that interleaves them with keys.
CUtensorMap head_map(const torch::Tensor& t, int box_rows, bool values = false) {
    GM_CHECK(t.is_cuda() && t.scalar_type() == torch::kBFloat16 && t.dim() == 4, "attention operands must be [B, T, H, D] bf16 CUDA tensors");
    const int64_t pitch = token_pitch(t);
    const int64_t head = head_pitch(t);
    GM_CHECK(t.stride(3) == 1 && (values ? head >= 64 && head % 8 == 0 : head == t.size(3)) && (t.size(0) == 1 || t.stride(0) == t.size(1) * pitch),
             "attention operands must be token-major with contiguous heads");
    return cached_map(t.data_ptr(), 2, (t.size(2) - 1) * head + t.size(3), t.size(1), t.size(0), pitch * 2, t.size(1) * pitch * 2, 64, box_rows, 128);
}

// Returns (out [B,T,H,64] bf16, lse [B,H,T] fp32).
const int* doc_start_ptr(const c10::optional<torch::Tensor>& doc_start, int64_t tokens) {
    if (!doc_start.has_value()) return nullptr;
    GM_CHECK(doc_start->is_cuda() && doc_start->scalar_type() == torch::kInt32 && doc_start->is_contiguous() && doc_start->numel() == tokens,
             "doc_start must be a contiguous int32 CUDA tensor with one entry per token");
    return doc_start->data_ptr<int>();
}

// `window_tensor`: optional 0-dim (or 1-element) int32 CUDA tensor holding the look-back; the kernels read it on the device, so the same
// (captured) launch follows a window schedule without a new host value (the reference's device-resident window,
// experiments/046-fa4-device-window.patch).
const int* window_word(const c10::optional<torch::Tensor>& window_tensor) {
    if (!window_tensor.has_value()) return nullptr;
    GM_CHECK(window_tensor->is_cuda() && window_tensor->scalar_type() == torch::kInt32 && window_tensor->numel() == 1,
             "window_tensor must be a one-element int32 CUDA tensor");
    return window_tensor->data_ptr<int>();
}

// `quantize`: also return the MXFP8 copy of out (payload uint8 [B*T, H*64], scale records), written by the kernel's epilogue.
// `single_tile`: keep the call on the kernel with one query tile per CTA (the other kernel is checked against it).
std::vector<torch::Tensor> attn_fwd(const torch::Tensor& q, const torch::Tensor& k, const torch::Tensor& v, int64_t window, double scale,
                                    double softcap, const c10::optional<torch::Tensor>& doc_start, bool quantize, bool single_tile,
                                    const c10::optional<torch::Tensor>& window_tensor) {
    c10::cuda::CUDAGuard guard(q.device());
    const int B = q.size(0), T = q.size(1), H = q.size(2), D = q.size(3), Hkv = k.size(2);
    GM_CHECK((D == 64 || D == 128) && k.size(3) == D && v.size(3) == 64 && T >= 1 && H % Hkv == 0,
             "attention kernel: query/key heads 64 or 128 wide, value heads 64 wide");
    gm::AttnParams p;
    std::memset(&p, 0, sizeof(p));
    p.batch = B; p.heads = H; p.seq_len = T; p.group = H / Hkv; p.qk_dim = D;
    p.v_head = p.dv_head = static_cast<int>(head_pitch(v));
    p.window = static_cast<int>(std::min<int64_t>(window, T));
    p.scale = static_cast<float>(scale);
    p.scale_log2e = static_cast<float>(scale * 1.4426950408889634);
    p.softcap = static_cast<float>(softcap);
    p.doc_start = doc_start_ptr(doc_start, static_cast<int64_t>(B) * T);
    auto out = gm::out_empty({B, T, H, 64}, q.options());
    auto lse = gm::out_empty({B, H, T}, q.options().dtype(torch::kFloat32));
    p.out = out.data_ptr(); p.out_stride = H * 64; p.lse = lse.data_ptr<float>();
    torch::Tensor oq, osf;
    if (quantize) {
        const int64_t rows = static_cast<int64_t>(B) * T, cols = static_cast<int64_t>(H) * 64;
        oq = gm::out_empty({rows, cols}, q.options().dtype(torch::kUInt8));
        osf = gm::out_empty({sf_records(rows, cols) * 512}, q.options().dtype(torch::kUInt8));
        p.out_q = oq.data_ptr<uint8_t>();
        p.out_sf = osf.data_ptr<uint8_t>();
    }
    p.status = status_tensor(q.device().index()).data_ptr<int>();
    p.single_tile = single_tile ? 1 : 0;
    p.window_ptr = window_word(window_tensor);
    cudaError_t e = gm::launch_attn_fwd(head_map(q, 128), head_map(k, 128), head_map(v, 128, true), p, current_stream());
    GM_CHECK(e == cudaSuccess, cudaGetErrorString(e));
    if (quantize) return {out, lse, oq, osf};
    return {out, lse};
}

// Backward.  `unpipelined`: keep the call on the kernel that issues its products in program order (the other is checked against it).
// q, k, v, out, d_out: [B,T,H(kv),64] bf16 views; lse [B,H,T].  dk, dv: [B,T,Hkv,64] bf16 views that are written
// (they may be column slices of a packed gradient buffer).  Returns dq as fp32 [B,T,H,64]; `dq_out`: a bf16 view of that shape
// (contiguous heads, e.g. the first columns of the same buffer) that gets its values as well.
torch::Tensor attn_bwd(const torch::Tensor& q, const torch::Tensor& k, const torch::Tensor& v, const torch::Tensor& out,
                       const torch::Tensor& d_out, const torch::Tensor& lse, torch::Tensor& dk, torch::Tensor& dv, int64_t window,
                       double scale, double softcap, const c10::optional<torch::Tensor>& doc_start, bool unpipelined,
                       const c10::optional<torch::Tensor>& window_tensor, const c10::optional<torch::Tensor>& dq_out) {
    c10::cuda::CUDAGuard guard(q.device());
    const int B = q.size(0), T = q.size(1), H = q.size(2), D = q.size(3), Hkv = k.size(2);
    GM_CHECK((D == 64 || D == 128) && k.size(3) == D && v.size(3) == 64 && T >= 1 && H % Hkv == 0,
             "attention kernel: query/key heads 64 or 128 wide, value heads 64 wide");
    GM_CHECK(dk.stride(3) == 1 && dk.stride(2) == D && dv.stride(3) == 1 && head_pitch(dv) % 8 == 0 && head_pitch(dv) >= 64 && token_pitch(dk) % 8 == 0 && token_pitch(dv) % 8 == 0,
             "dk/dv must be token-major views with contiguous heads and 16-byte aligned rows");
    GM_CHECK(out.stride(3) == 1 && out.stride(2) == 64 && d_out.stride(3) == 1 && d_out.stride(2) == 64, "out/d_out layout");
    gm::AttnParams p;
    std::memset(&p, 0, sizeof(p));
    p.batch = B; p.heads = H; p.seq_len = T; p.group = H / Hkv; p.qk_dim = D;
    p.v_head = p.dv_head = static_cast<int>(head_pitch(v));
    p.window = static_cast<int>(std::min<int64_t>(window, T));
    p.scale = static_cast<float>(scale);
    p.scale_log2e = static_cast<float>(scale * 1.4426950408889634);
    p.softcap = static_cast<float>(softcap);
    p.doc_start = doc_start_ptr(doc_start, static_cast<int64_t>(B) * T);
    p.lse = const_cast<float*>(lse.data_ptr<float>());
    auto delta = gm::out_empty({B, H, T}, lse.options());
    auto dq = gm::out_empty({B, T, H, D}, lse.options());
    p.delta = delta.data_ptr<float>();
    p.dq_accum = dq.data_ptr<float>();
    p.dk = dk.data_ptr(); p.dv = dv.data_ptr(); p.dv_head = static_cast<int>(head_pitch(dv)); p.dkv_stride = token_pitch(dk); p.dv_stride = token_pitch(dv);
    p.status = status_tensor(q.device().index()).data_ptr<int>();
    p.single_tile = unpipelined ? 1 : 0;
    p.window_ptr = window_word(window_tensor);
    const CUtensorMap& tdq = cached_map(dq.data_ptr(), 4, static_cast<uint64_t>(H) * D, T, B, static_cast<uint64_t>(H) * D * 4,
                                        static_cast<uint64_t>(T) * H * D * 4, 32, D == 64 && !unpipelined ? 32 : 128, 128);      // rows that leave at a time
    cudaError_t e = gm::launch_attn_bwd(head_map(q, 128), head_map(k, 128), head_map(v, 128, true), head_map(d_out, 128), tdq, p,
                                        d_out.data_ptr(), out.data_ptr(), token_pitch(d_out), token_pitch(out), delta.data_ptr<float>(),
                                        current_stream());
    GM_CHECK(e == cudaSuccess, cudaGetErrorString(e));
    if (dq_out.has_value()) {
        const torch::Tensor& o = *dq_out;
        GM_CHECK(o.is_cuda() && o.scalar_type() == torch::kBFloat16 && o.sizes() == q.sizes() && o.stride(3) == 1 && o.stride(2) == D && o.stride(1) % 8 == 0 &&
                 o.stride(0) == T * o.stride(1) && reinterpret_cast<uintptr_t>(o.data_ptr()) % 16 == 0, "dq_out: bf16 view of q's shape, contiguous heads, aligned rows");
        e = gm::launch_attn_dq_store(dq.data_ptr<float>(), o.data_ptr(), static_cast<long long>(B) * T, H * D, o.stride(1), current_stream());
        GM_CHECK(e == cudaSuccess, cudaGetErrorString(e));
    }
    return dq;
}

}  // namespace

namespace gm {
int* status_word(int device) { return status_tensor(device).data_ptr<int>(); }

void gemm_plain(const torch::Tensor& a, const torch::Tensor& b, torch::Tensor& d) {
    gemm_bf16(a, b, d, false, false, 1.0, 0.0, c10::nullopt, false, GEMM_DENSE, c10::nullopt, c10::nullopt, c10::nullopt, false, c10::nullopt, 0);
}
void gemm_by_expert(const torch::Tensor& a, const torch::Tensor& b, torch::Tensor& d, const torch::Tensor& tile_expert, const torch::Tensor& meta) {
    gemm_bf16(a, b, d, false, false, 1.0, 0.0, c10::nullopt, false, GEMM_GROUPED_M, tile_expert, meta, c10::nullopt, false, c10::nullopt, 0);
}
void gemm_fp32(const torch::Tensor& a, const torch::Tensor& b, torch::Tensor& d, bool accumulate) {
    gemm_run(a, b, d, false, false, 1.0, 0.0, c10::nullopt, accumulate, GEMM_DENSE, c10::nullopt, c10::nullopt, c10::nullopt, false, c10::nullopt, 0, false);
}
CUtensorMap rows_map(const void* base, uint64_t cols, uint64_t rows, uint64_t batch, uint64_t row_pitch, uint64_t batch_pitch) {
    return cached_map(base, 2, cols, rows, batch, row_pitch * 2, batch_pitch * 2, 64, 128, 128);
}
torch::Tensor attention_out(const torch::Tensor& q, const torch::Tensor& k, const torch::Tensor& v, int64_t window, double scale, double softcap,
                            const c10::optional<torch::Tensor>& doc_start) {
    return attn_fwd(q, k, v, window, scale, softcap, doc_start, false, false, c10::nullopt)[0];
}
}  // namespace gm

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("read_status", &read_status, "status word of the current device (0 = no bounded wait gave up)");
    m.def("reset_status", &reset_status);
    m.def("status_word_tensor", &status_word_tensor);
    m.def("gemm_bf16", &gemm_bf16, py::arg("a"), py::arg("b"), py::arg("d"), py::arg("a_mn") = false, py::arg("b_mn") = false,
          py::arg("alpha") = 1.0, py::arg("beta") = 0.0, py::arg("c") = py::none(), py::arg("accumulate") = false,
          py::arg("mode") = 0, py::arg("tile_expert") = py::none(), py::arg("num_m_tiles") = py::none(),
          py::arg("seg_ends") = py::none(), py::arg("symmetric") = false,
          py::arg("batch_sumsq") = py::none(), py::arg("scale_mode") = 0);
    m.def("bf16_splits", &bf16_splits, py::arg("m"), py::arg("n"), py::arg("k"), py::arg("narrow"), py::arg("sms"));
    m.def("polar_express", &polar_express, py::arg("x"), py::arg("sumsq"), py::arg("coeffs"));
    m.def("mxfp8_quantize", &mxfp8_quantize, py::arg("x"), py::arg("rows_limit") = py::none());
    m.def("mxfp8_quantize_weight", &mxfp8_quantize_weight);
    m.def("gemm_mxfp8", &gemm_mxfp8, py::arg("a"), py::arg("sfa"), py::arg("b"), py::arg("sfb"), py::arg("d"), py::arg("alpha") = 1.0,
          py::arg("tile_expert") = py::none(), py::arg("num_m_tiles") = py::none());
    m.def("attn_fwd", &attn_fwd, py::arg("q"), py::arg("k"), py::arg("v"), py::arg("window"), py::arg("scale"), py::arg("softcap") = 0.0,
          py::arg("doc_start") = py::none(), py::arg("quantize") = false, py::arg("single_tile") = false, py::arg("window_tensor") = py::none());
    m.def("attn_bwd", &attn_bwd, py::arg("q"), py::arg("k"), py::arg("v"), py::arg("out"), py::arg("d_out"), py::arg("lse"), py::arg("dk"),
          py::arg("dv"), py::arg("window"), py::arg("scale"), py::arg("softcap") = 0.0, py::arg("doc_start") = py::none(),
          py::arg("unpipelined") = false, py::arg("window_tensor") = py::none(), py::arg("dq_out") = py::none());
    gm::register_kernels(m);
}
