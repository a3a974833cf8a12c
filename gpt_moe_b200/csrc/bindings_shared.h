// Tensor-level functions of bindings.cpp that the composed calls of bindings_ops.cpp issue as well.
#pragma once
#include <cuda.h>
#include <torch/extension.h>

namespace gm {
// d = a b^T (bf16), dense; or grouped by expert: a [rows, K], b [E, N, K] with the tile table of `route`
void gemm_plain(const torch::Tensor& a, const torch::Tensor& b, torch::Tensor& d);
void gemm_by_expert(const torch::Tensor& a, const torch::Tensor& b, torch::Tensor& d, const torch::Tensor& tile_expert, const torch::Tensor& meta);
// d (+)= a b^T with an fp32 d, sums in the same order every time
void gemm_fp32(const torch::Tensor& a, const torch::Tensor& b, torch::Tensor& d, bool accumulate);
// map of a bf16 tensor [batch, rows, cols] (cols contiguous) with a 64 x 128 box, 128-byte swizzle
CUtensorMap rows_map(const void* base, uint64_t cols, uint64_t rows, uint64_t batch, uint64_t row_pitch, uint64_t batch_pitch);
torch::Tensor attention_out(const torch::Tensor& q, const torch::Tensor& k, const torch::Tensor& v, int64_t window, double scale, double softcap,
                            const c10::optional<torch::Tensor>& doc_start);
}  // namespace gm
