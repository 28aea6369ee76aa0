// Entry points shared by the translation units of the library: the C ABI's routing functions with the small per-call
// values (losses, their gradients) read and written on the device, as the layer driver (ffm_layer.cu) uses them.
#pragma once

#include "../../include/ffmoe.h"

namespace ffm {

// True where an address does not lie on a 16-byte boundary. The row and routing kernels load and store 16 bytes at a time, and an
// access off that boundary ends the context; the GEMMs' tensor maps refuse such operands themselves.
template <typename... P>
bool off_16_bytes(const P*... p) {
  return ((reinterpret_cast<uintptr_t>(p) | ...) & 15u) != 0;
}

// ffm_route_forward; aux = aux_scale * stats[E + 1], z = z_scale * stats[E], *zero = 0 (each skipped when null).
int route_forward_losses(const void* hidden, const void* gate_w, const float* expert_bias, int64_t N, int D, int E,
                         int top_k, int gating, float weight_scale, int pre_softmax, int n_group, int topk_group,
                         void* logits, float* topk_w, int32_t* topk_idx, float* lse, int32_t* counts,
                         int32_t* tile_start, int32_t* pos, int32_t* src, int64_t rows_cap, float* stats, float* aux,
                         float aux_scale, float* z, float z_scale, int32_t* zero, void* workspace,
                         size_t workspace_bytes, int32_t* status, ffm_stream_t stream);

// Gradients of the two losses: either the arrays of ffm_route_backward (gaux [E], gz scalar), or the upstream scalars
// (grad_aux, grad_z; null = no such term) with gaux[e] = counts[e] * (*grad_aux * aux_coef), gz = *grad_z * z_coef.
struct LossGrads {
  const float* gaux;
  const float* gz;
  const int32_t* counts;
  const float* grad_aux;
  const float* grad_z;
  float aux_coef;
  float z_coef;
};

int route_backward_losses(const float* gw, const float* topk_w, const int32_t* topk_idx, const void* logits,
                          const float* lse, const LossGrads& lg, const void* hidden, const void* gate_w, int64_t N,
                          int D, int E, int top_k, int gating, int accumulate, void* dH, void* dGate, void* workspace,
                          size_t workspace_bytes, int32_t* status, ffm_stream_t stream);

// ffm_grouped_gemm_wgrad_rows; with tile_start null the groups are equal ranges (in 128-row tiles) of the rows, a split of
// one dense contraction.
int grouped_wgrad(const void* A, const void* B, int groups, const int32_t* tile_start, const int32_t* counts,
                  int64_t rows_cap, int M, int Nout, float scale, void* dW, int32_t* status, ffm_stream_t stream);

// ffm_combine_forward_add2; with status_host (host memory the device can write) a non-zero *status is stored there.
int combine_forward_status(const void* Y, const int32_t* pos, const float* w, const void* addend, const void* addend2,
                           int64_t N, int top_k, int D, void* out, const int32_t* status, int32_t* status_host,
                           ffm_stream_t stream);

// out = a + b, bf16 values added in fp32 (n elements, a multiple of 8)
int add_bf16(const void* a, const void* b, int64_t n, void* out, ffm_stream_t stream);

}  // namespace ffm
