// Routing forward for sm_100a.
//
//   route_gate_topk   gate product (fp32 accumulate, bf16 round), scoring, iterative-argmax top-k (lowest index
//                     wins ties), renormalisation, logsumexp, per-block expert histogram and
//                     probability-mass partial sums.
//   route_scan        one block: per-expert exclusive scan of the block histograms, expert counts,
//                     128-row-aligned segment starts (tile_start) and the loss statistics, all summed in a
//                     fixed order so results do not depend on scheduling.
//   route_rank        stable rank of every routed slot inside its expert segment -> pos[] and src[].
//
// Tokens are assigned to blocks in contiguous chunks, so "block order, then warp order, then slot order"
// equals the (token, slot) order of a stable sort by expert id.
#include <atomic>

#include "ffm_common.cuh"
#include "ffm_internal.h"

namespace ffm {

namespace {

constexpr int ROUTE_THREADS = 256;
constexpr int ROUTE_WARPS = ROUTE_THREADS / 32;
constexpr int MAX_E = 256;

// What the last routing kernel derives from the statistics: aux = aux_scale * sum_e counts[e] * mass[e],
// z = z_scale * sum_n lse[n]^2, and a zeroed word (the count of dropped slots). Any pointer may be null.
struct LossOut {
  float* aux;
  float* z;
  int32_t* zero;
  float aux_scale;
  float z_scale;
};

struct RouteGrid {
  int blocks;
  int tokens_per_block;
};

// Tokens a block of the gate kernel handles per iteration, at least: 32 / slices of D with up to 32 experts, 16 / NG when
// the warps of a block share NG groups of 32 experts.
int route_granule(int E) { return E <= 32 ? 4 : (E <= 64 ? 8 : (E <= 128 ? 4 : 2)); }

RouteGrid route_grid(long long N, int granule = 16) {
  // Contiguous token chunks, a multiple of the granule, about four blocks per SM.
  long long target_blocks = 148 * 4;
  long long tpb = (N + target_blocks - 1) / target_blocks;
  tpb = ((tpb + granule - 1) / granule) * granule;
  if (tpb < granule) tpb = granule;
  RouteGrid g;
  g.tokens_per_block = static_cast<int>(tpb);
  g.blocks = static_cast<int>((N + tpb - 1) / tpb);
  if (g.blocks < 1) g.blocks = 1;
  return g;
}

// Sum GW per-lane partial accumulators across the warp; on return lane l holds the total of
// accumulator (l % GW) in a[0].
template <int GW>
__device__ __forceinline__ void transpose_reduce(float (&a)[GW], int lane) {
#pragma unroll
  for (int n = GW; n > 1; n >>= 1) {
    const int o = n >> 1;
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float lo = a[i], hi = a[i + o];
      const float send = upper ? lo : hi;
      const float keep = upper ? hi : lo;
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (int o = 16; o >= GW; o >>= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
}

__device__ __forceinline__ float dot8(const uint4& h, const uint4& w, float acc) {
  const float2 h0 = unpack_bf16x2(h.x), h1 = unpack_bf16x2(h.y), h2 = unpack_bf16x2(h.z), h3 = unpack_bf16x2(h.w);
  const float2 w0 = unpack_bf16x2(w.x), w1 = unpack_bf16x2(w.y), w2 = unpack_bf16x2(w.z), w3 = unpack_bf16x2(w.w);
  acc = fmaf(h0.x, w0.x, acc);
  acc = fmaf(h0.y, w0.y, acc);
  acc = fmaf(h1.x, w1.x, acc);
  acc = fmaf(h1.y, w1.y, acc);
  acc = fmaf(h2.x, w2.x, acc);
  acc = fmaf(h2.y, w2.y, acc);
  acc = fmaf(h3.x, w3.x, acc);
  acc = fmaf(h3.y, w3.y, acc);
  return acc;
}

struct RouteOpts {
  int gating;
  float weight_scale;
  int pre_softmax;  // softmax gating: probabilities over all experts before selection (DeepSeek-V3 style)
  int n_group;      // > 0: group-limited selection over n_group contiguous expert groups
  int topk_group;   // groups kept per token
};

// Arg-max of (value, expert) pairs over W lanes: greater value wins, equal values go to the lower expert index.
template <int W>
__device__ __forceinline__ void lanes_argmax(float& best, int& best_e) {
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
    if (ov > best || (ov == best && oe < best_e)) {
      best = ov;
      best_e = oe;
    }
  }
}

template <int W>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
  for (int o = W / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Scoring, selection, weights and statistics of one token by W lanes (8, 16 or 32; 32 / W tokens per warp side by side),
// whose bf16-rounded logits they hold: lane holds expert g * 32 + lane for NG > 1 (W == 32), expert lane % W for
// NG == 1 (E <= W). `lane` counts within the W lanes; lanes whose token does not exist take part in the shuffles with
// active == false and leave no trace.
template <int W, int NG>
__device__ __forceinline__ void route_token(const float (&logit)[NG], long long n, int lane, bool active, int E, int top_k,
                                            const RouteOpts& o, const float* __restrict__ bias,
                                            bf16* __restrict__ logits_out, float* __restrict__ topk_w,
                                            int32_t* __restrict__ topk_idx, float* __restrict__ lse_out,
                                            float (&mass)[NG], int (&cnt)[NG], float& zsum) {
  static_assert(NG == 1 || W == 32, "one expert per lane with fewer than 32 lanes");

  // logsumexp over all experts (z-loss, and the normaliser of pre-softmax scoring)
  float lmax = -INFINITY;
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    const int e = g * 32 + lane;
    if (e < E) {
      lmax = fmaxf(lmax, logit[g]);
      if (logits_out != nullptr && active) logits_out[n * E + e] = __float2bfloat16_rn(logit[g]);
    }
  }
#pragma unroll
  for (int s = W / 2; s > 0; s >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, s));
  float esum = 0.0f;
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    const int e = g * 32 + lane;
    if (e < E) esum += __expf(logit[g] - lmax);
  }
  esum = lanes_sum<W>(esum);
  const float lse = lmax + __logf(esum);
  if (lane == 0 && active) {
    lse_out[n] = lse;
    zsum += lse * lse;
  }

  float sel[NG];  // value used for selection
  float val[NG];  // unbiased value that becomes the weight (logit, probability or sigmoid score)
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    const int e = g * 32 + lane;
    const bool valid = e < E;
    const float lg = logit[g];
    float v;
    if (o.gating == FFM_GATING_SIGMOID) {
      v = sigmoid_rn(lg);
    } else if (o.pre_softmax) {
      v = __expf(lg - lse);
    } else {
      v = lg;
    }
    float sv = v;
    if (bias != nullptr && valid) sv = v + bias[e];
    val[g] = valid ? v : 0.0f;
    sel[g] = valid ? sv : -INFINITY;
  }
  if (o.gating == FFM_GATING_SIGMOID) {
#pragma unroll
    for (int g = 0; g < NG; ++g) mass[g] += active ? val[g] : 0.0f;
  }

  // ---- group-limited selection: keep the topk_group groups with the best sum of their top scores ----
  if (o.n_group > 0) {
    const int epg = E / o.n_group;
    const int per_group = top_k / o.topk_group;
    const bool use_sum = per_group > 1 && per_group <= epg;
    const int rounds = use_sum ? per_group : 1;
    float my_gscore = -INFINITY;  // lane gi holds the score of group gi
    for (int gi = 0; gi < o.n_group; ++gi) {
      float tmp[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        const int e = g * 32 + lane;
        tmp[g] = (e / epg == gi) ? sel[g] : -INFINITY;
      }
      float score = 0.0f;
      for (int r = 0; r < rounds; ++r) {
        float best = -INFINITY;
        int best_e = 0x7fffffff;
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          if (tmp[g] > best) {
            best = tmp[g];
            best_e = g * 32 + lane;
          }
        }
        lanes_argmax<W>(best, best_e);
        score = (r == 0) ? best : score + best;
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          if (g * 32 + lane == best_e) tmp[g] = -INFINITY;
        }
      }
      if (lane == gi) my_gscore = score;
    }
    unsigned keep = 0u;
    float gs = (lane < o.n_group) ? my_gscore : -INFINITY;
    for (int r = 0; r < o.topk_group; ++r) {
      float best = gs;
      int best_l = (gs == -INFINITY) ? 0x7fffffff : lane;
      lanes_argmax<W>(best, best_l);
      if (best_l < 32) keep |= 1u << best_l;
      if (lane == best_l) gs = -INFINITY;
    }
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const int e = g * 32 + lane;
      if (!((keep >> ((e / epg) & 31)) & 1u)) sel[g] = -INFINITY;
    }
  }

  // ---- top-k by iterative argmax, lowest index wins ties ----
  float my_val = 0.0f;
  int my_idx = 0;
  for (int j = 0; j < top_k; ++j) {
    float best = -INFINITY;
    int best_e = 0x7fffffff;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      if (sel[g] > best) {
        best = sel[g];
        best_e = g * 32 + lane;
      }
    }
    lanes_argmax<W>(best, best_e);
    // the holder of best_e publishes the unbiased value and retires the expert
    float v_pub = 0.0f;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      if (g * 32 + lane == best_e) {
        v_pub = val[g];
        sel[g] = -INFINITY;
      }
    }
    v_pub = __shfl_sync(0xffffffffu, v_pub, best_e & (W - 1), W);
    if (lane == j) {
      my_val = v_pub;
      my_idx = best_e < E ? best_e : -1;  // -1: nothing compares greater than -inf (NaN scores)
    }
  }

  // ---- weights over the k selected values (lanes 0..k-1) ----
  float w;
  if (o.gating == FFM_GATING_SOFTMAX && !o.pre_softmax) {
    float m = (lane < top_k) ? my_val : -INFINITY;
#pragma unroll
    for (int s = W / 2; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    const float ex = (lane < top_k) ? __expf(my_val - m) : 0.0f;
    const float den = lanes_sum<W>(ex);
    w = ex / den;
  } else {
    const float sc = (lane < top_k) ? my_val : 0.0f;
    const float den = lanes_sum<W>(sc) + 1e-6f;
    w = sc / den;
  }
  w *= o.weight_scale;
  if (lane < top_k && active) {
    topk_w[n * top_k + lane] = w;
    topk_idx[n * top_k + lane] = my_idx;
  }
  // ---- statistics: lane (e % 32) owns expert e ----
  for (int j = 0; j < top_k; ++j) {
    const int ej = __shfl_sync(0xffffffffu, my_idx, j, W);
    const float wj = __shfl_sync(0xffffffffu, w, j, W);
    const int own_lane = (NG > 1) ? (ej & 31) : ej;
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      if (active && lane == own_lane && g == ((NG > 1) ? (ej >> 5) : 0)) {
        cnt[g] += 1;
        if (o.gating == FFM_GATING_SOFTMAX) mass[g] += wj;
      }
    }
  }
}

// src[:] = -1 (padding), spread over the grid: the rank kernel later writes the rows in use.
__device__ __forceinline__ void fill_src(int32_t* __restrict__ src, long long rows_cap) {
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < rows_cap; i += step) src[i] = -1;
}

// Statistics of one block, summed over its warps in warp order. Lane l holds experts g * 32 + l.
template <int NG>
__device__ __forceinline__ void block_statistics(float (&s_mass)[ROUTE_WARPS][NG * 32], int (&s_cnt)[ROUTE_WARPS][NG * 32],
                                                 float (&s_z)[ROUTE_WARPS], const float (&mass)[NG],
                                                 const int (&cnt)[NG], float zsum, int E, int32_t* __restrict__ block_hist,
                                                 float* __restrict__ block_mass, float* __restrict__ block_z) {
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    s_mass[warp][g * 32 + lane] = mass[g];
    s_cnt[warp][g * 32 + lane] = cnt[g];
  }
  if (lane == 0) s_z[warp] = zsum;
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += ROUTE_THREADS) {
    float m = 0.0f;
    int c = 0;
    for (int w = 0; w < ROUTE_WARPS; ++w) {
      m += s_mass[w][e];
      c += s_cnt[w][e];
    }
    block_mass[static_cast<long long>(e) * gridDim.x + blockIdx.x] = m;
    block_hist[static_cast<long long>(e) * gridDim.x + blockIdx.x] = c;
  }
  if (threadIdx.x == 0) {
    float z = 0.0f;
    for (int w = 0; w < ROUTE_WARPS; ++w) z += s_z[w];
    block_z[blockIdx.x] = z;
  }
}

// Up to 32 experts: gate product, scoring and top-k in one kernel. `slices` warps (1, 2, 4 or 8, by the width of a row)
// split D for four tokens x eight experts, so that a row's chunks are all in flight at once and a block holds
// 32 / slices tokens; the slices are summed in order, and then W lanes (E <= W) route a token, 32 / W tokens per warp side
// by side, since that chain of shuffles is the longest part. With a token pair per warp (each lane walking a quarter to
// a sixteenth of the row) the kernel waited for memory. Before and after: 36 -> 31 us at 16384 tokens, E = 8, D = 1024;
// 13 -> 7 at 1999; 55 -> 48 at 8192, D = 4096; 17 -> 14 at 3001, E = 16; each with a memset of src less.
// Registers: with 64 (E <= 8) a block fits beside a CTA of the shared expert's GEMM; at 128, four tokens per pass, it is a
// little faster alone and 1 % slower in a layer with a shared expert.
constexpr int GATE_TG = 4;
constexpr int GATE_EG = 8;
constexpr int GATE_PASS = 2;  // tokens per pass: 16 accumulators, so that the kernel also fits beside a GEMM CTA
template <int W>
__global__ void __launch_bounds__(ROUTE_THREADS, W == 8 ? 4 : 3)
route_gate_topk(const bf16* __restrict__ hidden, const bf16* __restrict__ gate_w, const float* __restrict__ bias,
                long long N, int D, int E, int top_k, RouteOpts opts, int tokens_per_block, int slices,
                bf16* __restrict__ logits_out, float* __restrict__ topk_w, int32_t* __restrict__ topk_idx,
                float* __restrict__ lse_out, int32_t* __restrict__ block_hist, float* __restrict__ block_mass,
                float* __restrict__ block_z, int32_t* __restrict__ src, long long rows_cap) {
  __shared__ float s_mass[ROUTE_WARPS][32];
  __shared__ int s_cnt[ROUTE_WARPS][32];
  __shared__ float s_z[ROUTE_WARPS];
  __shared__ float s_part[ROUTE_WARPS][GATE_TG * GATE_EG];
  __shared__ float s_logit[ROUTE_WARPS * GATE_TG][33];
  static_assert(GATE_TG * GATE_EG <= 32, "one total per lane");

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const long long tok_begin = static_cast<long long>(blockIdx.x) * tokens_per_block;
  long long tok_end = tok_begin + tokens_per_block;
  if (tok_end > N) tok_end = N;
  const int chunks = D >> 3;  // 16-byte chunks per row
  const int groups = ROUTE_WARPS / slices;       // token groups of four per trip
  const int slice = warp % slices;
  const int tg = warp / slices;
  fill_src(src, rows_cap);

  float mass[1] = {0.0f};
  int cnt[1] = {0};
  float zsum = 0.0f;
  for (long long it0 = tok_begin; it0 < tok_end; it0 += groups * GATE_TG) {
    for (int e0 = 0; e0 < E; e0 += GATE_EG) {
#pragma unroll 1
      for (int p0 = 0; p0 < GATE_TG; p0 += GATE_PASS) {
        const bf16* h[GATE_PASS];
#pragma unroll
        for (int t = 0; t < GATE_PASS; ++t) {
          long long n = it0 + tg * GATE_TG + p0 + t;
          if (n >= tok_end) n = tok_end - 1;  // tokens past the end repeat the last one; their logits are not used
          h[t] = hidden + n * D;
        }
        float acc[GATE_PASS * GATE_EG];
#pragma unroll
        for (int i = 0; i < GATE_PASS * GATE_EG; ++i) acc[i] = 0.0f;
        for (int c = slice * 32 + lane; c < chunks; c += slices * 32) {
          uint4 hv[GATE_PASS];
#pragma unroll
          for (int t = 0; t < GATE_PASS; ++t) hv[t] = __ldg(reinterpret_cast<const uint4*>(h[t]) + c);
#pragma unroll
          for (int e = 0; e < GATE_EG; ++e) {
            const int ee = min(e0 + e, E - 1);
            const uint4 w = __ldg(reinterpret_cast<const uint4*>(gate_w + static_cast<long long>(ee) * D) + c);
#pragma unroll
            for (int t = 0; t < GATE_PASS; ++t) acc[t * GATE_EG + e] = dot8(hv[t], w, acc[t * GATE_EG + e]);
          }
        }
        transpose_reduce<GATE_PASS * GATE_EG>(acc, lane);
        if (lane < GATE_PASS * GATE_EG) s_part[warp][p0 * GATE_EG + lane] = acc[0];
      }
      __syncthreads();
      if (warp < groups) {
        float t = 0.0f;
        for (int i = 0; i < slices; ++i) t += s_part[warp * slices + i][lane];
        s_logit[warp * GATE_TG + lane / GATE_EG][e0 + lane % GATE_EG] = bf16_round(t);
      }
      __syncthreads();
    }
    constexpr int TPW = 32 / W;
    const int sub = lane % W;
    for (int t0 = warp * TPW; t0 < groups * GATE_TG && it0 + t0 < tok_end; t0 += ROUTE_WARPS * TPW) {
      const int t = t0 + lane / W;
      const float logit[1] = {sub < E ? s_logit[t][sub] : 0.0f};
      route_token<W, 1>(logit, it0 + t, sub, it0 + t < tok_end, E, top_k, opts, bias, logits_out, topk_w, topk_idx, lse_out,
                        mass, cnt, zsum);
    }
    __syncthreads();  // the logits are overwritten by the next trip
  }
  // lanes of the side-by-side tokens hold statistics of the same experts
#pragma unroll
  for (int o = W; o < 32; o <<= 1) {
    mass[0] += __shfl_xor_sync(0xffffffffu, mass[0], o);
    cnt[0] += __shfl_xor_sync(0xffffffffu, cnt[0], o);
    zsum += __shfl_xor_sync(0xffffffffu, zsum, o);
  }
  block_statistics<1>(s_mass, s_cnt, s_z, mass, cnt, zsum, E, block_hist, block_mass, block_z);
}

// Slices of D for rows of D elements: one 32-lane sweep of 16-byte chunks each, at most one per warp.
int gate_slices(int D) {
  const int chunks = D >> 3;
  return chunks <= 32 ? 1 : (chunks <= 64 ? 2 : (chunks <= 128 ? 4 : 8));
}

// More than 32 experts where the tensor-core gate GEMM does not apply: the warps of a block share the gate GEMM of a few
// token pairs. Warp w computes the 32 experts of group (w % NG) for pair (w / NG) and leaves the logits in shared
// memory; then warp t routes token t of the iteration. 8 / NG pairs per iteration keep every warp busy in the GEMM phase
// for any NG in {2, 4, 8}. Expert e = g * 32 + lane.
template <int NG>
__global__ void __launch_bounds__(ROUTE_THREADS, 1)
route_gate_topk_many(const bf16* __restrict__ hidden, const bf16* __restrict__ gate_w, const float* __restrict__ bias,
                     long long N, int D, int E, int top_k, RouteOpts opts, int tokens_per_block,
                     bf16* __restrict__ logits_out, float* __restrict__ topk_w, int32_t* __restrict__ topk_idx,
                     float* __restrict__ lse_out, int32_t* __restrict__ block_hist, float* __restrict__ block_mass,
                     float* __restrict__ block_z, int32_t* __restrict__ src, long long rows_cap) {
  __shared__ float s_mass[ROUTE_WARPS][NG * 32];
  __shared__ int s_cnt[ROUTE_WARPS][NG * 32];
  __shared__ float s_z[ROUTE_WARPS];
  constexpr int PAIRS = ROUTE_WARPS / NG;
  __shared__ float s_logit[2 * PAIRS][NG * 32];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const long long tok_begin = static_cast<long long>(blockIdx.x) * tokens_per_block;
  long long tok_end = tok_begin + tokens_per_block;
  if (tok_end > N) tok_end = N;
  const int chunks = D >> 3;  // 16-byte chunks per row
  fill_src(src, rows_cap);

  float mass[NG];
  int cnt[NG];
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    mass[g] = 0.0f;
    cnt[g] = 0;
  }
  float zsum = 0.0f;
  const int my_pair = warp / NG;
  const int my_group = warp % NG;
  for (long long it0 = tok_begin; it0 < tok_end; it0 += 2 * PAIRS) {
    const long long t0 = it0 + 2 * my_pair;
    if (t0 < tok_end) {
      const bool has1 = (t0 + 1) < tok_end;
      const uint4* h0p = reinterpret_cast<const uint4*>(hidden + t0 * D);
      const uint4* h1p = reinterpret_cast<const uint4*>(hidden + (has1 ? t0 + 1 : t0) * D);
      float acc0[32], acc1[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        acc0[e] = 0.0f;
        acc1[e] = 0.0f;
      }
      for (int c = lane; c < chunks; c += 32) {
        const uint4 a0 = __ldg(h0p + c);
        const uint4 a1 = __ldg(h1p + c);
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const int ee = my_group * 32 + e;
          if (ee < E) {
            const uint4 w = __ldg(reinterpret_cast<const uint4*>(gate_w + static_cast<long long>(ee) * D) + c);
            acc0[e] = dot8(a0, w, acc0[e]);
            acc1[e] = dot8(a1, w, acc1[e]);
          }
        }
      }
      transpose_reduce<32>(acc0, lane);
      transpose_reduce<32>(acc1, lane);
      s_logit[2 * my_pair][my_group * 32 + lane] = bf16_round(acc0[0]);
      s_logit[2 * my_pair + 1][my_group * 32 + lane] = bf16_round(acc1[0]);
    }
    __syncthreads();
    if (warp < 2 * PAIRS && it0 + warp < tok_end) {
      float logit[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) logit[g] = s_logit[warp][g * 32 + lane];
      route_token<32, NG>(logit, it0 + warp, lane, true, E, top_k, opts, bias, logits_out, topk_w, topk_idx, lse_out, mass,
                          cnt, zsum);
    }
    __syncthreads();
  }
  block_statistics<NG>(s_mass, s_cnt, s_z, mass, cnt, zsum, E, block_hist, block_mass, block_z);
}

// Scoring / top-k / statistics from logits that a GEMM already wrote (bf16 [N, E]): one warp per token, lane holds
// experts g * 32 + lane. Used when the gate GEMM runs on the tensor cores (many experts), where a CUDA-core dot
// product per (token, expert) would dominate the routing time.
template <int NG>
__global__ void __launch_bounds__(ROUTE_THREADS)
route_from_logits(const bf16* __restrict__ logits, const float* __restrict__ bias, long long N, int E, int top_k,
                  RouteOpts opts, int tokens_per_block, float* __restrict__ topk_w, int32_t* __restrict__ topk_idx,
                  float* __restrict__ lse_out, int32_t* __restrict__ block_hist, float* __restrict__ block_mass,
                  float* __restrict__ block_z, int32_t* __restrict__ src, long long rows_cap) {
  __shared__ float s_mass[ROUTE_WARPS][NG * 32];
  __shared__ int s_cnt[ROUTE_WARPS][NG * 32];
  __shared__ float s_z[ROUTE_WARPS];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const long long tok_begin = static_cast<long long>(blockIdx.x) * tokens_per_block;
  long long tok_end = tok_begin + tokens_per_block;
  if (tok_end > N) tok_end = N;
  fill_src(src, rows_cap);
  float mass[NG];
  int cnt[NG];
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    mass[g] = 0.0f;
    cnt[g] = 0;
  }
  float zsum = 0.0f;
  for (long long n = tok_begin + warp; n < tok_end; n += ROUTE_WARPS) {
    float logit[NG];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const int e = g * 32 + lane;
      logit[g] = (e < E) ? __bfloat162float(logits[n * E + e]) : 0.0f;
    }
    route_token<32, NG>(logit, n, lane, true, E, top_k, opts, bias, nullptr, topk_w, topk_idx, lse_out, mass, cnt, zsum);
  }
  block_statistics<NG>(s_mass, s_cnt, s_z, mass, cnt, zsum, E, block_hist, block_mass, block_z);
}

// Histogram of given expert ids with the same block chunking (expert-parallel receive side).
__global__ void __launch_bounds__(ROUTE_THREADS)
route_hist_ids(const int32_t* __restrict__ ids, long long T, int E, int slots_per_block,
               int32_t* __restrict__ block_hist, int32_t* __restrict__ status) {
  __shared__ int s_cnt[MAX_E];
  for (int e = threadIdx.x; e < E; e += ROUTE_THREADS) s_cnt[e] = 0;
  __syncthreads();
  const long long begin = static_cast<long long>(blockIdx.x) * slots_per_block;
  long long end = begin + slots_per_block;
  if (end > T) end = T;
  for (long long i = begin + threadIdx.x; i < end; i += ROUTE_THREADS) {
    const int e = ids[i];
    if (e >= 0 && e < E) {
      atomicAdd(&s_cnt[e], 1);
    } else {
      atomicCAS(status, 0, FFM_STATUS_BAD_INDEX);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += ROUTE_THREADS) block_hist[static_cast<long long>(e) * gridDim.x + blockIdx.x] = s_cnt[e];
}

// Segment starts (in 128-row tiles, always even) and the dot product of counts and probability masses, from per-expert
// totals in shared memory. One warp, eight consecutive experts per lane: a fixed order of sums.
__device__ __forceinline__ void finish_counts(const int* s_counts, const float* s_mass, float zsum, int E, int lane,
                                              int32_t* __restrict__ tile_start, float* __restrict__ stats,
                                              const LossOut& lo) {
  constexpr int PER = MAX_E / 32;
  int tiles[PER];
  int mine = 0;
  float dot = 0.0f;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane * PER + i;
    const int c = e < E ? s_counts[e] : 0;
    tiles[i] = ((c + 255) >> 8) << 1;  // segments start on multiples of 256 rows
    mine += tiles[i];
    if (e < E) dot += static_cast<float>(c) * s_mass[e];
  }
  int incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  int run = incl - mine;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane * PER + i;
    if (e < E) tile_start[e] = run;
    run += tiles[i];
    if (e + 1 == E) tile_start[E] = run;
  }
  dot = warp_sum(dot);
  if (lane == 0 && stats != nullptr) {
    stats[E] = zsum;
    stats[E + 1] = dot;
  }
  if (lane == 0) {
    if (lo.aux != nullptr) *lo.aux = dot * lo.aux_scale;
    if (lo.z != nullptr) *lo.z = zsum * lo.z_scale;
    if (lo.zero != nullptr) *lo.zero = 0;
  }
}

// One block of 32 warps. block_off[e][b] = sum_{b' < b} hist[e][b']; counts; tile_start; stats.
// One warp per expert, the lanes sweep its block histograms 32 at a time: the histograms are stored expert-major, so a
// sweep reads one 128-byte line (block-major, each lane touched its own line: with eight warps the kernel took 73 us at
// 512 blocks x 64 experts and 49 us at 64 x 256; now 15 us and, on the path for few tokens, part of route_finish_small). All
// sums keep a fixed order.
constexpr int SCAN_THREADS = 1024;
__global__ void __launch_bounds__(SCAN_THREADS)
route_scan(const int32_t* __restrict__ block_hist, const float* __restrict__ block_mass,
           const float* __restrict__ block_z, int blocks, int E, int32_t* __restrict__ block_off,
           int32_t* __restrict__ counts, int32_t* __restrict__ tile_start, float* __restrict__ stats, LossOut lo) {
  __shared__ int s_counts[MAX_E];
  __shared__ float s_mass[MAX_E];
  __shared__ float s_zsum;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  for (int e = warp; e < E; e += SCAN_THREADS / 32) {
    const long long row = static_cast<long long>(e) * blocks;
    int carry = 0;
    float m = 0.0f;
#pragma unroll 4
    for (int b0 = 0; b0 < blocks; b0 += 32) {
      const int b = b0 + lane;
      const int v = (b < blocks) ? block_hist[row + b] : 0;
      if (block_mass != nullptr && b < blocks) m += block_mass[row + b];
      int x = v;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += t;
      }
      if (b < blocks) block_off[row + b] = carry + x - v;
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
    m = warp_sum(m);
    if (lane == 0) {
      s_counts[e] = carry;
      s_mass[e] = m;
      counts[e] = carry;
      if (stats != nullptr) stats[e] = m;
    }
  }
  if (warp == SCAN_THREADS / 32 - 1) {
    float z = 0.0f;
    if (block_z != nullptr) {
      for (int b = lane; b < blocks; b += 32) z += block_z[b];
    }
    z = warp_sum(z);
    if (lane == 0) s_zsum = z;
  }
  __syncthreads();
  if (warp == 0) finish_counts(s_counts, s_mass, s_zsum, E, lane, tile_start, stats, lo);
}

// Stable rank inside each expert segment. Each warp owns a contiguous run of the block's slots.
__global__ void __launch_bounds__(ROUTE_THREADS)
route_rank(const int32_t* __restrict__ ids, long long T, int E, int slots_per_block,
           const int32_t* __restrict__ block_off, const int32_t* __restrict__ tile_start, long long rows_cap,
           int32_t* __restrict__ pos, int32_t* __restrict__ src, int32_t* __restrict__ status) {
  __shared__ int s_run[ROUTE_WARPS][MAX_E];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const long long begin = static_cast<long long>(blockIdx.x) * slots_per_block;
  long long end = begin + slots_per_block;
  if (end > T) end = T;
  const long long span = end > begin ? end - begin : 0;
  const long long per_warp = ((span + ROUTE_WARPS - 1) / ROUTE_WARPS + 31) / 32 * 32;
  const long long wb = begin + warp * per_warp;
  long long we = wb + per_warp;
  if (we > end) we = end;

  for (int e = lane; e < E; e += 32) s_run[warp][e] = 0;
  __syncwarp();
  // pass 1: per-warp counts
  for (long long i = wb + lane; i < we; i += 32) {
    const int e = ids[i];
    if (e >= 0 && e < E) atomicAdd(&s_run[warp][e], 1);
  }
  __syncthreads();
  // exclusive scan over warps, per expert, plus the block and segment bases
  for (int e = threadIdx.x; e < E; e += ROUTE_THREADS) {
    int run = tile_start[e] * 128 + block_off[static_cast<long long>(e) * gridDim.x + blockIdx.x];
    for (int w = 0; w < ROUTE_WARPS; ++w) {
      const int c = s_run[w][e];
      s_run[w][e] = run;
      run += c;
    }
  }
  __syncthreads();
  // pass 2: walk the run in order, 32 slots at a time
  for (long long i0 = wb; i0 < we; i0 += 32) {
    const long long i = i0 + lane;
    const bool active = i < we;
    int e = active ? ids[i] : -1;
    if (e < 0 || e >= E) e = -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const int leader = __ffs(same) - 1;
    const int rank = __popc(same & ((1u << lane) - 1u));
    int base = 0;
    if (e >= 0 && lane == leader) {
      base = s_run[warp][e];
      s_run[warp][e] = base + __popc(same);
    }
    base = __shfl_sync(0xffffffffu, base, leader);
    __syncwarp();
    if (active) {
      const long long r = static_cast<long long>(base) + rank;
      const bool placed = e >= 0 && r < rows_cap;
      pos[i] = placed ? static_cast<int32_t>(r) : -1;
      if (placed) {
        src[r] = static_cast<int32_t>(i);
      } else {
        atomicCAS(status, 0, FFM_STATUS_BAD_INDEX);
      }
    }
  }
}

// ---- few tokens (decode) -----------------------------------------------------------------------
// With a handful of tokens the kernels above leave the chip idle: one warp walks the whole row of a token pair (72 us
// at 7 tokens, D = 4096, E = 8), or one CTA pair walks the whole contraction of the tensor-core gate GEMM (46 us at 128
// tokens, D = 7168, E = 256), and scan and rank are two more launches. Here the gate product is spread over (token
// group x expert group) blocks whose eight warps split D, and one cluster does the rest.
constexpr int SMALL_TOKENS = 256;   // most tokens of this path
constexpr int SMALL_SLOTS = 4096;   // most routed slots (one block ranks them all)
constexpr int SMALL_TG = 4;         // tokens per gate block
constexpr int SMALL_EG = 8;         // experts per gate block
constexpr int FINISH_THREADS = 512;
constexpr int FINISH_WARPS = FINISH_THREADS / 32;
constexpr int FINISH_CLUSTER = 8;

// logits[n, e] = bf16(hidden[n, :] . gate_w[e, :]) in fp32, SMALL_EG experts x SMALL_TG tokens per block; also
// src[:] = -1. Sixteen experts per block read fewer bytes from L2 but take 165 registers, one block per SM, and leave
// the load latency exposed (42 us at 128 tokens, E = 256, D = 7168).
__global__ void __launch_bounds__(ROUTE_THREADS, 2)
route_gate_small(const bf16* __restrict__ hidden, const bf16* __restrict__ gate_w, int N, int D, int E,
                 bf16* __restrict__ logits, int32_t* __restrict__ src, long long rows_cap) {
  constexpr int EG = SMALL_EG;
  constexpr int ACC = EG * SMALL_TG;
  __shared__ float s_part[ROUTE_WARPS][ACC];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * SMALL_TG;
  const int e0 = blockIdx.y * EG;
  const int chunks = D >> 3;
  {
    const long long nthreads = static_cast<long long>(gridDim.x) * gridDim.y * ROUTE_THREADS;
    const long long tid = (static_cast<long long>(blockIdx.y) * gridDim.x + blockIdx.x) * ROUTE_THREADS + threadIdx.x;
    for (long long i = tid; i < rows_cap; i += nthreads) src[i] = -1;
  }
  float acc[ACC];
#pragma unroll
  for (int i = 0; i < ACC; ++i) acc[i] = 0.0f;
  for (int c = threadIdx.x; c < chunks; c += ROUTE_THREADS) {
    uint4 h[SMALL_TG];
#pragma unroll
    for (int t = 0; t < SMALL_TG; ++t) {
      const int n = min(n0 + t, N - 1);  // rows past the last token repeat it; their logits are not stored
      h[t] = __ldg(reinterpret_cast<const uint4*>(hidden + static_cast<long long>(n) * D) + c);
    }
#pragma unroll
    for (int e = 0; e < EG; ++e) {
      const int ee = min(e0 + e, E - 1);
      const uint4 w = __ldg(reinterpret_cast<const uint4*>(gate_w + static_cast<long long>(ee) * D) + c);
#pragma unroll
      for (int t = 0; t < SMALL_TG; ++t) acc[t * EG + e] = dot8(h[t], w, acc[t * EG + e]);
    }
  }
  static_assert(ACC == 32, "one total per lane");
  transpose_reduce<ACC>(acc, lane);
  s_part[warp][lane] = acc[0];
  __syncthreads();
  if (threadIdx.x < ACC) {
    const int n = n0 + threadIdx.x / EG;
    const int e = e0 + threadIdx.x % EG;
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < ROUTE_WARPS; ++w) t += s_part[w][threadIdx.x];
    if (n < N && e < E) logits[static_cast<long long>(n) * E + e] = __float2bfloat16_rn(t);
  }
}

// Scoring, top-k and statistics of every token (one warp each, spread over the cluster), then counts, segment starts
// and the stable rank of every slot in block 0. Launched as one cluster of gridDim.x blocks.
template <int NG>
__global__ void __launch_bounds__(FINISH_THREADS)
route_finish_small(const bf16* __restrict__ logits, const float* __restrict__ bias, int N, int E, int top_k,
                   RouteOpts opts, float* __restrict__ topk_w, int32_t* topk_idx, float* __restrict__ lse_out,
                   int32_t* block_hist, float* block_mass, float* block_z, int32_t* __restrict__ counts,
                   int32_t* __restrict__ tile_start, float* __restrict__ stats, long long rows_cap,
                   int32_t* __restrict__ pos, int32_t* __restrict__ src, int32_t* __restrict__ status, LossOut lo) {
  __shared__ float s_mass[FINISH_WARPS][NG * 32];
  __shared__ int s_cnt[FINISH_WARPS][NG * 32];
  __shared__ float s_z[FINISH_WARPS];
  __shared__ int s_counts[MAX_E];
  __shared__ float s_tot[MAX_E];
  __shared__ int s_start[MAX_E + 1];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int blocks = gridDim.x;
  const int per_block = (N + blocks - 1) / blocks;
  const int begin = blockIdx.x * per_block;
  const int end = min(begin + per_block, N);
  float mass[NG];
  int cnt[NG];
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    mass[g] = 0.0f;
    cnt[g] = 0;
  }
  float zsum = 0.0f;
  for (int n = begin + warp; n < end; n += FINISH_WARPS) {
    float logit[NG];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const int e = g * 32 + lane;
      logit[g] = (e < E) ? __bfloat162float(logits[static_cast<long long>(n) * E + e]) : 0.0f;
    }
    route_token<32, NG>(logit, n, lane, true, E, top_k, opts, bias, nullptr, topk_w, topk_idx, lse_out, mass, cnt, zsum);
  }
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    s_mass[warp][g * 32 + lane] = mass[g];
    s_cnt[warp][g * 32 + lane] = cnt[g];
  }
  if (lane == 0) s_z[warp] = zsum;
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += FINISH_THREADS) {
    float m = 0.0f;
    int c = 0;
    for (int w = 0; w < FINISH_WARPS; ++w) {
      m += s_mass[w][e];
      c += s_cnt[w][e];
    }
    block_mass[static_cast<long long>(e) * blocks + blockIdx.x] = m;
    block_hist[static_cast<long long>(e) * blocks + blockIdx.x] = c;
  }
  if (threadIdx.x == 0) {
    float z = 0.0f;
    for (int w = 0; w < FINISH_WARPS; ++w) z += s_z[w];
    block_z[blockIdx.x] = z;
  }
  // what the other blocks of the cluster wrote (ids, statistics) is visible to block 0 after this barrier
  __threadfence();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (blockIdx.x != 0) return;
  for (int e = threadIdx.x; e < E; e += FINISH_THREADS) {
    float m = 0.0f;
    int c = 0;
    for (int b = 0; b < blocks; ++b) {
      m += __ldcg(block_mass + static_cast<long long>(e) * blocks + b);
      c += __ldcg(block_hist + static_cast<long long>(e) * blocks + b);
    }
    s_counts[e] = c;
    s_tot[e] = m;
    counts[e] = c;
    stats[e] = m;
  }
  for (int i = threadIdx.x; i < FINISH_WARPS * NG * 32; i += FINISH_THREADS) (&s_cnt[0][0])[i] = 0;
  __syncthreads();
  if (warp == 0) {
    float z = 0.0f;
    for (int b = 0; b < blocks; ++b) z += __ldcg(block_z + b);
    finish_counts(s_counts, s_tot, z, E, lane, s_start, stats, lo);
  }
  // per-warp runs of slots, as in route_rank
  const int T = N * top_k;
  const int per_warp = ((T + FINISH_WARPS - 1) / FINISH_WARPS + 31) / 32 * 32;
  const int wb = warp * per_warp;
  const int we = min(wb + per_warp, T);
  for (int i = wb + lane; i < we; i += 32) {
    const int e = __ldcg(topk_idx + i);
    if (e >= 0 && e < E) atomicAdd(&s_cnt[warp][e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e <= E; e += FINISH_THREADS) {
    tile_start[e] = s_start[e];
    if (e < E) {
      int run = s_start[e] * 128;
      for (int w = 0; w < FINISH_WARPS; ++w) {
        const int c = s_cnt[w][e];
        s_cnt[w][e] = run;
        run += c;
      }
    }
  }
  __syncthreads();
  for (int i0 = wb; i0 < we; i0 += 32) {
    const int i = i0 + lane;
    const bool active = i < we;
    int e = active ? __ldcg(topk_idx + i) : -1;
    if (e < 0 || e >= E) e = -1;
    const unsigned same = __match_any_sync(0xffffffffu, e);
    const int leader = __ffs(same) - 1;
    const int rank = __popc(same & ((1u << lane) - 1u));
    int base = 0;
    if (e >= 0 && lane == leader) {
      base = s_cnt[warp][e];
      s_cnt[warp][e] = base + __popc(same);
    }
    base = __shfl_sync(0xffffffffu, base, leader);
    __syncwarp();
    if (active) {
      const int r = base + rank;
      const bool placed = e >= 0 && r < rows_cap;
      pos[i] = placed ? r : -1;
      if (placed) {
        src[r] = i;
      } else {
        atomicCAS(status, 0, FFM_STATUS_BAD_INDEX);
      }
    }
  }
}

struct RouteWorkspace {
  int32_t* block_hist;
  int32_t* block_off;
  float* block_mass;
  float* block_z;
  size_t bytes;
};

RouteWorkspace carve_workspace(void* base, int blocks, int E) {
  RouteWorkspace w;
  size_t off = 0;
  auto take = [&](size_t n) {
    size_t o = off;
    off += (n + 255) / 256 * 256;
    return o;
  };
  const size_t per = static_cast<size_t>(blocks) * E * 4;
  size_t o_hist = take(per), o_off = take(per), o_mass = take(per), o_z = take(static_cast<size_t>(blocks) * 4);
  uint8_t* b = static_cast<uint8_t*>(base);
  w.block_hist = reinterpret_cast<int32_t*>(b + o_hist);
  w.block_off = reinterpret_cast<int32_t*>(b + o_off);
  w.block_mass = reinterpret_cast<float*>(b + o_mass);
  w.block_z = reinterpret_cast<float*>(b + o_z);
  w.bytes = off;
  return w;
}

template <int NG>
int launch_finish_small(const bf16* logits, const float* bias, int N, int E, int top_k, const RouteOpts& opts,
                        float* topk_w, int32_t* topk_idx, float* lse, const RouteWorkspace& w, int32_t* counts,
                        int32_t* tile_start, float* stats, long long rows_cap, int32_t* pos, int32_t* src,
                        int32_t* status, const LossOut& lo, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  // up to one token per warp, a single block is enough; beyond, the tokens are spread over a cluster
  cfg.gridDim = dim3(N <= FINISH_WARPS ? 1 : FINISH_CLUSTER, 1, 1);
  cfg.blockDim = dim3(FINISH_THREADS, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cfg.gridDim.x;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, route_finish_small<NG>, logits, bias, N, E, top_k, opts, topk_w, topk_idx, lse,
                         w.block_hist, w.block_mass, w.block_z, counts, tile_start, stats, rows_cap, pos, src,
                         status, lo) != cudaSuccess) {
    cudaGetLastError();
    return FFM_ERR_LAUNCH;
  }
  return FFM_OK;
}

// Expert capacity: a routed slot whose rank inside its expert segment is >= capacity is dropped. One thread
// per token: dropped slots get weight 0 and their grouped row becomes a padding row (src = -1, so every later
// kernel sees zeros there); the kept weights are renormalised by their sum, or left at zero when nothing is kept.
__global__ void __launch_bounds__(ROUTE_THREADS)
route_capacity_kernel(float* __restrict__ topk_w, const int32_t* __restrict__ topk_idx, const int32_t* __restrict__ pos,
                      int32_t* __restrict__ src, const int32_t* __restrict__ tile_start, long long N, int top_k, int E,
                      int capacity, int32_t* __restrict__ dropped) {
  const long long n = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (n >= N) return;
  float sum = 0.0f;
  int ndrop = 0;
  for (int j = 0; j < top_k; ++j) {
    const long long i = n * top_k + j;
    const int e = topk_idx[i];
    if (e < 0 || e >= E) continue;
    const int r = pos[i] - tile_start[e] * 128;
    float w = topk_w[i];
    if (r >= capacity) {
      w = 0.0f;
      src[pos[i]] = -1;
      ++ndrop;
    }
    topk_w[i] = w;
    sum += w;
  }
  const float denom = sum + (sum > 0.0f ? 0.0f : 1.0f);
  for (int j = 0; j < top_k; ++j) topk_w[n * top_k + j] /= denom;
  if (ndrop > 0) atomicAdd(dropped, ndrop);
}

// ---- scratch for the allocation-free entry point ---------------------------------------------
// Lives in the library image: every GPU that loads libffmoe holds these bytes until the process exits.
// Sized for the stated maximum of ffm_group_rows_static: 592 blocks x 256 experts x 4 bytes, twice.
static __device__ __align__(256) unsigned char g_static_scratch[FFM_STATIC_SCRATCH_BYTES];

// Device address of g_static_scratch on the current device. In host code the array's name is only a
// stand-in for the symbol, not a pointer a kernel could use, so the address is asked for once per device
// (with that device current) and remembered.
int static_scratch_address(void** out) {
  static std::atomic<void*> cached[64];  // (zero-initialised; host threads may race here: same value either way)
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return FFM_ERR_LAUNCH;
  }
  void* p = cached[dev].load(std::memory_order_acquire);
  if (p == nullptr) {
    if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || p == nullptr) {
      cudaGetLastError();
      return FFM_ERR_LAUNCH;
    }
    cached[dev].store(p, std::memory_order_release);
  }
  *out = p;
  return FFM_OK;
}

}  // namespace

}  // namespace ffm

using namespace ffm;

// Few tokens: two launches. Whole routing, replayed, in us with two launches / with the kernels for many tokens: E = 256,
// D = 7168: 33 / 64 at 64 tokens, 47 / 68 at 128, 61 / 72 at 192, 66 / 72 at 224, 74 / 72 at 256; E = 256, D = 2048: 35 / 45 at
// 128, 51 / 49 at 256; E = 128, D = 7168: 49 / 61 at 256; E = 64, D = 2048: 27 / 31 at 256; E = 8, D = 1024: 16 / 16 at 256, D =
// 4096 18 / 20. So the line at 256 tokens is on the slower side, by 3 %, only at its very end with 256 experts; what grows
// beyond it is the gate product on CUDA cores, N E D multiply-adds.
static bool route_few_tokens(int64_t N, int top_k, bool has_logits) {
  return N > 0 && N <= SMALL_TOKENS && N * top_k <= SMALL_SLOTS && has_logits;
}

// Many experts: gate GEMM on the tensor cores (dense tcgen05 GEMM, fp32 accumulate, bf16 logits), then one
// scoring kernel. Few experts: everything in one warp-level kernel.
// (E = 32 included: one warp owning 32 experts keeps 64 accumulators per lane and ran at 0.12 TB/s)
static bool route_tensor_gate(int D, int E, bool has_logits) {
  return E >= 32 && D % 64 == 0 && E % 32 == 0 && has_logits;
}

extern "C" int ffm_route_forward_launches(int64_t N, int D, int E, int top_k, int has_logits) {
  if (route_few_tokens(N, top_k, has_logits != 0)) return 2;
  return N > 0 && route_tensor_gate(D, E, has_logits != 0) ? 4 : 3;
}

extern "C" int64_t ffm_rows_capacity(int64_t T, int E) {
  if (T < 0 || E < 1) return 0;
  return ((T + 255LL * E) / 256) * 256;
}

extern "C" size_t ffm_route_workspace_bytes(int64_t N, int E, int top_k) {
  (void)top_k;
  if (N < 0 || E < 1) return 0;
  // The same workspace serves ffm_group_rows over N * top_k slots, whose grid is never larger.
  RouteGrid g = route_grid(N > 0 ? N : 1, route_granule(E));
  RouteGrid g2 = route_grid(N > 0 ? N * (top_k > 0 ? top_k : 1) : 1);
  int blocks = g.blocks > g2.blocks ? g.blocks : g2.blocks;
  if (blocks < FINISH_CLUSTER) blocks = FINISH_CLUSTER;
  return carve_workspace(nullptr, blocks, E).bytes;
}

int ffm::route_forward_losses(const void* hidden, const void* gate_w, const float* expert_bias, int64_t N, int D, int E,
                              int top_k, int gating, float weight_scale, int pre_softmax, int n_group, int topk_group,
                              void* logits, float* topk_w, int32_t* topk_idx, float* lse, int32_t* counts,
                              int32_t* tile_start, int32_t* pos, int32_t* src, int64_t rows_cap, float* stats,
                              float* aux, float aux_scale, float* z, float z_scale, int32_t* zero, void* workspace,
                              size_t workspace_bytes, int32_t* status, ffm_stream_t stream) {
  const LossOut lo = {aux, z, zero, aux_scale, z_scale};
  if (!hidden || !gate_w || !topk_w || !topk_idx || !lse || !counts || !tile_start || !pos || !src || !stats ||
      !workspace || !status)
    return FFM_ERR_BAD_ARG;
  if (N < 0 || D <= 0 || E < 1 || top_k < 1) return FFM_ERR_BAD_ARG;
  if (gating != FFM_GATING_SOFTMAX && gating != FFM_GATING_SIGMOID) return FFM_ERR_BAD_ARG;
  if (D % 8 != 0 || E > MAX_E || top_k > E || top_k > 32) return FFM_ERR_UNSUPPORTED;
  if (n_group < 0 || (n_group > 0 && (topk_group < 1 || topk_group > n_group))) return FFM_ERR_BAD_ARG;
  if (n_group > 32 || (n_group > 0 && E % n_group != 0)) return FFM_ERR_UNSUPPORTED;
  if (n_group > 0 && topk_group * (E / n_group) < top_k) return FFM_ERR_BAD_ARG;  // the kept groups hold fewer experts
  if (rows_cap < ffm_rows_capacity(N * top_k, E)) return FFM_ERR_BAD_ARG;
  RouteOpts opts;
  opts.gating = gating;
  opts.weight_scale = weight_scale;
  opts.pre_softmax = (gating == FFM_GATING_SOFTMAX && pre_softmax) ? 1 : 0;
  opts.n_group = n_group;
  opts.topk_group = topk_group;
  if (workspace_bytes < ffm_route_workspace_bytes(N, E, top_k)) return FFM_ERR_WORKSPACE;
  if (N > 0 && off_16_bytes(hidden, gate_w)) return FFM_ERR_UNSUPPORTED;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bf16* h = static_cast<const bf16*>(hidden);
  const bf16* gw = static_cast<const bf16*>(gate_w);
  bf16* lg = static_cast<bf16*>(logits);
  if (route_few_tokens(N, top_k, lg != nullptr)) {
    const RouteWorkspace w = carve_workspace(workspace, FINISH_CLUSTER, E);
    const int n = static_cast<int>(N);
    const dim3 grid((n + SMALL_TG - 1) / SMALL_TG, (E + SMALL_EG - 1) / SMALL_EG, 1);
    route_gate_small<<<grid, ROUTE_THREADS, 0, s>>>(h, gw, n, D, E, lg, src, rows_cap);
    if (cudaGetLastError() != cudaSuccess) return FFM_ERR_LAUNCH;
#define FFM_FINISH_CASE(NG)                                                                                            \
  launch_finish_small<NG>(lg, expert_bias, n, E, top_k, opts, topk_w, topk_idx, lse, w, counts, tile_start, stats, \
                          rows_cap, pos, src, status, lo, s)
    if (E <= 32) return FFM_FINISH_CASE(1);
    if (E <= 64) return FFM_FINISH_CASE(2);
    if (E <= 128) return FFM_FINISH_CASE(4);
    return FFM_FINISH_CASE(8);
#undef FFM_FINISH_CASE
  }
  const bool tensor_gate = route_tensor_gate(D, E, lg != nullptr);
  const RouteGrid g = route_grid(N > 0 ? N : 1, tensor_gate || E > 32 ? route_granule(E) : 32 / gate_slices(D));
  RouteWorkspace w = carve_workspace(workspace, g.blocks, E);
  if (tensor_gate) {
    const int rc = ffm_grouped_gemm(hidden, gate_w, FFM_B_KMAJOR, 1, nullptr, N, D, E, 1.0f, logits, nullptr, 0, status,
                                    stream);
    if (rc != FFM_OK) return rc;
#define FFM_LOGIT_CASE(NG)                                                                                      \
  route_from_logits<NG><<<g.blocks, ROUTE_THREADS, 0, s>>>(lg, expert_bias, N, E, top_k, opts, g.tokens_per_block, \
                                                           topk_w, topk_idx, lse, w.block_hist, w.block_mass, w.block_z,  \
                                                           src, rows_cap)
    if (E <= 64) {
      FFM_LOGIT_CASE(2);
    } else if (E <= 128) {
      FFM_LOGIT_CASE(4);
    } else {
      FFM_LOGIT_CASE(8);
    }
#undef FFM_LOGIT_CASE
  } else {
#define FFM_ROUTE_CASE(NG)                                                                                          \
  route_gate_topk_many<NG><<<g.blocks, ROUTE_THREADS, 0, s>>>(h, gw, expert_bias, N, D, E, top_k, opts,             \
                                                              g.tokens_per_block, lg, topk_w, topk_idx, lse,       \
                                                              w.block_hist, w.block_mass, w.block_z, src, rows_cap)
    if (E <= 32) {
#define FFM_GATE_CASE(W)                                                                                              \
  FFM_PREFER_MAX_SHARED(route_gate_topk<W>);                                                                          \
  route_gate_topk<W><<<g.blocks, ROUTE_THREADS, 0, s>>>(h, gw, expert_bias, N, D, E, top_k, opts, g.tokens_per_block, \
                                                        gate_slices(D), lg, topk_w, topk_idx, lse, w.block_hist,     \
                                                        w.block_mass, w.block_z, src, rows_cap)
      if (E <= 8) {
        FFM_GATE_CASE(8);
      } else if (E <= 16) {
        FFM_GATE_CASE(16);
      } else {
        FFM_GATE_CASE(32);
      }
#undef FFM_GATE_CASE
    } else if (E <= 64) {
      FFM_ROUTE_CASE(2);
    } else if (E <= 128) {
      FFM_ROUTE_CASE(4);
    } else {
      FFM_ROUTE_CASE(8);
    }
#undef FFM_ROUTE_CASE
  }
  FFM_PREFER_MAX_SHARED(route_scan);
  route_scan<<<1, SCAN_THREADS, 0, s>>>(w.block_hist, w.block_mass, w.block_z, g.blocks, E, w.block_off, counts,
                                         tile_start, stats, lo);
  route_rank<<<g.blocks, ROUTE_THREADS, 0, s>>>(topk_idx, N * top_k, E, g.tokens_per_block * top_k, w.block_off,
                                                tile_start, rows_cap, pos, src, status);
  return cudaGetLastError() == cudaSuccess ? FFM_OK : FFM_ERR_LAUNCH;
}

extern "C" int ffm_route_forward(const void* hidden, const void* gate_w, const float* expert_bias, int64_t N, int D,
                                 int E, int top_k, int gating, float weight_scale, int pre_softmax, int n_group,
                                 int topk_group, void* logits, float* topk_w,
                                 int32_t* topk_idx, float* lse, int32_t* counts, int32_t* tile_start, int32_t* pos,
                                 int32_t* src, int64_t rows_cap, float* stats, void* workspace,
                                 size_t workspace_bytes, int32_t* status, ffm_stream_t stream) {
  return ffm::route_forward_losses(hidden, gate_w, expert_bias, N, D, E, top_k, gating, weight_scale, pre_softmax, n_group,
                                   topk_group, logits, topk_w, topk_idx, lse, counts, tile_start, pos, src, rows_cap,
                                   stats, nullptr, 0.0f, nullptr, 0.0f, nullptr, workspace, workspace_bytes, status,
                                   stream);
}

extern "C" int ffm_group_rows(const int32_t* expert_ids, int64_t T, int E, int32_t* counts, int32_t* tile_start,
                              int32_t* pos, int32_t* src, int64_t rows_cap, void* workspace, size_t workspace_bytes,
                              int32_t* status, ffm_stream_t stream) {
  if (!expert_ids || !counts || !tile_start || !pos || !src || !workspace || !status) return FFM_ERR_BAD_ARG;
  if (T < 0 || E < 1) return FFM_ERR_BAD_ARG;
  if (E > MAX_E) return FFM_ERR_UNSUPPORTED;
  if (rows_cap < ffm_rows_capacity(T, E)) return FFM_ERR_BAD_ARG;
  const RouteGrid g = route_grid(T > 0 ? T : 1);
  if (workspace_bytes < carve_workspace(nullptr, g.blocks, E).bytes) return FFM_ERR_WORKSPACE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(src, 0xFF, static_cast<size_t>(rows_cap) * 4, s) != cudaSuccess) return FFM_ERR_LAUNCH;
  RouteWorkspace w = carve_workspace(workspace, g.blocks, E);
  route_hist_ids<<<g.blocks, ROUTE_THREADS, 0, s>>>(expert_ids, T, E, g.tokens_per_block, w.block_hist, status);
  route_scan<<<1, SCAN_THREADS, 0, s>>>(w.block_hist, nullptr, nullptr, g.blocks, E, w.block_off, counts, tile_start,
                                         nullptr, LossOut{});
  route_rank<<<g.blocks, ROUTE_THREADS, 0, s>>>(expert_ids, T, E, g.tokens_per_block, w.block_off, tile_start,
                                                rows_cap, pos, src, status);
  return cudaGetLastError() == cudaSuccess ? FFM_OK : FFM_ERR_LAUNCH;
}

extern "C" int ffm_group_rows_static(const int32_t* expert_ids, int64_t T, int E, int32_t* counts,
                                     int32_t* tile_start, int32_t* pos, int32_t* src, int64_t rows_cap,
                                     int32_t* status, ffm_stream_t stream) {
  if (!expert_ids || !counts || !tile_start || !pos || !src || !status) return FFM_ERR_BAD_ARG;
  if (T < 0 || E < 1) return FFM_ERR_BAD_ARG;
  if (E > FFM_STATIC_MAX_EXPERTS || T > FFM_STATIC_MAX_ROWS) return FFM_ERR_STATIC_LIMIT;
  if (rows_cap < ffm_rows_capacity(T, E)) return FFM_ERR_BAD_ARG;
  const RouteGrid g = route_grid(T > 0 ? T : 1);
  const size_t per = (static_cast<size_t>(g.blocks) * E * 4 + 255) / 256 * 256;
  if (2 * per > FFM_STATIC_SCRATCH_BYTES) return FFM_ERR_STATIC_LIMIT;
  void* base = nullptr;
  const int rc = static_scratch_address(&base);
  if (rc != FFM_OK) return rc;
  // Every word of the scratch that the scan and rank kernels read is written by the histogram kernel of
  // this same call, so nothing left over from an earlier call is ever consumed and no clearing is needed.
  int32_t* block_hist = reinterpret_cast<int32_t*>(base);
  int32_t* block_off = reinterpret_cast<int32_t*>(static_cast<unsigned char*>(base) + per);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(src, 0xFF, static_cast<size_t>(rows_cap) * 4, s) != cudaSuccess) return FFM_ERR_LAUNCH;
  route_hist_ids<<<g.blocks, ROUTE_THREADS, 0, s>>>(expert_ids, T, E, g.tokens_per_block, block_hist, status);
  route_scan<<<1, SCAN_THREADS, 0, s>>>(block_hist, nullptr, nullptr, g.blocks, E, block_off, counts, tile_start,
                                         nullptr, LossOut{});
  route_rank<<<g.blocks, ROUTE_THREADS, 0, s>>>(expert_ids, T, E, g.tokens_per_block, block_off, tile_start, rows_cap,
                                                pos, src, status);
  return cudaGetLastError() == cudaSuccess ? FFM_OK : FFM_ERR_LAUNCH;
}

namespace ffm {
namespace {

// Positions of the routed rows in the grouped order with the 256-row padding squeezed out (the order in which an
// expert-parallel rank sends them), and the inverse map. Every block rebuilds the per-expert shift in shared memory.
__global__ void __launch_bounds__(ROUTE_THREADS)
compact_positions_kernel(const int32_t* __restrict__ pos, const int32_t* __restrict__ topk_idx,
                         const int32_t* __restrict__ counts, const int32_t* __restrict__ tile_start, long long T, int E,
                         int32_t* __restrict__ cpos, int32_t* __restrict__ src_c) {
  __shared__ int s_shift[MAX_E];  // padded position minus compact position for rows of expert e
  __shared__ int s_rows;          // slots with a row: all T unless some have no expert
  if (threadIdx.x == 0) {
    int before = 0;
    for (int e = 0; e < E; ++e) {
      s_shift[e] = tile_start[e] * 128 - before;
      before += counts[e];
    }
    s_rows = before;
  }
  __syncthreads();
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < T) {
    const int e = topk_idx[i];
    const bool placed = e >= 0 && e < E && pos[i] >= 0;
    const int c = placed ? pos[i] - s_shift[e] : -1;
    cpos[i] = c;
    if (placed) src_c[c] = static_cast<int32_t>(i);
    if (i >= s_rows) src_c[i] = -1;
  }
}

}  // namespace
}  // namespace ffm

extern "C" int ffm_compact_positions(const int32_t* pos, const int32_t* topk_idx, const int32_t* counts,
                                     const int32_t* tile_start, int64_t T, int E, int32_t* cpos, int32_t* src_c,
                                     ffm_stream_t stream) {
  if (!pos || !topk_idx || !counts || !tile_start || !cpos || !src_c) return FFM_ERR_BAD_ARG;
  if (T < 0 || E < 1) return FFM_ERR_BAD_ARG;
  if (E > ffm::MAX_E) return FFM_ERR_UNSUPPORTED;
  if (T == 0) return FFM_OK;
  const int blocks = static_cast<int>((T + ffm::ROUTE_THREADS - 1) / ffm::ROUTE_THREADS);
  ffm::compact_positions_kernel<<<blocks, ffm::ROUTE_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      pos, topk_idx, counts, tile_start, T, E, cpos, src_c);
  return cudaGetLastError() == cudaSuccess ? FFM_OK : FFM_ERR_LAUNCH;
}

extern "C" int ffm_route_apply_capacity(float* topk_w, const int32_t* topk_idx, const int32_t* pos, int32_t* src,
                                        const int32_t* tile_start, int64_t N, int top_k, int E, int capacity,
                                        int32_t* dropped_count, ffm_stream_t stream) {
  if (!topk_w || !topk_idx || !pos || !src || !tile_start || !dropped_count) return FFM_ERR_BAD_ARG;
  if (N < 0 || top_k < 1 || E < 1 || capacity < 0) return FFM_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(dropped_count, 0, 4, s) != cudaSuccess) return FFM_ERR_LAUNCH;
  if (N == 0) return FFM_OK;
  const int blocks = static_cast<int>((N + ROUTE_THREADS - 1) / ROUTE_THREADS);
  route_capacity_kernel<<<blocks, ROUTE_THREADS, 0, s>>>(topk_w, topk_idx, pos, src, tile_start, N, top_k, E, capacity,
                                                         dropped_count);
  return cudaGetLastError() == cudaSuccess ? FFM_OK : FFM_ERR_LAUNCH;
}
