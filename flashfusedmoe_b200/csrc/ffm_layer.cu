// Launch sequence of the single-GPU layer, forward and backward (host code only).
//
// One call enqueues a whole pass: 5 to 13 launches forward, 9 to 19 backward, and the events that fork and join the side
// streams. From Python, each launch cost a ctypes call with its argument checks, an output allocation and, at a fork, stream and event objects:
// 230 us for a forward pass and 600 us for a backward pass however small, more than the GPU needed at up to a few
// thousand tokens.
//
// Every launch waits for the end of the one before it on its stream. Placed ahead of that end (programmatic stream
// serialization) a forward pass is up to 3 % faster (4096 tokens on 64 experts 663 us instead of 681). But in loops of training
// calls that filled the launch queue (3001 tokens on 16 experts) two of six runs did not come to an end, with events that other
// streams wait for between such launches. No cause was found in the kernels, and a library cannot keep events from between its
// launches: the calls release the interpreter's lock, and the allocator records events of its own.
#include <cuda_runtime.h>

#include "../../include/ffmoe.h"
#include "ffm_internal.h"

namespace ffm {

namespace {

// An event for one fork or join, created when it is first recorded. Destroying it with the record still pending is
// allowed (its resources go once it is done), also while the stream is being captured.
class Event {
 public:
  Event() = default;
  ~Event() {
    if (ok_) cudaEventDestroy(e_);
  }
  Event(const Event&) = delete;
  Event& operator=(const Event&) = delete;
  bool record(ffm_stream_t s) {
    if (!ok_) ok_ = cudaEventCreateWithFlags(&e_, cudaEventDisableTiming) == cudaSuccess;
    return ok_ && cudaEventRecord(e_, static_cast<cudaStream_t>(s)) == cudaSuccess;
  }
  bool wait(ffm_stream_t s) { return ok_ && cudaStreamWaitEvent(static_cast<cudaStream_t>(s), e_, 0) == cudaSuccess; }
  // `to` goes on after what `from` holds now
  bool order(ffm_stream_t from, ffm_stream_t to) { return record(from) && wait(to); }

 private:
  cudaEvent_t e_ = nullptr;
  bool ok_ = false;
};

// Runs launch sites: timing events around each when the caller asked for them, launch count, first error.
class Sites {
 public:
  Sites(const int64_t* timer, int64_t* launched) : timer_(timer), launched_(launched) {
    for (int i = 0; i < 3; ++i) launched_[i] = 0;
  }
  template <typename F>
  void run(int site, int kernels, ffm_stream_t stream, F&& launch) {
    if (rc_ != FFM_OK) return;
    mark(2 * site, stream);
    rc_ = launch();
    mark(2 * site + 1, stream);
    launched_[0] += kernels;
    launched_[1] |= int64_t{1} << site;
    if (rc_ != FFM_OK) launched_[2] = site;
  }
  void require(bool ok) {
    if (!ok && rc_ == FFM_OK) {
      cudaGetLastError();
      rc_ = FFM_ERR_LAUNCH;
      launched_[2] = -1;
    }
  }
  int rc() const { return rc_; }

 private:
  void mark(int i, ffm_stream_t stream) {
    if (timer_ == nullptr) return;
    cudaEventRecord(reinterpret_cast<cudaEvent_t>(timer_[i]), static_cast<cudaStream_t>(stream));
  }
  const int64_t* timer_;
  int64_t* launched_;
  int rc_ = FFM_OK;
};

// Callers pack the argument blocks by hand, eight bytes a field; tests/test_cabi_cpu.py compares the packing with the
// header's field list and with these sizes.
static_assert(sizeof(ffm_layer_forward_args) == 68 * 8, "a field was added or removed");
static_assert(sizeof(ffm_layer_backward_args) == 67 * 8, "a field was added or removed");

// Combinations of few_rows that would leave a buffer unwritten that a later launch reads: the decode GEMMs store no
// pre-activations, and the one chain, which permutes nothing, needs both of them, the shared expert inside and every
// routed row in use.
bool bad_few_rows(const ffm_layer_forward_args& a) {
  const int64_t both = FFM_FEW_DECODE_UP | FFM_FEW_DECODE_DOWN;
  const bool decode = (a.few_rows & (both | FFM_FEW_DECODE_SHARED)) != 0;
  if (a.few_rows & ~int64_t{FFM_FEW_TILES | both | FFM_FEW_DECODE_SHARED | FFM_FEW_ONE_CHAIN}) return true;
  if (decode && (a.need_grad || a.preact != nullptr || a.s_preact != nullptr)) return true;
  if ((a.few_rows & both) && a.fp8) return true;
  if (!(a.few_rows & FFM_FEW_ONE_CHAIN)) return false;
  return (a.few_rows & both) != both || a.capacity >= 0 || (a.Hs > 0 && !(a.few_rows & FFM_FEW_DECODE_SHARED));
}

}  // namespace

}  // namespace ffm

using namespace ffm;

extern "C" int64_t ffm_layer_args_bytes(int backward) {
  return backward ? sizeof(ffm_layer_backward_args) : sizeof(ffm_layer_forward_args);
}

extern "C" int ffm_layer_forward(const ffm_layer_forward_args* args) {
  if (args == nullptr || args->launched == nullptr) return FFM_ERR_BAD_ARG;
  const ffm_layer_forward_args& a = *args;
  if (bad_few_rows(a)) {
    for (int i = 0; i < 3; ++i) a.launched[i] = i == 2 ? FFM_FWD_UP : 0;
    return FFM_ERR_BAD_ARG;
  }
  const int D = static_cast<int>(a.D), E = static_cast<int>(a.E), H = static_cast<int>(a.H), k = static_cast<int>(a.top_k);
  const int Hs = static_cast<int>(a.Hs);
  const int act = static_cast<int>(a.activation);
  ffm_stream_t st = a.stream;
  ffm_stream_t sh = a.overlap ? a.shared_stream : a.stream;
  Sites sites(a.timer, a.launched);
  Event fork, shared_done;

  // shared expert: beside the routing kernels, which leave the tensor cores idle; in a decode-sized call it is one more
  // group of the expert GEMMs
  const bool one_chain = (a.few_rows & FFM_FEW_ONE_CHAIN) != 0;
  const bool shared_inside = Hs > 0 && one_chain;
  const bool shared_beside = Hs > 0 && !shared_inside;
  if (shared_beside) {
    if (sh != st) sites.require(fork.order(st, sh));
    sites.run(FFM_FWD_SHARED_UP, 1, sh, [&] {
      if (a.few_rows & FFM_FEW_DECODE_SHARED) {
        return ffm_decode_up(nullptr, nullptr, a.hidden, a.N, D, k, 0, nullptr, nullptr, 0, nullptr, 0, 0, nullptr, a.sw_gate,
                             a.sw_up, Hs, static_cast<int>(a.shared_activation), a.s_act, a.status, sh);
      }
      return ffm_grouped_gemm_glu(a.hidden, a.sw_gate, a.sw_up, Hs, 1, nullptr, a.N, D, Hs,
                                  static_cast<int>(a.shared_activation), a.s_act, a.s_preact, nullptr, 0, a.status, sh);
    });
    sites.run(FFM_FWD_SHARED_DOWN, 1, sh, [&] {
      if (a.few_rows & FFM_FEW_DECODE_SHARED) {
        return ffm_decode_down(nullptr, 0, 0, 0, nullptr, nullptr, k, nullptr, D, nullptr, a.s_act, a.N, Hs, a.sw_down,
                               a.s_out, a.status, sh);
      }
      return ffm_grouped_gemm(a.s_act, a.sw_down, FFM_B_KMAJOR, 1, nullptr, a.N, Hs, D, 1.0f, a.s_out, nullptr, 0,
                              a.status, sh);
    });
    if (sh != st) sites.require(shared_done.record(sh));
  }

  sites.run(FFM_FWD_ROUTE, ffm_route_forward_launches(a.N, D, E, k, a.logits != nullptr), st, [&] {
    return route_forward_losses(a.hidden_route, a.gate, a.expert_bias, a.N, D, E, k, static_cast<int>(a.gating),
                                static_cast<float>(a.weight_scale), static_cast<int>(a.pre_softmax),
                                static_cast<int>(a.n_group), static_cast<int>(a.topk_group), a.logits, a.topk_w,
                                a.topk_idx, a.lse, a.counts, a.tile_start, a.pos, a.src, a.rows_cap, a.stats, a.aux,
                                static_cast<float>(a.aux_scale), a.z, static_cast<float>(a.z_scale), a.dropped,
                                a.workspace, static_cast<size_t>(a.workspace_bytes), a.status, st);
  });
  if (a.capacity >= 0) {
    sites.run(FFM_FWD_CAPACITY, 1, st, [&] {
      return ffm_route_apply_capacity(a.topk_w, a.topk_idx, a.pos, a.src, a.tile_start, a.N, k, E,
                                      static_cast<int>(a.capacity), a.dropped, st);
    });
  }
  // Without a backward pass nothing sums over the padding rows, so they are not zeroed -- except with capacity dropping: a
  // dropped slot keeps its grouped row (now a padding row) with weight 0, and 0 * (whatever the GEMMs make of
  // uninitialised memory, possibly NaN) would reach the output through the combine.
  if (!one_chain) {
    sites.run(FFM_FWD_PERMUTE, 1, st, [&] {
      return ffm_permute_rows(a.hidden, a.src, a.rows_cap, k, D, a.need_grad || a.capacity >= 0 ? 1 : 0, a.Xg, st);
    });
  }
  const int32_t* valid = (a.few_rows & FFM_FEW_TILES) ? a.counts : nullptr;
  const int tile_rows = (a.few_rows & FFM_FEW_TILES) ? 128 : 0;
  if (a.fp8) {
    sites.run(FFM_FWD_QUANT_X, 1, st, [&] { return ffm_quantize_rows_e4m3(a.Xg, a.rows_cap, D, a.xq, a.x_scale, st); });
    sites.run(FFM_FWD_UP, 1, st, [&] {
      return ffm_grouped_gemm_glu_fp8(a.xq, a.x_scale, a.w_up_q, static_cast<const float*>(a.w_up_scale), E, a.tile_start,
                                      a.rows_cap, D, H, act, a.act, a.preact, 0, a.status, st);
    });
    sites.run(FFM_FWD_QUANT_ACT, 1, st, [&] { return ffm_quantize_rows_e4m3(a.act, a.rows_cap, H, a.aq, a.a_scale, st); });
    sites.run(FFM_FWD_DOWN, 1, st, [&] {
      return ffm_grouped_gemm_fp8(a.aq, a.a_scale, a.w_down_q, static_cast<const float*>(a.w_down_scale), E, a.tile_start,
                                  a.rows_cap, H, D, a.Y, 0, a.status, st);
    });
  } else {
    const void* up_rows = static_cast<const char*>(a.w_up) + a.H * a.D * 2;
    sites.run(FFM_FWD_UP, 1, st, [&] {
      if (a.few_rows & FFM_FEW_DECODE_UP) {
        return ffm_decode_up(one_chain ? a.hidden : a.Xg, one_chain ? a.src : nullptr, a.hidden, a.N, D, k, E, a.tile_start,
                             a.counts, a.rows_cap, a.w_up, H, act, a.act, a.sw_gate, a.sw_up, shared_inside ? Hs : 0,
                             static_cast<int>(a.shared_activation), a.s_act, a.status, st);
      }
      return ffm_grouped_gemm_glu(a.Xg, a.w_up, up_rows, 2 * a.H, E, a.tile_start, a.rows_cap, D, H, act, a.act, a.preact,
                                  valid, tile_rows, a.status, st);
    });
    sites.run(FFM_FWD_DOWN, 1, st, [&] {
      if (a.few_rows & FFM_FEW_DECODE_DOWN) {
        return ffm_decode_down(a.act, a.rows_cap, H, E, a.tile_start, a.counts, k, a.w_down, D, a.Y, a.s_act, a.N,
                               shared_inside ? Hs : 0, a.sw_down, a.s_out, a.status, st);
      }
      return ffm_grouped_gemm(a.act, a.w_down, FFM_B_KMAJOR, E, a.tile_start, a.rows_cap, H, D, 1.0f, a.Y, valid, tile_rows,
                              a.status, st);
    });
  }
  if (a.addend_ready != nullptr) {
    sites.require(cudaStreamWaitEvent(static_cast<cudaStream_t>(st), static_cast<cudaEvent_t>(a.addend_ready), 0) ==
                  cudaSuccess);
  }
  if (shared_beside && sh != st) sites.require(shared_done.wait(st));
  const void* add = Hs > 0 ? a.s_out : a.addend;
  sites.run(FFM_FWD_COMBINE, 1, st, [&] {
    return combine_forward_status(a.Y, a.pos, a.topk_w, add, nullptr, a.N, k, D, a.out, a.status, a.status_host, st);
  });
  return sites.rc();
}

// Two GEMMs never share an SM, so the GEMMs stay in one chain and each HBM-bound kernel is paired with a GEMM that does
// not depend on it:
//   stream:  combine backward -> dAct GEMM (GLU backward in its epilogue) -> dW_down -> dX -> un-permute (+ routing term,
//            + the shared expert's input gradient)
//   shared:  the shared expert's backward; it needs the output gradient alone, so it starts with the pass
//   small:   sum of the two partial products of the shared dW_down, which nothing waits for until the end
//   route:   routing backward (fills the gaps between GEMMs)
//   gemm:    (after dX) dW_up
extern "C" int ffm_layer_backward(const ffm_layer_backward_args* args) {
  if (args == nullptr || args->launched == nullptr) return FFM_ERR_BAD_ARG;
  const ffm_layer_backward_args& a = *args;
  const int D = static_cast<int>(a.D), E = static_cast<int>(a.E), H = static_cast<int>(a.H), k = static_cast<int>(a.top_k);
  const int Hs = static_cast<int>(a.Hs);
  const int act = static_cast<int>(a.activation), s_activation = static_cast<int>(a.shared_activation);
  const bool overlap = a.overlap != 0;
  ffm_stream_t st = a.stream;
  ffm_stream_t sh = overlap ? a.shared_stream : st;
  ffm_stream_t rt = overlap ? a.route_stream : st;
  ffm_stream_t gm = overlap ? a.gemm_stream : st;
  ffm_stream_t sm = overlap ? a.small_stream : st;
  Sites sites(a.timer, a.launched);
  Event start, sum_fork, sum_done, shared_done, rows_done, route_done, dx_done, join;

  if (a.recompute) {
    // recompute the three large tensors with the same kernels: bit-identical to the forward pass
    const void* up_rows = static_cast<const char*>(a.w_up) + a.H * a.D * 2;
    sites.run(FFM_BWD_RE_UP, 1, st, [&] {
      return ffm_grouped_gemm_glu(a.Xg, a.w_up, up_rows, 2 * a.H, E, a.tile_start, a.rows_cap, D, H, act, a.act, a.preact,
                                  nullptr, 0, a.status, st);
    });
    sites.run(FFM_BWD_RE_DOWN, 1, st, [&] {
      return ffm_grouped_gemm(a.act, a.w_down, FFM_B_KMAJOR, E, a.tile_start, a.rows_cap, H, D, 1.0f, a.Y, nullptr, 0,
                              a.status, st);
    });
  }
  if (Hs > 0 && overlap) sites.require(start.record(st));
  // first in launch order: the routed GEMMs wait for it, the shared expert's do not
  sites.run(FFM_BWD_COMBINE, 1, st, [&] {
    if (a.zero_gw && cudaMemsetAsync(a.gw, 0, static_cast<size_t>(a.N) * k * 4, static_cast<cudaStream_t>(st)) != cudaSuccess)
      return FFM_ERR_LAUNCH;
    return ffm_combine_backward(a.go, a.Y, a.topk_w, a.src, a.rows_cap, k, D, a.gYw, a.gw, st);
  });

  if (Hs > 0) {
    if (overlap) sites.require(start.wait(sh));
    const int split = static_cast<int>(a.shared_split);
    void* parts = split == 2 ? a.s_parts : a.s_d_down;
    if (a.fused_glu) {
      sites.run(FFM_BWD_S_DACT, 1, sh, [&] {
        return ffm_grouped_gemm_dact_glu_backward(a.go, a.sw_down, 1, nullptr, a.N, D, Hs, s_activation, a.s_preact, a.s_gU,
                                                  0, a.status, sh);
      });
    } else {
      sites.run(FFM_BWD_S_DACT, 1, sh, [&] {
        return ffm_grouped_gemm(a.go, a.sw_down, FFM_B_NMAJOR, 1, nullptr, a.N, D, Hs, 1.0f, a.s_d_act, nullptr, 0, a.status,
                                sh);
      });
      sites.run(FFM_BWD_S_GLU, 1, sh, [&] {
        return ffm_glu_backward(a.s_d_act, a.s_preact, nullptr, 1, a.N, Hs, s_activation, a.s_gU, sh);
      });
    }
    sites.run(FFM_BWD_S_WDOWN, 1, sh, [&] {
      return grouped_wgrad(a.go, a.s_act, split, nullptr, nullptr, a.N, D, Hs, 1.0f, parts, a.status, sh);
    });
    if (split == 2) {
      if (overlap) sites.require(sum_fork.order(sh, sm));
      const int64_t n = a.D * a.Hs;
      sites.run(FFM_BWD_S_SUM, 1, sm, [&] { return add_bf16(parts, static_cast<char*>(parts) + n * 2, n, a.s_d_down, sm); });
      if (overlap) sites.require(sum_done.record(sm));
    }
    sites.run(FFM_BWD_S_DX, 1, sh, [&] {
      return ffm_dense_gemm_two(a.s_gU, a.sw_gate, Hs, a.sw_up, a.N, 2 * Hs, D, a.s_dx, a.status, sh);
    });
    sites.run(FFM_BWD_S_WUP, 1, sh, [&] {
      return grouped_wgrad(a.s_gU, a.hidden, 1, nullptr, nullptr, a.N, 2 * Hs, D, 1.0f, a.s_d_gate_up, a.status, sh);
    });
    if (overlap) {
      if (split == 2) sites.require(sum_done.wait(sh));
      sites.require(shared_done.record(sh));
    }
  }

  LossGrads lg = {};
  lg.counts = a.counts;
  lg.grad_aux = a.grad_aux;
  lg.grad_z = a.grad_z;
  lg.aux_coef = static_cast<float>(a.aux_coef);
  lg.z_coef = static_cast<float>(a.z_coef);
  if (overlap) sites.require(rows_done.order(st, rt));
  const int route_kernels = ffm_route_backward_launches(a.N, D, E, static_cast<int>(a.gating), a.grad_aux != nullptr,
                                                        a.grad_z != nullptr, 0);
  sites.run(FFM_BWD_ROUTE, route_kernels, rt, [&] {
    return route_backward_losses(a.gw, a.topk_w, a.topk_idx, a.logits, a.lse, lg, a.hidden, a.gate, a.N, D, E, k,
                                 static_cast<int>(a.gating), 0, a.dH_route, a.d_gate, a.workspace,
                                 static_cast<size_t>(a.workspace_bytes), a.status, rt);
  });
  if (overlap) sites.require(route_done.record(rt));

  if (a.fused_glu) {
    sites.run(FFM_BWD_DACT, 1, st, [&] {
      return ffm_grouped_gemm_dact_glu_backward(a.gYw, a.w_down, E, a.tile_start, a.rows_cap, D, H, act, a.preact, a.gU, 0,
                                                a.status, st);
    });
    sites.run(FFM_BWD_WDOWN, 1, st, [&] {
      return grouped_wgrad(a.gYw, a.act, E, a.tile_start, a.counts, a.rows_cap, D, H, 1.0f, a.d_w_down, a.status, st);
    });
  } else {
    sites.run(FFM_BWD_DACT, 1, st, [&] {
      return ffm_grouped_gemm(a.gYw, a.w_down, FFM_B_NMAJOR, E, a.tile_start, a.rows_cap, D, H, 1.0f, a.d_act, nullptr, 0,
                              a.status, st);
    });
    if (overlap) {
      // the GLU backward rides on extra warps of the dW_down GEMM (one launch)
      sites.run(FFM_BWD_WDOWN, 1, st, [&] {
        return ffm_grouped_gemm_wgrad_glu_backward(a.gYw, a.act, E, a.tile_start, a.rows_cap, D, H, 1.0f, a.d_w_down, a.d_act,
                                                   a.preact, a.rows_cap, H, act, a.gU, a.status, st);
      });
    } else {
      sites.run(FFM_BWD_GLU, 1, st, [&] {
        return ffm_glu_backward(a.d_act, a.preact, a.tile_start, E, a.rows_cap, H, act, a.gU, st);
      });
      sites.run(FFM_BWD_WDOWN, 1, st, [&] {
        return grouped_wgrad(a.gYw, a.act, E, a.tile_start, a.counts, a.rows_cap, D, H, 1.0f, a.d_w_down, a.status, st);
      });
    }
  }
  sites.run(FFM_BWD_DX, 1, st, [&] {
    return ffm_grouped_gemm(a.gU, a.w_up, FFM_B_NMAJOR, E, a.tile_start, a.rows_cap, 2 * H, D, 1.0f, a.dXg, nullptr, 0,
                            a.status, st);
  });
  if (overlap) sites.require(dx_done.order(st, gm));
  sites.run(FFM_BWD_WUP, 1, gm, [&] {
    return grouped_wgrad(a.gU, a.Xg, E, a.tile_start, a.counts, a.rows_cap, 2 * H, D, 1.0f, a.d_w_up, a.status, gm);
  });
  if (overlap) {
    sites.require(join.record(gm));
    sites.require(route_done.wait(st));
    if (Hs > 0) sites.require(shared_done.wait(st));
  }
  sites.run(FFM_BWD_UNPERMUTE, 1, st, [&] {
    return ffm_combine_forward_add2(a.dXg, a.pos, nullptr, a.dH_route, Hs > 0 ? a.s_dx : nullptr, a.N, k, D, a.dH, st);
  });
  if (overlap) sites.require(join.wait(st));
  return sites.rc();
}

extern "C" int ffm_status_copy(const int32_t* status, int32_t* host, ffm_stream_t stream, ffm_stream_t side_stream,
                               void* ready, void* done) {
  if (!status || !host || !ready || !done) return FFM_ERR_BAD_ARG;
  cudaStream_t side = static_cast<cudaStream_t>(side_stream);
  const bool ok = cudaEventRecord(static_cast<cudaEvent_t>(ready), static_cast<cudaStream_t>(stream)) == cudaSuccess &&
                  cudaStreamWaitEvent(side, static_cast<cudaEvent_t>(ready), 0) == cudaSuccess &&
                  cudaMemcpyAsync(host, status, 4, cudaMemcpyDeviceToHost, side) == cudaSuccess &&
                  cudaEventRecord(static_cast<cudaEvent_t>(done), side) == cudaSuccess;
  if (!ok) cudaGetLastError();
  return ok ? FFM_OK : FFM_ERR_LAUNCH;
}
