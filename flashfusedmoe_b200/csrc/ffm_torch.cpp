// The single-GPU layer's passes for torch tensors: operand checks and casts, output and scratch allocations and the
// argument block of ffm_layer_forward / ffm_layer_backward, in one call from Python each way.
//
// From Python these cost more host time than the GPU needs for a small call: a decode step of one token (8 experts and a shared
// one) took 91 us of host time, 15 of them in the library with its five launches; now 62 to 70, while the GPU needs 31
// (replayed from a graph). See fused_moe.py for what stays there (validation, losses, the autograd function).
#include <torch/extension.h>

#include <initializer_list>
#include <optional>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/ffmoe.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

// libffmoe.so is loaded by the Python package, by path, and its functions are handed over (bind): linked by name, a second
// copy of the package in one process would get the first one's library.
decltype(&ffm_layer_forward) forward_pass = nullptr;
decltype(&ffm_layer_backward) backward_pass = nullptr;
decltype(&ffm_rows_capacity) rows_capacity = nullptr;
decltype(&ffm_route_workspace_bytes) forward_workspace = nullptr;
decltype(&ffm_route_backward_workspace_bytes) backward_workspace = nullptr;
decltype(&ffm_cast_many) cast_many = nullptr;

void bind(uintptr_t forward, uintptr_t backward, uintptr_t capacity, uintptr_t forward_ws, uintptr_t backward_ws,
          uintptr_t cast) {
  forward_pass = reinterpret_cast<decltype(forward_pass)>(forward);
  backward_pass = reinterpret_cast<decltype(backward_pass)>(backward);
  rows_capacity = reinterpret_cast<decltype(rows_capacity)>(capacity);
  forward_workspace = reinterpret_cast<decltype(forward_workspace)>(forward_ws);
  backward_workspace = reinterpret_cast<decltype(backward_workspace)>(backward_ws);
  cast_many = reinterpret_cast<decltype(cast_many)>(cast);
}

constexpr int64_t ALIGN = 256;
// Scratch buffers from this size on are allocations of their own: one block for all of them would be larger than anything
// a program frees again, so that the allocator could not serve it from what it holds.
constexpr int64_t OWN_ALLOCATION = 16 << 20;

int64_t aligned(int64_t n) { return (n + ALIGN - 1) / ALIGN * ALIGN; }

const Tensor& require(const Tensor& t, at::ScalarType dtype, const char* name) {
  if (!t.is_cuda()) {
    throw std::runtime_error(std::string(name) + " must be a CUDA tensor: flashfusedmoe_b200 has no CPU path");
  }
  if (t.scalar_type() != dtype) {
    throw py::type_error(std::string(name) + " must be " + c10::toString(dtype) + ", got " + c10::toString(t.scalar_type()));
  }
  if (!t.is_contiguous()) throw py::value_error(std::string(name) + " must be contiguous");
  return t;
}

// Conversions between fp32 and bf16, collected and run in one launch.
class Casts {
 public:
  static bool takes(const Tensor& t) {
    return t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous() && !t.is_neg() && !t._is_zerotensor() &&
           t.numel() > 0 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  }
  void add(const void* src, void* dst, int64_t elements) {
    if (count_ == FFM_CAST_MAX) throw std::logic_error("more tensors than one launch converts");
    src_[count_] = src;
    dst_[count_] = dst;
    elements_[count_++] = elements;
  }
  // kernels enqueued
  int64_t run(bool to_bf16, int64_t stream) {
    if (count_ == 0) return 0;
    const int rc = cast_many(count_, src_, dst_, elements_, to_bf16, reinterpret_cast<ffm_stream_t>(stream));
    if (rc != FFM_OK) throw std::runtime_error("libffmoe ffm_cast_many failed: " + std::to_string(rc));
    return 1;
  }

 private:
  const void* src_[FFM_CAST_MAX];
  void* dst_[FFM_CAST_MAX];
  int64_t elements_[FFM_CAST_MAX];
  int count_ = 0;
};

// t in the compute type, contiguous, with its values in memory (no negation pending); an fp32 tensor's cast may only be entered
// in `casts`
Tensor computed(const Tensor& t, const char* name, Casts* casts = nullptr) {
  if (casts != nullptr && t.scalar_type() == at::kFloat && Casts::takes(t)) {
    const Tensor c = at::empty(t.sizes(), t.options().dtype(at::kBFloat16));
    casts->add(t.data_ptr(), c.data_ptr(), t.numel());
    return c;
  }
  Tensor c = t.scalar_type() == at::kBFloat16 ? t : t.to(at::kBFloat16);
  if (!c.is_contiguous()) c = c.contiguous();
  if (c.is_neg()) c = c.resolve_neg();
  return require(c, at::kBFloat16, name);
}

Tensor computed(const OptTensor& t, const char* name, Casts* casts) {
  return t.has_value() ? computed(*t, name, casts) : Tensor();
}

template <typename T = void>
T* ptr(const Tensor& t) {
  return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr;
}

template <typename T>
T* at_address(int64_t a) {
  return reinterpret_cast<T*>(a);
}

// Device addresses of scratch buffers of the given byte sizes, 256-byte aligned (null for a size of 0). Small ones share
// one allocation. Holds the tensors.
class Scratch {
 public:
  Scratch(const at::TensorOptions& bytes, std::initializer_list<int64_t> sizes) {
    int64_t shared = 0;
    for (int64_t n : sizes) shared += n < OWN_ALLOCATION ? aligned(n) : 0;
    char* base = nullptr;
    if (shared > 0) {
      held_.push_back(at::empty({shared}, bytes));
      base = static_cast<char*>(held_.back().data_ptr());
    }
    for (int64_t n : sizes) {
      if (n <= 0) {
        where_.push_back(nullptr);
      } else if (n >= OWN_ALLOCATION) {
        held_.push_back(at::empty({n}, bytes));
        where_.push_back(static_cast<char*>(held_.back().data_ptr()));
      } else {
        where_.push_back(base);
        base += aligned(n);
      }
    }
  }
  // the buffers in the order of their sizes
  template <typename T = void>
  T* take() {
    return reinterpret_cast<T*>(where_[next_++]);
  }

 private:
  std::vector<Tensor> held_;
  std::vector<char*> where_;
  size_t next_ = 0;
};

// The routing results that the backward pass reads, in one buffer.
struct RoutingLayout {
  int64_t topk_w, topk_idx, logits, lse, tile_start, pos, src, stats, bytes;
  RoutingLayout(int64_t N, int64_t E, int64_t k, int64_t rows) {
    const int64_t T = N * k;
    int64_t end = 0;
    auto next = [&end](int64_t n) {
      const int64_t here = end;
      end += aligned(n);
      return here;
    };
    topk_w = next(T * 4);
    topk_idx = next(T * 4);
    logits = next(N * E * 2);
    lse = next(N * 4);
    tile_start = next((E + 1) * 4);
    pos = next(T * 4);
    src = next((rows > 1 ? rows : 1) * 4);
    stats = next((E + 2) * 4);
    bytes = end > ALIGN ? end : ALIGN;
  }
};

// return code, kernels enqueued, mask of the sites that ran, site of an error
py::tuple outcome(int rc, const int64_t (&launched)[3]) {
  return py::make_tuple(rc, launched[0], launched[1], launched[2]);
}

py::object handed(const Tensor& t) { return t.defined() ? py::cast(t) : py::none(); }

// (outcome, out, aux, z, counts, dropped, [what the backward pass needs, or nothing])
py::tuple layer_forward(const Tensor& hidden, const Tensor& gate, const Tensor& w_up, const Tensor& w_down,
                        const OptTensor& addend, const OptTensor& sw_gate, const OptTensor& sw_up, const OptTensor& sw_down,
                        const OptTensor& expert_bias, const OptTensor& w_up_q, const OptTensor& w_up_scale,
                        const OptTensor& w_down_q, const OptTensor& w_down_scale, int64_t top_k, int64_t gating,
                        int64_t activation, int64_t shared_activation, bool pre_softmax, int64_t n_group, int64_t topk_group,
                        int64_t capacity, bool need_grad, bool recompute, int64_t few, bool overlap, double jitter,
                        double weight_scale, double aux_scale, double z_scale, int64_t status, int64_t status_host,
                        int64_t stream, int64_t shared_stream, int64_t addend_ready, int64_t timer) {
  Casts casts;
  const Tensor h = computed(hidden, "hidden", &casts), g = computed(gate, "gate weight", &casts),
               wu = computed(w_up, "w_up", &casts), wd = computed(w_down, "w_down", &casts),
               add = computed(addend, "addend", &casts), swg = computed(sw_gate, "shared expert weight", &casts),
               swu = computed(sw_up, "shared expert weight", &casts),
               swd = computed(sw_down, "shared expert weight", &casts);
  const int64_t cast_launches = casts.run(true, stream);
  const int64_t N = h.size(0), D = h.size(1), E = g.size(0), H = wu.size(1) / 2, Hs = swg.defined() ? swg.size(0) : 0;
  const bool keep = need_grad && !recompute, fp8 = w_up_q.has_value();
  // what the router sees; the noise is drawn as the reference draws it (fused_moe.py:329-332)
  Tensor h_route = h;
  if (jitter > 0.0) h_route = h * at::empty_like(h).uniform_(1.0 - jitter, 1.0 + jitter);
  Tensor bias;
  if (expert_bias.has_value()) bias = require(expert_bias->to(at::kFloat).contiguous().resolve_neg(), at::kFloat, "expert_bias");

  const int64_t rows = rows_capacity(N * top_k, static_cast<int>(E));
  const int64_t ws_bytes = static_cast<int64_t>(forward_workspace(N, static_cast<int>(E), static_cast<int>(top_k)));
  const RoutingLayout layout(N, E, top_k, rows);
  const at::TensorOptions b16 = h.options(), i32 = b16.dtype(at::kInt), f32 = b16.dtype(at::kFloat),
                          u8 = b16.dtype(at::kByte);
  const Tensor out = at::empty({N, D}, b16), counts = at::empty({E}, i32), aux = at::empty({}, f32), z = at::empty({}, f32),
               dropped = at::empty({1}, i32);
  // Kept for the backward pass: tensors; everything else is scratch. All of it is allocated on the current stream, which
  // the side streams are forked from and joined to inside the call.
  Tensor routing, Xg, pre, act, Y, s_act, s_pre;
  if (need_grad) {
    routing = at::empty({layout.bytes}, u8);
    Xg = at::empty({rows, D}, b16);
    if (Hs > 0) {
      s_act = at::empty({N, Hs}, b16);
      s_pre = at::empty({N, 2 * Hs}, b16);
    }
  }
  if (keep) {
    pre = at::empty({rows, 2 * H}, b16);
    act = at::empty({rows, H}, b16);
    Y = at::empty({rows, D}, b16);
  }
  Scratch scratch(u8, {need_grad ? 0 : layout.bytes, need_grad ? 0 : rows * D * 2, need_grad ? 0 : N * Hs * 2,
                       keep ? 0 : rows * H * 2, keep ? 0 : rows * D * 2, Hs > 0 ? N * D * 2 : 0, ws_bytes,
                       fp8 ? rows * D : 0, fp8 ? rows * 4 : 0, fp8 ? rows * H : 0, fp8 ? rows * 4 : 0});

  int64_t launched[3] = {0, 0, 0};
  ffm_layer_forward_args a = {};
  a.N = N;
  a.D = D;
  a.E = E;
  a.top_k = top_k;
  a.H = H;
  a.Hs = Hs;
  a.rows_cap = rows;
  a.gating = gating;
  a.activation = activation;
  a.shared_activation = shared_activation;
  a.pre_softmax = pre_softmax;
  a.n_group = n_group;
  a.topk_group = topk_group;
  a.capacity = capacity;
  a.need_grad = need_grad;
  a.few_rows = few;
  a.fp8 = fp8;
  a.overlap = overlap;
  a.weight_scale = weight_scale;
  a.aux_scale = aux_scale;
  a.z_scale = z_scale;
  a.hidden = ptr(h);
  a.hidden_route = ptr(h_route);
  a.gate = ptr(g);
  a.w_up = ptr(wu);
  a.w_down = ptr(wd);
  a.expert_bias = ptr<float>(bias);
  a.addend = ptr(add);
  a.sw_gate = ptr(swg);
  a.sw_up = ptr(swu);
  a.sw_down = ptr(swd);
  if (fp8) {
    a.w_up_q = ptr(*w_up_q);
    a.w_up_scale = ptr<float>(w_up_scale.value());
    a.w_down_q = ptr(w_down_q.value());
    a.w_down_scale = ptr<float>(w_down_scale.value());
  }
  char* rt = scratch.take<char>();
  if (need_grad) rt = ptr<char>(routing);
  void* const scratch_xg = scratch.take();
  void* const scratch_sact = scratch.take();
  void* const scratch_act = scratch.take();
  void* const scratch_y = scratch.take();
  a.s_out = scratch.take();
  a.workspace = scratch.take();
  a.xq = scratch.take();
  a.x_scale = scratch.take<float>();
  a.aq = scratch.take();
  a.a_scale = scratch.take<float>();
  a.workspace_bytes = ws_bytes;
  a.topk_w = reinterpret_cast<float*>(rt + layout.topk_w);
  a.topk_idx = reinterpret_cast<int32_t*>(rt + layout.topk_idx);
  a.logits = rt + layout.logits;
  a.lse = reinterpret_cast<float*>(rt + layout.lse);
  a.counts = ptr<int32_t>(counts);
  a.tile_start = reinterpret_cast<int32_t*>(rt + layout.tile_start);
  a.pos = reinterpret_cast<int32_t*>(rt + layout.pos);
  a.src = reinterpret_cast<int32_t*>(rt + layout.src);
  a.stats = reinterpret_cast<float*>(rt + layout.stats);
  a.aux = ptr<float>(aux);
  a.z = ptr<float>(z);
  a.dropped = ptr<int32_t>(dropped);
  a.Xg = need_grad ? ptr(Xg) : scratch_xg;
  a.preact = ptr(pre);
  a.act = keep ? ptr(act) : scratch_act;
  a.Y = keep ? ptr(Y) : scratch_y;
  a.s_act = need_grad ? ptr(s_act) : scratch_sact;
  a.s_preact = ptr(s_pre);
  a.out = ptr(out);
  a.status = at_address<int32_t>(status);
  a.status_host = at_address<int32_t>(status_host);
  a.stream = at_address<void>(stream);
  a.shared_stream = at_address<void>(shared_stream);
  a.addend_ready = at_address<void>(addend_ready);
  a.timer = at_address<const int64_t>(timer);
  a.launched = launched;
  int rc;
  {
    py::gil_scoped_release released;
    rc = forward_pass(&a);
  }
  launched[0] += cast_launches;
  py::list saved;
  if (need_grad) {
    for (const Tensor& t : {h, g, wu, wd, routing, counts, Xg, pre, act, Y, s_act, s_pre, swg, swu, swd}) {
      saved.append(handed(t));
    }
  }
  return py::make_tuple(outcome(rc, launched), out, aux, z, counts, dropped, saved);
}

// (outcome, dH, d_gate, d_w_up, d_w_down, shared gate, up and down gradients or None, grad_out as computed with). Gradients
// are in the compute type; with bit i of fp32_mask set the i-th of those four, of gate and up together (4) or of down (5) is
// fp32.
py::tuple layer_backward(const OptTensor& grad_out, const OptTensor& grad_aux, const OptTensor& grad_z, const Tensor& h,
                         const Tensor& g, const Tensor& wu, const Tensor& wd, const Tensor& routing, const Tensor& counts,
                         const Tensor& Xg, const OptTensor& pre, const OptTensor& act, const OptTensor& Y,
                         const OptTensor& s_act, const OptTensor& s_pre, const OptTensor& swg, const OptTensor& swu,
                         const OptTensor& swd, int64_t top_k, int64_t gating, int64_t activation, int64_t shared_activation,
                         bool capacity, bool fused, bool overlap, double aux_coef, double z_coef, int64_t status,
                         int64_t stream, int64_t shared_stream, int64_t route_stream, int64_t gemm_stream,
                         int64_t small_stream, int64_t timer, int64_t fp32_mask) {
  // saved-tensor hooks may have handed back other tensors than were saved
  for (const Tensor* t : {&h, &g, &wu, &wd, &Xg}) require(*t, at::kBFloat16, "saved tensor");
  for (const OptTensor* t : {&pre, &act, &Y, &s_act, &s_pre, &swg, &swu, &swd}) {
    if (t->has_value()) require(**t, at::kBFloat16, "saved tensor");
  }
  require(routing, at::kByte, "saved tensor");
  require(counts, at::kInt, "saved tensor");
  const bool shared = swg.has_value(), kept = pre.has_value();
  const int64_t N = h.size(0), D = h.size(1), E = g.size(0), H = wu.size(1) / 2, Hs = shared ? swg->size(0) : 0;
  const int64_t rows = rows_capacity(N * top_k, static_cast<int>(E));
  const int64_t ws_bytes = static_cast<int64_t>(backward_workspace(N, static_cast<int>(D), static_cast<int>(E)));
  const RoutingLayout layout(N, E, top_k, rows);
  const at::TensorOptions b16 = h.options(), u8 = b16.dtype(at::kByte);
  // computed() also densifies expanded (stride-0) gradients
  const Tensor go = grad_out.has_value() ? computed(*grad_out, "go") : at::zeros({N, D}, b16);
  Tensor gaux, gz;
  if (grad_aux.has_value()) gaux = grad_aux->to(at::kFloat).resolve_neg();
  if (grad_z.has_value()) gz = grad_z->to(at::kFloat).resolve_neg();
  // [D, Hs] has few output tiles (32 CTA-pair tiles at D = 1024, Hs = 2048 for 74 pairs): split the token dimension in two
  // halves, each accumulated in fp32, and add the two bf16 results
  const int64_t split = (N + 127) / 128 >= 64 && (D / 256) * ((Hs + 255) / 256) <= 40 ? 2 : 1;

  // Gradients of fp32 tensors are computed in bf16 like the others, in scratch, and converted in one launch at the end.
  struct Grad {
    Tensor t;             // as it is handed back
    int64_t scratch = 0;  // bytes of the bf16 values where they are computed elsewhere
  };
  auto gradient = [&](int i, at::IntArrayRef shape) {
    Grad gr;
    const bool wide = (fp32_mask >> i & 1) != 0;
    gr.t = at::empty(shape, wide ? b16.dtype(at::kFloat) : b16);
    gr.scratch = wide ? gr.t.numel() * 2 : 0;
    return gr;
  };
  const Grad dH = gradient(0, {N, D}), d_gate = gradient(1, {E, D}), d_wu = gradient(2, {E, 2 * H, D}),
             d_wd = gradient(3, {E, D, H});
  Grad s_dw, s_dwd;
  Tensor s_gate, s_up;  // the halves of s_dw
  if (shared) {
    if ((fp32_mask >> 4 & 1) != 0) {
      s_dw.scratch = 2 * Hs * D * 2;
      s_gate = at::empty({Hs, D}, b16.dtype(at::kFloat));
      s_up = at::empty({Hs, D}, b16.dtype(at::kFloat));
    } else {
      s_dw.t = at::empty({2 * Hs, D}, b16);
      s_gate = s_dw.t.narrow(0, 0, Hs);
      s_up = s_dw.t.narrow(0, Hs, Hs);
    }
    s_dwd = gradient(5, {D, Hs});
  }
  Scratch scratch(u8, {dH.scratch, d_gate.scratch, d_wu.scratch, d_wd.scratch, s_dw.scratch, s_dwd.scratch,
                       rows * D * 2, N * top_k * 4, rows * 4 * H, rows * D * 2, N * D * 2, ws_bytes,
                       fused ? 0 : rows * H * 2, N * Hs * 4, fused ? 0 : N * Hs * 2, shared ? N * D * 2 : 0,
                       split == 2 ? 2 * D * Hs * 2 : 0, kept ? 0 : rows * H * 4, kept ? 0 : rows * H * 2,
                       kept ? 0 : rows * D * 2});

  int64_t launched[3] = {0, 0, 0};
  ffm_layer_backward_args a = {};
  a.N = N;
  a.D = D;
  a.E = E;
  a.top_k = top_k;
  a.H = H;
  a.Hs = Hs;
  a.rows_cap = rows;
  a.gating = gating;
  a.activation = activation;
  a.shared_activation = shared_activation;
  a.recompute = !kept;
  a.zero_gw = capacity;
  a.fused_glu = fused;
  a.overlap = overlap;
  a.shared_split = split;
  a.aux_coef = aux_coef;
  a.z_coef = z_coef;
  a.go = ptr(go);
  a.hidden = ptr(h);
  a.gate = ptr(g);
  a.w_up = ptr(wu);
  a.w_down = ptr(wd);
  if (shared) {
    a.sw_gate = ptr(*swg);
    a.sw_up = ptr(swu.value());
    a.sw_down = ptr(swd.value());
    a.s_act = ptr(s_act.value());
    a.s_preact = ptr(s_pre.value());
  }
  a.grad_aux = ptr<float>(gaux);
  a.grad_z = ptr<float>(gz);
  char* rt = ptr<char>(routing);
  a.topk_w = reinterpret_cast<float*>(rt + layout.topk_w);
  a.topk_idx = reinterpret_cast<int32_t*>(rt + layout.topk_idx);
  a.logits = rt + layout.logits;
  a.lse = reinterpret_cast<float*>(rt + layout.lse);
  a.counts = ptr<int32_t>(counts);
  a.tile_start = reinterpret_cast<int32_t*>(rt + layout.tile_start);
  a.pos = reinterpret_cast<int32_t*>(rt + layout.pos);
  a.src = reinterpret_cast<int32_t*>(rt + layout.src);
  a.Xg = ptr(Xg);
  Casts casts;
  auto place = [&](const Grad& gr) {
    void* narrow = scratch.take();
    if (narrow == nullptr) return ptr(gr.t);
    if (gr.t.defined()) casts.add(narrow, gr.t.data_ptr(), gr.t.numel());
    return narrow;
  };
  a.dH = place(dH);
  a.d_gate = place(d_gate);
  a.d_w_up = place(d_wu);
  a.d_w_down = place(d_wd);
  a.s_d_gate_up = place(s_dw);
  if (s_dw.scratch > 0) {
    casts.add(a.s_d_gate_up, s_gate.data_ptr(), Hs * D);
    casts.add(static_cast<char*>(a.s_d_gate_up) + Hs * D * 2, s_up.data_ptr(), Hs * D);
  }
  a.s_d_down = place(s_dwd);
  a.gYw = scratch.take();
  a.gw = scratch.take<float>();
  a.gU = scratch.take();
  a.dXg = scratch.take();
  a.dH_route = scratch.take();
  a.workspace = scratch.take();
  a.d_act = scratch.take();
  a.s_gU = scratch.take();
  a.s_d_act = scratch.take();
  a.s_dx = scratch.take();
  a.s_parts = scratch.take();
  a.preact = scratch.take();
  a.act = scratch.take();
  a.Y = scratch.take();
  if (kept) {
    a.preact = ptr(*pre);
    a.act = ptr(act.value());
    a.Y = ptr(Y.value());
  }
  a.workspace_bytes = ws_bytes;
  a.status = at_address<int32_t>(status);
  a.stream = at_address<void>(stream);
  a.shared_stream = at_address<void>(shared_stream);
  a.route_stream = at_address<void>(route_stream);
  a.gemm_stream = at_address<void>(gemm_stream);
  a.small_stream = at_address<void>(small_stream);
  a.timer = at_address<const int64_t>(timer);
  a.launched = launched;
  int rc;
  {
    py::gil_scoped_release released;
    rc = backward_pass(&a);
  }
  if (rc == FFM_OK) launched[0] += casts.run(false, stream);
  return py::make_tuple(outcome(rc, launched), dH.t, d_gate.t, d_wu.t, d_wd.t, handed(s_gate), handed(s_up),
                        handed(s_dwd.t), go);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("bind", &bind);
  m.def("layer_forward", &layer_forward);
  m.def("layer_backward", &layer_backward);
}
