// The autograd boundary in native code: what attention.py does around the C ABI (evoattn.h), as a
// torch::autograd::Function.  A call of the op on a small problem is bound by the host: parsing,
// allocations, tensor views and autograd nodes in Python cost five to ten times what the kernels take
// (B=4, N_res=32: forward 58 us a call from Python, 8 us on the device), and backward has to take the
// interpreter lock on autograd's own thread.  Here a call reads sizes and strides, allocates its
// results and goes straight to the library; no view is created for a layout.
//
// Same semantics as the Python boundary (dsevoformer-triton/evoformer.py:633-862): the reinterpreting
// head layout or the true one, None for mask and bias, additive or boolean masks, gating, both bias
// layouts.  The N_seq-sharded op, which exchanges d(pair_bias) in its backward, and a call that is being
// traced stay in Python and take their checks and the preparation of their inputs from here.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <atomic>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "evoattn.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

std::atomic<int> g_force_generic{0};
std::atomic<int> g_fwd_launches{0}, g_bwd_launches{0}, g_fwd_path{0}, g_bwd_path{0};

// One int32 per device that kernels set when they give up a bounded wait.
constexpr int kMaxDevices = 64;
std::mutex g_status_mutex;
std::atomic<int32_t*> g_status_ptr[kMaxDevices];
Tensor* g_status[kMaxDevices] = {};  // (never destroyed: the CUDA context may be gone before they would be)

int32_t* status_ptr(c10::Device dev) {
  const int i = dev.index();
  TORCH_CHECK(i >= 0 && i < kMaxDevices, "device index out of range");
  if (int32_t* p = g_status_ptr[i].load(std::memory_order_acquire)) return p;
  std::lock_guard<std::mutex> lock(g_status_mutex);
  if (!g_status[i]) {
    g_status[i] = new Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(dev)));
    g_status_ptr[i].store(g_status[i]->data_ptr<int32_t>(), std::memory_order_release);
  }
  return g_status_ptr[i].load(std::memory_order_acquire);
}
Tensor status_word(int64_t index) {
  status_ptr(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(index)));
  return *g_status[index];
}

void check(int rc, const char* what) {
  if (rc != EVOATTN_OK) throw std::runtime_error(std::string(what) + " failed: " + evoattn_strerror(rc) + " (status " + std::to_string(rc) + ")");
}

int dtype_code(at::ScalarType t) { return t == at::kBFloat16 ? EVOATTN_BF16 : t == at::kHalf ? EVOATTN_FP16 : EVOATTN_FP32; }
bool known(at::ScalarType t) { return t == at::kBFloat16 || t == at::kHalf || t == at::kFloat; }

struct Dims {
  int64_t B, S, R, H, D;
  explicit Dims(const Tensor& q) : B(q.size(0)), S(q.size(1)), R(q.size(2)), H(q.size(3)), D(q.size(4)) {}
};

// Element strides of (b,h,s,r) of the attention view [B,H,S,R,D] of x [B,S,R,H,D]: the buffer
// reinterpreted (evoformer.py:648-650), or the true head axis.
void view_strides(const Tensor& x, const Dims& d, bool true_layout, int64_t* st) {
  if (true_layout) {
    st[0] = x.stride(0); st[1] = x.stride(3); st[2] = x.stride(1); st[3] = x.stride(2);
  } else {
    st[3] = d.D; st[2] = d.R * d.D; st[1] = d.S * d.R * d.D; st[0] = d.H * d.S * d.R * d.D;
  }
}
Tensor operand(const Tensor& x, bool true_layout) {
  if (true_layout ? x.stride(4) == 1 : x.is_contiguous()) return x;
  return x.contiguous();
}

void fill(evoattn_fwd_params* p, const Dims& d, bool tl, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o,
          const Tensor& lse, const Tensor& mask, const Tensor& bias, const Tensor& gate) {
  p->dtype = dtype_code(q.scalar_type());
  p->B = (int32_t)d.B; p->H = (int32_t)d.H; p->S = (int32_t)d.S; p->R = (int32_t)d.R; p->D = (int32_t)d.D;
  p->scale = (float)(1.0 / std::sqrt((double)d.D));  // evoformer.py:646
  p->flags = g_force_generic.load(std::memory_order_relaxed) ? EVOATTN_FLAG_FORCE_GENERIC : 0;
  p->q = q.data_ptr(); p->k = k.data_ptr(); p->v = v.data_ptr(); p->o = o.data_ptr();
  p->lse = lse.data_ptr<float>();
  view_strides(q, d, tl, p->q_stride);
  view_strides(k, d, tl, p->k_stride);
  view_strides(v, d, tl, p->v_stride);
  view_strides(o, d, tl, p->o_stride);
  if (mask.defined()) {
    p->mask = mask.data_ptr();
    p->mask_kind = mask.scalar_type() == at::kBool ? EVOATTN_MASK_BOOL
                   : mask.scalar_type() == at::kFloat ? EVOATTN_MASK_ADD_F32 : EVOATTN_MASK_ADD_SAME;
    const int last = (int)mask.dim() - 1;  // [B,S,1,1,R], or [B,S,R]
    p->mask_stride[0] = mask.stride(0); p->mask_stride[1] = mask.stride(1); p->mask_stride[2] = mask.stride(last);
  }
  if (bias.defined()) {
    p->bias = bias.data_ptr();
    p->bias_dtype = bias.scalar_type() == at::kFloat ? EVOATTN_BIAS_F32 : EVOATTN_BIAS_SAME;
    const int n = (int)bias.dim();  // [B,1,H,R,R], or [B,H,R,>=R]
    p->bias_stride[0] = bias.stride(0); p->bias_stride[1] = bias.stride(n - 3); p->bias_stride[2] = bias.stride(n - 2);
  }
  p->status = status_ptr(q.device());
  if (gate.defined()) {
    p->gate = gate.data_ptr();
    view_strides(gate, d, tl, p->gate_stride);
  }
}

// The residue mask as the kernels take it: bool, fp32 or the type of Q.
Tensor kernel_mask(const Tensor& m, const Dims& d, at::ScalarType qt) {
  if (!m.defined()) return m;
  Tensor r = m;
  const bool plain = m.dim() == 5 && m.size(0) == d.B && m.size(1) == d.S && m.size(2) == 1 && m.size(3) == 1 && m.size(4) == d.R;
  if (!plain) r = m.reshape({d.B, d.S, d.R});
  const at::ScalarType t = r.scalar_type();
  return (t == at::kBool || t == at::kFloat || t == qt) ? r : r.to(at::kFloat);
}

// The pair bias as the kernels take it: fp32 or the type of Q, last axis contiguous, and (where the
// tensor-core kernels apply) rows that tensor maps can read.
Tensor kernel_bias(const Tensor& pb, const Dims& d, at::ScalarType qt, bool heads_last, cudaStream_t st) {
  if (!pb.defined()) return pb;
  Tensor b = pb;
  if (b.scalar_type() != at::kFloat && b.scalar_type() != qt) b = b.to(at::kFloat);
  const int es = (int)b.element_size(), per = 16 / es;
  const int64_t ld = (d.R + per - 1) / per * per;
  if (heads_last) {
    TORCH_CHECK(b.dim() == 4 && b.size(0) == d.B && b.size(1) == d.R && b.size(2) == d.R && b.size(3) == d.H,
                "a heads-last pair bias has the shape [B, N_res, N_res, H]");
    b = b.contiguous();
    Tensor r = at::empty({d.B, d.H, d.R, ld}, b.options());
    check(evoattn_bias_to_heads_first_ld(b.data_ptr(), r.data_ptr(), dtype_code(b.scalar_type()), (int)d.B, (int)d.H, (int)d.R,
                                         (int)ld, st), "evoattn_bias_to_heads_first_ld");
    return r;
  }
  const bool plain = b.dim() == 5 && b.size(0) == d.B && b.size(1) == 1 && b.size(2) == d.H && b.size(3) == d.R && b.size(4) == d.R;
  if (!plain) b = b.reshape({d.B, d.H, d.R, d.R});
  if (b.stride(-1) != 1) b = b.contiguous();
  if (qt == at::kFloat || d.D > 64 || d.D % 8 != 0 || d.R > 2048) return b;
  const int n = (int)b.dim();
  const int64_t s[3] = {b.stride(0), b.stride(n - 3), b.stride(n - 2)};
  if (((uintptr_t)b.data_ptr() & 15) == 0 && (s[0] * es) % 16 == 0 && (s[1] * es) % 16 == 0 && (s[2] * es) % 16 == 0) return b;
  Tensor r = at::empty({d.B, d.H, d.R, ld}, b.options());
  check(evoattn_bias_pad_rows(b.data_ptr(), s, r.data_ptr(), dtype_code(b.scalar_type()), (int)d.B, (int)d.H, (int)d.R, (int)ld,
                              st), "evoattn_bias_pad_rows");
  return r;
}

using Maybe = c10::optional<Tensor>;

[[noreturn]] void raise(PyObject* type, const char* text) {
  PyErr_SetString(type, text);
  throw py::error_already_set();
}

// Everything a kernel is given an address of is checked here: on Q's device, of a size that its strides
// are read for.
void check_call(const Tensor& Q, const Tensor& K, const Tensor& V, const Maybe& mask, const Maybe& bias, const Maybe& gate) {
  const auto beside_q = [&](const Tensor& t, const char* name) {
    if (t.device() != Q.device())
      raise(PyExc_RuntimeError, (std::string(name) + " is on " + t.device().str() + ", Q on " + Q.device().str()).c_str());
  };
  if (mask) beside_q(*mask, "res_mask");
  if (bias) beside_q(*bias, "pair_bias");
  if (gate) beside_q(*gate, "gate");
  for (const Tensor* t : {&Q, &K, &V})
    if (!t->is_cuda()) raise(PyExc_RuntimeError, "EvoformerAttention runs on CUDA tensors only; there is no CPU fallback");
  beside_q(K, "K");
  beside_q(V, "V");
  if (Q.dim() != 5) raise(PyExc_ValueError, "Q must have the shape [B, N_seq, N_res, H, D]");
  if (K.size(-1) != Q.size(-1) || V.size(-1) != Q.size(-1))
    raise(PyExc_AssertionError, "Q, K, V must share the head dimension");  // evoformer.py:642-643
  if (!known(Q.scalar_type()) || K.scalar_type() != Q.scalar_type() || V.scalar_type() != Q.scalar_type())
    raise(PyExc_TypeError, "Q, K, V must share one dtype out of bfloat16, float16, float32");
  if (K.sizes() != Q.sizes() || V.sizes() != Q.sizes()) raise(PyExc_RuntimeError, "Q, K, V must have one shape");
  if (gate && (gate->sizes() != Q.sizes() || gate->scalar_type() != Q.scalar_type()))
    raise(PyExc_TypeError, "gate must have the shape and dtype of Q");
}

// The inputs of a call as the kernels take them.
struct Operands {
  Tensor q, k, v, mask, bias, gate;
  Operands(const Tensor& Q, const Tensor& K, const Tensor& V, const Maybe& mask_in, const Maybe& bias_in, const Maybe& gate_in,
           bool true_layout, bool heads_last, cudaStream_t st)
      : q(operand(Q, true_layout)), k(operand(K, true_layout)), v(operand(V, true_layout)),
        mask(kernel_mask(mask_in.value_or(Tensor()), Dims(Q), Q.scalar_type())),
        bias(kernel_bias(bias_in.value_or(Tensor()), Dims(Q), Q.scalar_type(), heads_last, st)),
        gate(gate_in ? operand(*gate_in, true_layout) : Tensor()) {}
};

struct Attention : public torch::autograd::Function<Attention> {

  static Tensor forward(AutogradContext* ctx, const Tensor& Q, const Tensor& K, const Tensor& V, const Maybe& mask_in,
                        const Maybe& bias_in, const Maybe& gate_in, bool true_layout, bool heads_last) {
    const Dims d(Q);
    const Tensor res_mask = mask_in.value_or(Tensor()), pair_bias = bias_in.value_or(Tensor());
    const c10::cuda::CUDAGuard guard(Q.device());
    const cudaStream_t st = at::cuda::getCurrentCUDAStream().stream();
    const Operands x(Q, K, V, mask_in, bias_in, gate_in, true_layout, heads_last, st);
    const Tensor &q = x.q, &k = x.k, &v = x.v, &mask = x.mask, &bias = x.bias, &gate = x.gate;
    Tensor o = at::empty({d.B, d.S, d.R, d.H, d.D}, q.options());
    Tensor lse = at::empty({d.B, d.H, d.S, d.R}, q.options().dtype(at::kFloat));
    evoattn_fwd_params p{};
    fill(&p, d, true_layout, q, k, v, o, lse, mask, bias, gate);
    check(evoattn_fwd(&p, st), "evoattn_fwd");
    g_fwd_launches = evoattn_last_launch_count();
    g_fwd_path = evoattn_last_path();
    ctx->save_for_backward({q, k, v, mask, bias, gate, o, lse});  // evoformer.py:729
    auto& sd = ctx->saved_data;
    sd["layout"] = (int64_t)((true_layout ? 1 : 0) | (heads_last ? 2 : 0));
    if (pair_bias.defined()) sd["bias"] = std::vector<int64_t>(pair_bias.sizes().vec()), sd["bias_t"] = (int64_t)pair_bias.scalar_type();
    if (res_mask.defined() && res_mask.is_floating_point())
      sd["mask"] = std::vector<int64_t>(res_mask.sizes().vec()), sd["mask_t"] = (int64_t)res_mask.scalar_type();
    return o;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k = s[1], &v = s[2], &mask = s[3], &bias = s[4], &gate = s[5], &o = s[6], &lse = s[7];
    auto& sd = ctx->saved_data;
    const int64_t layout = sd["layout"].toInt();
    const bool tl = layout & 1, heads_last = layout & 2;
    const Dims d(q);
    const c10::cuda::CUDAGuard guard(q.device());
    const cudaStream_t st = at::cuda::getCurrentCUDAStream().stream();
    Tensor dO = grads[0];
    if (dO.scalar_type() != q.scalar_type()) dO = dO.to(q.scalar_type());
    dO = operand(dO, tl);  // the reference asserts contiguity instead (evoformer.py:747)
    evoattn_bwd_params p{};
    fill(&p.fwd, d, tl, q, k, v, o, lse, mask, bias, gate);
    Tensor dq = at::empty({d.B, d.S, d.R, d.H, d.D}, q.options());
    Tensor dk = at::empty({d.B, d.S, d.R, d.H, d.D}, q.options());
    Tensor dv = at::empty({d.B, d.S, d.R, d.H, d.D}, q.options());
    p.d_o = dO.data_ptr(); p.dq = dq.data_ptr(); p.dk = dk.data_ptr(); p.dv = dv.data_ptr();
    view_strides(dO, d, tl, p.do_stride);
    view_strides(dq, d, tl, p.dq_stride);
    view_strides(dk, d, tl, p.dk_stride);
    view_strides(dv, d, tl, p.dv_stride);
    Tensor dgate, dmask, dbias;
    // edges of the node: Q, K, V, then those of mask, bias and gate that were given
    const size_t edge_mask = 3, edge_bias = mask.defined() ? 4 : 3;
    if (gate.defined()) {
      dgate = at::empty({d.B, d.S, d.R, d.H, d.D}, q.options());
      p.dgate = dgate.data_ptr();
      view_strides(dgate, d, tl, p.dgate_stride);
    }
    if (bias.defined() && ctx->needs_input_grad(edge_bias)) {
      const at::ScalarType want = (at::ScalarType)sd["bias_t"].toInt();
      const at::ScalarType t = known(want) ? want : at::kFloat;
      dbias = at::empty(sd["bias"].toIntVector(), q.options().dtype(t));
      if (t == at::kFloat && !heads_last) {
        p.dbias = dbias.data_ptr<float>();
      } else {  // the sum over N_seq stays in fp32 until this one cast (evoformer.py:860 casts to dO's type first)
        p.dbias_cast = dbias.data_ptr();
        p.dbias_cast_dtype = dtype_code(t);
        p.dbias_cast_heads_last = heads_last;
      }
    }
    // an additive mask that asks for a gradient gets one (DS4Sci returns gradients for both biases; the
    // reference returns None, evoformer.py:862)
    if (mask.defined() && mask.is_floating_point() && sd.count("mask") && ctx->needs_input_grad(edge_mask)) {
      dmask = at::empty({d.B, d.S, d.R}, q.options().dtype(at::kFloat));
      p.dmask = dmask.data_ptr<float>();
    }
    const size_t need = evoattn_bwd_workspace_bytes(&p);
    Tensor ws = at::empty({(int64_t)(need ? need : 1)}, q.options().dtype(at::kByte));
    p.workspace = ws.data_ptr();
    p.workspace_bytes = need;
    check(evoattn_bwd(&p, st), "evoattn_bwd");
    g_bwd_launches = evoattn_last_launch_count();
    g_bwd_path = evoattn_last_path();
    if (dbias.defined()) {
      const at::ScalarType want = (at::ScalarType)sd["bias_t"].toInt();
      if (dbias.scalar_type() != want) dbias = dbias.to(want);
    }
    if (dmask.defined()) dmask = dmask.reshape(sd["mask"].toIntVector()).to((at::ScalarType)sd["mask_t"].toInt());
    return {dq, dk, dv, dmask, dbias, dgate, Tensor(), Tensor()};
  }
};

Tensor attention(const Tensor& Q, const Tensor& K, const Tensor& V, const Maybe& mask, const Maybe& bias, const Maybe& gate,
                 bool true_layout, bool heads_last) {
  // A tracer would record this call as the allocation of its result; it takes the Python Function as one node.
  if (torch::jit::tracer::isTracing())
    return py::module_::import("evoformer_triton_b200.attention").attr("_python_boundary")(Q, K, V, mask, bias, gate, true_layout, heads_last).cast<Tensor>();
  check_call(Q, K, V, mask, bias, gate);
  return Attention::apply(Q, K, V, mask, bias, gate, true_layout, heads_last);
}

// What the Python boundary hands to the C ABI: the checks and the preparation are these.
std::vector<Tensor> prepare_call(const Tensor& Q, const Tensor& K, const Tensor& V, const Maybe& mask, const Maybe& bias,
                                 const Maybe& gate, bool true_layout, bool heads_last) {
  check_call(Q, K, V, mask, bias, gate);
  const c10::cuda::CUDAGuard guard(Q.device());
  const Operands x(Q, K, V, mask, bias, gate, true_layout, heads_last, at::cuda::getCurrentCUDAStream().stream());
  return {x.q, x.k, x.v, x.mask, x.bias, x.gate};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("attention", &attention);
  m.def("prepare_call", &prepare_call);
  m.def("status_word", &status_word);
  m.def("status_words", [] {
    std::lock_guard<std::mutex> lock(g_status_mutex);
    std::vector<Tensor> all;
    for (Tensor* t : g_status)
      if (t) all.push_back(*t);
    return all;
  });
  m.def("force_generic", [](bool on) { g_force_generic = on ? 1 : 0; });
  m.def("launch_counts", [] { return std::make_pair(g_fwd_launches.load(), g_bwd_launches.load()); });
  m.def("paths", [] { return std::make_pair(g_fwd_path.load(), g_bwd_path.load()); });
  // (the calls that attention.py makes itself, for the sharded op, are recorded here too)
  m.def("note_fwd", [](int launches, int path) { g_fwd_launches = launches; g_fwd_path = path; });
  m.def("note_bwd", [](int launches, int path) { g_bwd_launches = launches; g_bwd_path = path; });
  m.def("abi_version", [] { return evoattn_abi_version(); });
}
