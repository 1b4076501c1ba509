// Torch operators over the C ABI: outputs are allocated, arguments marshalled and the library called without going through
// Python.  rewy_b200::family_bwd is the whole-family backward (include/rewy_b200.h: rewy_{kda,gdn2,gdn,delta}_bwd),
// rewy_b200::chunk_fwd the forward (rewy_chunk_fwd).  Inputs are contiguous CUDA tensors of one device in the types of
// RewyBwdArgs / RewyFwdArgs; the launches go to torch's current stream, on which outputs and workspace are allocated, so the
// caching allocator's stream-ordered reuse keeps them valid.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/autograd_not_implemented_fallback.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/library.h>
#include <tuple>
#include "../../include/rewy_b200.h"

namespace {
using at::Tensor;
using OptTensor = std::optional<Tensor>;

const void* in(const Tensor& t) { return t.data_ptr(); }
const void* in(const OptTensor& t) { return t.has_value() ? t->data_ptr() : nullptr; }
const float* in32(const OptTensor& t) { return t.has_value() ? static_cast<const float*>(t->data_ptr()) : nullptr; }

void check(int status, const char* what) {
  TORCH_CHECK(status == REWY_OK, "rewy_b200 ", what, " failed with status ", status, ": ", rewy_last_error());
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> family_bwd(
    int64_t family, int64_t policy, bool out_f32, int64_t intra_passes, bool state_v_first, double scale, const Tensor& q,
    const Tensor& k, const Tensor& v, const Tensor& d_o, const Tensor& Akk, Tensor workspace, const OptTensor& g,
    const OptTensor& beta, const OptTensor& b_gate, const OptTensor& w_gate, const OptTensor& Aqk, const OptTensor& h0,
    const OptTensor& dht, const OptTensor& w, const OptTensor& qg, const OptTensor& kg, const OptTensor& v_new,
    const OptTensor& h, const OptTensor& cu_seqlens) {
  const c10::cuda::CUDAGuard guard(q.device());
  const auto B = k.size(0), T = k.size(1), H = k.size(2);
  const auto f32 = q.options().dtype(at::kFloat), bf16 = q.options().dtype(at::kBFloat16), odt = out_f32 ? f32 : bf16;
  const bool vec = family == REWY_GDN2;
  auto none = [&] { return at::empty({0}, f32); };
  auto big = [&](const at::TensorOptions& o) { return at::empty({B, T, H, 128}, o); };
  Tensor dq = big(odt), dk = big(odt), dv = big(bf16), dg = g.has_value() ? at::empty_like(*g) : none();
  Tensor dbeta = vec ? none() : at::empty({B, T, H}, f32), db = vec ? big(odt) : none(), dw = vec ? big(odt) : none();
  Tensor dh0 = h0.has_value() ? at::empty_like(*h0) : none();
  RewyBwdArgs a{};
  a.family = (int32_t)family; a.policy = (int32_t)policy; a.B = (int32_t)B; a.T = (int32_t)T; a.H = (int32_t)H;
  a.out_dtype = out_f32 ? REWY_OUT_F32 : REWY_OUT_BF16;
  a.intra_passes = (int32_t)intra_passes; a.state_v_first = state_v_first; a.scale = (float)scale;
  a.q = in(q); a.k = in(k); a.v = in(v); a.g = in32(g); a.beta = in32(beta); a.b_gate = in(b_gate); a.w_gate = in(w_gate);
  a.Aqk = in(Aqk); a.Akk = in(Akk); a.h0 = in32(h0); a.d_o = in(d_o); a.dht = in32(dht);
  a.w = in(w); a.qg = in(qg); a.kg = in(kg); a.v_new = in(v_new); a.h = in(h);
  a.dq = dq.data_ptr(); a.dk = dk.data_ptr(); a.dv = dv.data_ptr();
  a.dg = g.has_value() ? dg.data_ptr<float>() : nullptr;
  a.dbeta = vec ? nullptr : dbeta.data_ptr<float>();
  a.db_gate = vec ? db.data_ptr() : nullptr; a.dw_gate = vec ? dw.data_ptr() : nullptr;
  a.dh0 = h0.has_value() ? dh0.data_ptr<float>() : nullptr;
  if (cu_seqlens.has_value()) {  // int32, on the device, [sequences + 1]
    a.cu_seqlens = cu_seqlens->data_ptr<int32_t>();
    a.num_seqs = (int32_t)cu_seqlens->numel() - 1;
  }
  a.workspace = workspace.data_ptr();
  a.workspace_bytes = workspace.nbytes();
  if (!workspace.is_inference()) workspace.unsafeGetTensorImpl()->bump_version();  // written, as the schema says
  const auto st = at::cuda::getCurrentCUDAStream().stream();
  switch (family) {
    case REWY_KDA: check(rewy_kda_bwd(&a, st), "rewy_kda_bwd"); break;
    case REWY_GDN2: check(rewy_gdn2_bwd(&a, st), "rewy_gdn2_bwd"); break;
    case REWY_GDN: check(rewy_gdn_bwd(&a, st), "rewy_gdn_bwd"); break;
    default: check(rewy_delta_bwd(&a, st), "rewy_delta_bwd"); break;
  }
  return {dq, dk, dv, dg, dbeta, db, dw, dh0};
}

// (o, final_state, Aqk, Akk, w, u, qg, kg, v_new, h, ctrl); without a gate qg and kg are q and k and come back empty
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> chunk_fwd(
    int64_t family, bool state_v_first, bool output_final_state, double scale, const Tensor& q, const Tensor& k, const Tensor& v,
    const OptTensor& g, const OptTensor& beta, const OptTensor& b_gate, const OptTensor& w_gate, const OptTensor& h0,
    const OptTensor& cu_seqlens) {
  const c10::cuda::CUDAGuard guard(q.device());
  const auto B = k.size(0), T = k.size(1), H = k.size(2);
  const auto bf16 = q.options(), f32 = bf16.dtype(at::kFloat);
  const bool gateless = family == REWY_DELTA;
  auto big = [&] { return at::empty({B, T, H, 128}, bf16); };
  auto a64 = [&] { return at::empty({B, T, H, 64}, bf16); };
  auto none = [&] { return at::empty({0}, bf16); };
  const int64_t seqs = cu_seqlens.has_value() ? cu_seqlens->numel() - 1 : B;
  Tensor o = big(), Aqk = a64(), Akk = a64(), w = big(), u = big(), qg = gateless ? none() : big(), kg = gateless ? none() : big();
  Tensor v_new = big(), h = at::empty({B, T / 64, H, 128, 128}, bf16), ctrl = at::empty({2}, bf16.dtype(at::kInt));
  Tensor fin = output_final_state ? at::empty({seqs, H, 128, 128}, f32) : at::empty({0}, f32);
  RewyFwdArgs a{};
  a.family = (int32_t)family; a.B = (int32_t)B; a.T = (int32_t)T; a.H = (int32_t)H; a.state_v_first = state_v_first;
  a.scale = (float)scale;
  a.q = in(q); a.k = in(k); a.v = in(v); a.g = in32(g); a.beta = in32(beta); a.b_gate = in(b_gate); a.w_gate = in(w_gate);
  a.h0 = in32(h0);
  a.o = o.data_ptr(); a.final_state = output_final_state ? fin.data_ptr<float>() : nullptr;
  a.Aqk = Aqk.data_ptr(); a.Akk = Akk.data_ptr(); a.w = w.data_ptr(); a.u = u.data_ptr();
  a.qg = gateless ? const_cast<void*>(in(q)) : qg.data_ptr(); a.kg = gateless ? const_cast<void*>(in(k)) : kg.data_ptr();
  a.v_new = v_new.data_ptr(); a.h = h.data_ptr(); a.ctrl = ctrl.data_ptr();
  if (cu_seqlens.has_value()) {
    a.cu_seqlens = cu_seqlens->data_ptr<int32_t>();
    a.num_seqs = (int32_t)seqs;
  }
  check(rewy_chunk_fwd(&a, at::cuda::getCurrentCUDAStream().stream()), "rewy_chunk_fwd");
  return {o, fin, Aqk, Akk, w, u, qg, kg, v_new, h, ctrl};
}

// Inside the backward of an autograd function: the gradients it gives, tied to the function's inputs by a node that raises.
std::vector<Tensor> first_order(at::TensorList grads) {
  std::vector<Tensor> out(grads.begin(), grads.end());
  const auto current = torch::autograd::get_current_node();
  if (current == nullptr) return out;
  auto edges = current->next_edges();
  const auto error = std::make_shared<torch::autograd::Error>("derivative for rewy_b200::family_bwd is not implemented", std::move(edges));
  for (Tensor& t : out) {
    t = t.detach();
    torch::autograd::create_gradient_edge(t, error);
  }
  return out;
}

}  // namespace

// (the schemas are defined in rewy_b200/backward.py)
TORCH_LIBRARY_IMPL(rewy_b200, CUDA, m) {
  m.impl("family_bwd", &family_bwd);
  m.impl("chunk_fwd", &chunk_fwd);
}
TORCH_LIBRARY_IMPL(rewy_b200, Autograd, m) {  // differentiating through them raises
  m.impl("family_bwd", torch::autograd::autogradNotImplementedFallback());
  m.impl("chunk_fwd", torch::autograd::autogradNotImplementedFallback());
}
TORCH_LIBRARY_IMPL(rewy_b200, CompositeImplicitAutograd, m) { m.impl("first_order", &first_order); }
