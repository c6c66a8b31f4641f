// The host path of the differentiable ops: tensors in, one C-ABI call per direction, autograd nodes.
//
// A small call of this library is a few microseconds on the GPU, so what a user waits for is the code in front of the
// launch.  Filling the ABI's structs through ctypes, allocating through keyword arguments and running a Python
// autograd.Function cost 20 us for a decode step and about 200 us for a forward + backward; the same steps here cost
// a few.  Nothing is computed in this file and nothing is kept between calls.
//
// Python keeps the argument checks that name shapes (AssertionError) and the reference's signatures; what arrives here
// has consistent shapes.  Tensors are made contiguous here.
#include "common.h"

using namespace tops_torch;

namespace {

// ---------------------------------------------------------------------------------------------------
// chunked GLA and simple_gla
// ---------------------------------------------------------------------------------------------------
tops_chunk_problem chunk_problem(const ChunkShape& s, const Tensor& q, const Tensor& v, const Tensor& gate) {
  tops_chunk_problem pb{};
  pb.B = (int)q.size(0); pb.T = (int)q.size(1); pb.H = (int)q.size(2); pb.K = (int)q.size(3); pb.V = (int)v.size(3);
  pb.chunk = s.chunk; pb.dtype = code_of(q); pb.gate_dtype = gate.defined() ? code_of(gate) : TOPS_F32;
  pb.gate_kind = s.kind; pb.impl = TOPS_IMPL_AUTO; pb.scale = (float)s.scale;
  if (!s.cu.empty()) { pb.cu_seqlens_host = s.cu.data(); pb.N = (int)s.cu.size() - 1; }
  return pb;
}
// the generic kernels read the boundaries of a packed batch from the device
Tensor device_boundaries(const ChunkShape& s, tops_chunk_problem& pb, const Call& c) {
  Tensor t = at::tensor(at::ArrayRef<int32_t>(s.cu), at::TensorOptions().dtype(at::kInt)).to(c.dev);
  pb.cu_seqlens = t.data_ptr<int32_t>();
  return t;
}

struct ChunkNode : public OpNode {
  ChunkShape s;
  bool has_h0 = false;
  variable_list apply(variable_list&& grads) override {
    variable_list t;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      t = unpack();
    }
    const Tensor &q = t[0], &k = t[1], &v = t[2], &gate = t[3], &h0 = t[4], &hs = t[5];
    Call c(q);
    const auto type = q.scalar_type();
    const bool stored = s.kind == TOPS_GATE_PER_CHANNEL || s.kind == TOPS_GATE_SCALAR;
    Tensor qc = c.in(q), kc = c.in(k), vc = c.in(v);
    Tensor gc = s.kind == TOPS_GATE_GAMMA ? c.in_as(gate, at::kFloat) : c.in(gate);
    Tensor h0c = c.in_as(h0, at::kFloat);
    Tensor doc = cotangent(grads[0], v, type, c);
    Tensor dht = grads.size() > 1 ? c.in_as(grads[1], at::kFloat) : Tensor();
    tops_chunk_bwd_params p{};
    p.pb = chunk_problem(s, q, v, gc);
    const bool fast = tops_b200_chunk_selected_impl(&p.pb) == TOPS_IMPL_SM100;
    Tensor cu_dev;
    if (!fast && !s.cu.empty()) cu_dev = device_boundaries(s, p.pb, c);
    // the tcgen05 kernels write the primals' dtypes, the generic ones fp32 for chunked GLA (cast below)
    const auto grad_type = (fast || s.kind == TOPS_GATE_SCALAR || s.kind == TOPS_GATE_GAMMA) ? type : at::kFloat;
    const auto dg_type = (fast && s.kind == TOPS_GATE_PER_CHANNEL) ? gate.scalar_type() : at::kFloat;
    Tensor dq = c.empty(q.sizes(), grad_type), dk = c.empty(k.sizes(), grad_type), dv = c.empty(v.sizes(), type), dg, dh0;
    if (stored && task_should_compute_output(3)) dg = c.empty(gate.sizes(), dg_type);
    if (has_h0) dh0 = c.empty(h0.sizes(), at::kFloat);
    p.q = ptr(qc); p.k = ptr(kc); p.v = ptr(vc); p.g = ptr(gc); p.h0 = ptr<float>(h0c); p.do_ = ptr(doc); p.dht = ptr<float>(dht);
    p.dq = ptr(dq); p.dk = ptr(dk); p.dv = ptr(dv); p.dg = ptr(dg); p.dh0 = ptr<float>(dh0);
    p.grad_dtype = code_of(grad_type); p.dg_dtype = code_of(dg_type); p.h_saved = ptr(hs);
    p.saved_bytes = hs.defined() ? hs.nbytes() : 0;
    const size_t need = tops_b200_chunk_bwd_workspace_bytes(&p);
    Tensor ws = c.bytes(need);
    check(tops_b200_chunk_gla_bwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "chunk_gla_bwd");
    check_device_word("chunk backward");
    if (grad_type != type) { dq = dq.to(type); dk = dk.to(type); }
    if (dg.defined() && dg.scalar_type() != gate.scalar_type()) dg = dg.to(gate.scalar_type());
    if (s.kind == TOPS_GATE_GAMMA && task_should_compute_output(3)) dg = at::zeros_like(gate);   // a constant decay gets a zero cotangent
    if (dh0.defined() && h0.scalar_type() != at::kFloat) dh0 = dh0.to(h0.scalar_type());
    return {dq, dk, dv, dg, dh0};
  }
};

std::tuple<Tensor, OptTensor> chunk(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& gate_, int kind,
                                    const OptTensor& h0_, double scale, bool want_ht, std::vector<int32_t> cu, int chunk_len) {
  Call c(q);
  const Tensor gate = opt(gate_), h0 = opt(h0_);
  ChunkShape s;
  s.kind = kind; s.chunk = chunk_len; s.scale = scale; s.cu = std::move(cu);
  s.N = s.cu.empty() ? (int)q.size(0) : (int)s.cu.size() - 1;
  Tensor qc = c.in(q), kc = c.in(k), vc = c.in(v);
  Tensor gc = kind == TOPS_GATE_GAMMA ? c.in_as(gate, at::kFloat) : c.in(gate);
  Tensor h0c = c.in_as(h0, at::kFloat);
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3), V = v.size(3);
  Tensor o = c.empty({B, T, H, V}, v.scalar_type()), ht, hs;
  if (want_ht) ht = c.empty({s.N, H, K, V}, at::kFloat);
  tops_chunk_fwd_params p{};
  // the results do not depend on the chunk length beyond where roundings fall: a problem the tcgen05 kernels take runs
  // with their 64, every other one with the length it asks for (the CUDA-core kernels lose strong gates in longer chunks)
  s.chunk = 64;
  p.pb = chunk_problem(s, q, v, gc);
  if (tops_b200_chunk_selected_impl(&p.pb) != TOPS_IMPL_SM100) p.pb.chunk = s.chunk = chunk_len;
  p.q = ptr(qc); p.k = ptr(kc); p.v = ptr(vc); p.g = ptr(gc); p.h0 = ptr<float>(h0c); p.o = ptr(o); p.ht = ptr<float>(ht);
  const bool keep = wants_grad(q, k, v, gate, h0);
  Tensor cu_dev;
  if (keep) {   // the tcgen05 forward keeps its chunk-start states for the backward
    const size_t n = tops_b200_chunk_saved_bytes(&p.pb);
    if (n) {
      hs = c.empty({(int64_t)(n / 2)}, at::kBFloat16);
      p.saved_out = ptr(hs);
      p.saved_bytes = hs.nbytes();
    }
  }
  if (!s.cu.empty() && tops_b200_chunk_selected_impl(&p.pb) != TOPS_IMPL_SM100) cu_dev = device_boundaries(s, p.pb, c);
  Tensor ws = c.bytes(tops_b200_chunk_fwd_workspace_bytes(&p));
  check(tops_b200_chunk_gla_fwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "chunk_gla_fwd");
  if (keep) {
    auto node = make_node<ChunkNode>(q, k, v, gate, h0);
    node->s = std::move(s);
    node->has_h0 = h0.defined();
    node->keep({q, k, v, gate, h0, hs});
    attach(o, node);
    attach(ht, node);
  }
  return {o, ht.defined() ? OptTensor(ht) : std::nullopt};
}

// ---------------------------------------------------------------------------------------------------
// token recurrence (GLA)
// ---------------------------------------------------------------------------------------------------
tops_recurrent_fwd_params rec_fwd_params(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gk, const Tensor& gv,
                                         double scale, bool reverse, at::ScalarType o_type) {
  tops_recurrent_fwd_params p{};
  p.B = (int)q.size(0); p.T = (int)q.size(1); p.H = (int)q.size(2); p.K = (int)q.size(3); p.V = (int)v.size(3);
  p.dtype = code_of(q); p.gate_dtype = gk.defined() ? code_of(gk) : gv.defined() ? code_of(gv) : TOPS_F32;
  p.o_dtype = code_of(o_type); p.reverse = reverse; p.scale = (float)scale;
  p.q = ptr(q); p.k = ptr(k); p.v = ptr(v); p.gk = ptr(gk); p.gv = ptr(gv);
  return p;
}

struct RecNode : public OpNode {
  double scale = 1.0;
  bool reverse = false;
  std::vector<int32_t> cu;
  variable_list apply(variable_list&& grads) override {
    variable_list t;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      t = unpack();
    }
    const Tensor &q = t[0], &k = t[1], &v = t[2], &gk = t[3], &gv = t[4], &h0 = t[5], &o32 = t[6];
    Call c(q);
    Tensor qc = c.in(q), kc = c.in(k), vc = c.in(v), gkc = c.in(gk), gvc = c.in(gv), h0c = c.in_as(h0, at::kFloat);
    Tensor doc = cotangent(grads[0], v, q.scalar_type(), c);
    Tensor dht = grads.size() > 1 ? c.in_as(grads[1], at::kFloat) : Tensor();
    Tensor dq = c.empty_as(q), dk = c.empty_as(k), dv = c.empty_as(v), dgk, dgv, dh0, cu_dev;
    if (gk.defined()) dgk = c.empty_as(gk);
    if (gv.defined()) dgv = c.empty_as(gv);
    if (h0.defined()) dh0 = c.empty(h0.sizes(), at::kFloat);
    tops_recurrent_bwd_params p{};
    p.B = (int)q.size(0); p.T = (int)q.size(1); p.H = (int)q.size(2); p.K = (int)q.size(3); p.V = (int)v.size(3);
    p.dtype = code_of(q); p.gate_dtype = gk.defined() ? code_of(gk) : gv.defined() ? code_of(gv) : TOPS_F32;
    p.reverse = reverse; p.scale = (float)scale;
    p.q = ptr(qc); p.k = ptr(kc); p.v = ptr(vc); p.gk = ptr(gkc); p.gv = ptr(gvc); p.o = ptr<float>(o32); p.do_ = ptr(doc);
    p.h0 = ptr<float>(h0c); p.dht = ptr<float>(dht); p.dq = ptr(dq); p.dk = ptr(dk); p.dv = ptr(dv); p.dgk = ptr(dgk);
    p.dgv = ptr(dgv); p.dh0 = ptr<float>(dh0); p.N = p.B;
    if (!cu.empty()) {
      cu_dev = at::tensor(at::ArrayRef<int32_t>(cu), at::TensorOptions().dtype(at::kInt)).to(c.dev);
      p.cu_seqlens = cu_dev.data_ptr<int32_t>();
      p.N = (int)cu.size() - 1;
    }
    Tensor ws = c.bytes(tops_b200_fused_recurrent_gla_bwd_workspace_bytes(&p));
    check(tops_b200_fused_recurrent_gla_bwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "fused_recurrent_gla_bwd");
    if (dh0.defined() && h0.scalar_type() != at::kFloat) dh0 = dh0.to(h0.scalar_type());
    return {dq, dk, dv, dgk, dgv, dh0};
  }
};

std::tuple<Tensor, OptTensor> recurrent(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& gk_, const OptTensor& gv_,
                                        double scale, const OptTensor& h0_, bool want_ht, bool reverse, std::vector<int32_t> cu) {
  Call c(q);
  const Tensor gk = opt(gk_), gv = opt(gv_), h0 = opt(h0_);
  Tensor qc = c.in(q), kc = c.in(k), vc = c.in(v), gkc = c.in(gk), gvc = c.in(gv), h0c = c.in_as(h0, at::kFloat);
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3), V = v.size(3);
  const int64_t N = cu.empty() ? B : (int64_t)cu.size() - 1;
  const bool grad = wants_grad(q, k, v, gk, gv, h0);
  // the fp32 outputs are only needed by the gradient of gv
  const auto o_type = grad && gv.defined() ? at::kFloat : q.scalar_type();
  Tensor o = c.empty({B, T, H, V}, o_type), ht, cu_dev;
  if (want_ht) ht = c.empty({N, H, K, V}, at::kFloat);
  tops_recurrent_fwd_params p = rec_fwd_params(qc, kc, vc, gkc, gvc, scale, reverse, o_type);
  p.state_in = ptr<float>(h0c); p.state_out = ptr<float>(ht); p.o = ptr(o); p.N = (int)N;
  if (!cu.empty()) {
    cu_dev = at::tensor(at::ArrayRef<int32_t>(cu), at::TensorOptions().dtype(at::kInt)).to(c.dev);
    p.cu_seqlens = cu_dev.data_ptr<int32_t>();
  }
  check(tops_b200_fused_recurrent_gla_fwd(&p, c.stream()), "fused_recurrent_gla_fwd");
  Tensor o32 = o;
  if (o_type != q.scalar_type()) o = o.to(q.scalar_type());
  if (grad) {
    auto node = make_node<RecNode>(q, k, v, gk, gv, h0);
    node->scale = scale; node->reverse = reverse; node->cu = std::move(cu);
    if (gv.defined() && o32.is_same(o)) o32 = o.detach();   // (fp32 q: the output itself; saved without its history)
    node->keep({q, k, v, gk, gv, h0, gv.defined() ? o32 : Tensor()});
    attach(o, node);
    attach(ht, node);
  }
  return {o, ht.defined() ? OptTensor(ht) : std::nullopt};
}

// one call of a decode loop: `state` fp32 [B,H,K,V] is updated in place
Tensor recurrent_decode(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& gk_, const OptTensor& gv_, double scale,
                        const Tensor& state) {
  Call c(q);
  Tensor qc = c.in(q), kc = c.in(k), vc = c.in(v), gk = c.in(gk_), gv = c.in(gv_);
  Tensor o = c.empty({q.size(0), q.size(1), q.size(2), v.size(3)}, q.scalar_type());
  tops_recurrent_fwd_params p = rec_fwd_params(qc, kc, vc, gk, gv, scale, false, q.scalar_type());
  p.state_in = p.state_out = c.state(state); p.o = ptr(o); p.N = p.B;
  check(tops_b200_fused_recurrent_gla_fwd(&p, c.stream()), "fused_recurrent_gla_fwd");
  return o;
}

// ---------------------------------------------------------------------------------------------------
// KDA
// ---------------------------------------------------------------------------------------------------
tops_chunk_kda_fwd_params kda_chunk_params(const Tensor& q, const Tensor& v, const Tensor& g, double scale) {
  tops_chunk_kda_fwd_params p{};
  p.B = (int)q.size(0); p.T = (int)q.size(1); p.H = (int)q.size(2); p.K = (int)q.size(3); p.V = (int)v.size(3); p.chunk = 64;
  p.dtype = code_of(q); p.gate_dtype = code_of(g); p.scale = (float)scale;
  return p;
}

struct KdaNode : public OpNode {
  double scale = 1.0;
  bool chunked = false;
  variable_list apply(variable_list&& grads) override {
    variable_list t;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      t = unpack();
    }
    const Tensor &q = t[0], &k = t[1], &v = t[2], &g = t[3], &beta = t[4], &h0 = t[5];
    Call c(q);
    const auto type = q.scalar_type();
    Tensor qc = c.in(q), kc = c.in(k), vc = c.in(v), gc = c.in(g), bc = c.in_as(beta, type), h0c = c.in_as(h0, at::kFloat);
    Tensor doc = cotangent(grads[0], v, type, c);
    Tensor dht = grads.size() > 1 ? c.in_as(grads[1], at::kFloat) : Tensor();
    Tensor dq = c.empty_as(q), dk = c.empty_as(k), dv = c.empty_as(v), dg, db = c.empty(beta.sizes(), type), dh0;
    if (h0.defined()) dh0 = c.empty(h0.sizes(), at::kFloat);
    if (chunked) {
      dg = c.empty(g.sizes(), type);
      tops_chunk_kda_bwd_params p{};
      p.B = (int)q.size(0); p.T = (int)q.size(1); p.H = (int)q.size(2); p.K = (int)q.size(3); p.V = (int)v.size(3); p.chunk = 64;
      p.dtype = code_of(q); p.gate_dtype = code_of(g); p.scale = (float)scale;
      p.q = ptr(qc); p.k = ptr(kc); p.v = ptr(vc); p.g = ptr(gc); p.beta = ptr(bc); p.do_ = ptr(doc); p.dht = ptr<float>(dht);
      p.saved = ptr(t[6]);
      p.dq = ptr(dq); p.dk = ptr(dk); p.dg = ptr(dg); p.dbeta = ptr(db); p.dv = ptr(dv); p.dh0 = ptr<float>(dh0);
      p.grad_dtype = code_of(type);
      Tensor ws = c.bytes(tops_b200_chunk_kda_bwd_workspace_bytes(&p));
      check(tops_b200_chunk_kda_bwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "chunk_kda_bwd");
      check_device_word("chunk_kda backward");
      if (g.scalar_type() != type) dg = dg.to(g.scalar_type());
    } else {
      if (q.size(3) > 128 || v.size(3) > 128) raise_assertion("the KDA backward kernel takes K, V <= 128");
      dg = c.empty_as(g);
      tops_kda_bwd_params p{};
      p.B = (int)q.size(0); p.T = (int)q.size(1); p.H = (int)q.size(2); p.K = (int)q.size(3); p.V = (int)v.size(3);
      p.dtype = code_of(q); p.gate_dtype = code_of(g); p.scale = (float)scale;
      p.q = ptr(qc); p.k = ptr(kc); p.v = ptr(vc); p.g = ptr(gc); p.beta = ptr(bc); p.h0 = ptr<float>(h0c); p.do_ = ptr(doc);
      p.dht = ptr<float>(dht); p.dq = ptr(dq); p.dk = ptr(dk); p.dv = ptr(dv); p.dg = ptr(dg); p.dbeta = ptr(db); p.dh0 = ptr<float>(dh0);
      Tensor ws = c.bytes(tops_b200_kda_bwd_workspace_bytes(&p));
      check(tops_b200_kda_bwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "kda_bwd");
    }
    if (beta.scalar_type() != type) db = db.to(beta.scalar_type());
    if (dh0.defined() && h0.scalar_type() != at::kFloat) dh0 = dh0.to(h0.scalar_type());
    return {dq, dk, dv, dg, db, dh0};
  }
};

Tensor kda_run(const Call& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, double scale,
               const float* h0, float* ht) {
  Tensor o = c.empty(v.sizes(), q.scalar_type());
  tops_kda_fwd_params p{};
  p.B = (int)q.size(0); p.T = (int)q.size(1); p.H = (int)q.size(2); p.K = (int)q.size(3); p.V = (int)v.size(3);
  p.dtype = code_of(q); p.gate_dtype = code_of(g); p.scale = (float)scale;
  p.q = ptr(q); p.k = ptr(k); p.v = ptr(v); p.g = ptr(g); p.beta = ptr(beta); p.h0 = h0; p.o = ptr(o); p.ht = ht;
  check(tops_b200_kda_fwd(&p, c.stream()), "kda_fwd");
  return o;
}

// `chunked`: use the tensor-core kernels where they take the problem
std::tuple<Tensor, OptTensor> kda(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, double scale,
                                  const OptTensor& h0_, bool want_ht, bool chunked) {
  Call c(q);
  const Tensor h0 = opt(h0_);
  const auto type = q.scalar_type();
  Tensor qc = c.in(q), kc = c.in(k), vc = c.in(v), gc = c.in(g), bc = c.in_as(beta, type), h0c = c.in_as(h0, at::kFloat);
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3), V = v.size(3);
  const bool grad = wants_grad(q, k, v, g, beta, h0);
  Tensor ht, o, saved, ws;
  if (want_ht) ht = c.empty({B, H, K, V}, at::kFloat);
  tops_chunk_kda_fwd_params p = kda_chunk_params(q, v, g, scale);
  chunked = chunked && tops_b200_chunk_kda_supported(&p) != 0;
  if (chunked) {
    o = c.empty({B, T, H, V}, type);
    if (grad) {
      saved = c.bytes(tops_b200_chunk_kda_saved_bytes(&p));
    } else {
      ws = c.bytes(tops_b200_chunk_kda_fwd_workspace_bytes(&p));
      p.workspace = ptr(ws); p.workspace_bytes = (size_t)ws.numel();
    }
    p.q = ptr(qc); p.k = ptr(kc); p.v = ptr(vc); p.g = ptr(gc); p.beta = ptr(bc); p.h0 = ptr<float>(h0c); p.o = ptr(o);
    p.ht = ptr<float>(ht); p.saved = ptr(saved);
    check(tops_b200_chunk_kda_fwd(&p, c.stream()), "chunk_kda_fwd");
  } else {
    o = kda_run(c, qc, kc, vc, gc, bc, scale, ptr<float>(h0c), ptr<float>(ht));
  }
  if (grad) {
    auto node = make_node<KdaNode>(q, k, v, g, beta, h0);
    node->scale = scale; node->chunked = chunked;
    node->keep({q, k, v, g, beta, h0, saved});
    attach(o, node);
    attach(ht, node);
  }
  return {o, ht.defined() ? OptTensor(ht) : std::nullopt};
}

Tensor kda_decode(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, double scale,
                  const Tensor& state) {
  Call c(q);
  return kda_run(c, c.in(q), c.in(k), c.in(v), c.in(g), c.in_as(beta, q.scalar_type()), scale, c.state(state), c.state(state));
}

// ---------------------------------------------------------------------------------------------------
// gates
// ---------------------------------------------------------------------------------------------------
struct GateLaw { int kind = 0; double lower_bound = 0, normalizer = 1, clamp = 0; bool has_clamp = false; };
tops_gate_act_params gate_params(const GateLaw& l, const Tensor& g, const Tensor& A, const Tensor& b, at::ScalarType out_type) {
  tops_gate_act_params p{};
  const int64_t H = g.size(-2), K = g.size(-1);
  p.rows = g.numel() / (H * K); p.H = (int)H; p.K = (int)K; p.kind = l.kind; p.dtype = code_of(g); p.out_dtype = code_of(out_type);
  p.g = ptr(g); p.A_log = ptr<float>(A); p.dt_bias = ptr<float>(b); p.lower_bound = (float)l.lower_bound;
  p.normalizer = (float)l.normalizer; p.clamp_min = (float)l.clamp; p.has_clamp_min = l.has_clamp;
  return p;
}
// head-wise parameters of fewer heads are repeated: fp32 [H] and [H*K]
Tensor expand_A(const Call& c, const Tensor& A, int64_t H) {
  Tensor a = c.in_as(A, at::kFloat);
  return a.size(0) == H ? a : a.repeat_interleave(H / a.size(0)).contiguous();
}
Tensor expand_bias(const Call& c, const Tensor& bias, int64_t base, int64_t H, int64_t K) {
  if (!bias.defined()) return bias;
  Tensor b = c.in_as(bias, at::kFloat);
  return b.size(0) == H * K ? b : b.reshape({base, K}).repeat_interleave(H / base, 0).reshape({-1}).contiguous();
}

struct GateNode : public OpNode {
  GateLaw law;
  variable_list apply(variable_list&& grads) override {
    variable_list t;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      t = unpack();
    }
    const Tensor &g = t[0], &A_log = t[1], &bias = t[2];
    if (!grads[0].defined()) return variable_list(A_log.defined() ? 3 : 1);
    Call c(g);
    const int64_t H = g.size(-2), K = g.size(-1);
    Tensor gc = c.in(g), dy = c.in(grads[0]), dg = c.empty_as(g), A, b, dA, db;
    if (A_log.defined()) {
      A = expand_A(c, A_log, H);
      b = expand_bias(c, bias, A_log.size(0), H, K);
      dA = c.empty({H}, at::kFloat);
      if (b.defined()) db = c.empty({H * K}, at::kFloat);
    }
    tops_gate_act_bwd_params p{};
    p.fwd = gate_params(law, gc, A, b, gc.scalar_type());
    p.dy = ptr(dy); p.dy_dtype = code_of(dy); p.dg = ptr(dg); p.dA_log = ptr<float>(dA); p.dbias = ptr<float>(db);
    Tensor ws = c.bytes(tops_b200_gate_act_bwd_workspace_bytes(&p));
    check(tops_b200_gate_act_bwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "gate_act_bwd");
    if (!A_log.defined()) return {dg};
    const int64_t base = A_log.size(0);
    if (base != H) dA = dA.reshape({base, H / base}).sum(1);
    if (dA.scalar_type() != A_log.scalar_type()) dA = dA.to(A_log.scalar_type());
    if (db.defined()) {
      if (bias.size(0) != H * K) db = db.reshape({base, H / base, K}).sum(1).reshape({-1});
      if (db.scalar_type() != bias.scalar_type()) db = db.to(bias.scalar_type());
    }
    return {dg, dA, db};
  }
};

Tensor gate(const Tensor& g, const OptTensor& A_, const OptTensor& bias_, int kind, double lower_bound, double normalizer,
            std::optional<double> clamp, std::optional<at::ScalarType> out_type_) {
  Call c(g);
  const Tensor A_log = opt(A_), bias = opt(bias_);
  const auto out_type = out_type_.value_or(g.scalar_type());
  const int64_t H = g.size(-2), K = g.size(-1);
  Tensor gc = c.in(g), A, b, out = c.empty(g.sizes(), out_type);
  if (A_log.defined()) { A = expand_A(c, A_log, H); b = expand_bias(c, bias, A_log.size(0), H, K); }
  GateLaw law{kind, lower_bound, normalizer, clamp.value_or(0.0), clamp.has_value()};
  tops_gate_act_params p = gate_params(law, gc, A, b, out_type);
  p.out = ptr(out);
  check(tops_b200_gate_act_fwd(&p, c.stream()), "gate_act_fwd");
  if (wants_grad(g, A_log, bias)) {
    auto node = A_log.defined() ? make_node<GateNode>(g, A_log, bias) : make_node<GateNode>(g);
    node->law = law;
    node->keep({g, A_log, bias});
    attach(out, node);
  }
  return out;
}

// ---------------------------------------------------------------------------------------------------
// norms
// ---------------------------------------------------------------------------------------------------
tops_norm_params norm_params(const Tensor& x, double eps) {
  tops_norm_params p{};
  const int64_t D = x.size(-1);
  p.rows = x.numel() / D; p.D = (int)D; p.dtype = code_of(x); p.eps = (float)eps; p.x = ptr(x);
  return p;
}

struct L2Node : public OpNode {
  double eps = 1e-6;
  variable_list apply(variable_list&& grads) override {
    variable_list t;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      t = unpack();
    }
    if (!grads[0].defined()) return variable_list(1);
    Call c(t[0]);
    Tensor x = c.in(t[0]), dy = c.in_as(grads[0], x.scalar_type()), dx = c.empty_as(x);
    tops_norm_params p = norm_params(x, eps);
    p.dy = ptr(dy); p.dx = ptr(dx);
    check(tops_b200_l2norm_bwd(&p, c.stream()), "l2norm_bwd");
    return {dx};
  }
};
Tensor l2norm(const Tensor& x, double eps) {
  Call c(x);
  Tensor xc = c.in(x), y = c.empty_as(x);
  tops_norm_params p = norm_params(xc, eps);
  p.y = ptr(y);
  check(tops_b200_l2norm_fwd(&p, c.stream()), "l2norm_fwd");
  if (wants_grad(x)) {
    auto node = make_node<L2Node>(x);
    node->eps = eps;
    node->keep({x});
    attach(y, node);
  }
  return y;
}

struct RmsNode : public OpNode {
  double eps = 1e-5;
  variable_list apply(variable_list&& grads) override {
    variable_list t;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      t = unpack();
    }
    if (!grads[0].defined()) return variable_list(3);
    Call c(t[0]);
    Tensor x = c.in(t[0]), g = c.in(t[1]), w = c.in_as(t[2], at::kFloat), dy = c.in_as(grads[0], x.scalar_type());
    Tensor dx = c.empty_as(x), dg = c.empty_as(g), dw;
    if (w.defined()) dw = c.empty({x.size(-1)}, at::kFloat);
    tops_norm_params p = norm_params(x, eps);
    p.gate = ptr(g); p.weight = ptr<float>(w); p.dy = ptr(dy); p.dx = ptr(dx); p.dgate = ptr(dg); p.dweight = ptr<float>(dw);
    Tensor ws = c.bytes(tops_b200_rmsnorm_gated_bwd_workspace_bytes(&p));
    check(tops_b200_rmsnorm_gated_bwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "rmsnorm_gated_bwd");
    if (dw.defined() && t[2].scalar_type() != at::kFloat) dw = dw.to(t[2].scalar_type());
    return {dx, dg, dw};
  }
};
Tensor rmsnorm_gated(const Tensor& x, const Tensor& g, const OptTensor& w_, double eps) {
  Call c(x);
  const Tensor weight = opt(w_);
  Tensor xc = c.in(x), gc = c.in(g), w = c.in_as(weight, at::kFloat), y = c.empty_as(x);
  tops_norm_params p = norm_params(xc, eps);
  p.gate = ptr(gc); p.weight = ptr<float>(w); p.y = ptr(y);
  check(tops_b200_rmsnorm_gated_fwd(&p, c.stream()), "rmsnorm_gated_fwd");
  if (wants_grad(x, g, weight)) {
    auto node = make_node<RmsNode>(x, g, weight);
    node->eps = eps;
    node->keep({x, g, weight});
    attach(y, node);
  }
  return y;
}

}  // namespace

PYBIND11_MODULE(_torch_ops, m) {
  m.def("configure", [](py::object module) { g_module = module.inc_ref().ptr(); });
  m.def("chunk", &chunk);
  m.def("recurrent", &recurrent);
  m.def("recurrent_decode", &recurrent_decode);
  m.def("kda", &kda);
  m.def("kda_decode", &kda_decode);
  m.def("gate", &gate);
  m.def("l2norm", &l2norm);
  m.def("rmsnorm_gated", &rmsnorm_gated);
  m.def("gla_layer", &gla_layer);
  m.def("gla_layer_takes", &gla_layer_takes);
}
