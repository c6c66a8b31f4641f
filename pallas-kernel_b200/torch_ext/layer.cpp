// The GLA layer's forward and backward as one autograd node.
//
// Through torch modules a layer step is some 45 launches with 10 - 15 us of host work in front of most of them: at the
// default sizes (hidden 1024, 4 x 2048 tokens) the GPU waited for the host half of the time, at small ones always.
// Here the projections are plain matrix products of the flattened tokens (the same library GEMMs, for training the same
// calls the modules made, so q, k and v keep their bits), the low-rank gate is one kernel, and the backward lets every
// gradient kernel write its columns of ONE matrix [tokens, 2 K + 2 V + rank]: the input's gradient and the five input
// weights' gradients are then one product each instead of five products and four additions.  Without gradients the
// input weights are packed the same way and the attention reads its columns of the product's rows in place; up to 64
// tokens (a decode step) the projections run in the few-row kernel.
#include "common.h"

namespace tops_torch {
namespace {

struct Dims {
  int64_t B = 0, T = 0, n = 0, hid = 0, K = 0, V = 0, R = 0, H = 0;
  int64_t cols() const { return 2 * K + 2 * V + R; }
};
struct Law { double eps = 1e-5, normalizer = 16.0, clamp = 0.0; bool has_clamp = false; };

char* at_col(const Tensor& t, int64_t col) { return reinterpret_cast<char*>(t.data_ptr()) + col * 2; }

void lowrank_gate(const Call& c, const Dims& d, const Law& l, const void* low, int64_t low_pitch, const Tensor& W, const Tensor& b,
                  const Tensor& x, const Tensor& y) {
  tops_lowrank_gate_params p{};
  p.rows = d.n; p.low_pitch = low_pitch; p.R = (int)d.R; p.N = (int)d.K; p.dtype = TOPS_BF16;
  p.low = low; p.W = ptr(W); p.bias = ptr(b); p.normalizer = (float)l.normalizer; p.clamp_min = (float)l.clamp;
  p.has_clamp_min = l.has_clamp; p.x = ptr(x); p.y = ptr(y);
  check(tops_b200_lowrank_gate_fwd(&p, c.stream()), "lowrank_gate_fwd");
}
void norm_fwd(const Call& c, const Dims& d, const Law& l, const Tensor& o, const void* gate, int64_t gate_pitch, const Tensor& w,
              const Tensor& y) {
  tops_norm_params p{};
  p.rows = d.n * d.H; p.D = (int)(d.V / d.H); p.dtype = TOPS_BF16; p.eps = (float)l.eps; p.x = ptr(o); p.gate = gate;
  p.weight = ptr<float>(w); p.weight_dtype = w.defined() ? code_of(w) : TOPS_F32; p.y = ptr(y); p.gate_pitch = gate_pitch;
  p.heads = (int)d.H;
  check(tops_b200_rmsnorm_gated_fwd(&p, c.stream()), "rmsnorm_gated_fwd");
}
tops_chunk_problem problem(const Dims& d, const std::vector<int32_t>& cu) {
  tops_chunk_problem pb{};
  pb.B = (int)d.B; pb.T = (int)d.T; pb.H = (int)d.H; pb.K = (int)(d.K / d.H); pb.V = (int)(d.V / d.H); pb.chunk = 64;
  pb.dtype = pb.gate_dtype = TOPS_BF16; pb.gate_kind = TOPS_GATE_PER_CHANNEL; pb.impl = TOPS_IMPL_AUTO;
  pb.scale = (float)(1.0 / std::sqrt((double)(d.K / d.H)));
  if (!cu.empty()) { pb.cu_seqlens_host = cu.data(); pb.N = (int)cu.size() - 1; }
  return pb;
}

struct LayerNode : public OpNode {
  Dims d;
  Law law;
  std::vector<int32_t> cu;
  variable_list apply(variable_list&& grads) override {
    variable_list t;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      t = unpack();
    }
    const Tensor &x = t[0], &Wq = t[1], &Wk = t[2], &Wv = t[3], &Wg = t[4], &Wlow = t[5], &Wgk = t[6], &bgk = t[7], &nw = t[8],
                 &Wo = t[9], &h0 = t[10], &q = t[11], &k = t[12], &v = t[13], &g = t[14], &low = t[15], &raw = t[16], &gk = t[17],
                 &o = t[18], &on = t[19], &hs = t[20];
    at::NoGradGuard no_grad;
    Call c(x);
    const int64_t cols = d.cols();
    Tensor dout = cotangent(grads[0], x, at::kBFloat16, c).view({d.n, d.hid});
    Tensor dht = grads.size() > 1 ? c.in_as(grads[1], at::kFloat) : Tensor();
    Tensor x2 = x.view({d.n, d.hid});
    Tensor dWo;
    if (task_should_compute_output(9)) dWo = at::mm(dout.t(), on);
    Tensor don = at::mm(dout, Wo);
    // columns of dY: dq | dk | dv | dg | dlow
    Tensor dY = c.empty({d.n, cols}, at::kBFloat16);
    Tensor d_o = c.empty({d.n, d.V}, at::kBFloat16), dnw;
    {
      tops_norm_params p{};
      p.rows = d.n * d.H; p.D = (int)(d.V / d.H); p.dtype = TOPS_BF16; p.eps = (float)law.eps; p.x = ptr(o); p.gate = ptr(g);
      p.weight = ptr<float>(nw); p.weight_dtype = nw.defined() ? code_of(nw) : TOPS_F32; p.heads = (int)d.H;
      p.dy = ptr(don); p.dx = ptr(d_o); p.dgate = at_col(dY, 2 * d.K + d.V); p.dgate_pitch = cols;
      if (nw.defined()) { dnw = c.empty({d.V / d.H}, at::kFloat); p.dweight = ptr<float>(dnw); }
      Tensor ws = c.bytes(tops_b200_rmsnorm_gated_bwd_workspace_bytes(&p));
      check(tops_b200_rmsnorm_gated_bwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "rmsnorm_gated_bwd");
      if (dnw.defined() && nw.scalar_type() != at::kFloat) dnw = dnw.to(nw.scalar_type());
    }
    Tensor dgk = c.empty({d.n, d.K}, at::kBFloat16), dh0;
    {
      Tensor h0c = c.in_as(h0, at::kFloat);
      tops_chunk_bwd_params p{};
      p.pb = problem(d, cu);
      if (h0.defined()) dh0 = c.empty(h0.sizes(), at::kFloat);
      p.q = ptr(q); p.k = ptr(k); p.v = ptr(v); p.g = ptr(gk); p.h0 = ptr<float>(h0c); p.do_ = ptr(d_o); p.dht = ptr<float>(dht);
      p.dq = at_col(dY, 0); p.dk = at_col(dY, d.K); p.dv = at_col(dY, 2 * d.K); p.dg = ptr(dgk); p.dh0 = ptr<float>(dh0);
      p.grad_dtype = p.dg_dtype = TOPS_BF16; p.h_saved = ptr(hs); p.saved_bytes = hs.nbytes(); p.grad_pitch = cols;
      Tensor ws = c.bytes(tops_b200_chunk_bwd_workspace_bytes(&p));
      check(tops_b200_chunk_gla_bwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "chunk_gla_bwd");
      check_device_word("layer backward");
      if (dh0.defined() && h0.scalar_type() != at::kFloat) dh0 = dh0.to(h0.scalar_type());
    }
    Tensor draw = c.empty({d.n, d.K}, at::kBFloat16), dWgk, dbgk;
    {
      tops_gate_act_bwd_params p{};
      p.fwd.rows = d.n; p.fwd.H = 1; p.fwd.K = (int)d.K; p.fwd.kind = TOPS_GATE_ACT_LOG_SIGMOID; p.fwd.dtype = p.fwd.out_dtype = TOPS_BF16;
      p.fwd.g = ptr(raw); p.fwd.normalizer = (float)law.normalizer; p.fwd.clamp_min = (float)law.clamp; p.fwd.has_clamp_min = law.has_clamp;
      p.dy = ptr(dgk); p.dy_dtype = TOPS_BF16; p.dg = ptr(draw);
      if (task_should_compute_output(7)) { dbgk = c.empty({d.K}, at::kFloat); p.dbias = ptr<float>(dbgk); }   // column sums of draw
      Tensor ws = c.bytes(tops_b200_gate_act_bwd_workspace_bytes(&p));
      check(tops_b200_gate_act_bwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "gate_act_bwd");
    }
    if (task_should_compute_output(6)) dWgk = at::mm(draw.t(), low);
    if (dbgk.defined()) dbgk = dbgk.to(at::kBFloat16);
    Tensor dlow = dY.narrow(1, cols - d.R, d.R);
    at::mm_out(dlow, draw, Wgk);
    Tensor dx, dWq, dWk, dWv, dWg, dWlow;
    if (task_should_compute_output(0)) dx = at::mm(dY, at::cat({Wq, Wk, Wv, Wg, Wlow}, 0)).view(x.sizes());
    if (task_should_compute_output(1) || task_should_compute_output(2) || task_should_compute_output(3) || task_should_compute_output(4) ||
        task_should_compute_output(5)) {
      const Tensor dW = at::mm(dY.t(), x2);
      dWq = dW.narrow(0, 0, d.K); dWk = dW.narrow(0, d.K, d.K); dWv = dW.narrow(0, 2 * d.K, d.V);
      dWg = dW.narrow(0, 2 * d.K + d.V, d.V); dWlow = dW.narrow(0, 2 * d.K + 2 * d.V, d.R);
    }
    return {dx, dWq, dWk, dWv, dWg, dWlow, dWgk, dbgk, dnw, dWo, dh0};
  }
};

// up to 64 tokens, no gradients: few-row projections, token recurrence
std::tuple<Tensor, OptTensor> step(const Call& c, const Dims& d, const Law& l, const Tensor& x, const Tensor& Wq, const Tensor& Wk,
                                   const Tensor& Wv, const Tensor& Wg, const Tensor& Wlow, const Tensor& Wgk, const Tensor& bgk,
                                   const Tensor& nw, const Tensor& Wo, const Tensor& h0, bool want_state, const std::vector<int32_t>& cu) {
  const int64_t cols = d.cols(), N = cu.empty() ? d.B : (int64_t)cu.size() - 1;
  Tensor Y = c.empty({d.n, cols}, at::kBFloat16);
  {
    tops_skinny_linear_params p{};
    p.rows = (int)d.n; p.K = (int)d.hid; p.x_pitch = d.hid; p.x = ptr(x);
    const Tensor* w[5] = {&Wq, &Wk, &Wv, &Wg, &Wlow};
    int64_t col = 0;
    for (const Tensor* t : w) {
      const int i = p.count++;
      p.W[i] = ptr(*t); p.N[i] = (int)t->size(0); p.y[i] = at_col(Y, col); p.y_pitch[i] = cols;
      col += t->size(0);
    }
    check(tops_b200_skinny_linear(&p, c.stream()), "skinny_linear");
  }
  Tensor gk = c.empty({d.n, d.K}, at::kBFloat16);
  lowrank_gate(c, d, l, at_col(Y, cols - d.R), cols, Wgk, bgk, Tensor(), gk);
  Tensor o = c.empty({d.n, d.V}, at::kBFloat16), ht, cu_dev;
  if (want_state) ht = c.empty({N, d.H, d.K / d.H, d.V / d.H}, at::kFloat);
  {
    Tensor h0c = c.in_as(h0, at::kFloat);
    tops_recurrent_fwd_params p{};
    p.B = (int)d.B; p.T = (int)d.T; p.H = (int)d.H; p.K = (int)(d.K / d.H); p.V = (int)(d.V / d.H);
    p.dtype = p.gate_dtype = p.o_dtype = TOPS_BF16; p.scale = (float)(1.0 / std::sqrt((double)(d.K / d.H)));
    p.q = at_col(Y, 0); p.k = at_col(Y, d.K); p.v = at_col(Y, 2 * d.K); p.gk = ptr(gk); p.pitch = cols;
    p.state_in = ptr<float>(h0c); p.state_out = ptr<float>(ht); p.o = ptr(o); p.N = (int)N;
    if (!cu.empty()) {
      cu_dev = at::tensor(at::ArrayRef<int32_t>(cu), at::TensorOptions().dtype(at::kInt)).to(c.dev);
      p.cu_seqlens = cu_dev.data_ptr<int32_t>();
    }
    check(tops_b200_fused_recurrent_gla_fwd(&p, c.stream()), "fused_recurrent_gla_fwd");
  }
  Tensor on = c.empty({d.n, d.V}, at::kBFloat16), out = c.empty({d.B, d.T, d.hid}, at::kBFloat16);
  norm_fwd(c, d, l, o, at_col(Y, 2 * d.K + d.V), cols, nw, on);
  tops_skinny_linear_params p{};
  p.rows = (int)d.n; p.K = (int)d.V; p.x_pitch = d.V; p.x = ptr(on); p.count = 1; p.W[0] = ptr(Wo); p.N[0] = (int)d.hid;
  p.y[0] = ptr(out); p.y_pitch[0] = d.hid;
  check(tops_b200_skinny_linear(&p, c.stream()), "skinny_linear");
  return {out, ht.defined() ? OptTensor(ht) : std::nullopt};
}

// more tokens, no gradients: packed input projection, attention on its columns
std::tuple<Tensor, OptTensor> prompt(const Call& c, const Dims& d, const Law& l, const Tensor& x, const Tensor& Wq, const Tensor& Wk,
                                     const Tensor& Wv, const Tensor& Wg, const Tensor& Wlow, const Tensor& Wgk, const Tensor& bgk,
                                     const Tensor& nw, const Tensor& Wo, const Tensor& h0, bool want_state, const std::vector<int32_t>& cu) {
  const int64_t cols = d.cols(), N = cu.empty() ? d.B : (int64_t)cu.size() - 1;
  Tensor Y = at::mm(x.view({d.n, d.hid}), at::cat({Wq, Wk, Wv, Wg, Wlow}, 0).t());
  Tensor gk = c.empty({d.n, d.K}, at::kBFloat16);
  lowrank_gate(c, d, l, at_col(Y, cols - d.R), cols, Wgk, bgk, Tensor(), gk);
  Tensor o = c.empty({d.n, d.V}, at::kBFloat16), ht;
  if (want_state) ht = c.empty({N, d.H, d.K / d.H, d.V / d.H}, at::kFloat);
  {
    Tensor h0c = c.in_as(h0, at::kFloat);
    tops_chunk_fwd_params p{};
    p.pb = problem(d, cu);
    p.q = at_col(Y, 0); p.k = at_col(Y, d.K); p.v = at_col(Y, 2 * d.K); p.g = ptr(gk); p.h0 = ptr<float>(h0c); p.o = ptr(o);
    p.ht = ptr<float>(ht); p.pitch = cols;
    Tensor ws = c.bytes(tops_b200_chunk_fwd_workspace_bytes(&p));
    check(tops_b200_chunk_gla_fwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "chunk_gla_fwd");
  }
  Tensor on = c.empty({d.n, d.V}, at::kBFloat16);
  norm_fwd(c, d, l, o, at_col(Y, 2 * d.K + d.V), cols, nw, on);
  return {at::mm(on, Wo.t()).view({d.B, d.T, d.hid}), ht.defined() ? OptTensor(ht) : std::nullopt};
}

}  // namespace

// bf16 on the GPU at sizes every kernel of the path takes, and weights that fit the input and one another: nothing below
// checks a shape, the few-row kernel reads hid columns of every row whatever a weight holds.  (What does not fit goes
// through the modules, which refuse it by name.)
bool gla_layer_takes(const Tensor& x, const Tensor& Wq, const Tensor& Wk, const Tensor& Wv, const Tensor& Wg, const Tensor& Wlow,
                     const Tensor& Wgk, const Tensor& bgk, const OptTensor& nw, const Tensor& Wo, int heads, bool recurrent) {
  if (!x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.dim() != 3) return false;
  const int64_t hid = x.size(2), key_dim = Wq.size(0), value_dim = Wv.size(0), rank = Wlow.size(0);
  auto like = [&](const Tensor& w, at::IntArrayRef sizes) {
    return w.scalar_type() == at::kBFloat16 && w.device() == x.device() && w.sizes() == sizes && w.is_contiguous() &&
           (reinterpret_cast<uintptr_t>(w.data_ptr()) & 15) == 0;
  };
  if (!like(Wq, {key_dim, hid}) || !like(Wk, {key_dim, hid}) || !like(Wv, {value_dim, hid}) || !like(Wg, {value_dim, hid}) ||
      !like(Wlow, {rank, hid}) || !like(Wgk, {key_dim, rank}) || !like(bgk, {key_dim}) || !like(Wo, {hid, value_dim}))
    return false;
  if (key_dim % heads != 0 || value_dim % heads != 0) return false;
  if (nw.has_value() && (nw->device() != x.device() || nw->dim() != 1 || nw->size(0) != value_dim / heads || !nw->is_contiguous() ||
                         (reinterpret_cast<uintptr_t>(nw->data_ptr()) & 15) != 0 ||
                         (nw->scalar_type() != at::kFloat && nw->scalar_type() != at::kBFloat16 && nw->scalar_type() != at::kHalf)))
    return false;
  const int64_t K = key_dim / heads, V = value_dim / heads, n = x.size(0) * x.size(1);
  if (n < 1 || x.size(2) % 32 != 0 || key_dim % 8 != 0 || value_dim % 32 != 0 || rank < 8 || rank > 64 || rank % 8 != 0) return false;
  if (V % 4 != 0 || V > 1024) return false;
  if (recurrent) return n <= 64 && K <= 256 && !at::GradMode::is_enabled();
  tops_chunk_problem pb{};
  pb.B = (int)x.size(0); pb.T = (int)x.size(1); pb.H = heads; pb.K = (int)K; pb.V = (int)V; pb.chunk = 64; pb.dtype = pb.gate_dtype = TOPS_BF16;
  pb.gate_kind = TOPS_GATE_PER_CHANNEL; pb.impl = TOPS_IMPL_AUTO; pb.scale = 1.f;
  return tops_b200_chunk_selected_impl(&pb) == TOPS_IMPL_SM100 && K >= 32 && K <= 128 && K % 8 == 0 && V >= 32 && V % 8 == 0;
}

std::tuple<Tensor, OptTensor> gla_layer(const Tensor& x_, const Tensor& Wq, const Tensor& Wk, const Tensor& Wv, const Tensor& Wg,
                                        const Tensor& Wlow, const Tensor& Wgk, const Tensor& bgk, const OptTensor& norm_weight,
                                        const Tensor& Wo, int heads, double eps, double normalizer, std::optional<double> clamp,
                                        const OptTensor& state, bool want_state, std::vector<int32_t> cu, bool recurrent) {
  Call c(x_);
  const Tensor nw = opt(norm_weight), h0 = opt(state);
  Dims d;
  d.B = x_.size(0); d.T = x_.size(1); d.n = d.B * d.T; d.hid = x_.size(2); d.K = Wq.size(0); d.V = Wv.size(0); d.R = Wlow.size(0); d.H = heads;
  const Law l{eps, normalizer, clamp.value_or(0.0), clamp.has_value()};
  const bool grad = wants_grad(x_, Wq, Wk, Wv, Wg, Wlow, Wgk, bgk, nw, Wo, h0);
  if (!grad) {
    const Tensor x = c.in(x_);
    return recurrent ? step(c, d, l, x, c.in(Wq), c.in(Wk), c.in(Wv), c.in(Wg), c.in(Wlow), c.in(Wgk), c.in(bgk), c.in(nw), c.in(Wo), h0, want_state, cu)
                     : prompt(c, d, l, x, Wq, Wk, Wv, Wg, Wlow, c.in(Wgk), c.in(bgk), c.in(nw), Wo, h0, want_state, cu);
  }
  TORCH_CHECK(!recurrent, "the token recurrence of the layer is differentiated through its module");
  Tensor x, q, k, v, g, low, raw, gk, o, on, out, ht, hs;
  {
    at::NoGradGuard no_grad;
    x = c.in(x_);
    const Tensor x2 = x.view({d.n, d.hid});
    q = at::mm(x2, Wq.t()); k = at::mm(x2, Wk.t()); v = at::mm(x2, Wv.t()); g = at::mm(x2, Wg.t()); low = at::mm(x2, Wlow.t());
    raw = c.empty({d.n, d.K}, at::kBFloat16);
    gk = c.empty({d.n, d.K}, at::kBFloat16);
    lowrank_gate(c, d, l, ptr(low), d.R, c.in(Wgk), c.in(bgk), raw, gk);
    o = c.empty({d.n, d.V}, at::kBFloat16);
    const int64_t N = cu.empty() ? d.B : (int64_t)cu.size() - 1;
    if (want_state) ht = c.empty({N, d.H, d.K / d.H, d.V / d.H}, at::kFloat);
    Tensor h0c = c.in_as(h0, at::kFloat);
    tops_chunk_fwd_params p{};
    p.pb = problem(d, cu);
    p.q = ptr(q); p.k = ptr(k); p.v = ptr(v); p.g = ptr(gk); p.h0 = ptr<float>(h0c); p.o = ptr(o); p.ht = ptr<float>(ht);
    hs = c.empty({(int64_t)(tops_b200_chunk_saved_bytes(&p.pb) / 2)}, at::kBFloat16);
    p.saved_out = ptr(hs);
    p.saved_bytes = hs.nbytes();
    Tensor ws = c.bytes(tops_b200_chunk_fwd_workspace_bytes(&p));
    check(tops_b200_chunk_gla_fwd(&p, ws.data_ptr(), (size_t)ws.numel(), c.stream()), "chunk_gla_fwd");
    on = c.empty({d.n, d.V}, at::kBFloat16);
    norm_fwd(c, d, l, o, ptr(g), 0, c.in(nw), on);
    // (not a view: autograd refuses in-place operations on a view made without gradients)
    out = c.empty({d.B, d.T, d.hid}, at::kBFloat16);
    Tensor rows = out.view({d.n, d.hid});
    at::mm_out(rows, on, Wo.t());
  }
  auto node = make_node<LayerNode>(x_, Wq, Wk, Wv, Wg, Wlow, Wgk, bgk, nw, Wo, h0);
  node->d = d; node->law = l; node->cu = std::move(cu);
  node->keep({x, Wq, Wk, Wv, Wg, Wlow, Wgk, bgk, nw, Wo, h0, q, k, v, g, low, raw, gk, o, on, hs});
  attach(out, node);
  attach(ht, node);
  return {out, ht.defined() ? OptTensor(ht) : std::nullopt};
}

}  // namespace tops_torch
