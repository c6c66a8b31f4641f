// The steps either side of the attention kernels: gate activations (and their backward with the
// parameter reductions), q/k L2 normalisation, and the gated RMS norm of the output.  All are one pass
// over HBM: every input is read once and every output written once.  Column reductions (dA_log, d dt_bias,
// d weight) go through per-block partial sums that a second kernel adds in a fixed order.
//
// All of them are bound by how many bytes a thread keeps in flight: at 6.5 TB/s and about 0.8 us of latency an
// SM needs some 35 KB of loads outstanding.  So a thread moves VW = 8 elements per access (16 bytes of bf16) and
// issues the loads of U rows before it uses the first; rows narrower than a warp share it, LPR lanes each.
// The form before, one row per warp and one 8-byte access at a time, reached 0.9 - 2.2 TB/s.  On
// [8, 4096, 16, 128] bf16 (134 MB per tensor), us per launch before -> now: l2norm forward 150 -> 46 (5.9 TB/s),
// backward 440 -> 64 (6.3); gated RMS norm forward 250 -> 65 (6.2), backward 530 -> 117 (5.7); KDA gate forward
// 230 -> 56 (4.8), backward 220 -> 87 (4.6), log-sigmoid gate backward -> 68 (5.9).  The KDA gate is the one that
// arithmetic holds back: about 25 instructions per element on top of its two or three memory accesses.
#include <type_traits>

#include "elementwise.cuh"

namespace tops {
namespace elementwise {
namespace {

// VW consecutive elements of T as they lie in memory (loads stay in this form until they are used: half the
// registers of the widened values) and as floats
template <class T, int VW> struct Vec;
template <int VW> struct Vec<float, VW> {
  struct Raw { float4 x[VW / 4]; };
  static __device__ __forceinline__ void load(const float* p, Raw& r) {
#pragma unroll
    for (int i = 0; i < VW / 4; ++i) r.x[i] = reinterpret_cast<const float4*>(p)[i];
  }
  static __device__ __forceinline__ void clear(Raw& r) {
#pragma unroll
    for (int i = 0; i < VW / 4; ++i) r.x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  static __device__ __forceinline__ void widen(const Raw& r, float (&v)[VW]) {
#pragma unroll
    for (int i = 0; i < VW / 4; ++i) { v[4 * i] = r.x[i].x; v[4 * i + 1] = r.x[i].y; v[4 * i + 2] = r.x[i].z; v[4 * i + 3] = r.x[i].w; }
  }
  static __device__ __forceinline__ void load(const float* p, float (&v)[VW]) {
    Raw r;
    load(p, r);
    widen(r, v);
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[VW]) {
#pragma unroll
    for (int i = 0; i < VW; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
  }
};
template <class T> struct Pair;
template <> struct Pair<__nv_bfloat16> {
  static __device__ __forceinline__ float2 get(uint32_t x) { return make_float2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u)); }
  static __device__ __forceinline__ uint32_t put(float a, float b) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&t);
  }
};
template <> struct Pair<__half> {
  static __device__ __forceinline__ float2 get(uint32_t x) { return __half22float2(*reinterpret_cast<const __half2*>(&x)); }
  static __device__ __forceinline__ uint32_t put(float a, float b) {
    const __half2 t = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&t);
  }
};
template <class T, int VW> struct HalfVec {
  struct Raw { uint32_t w[VW / 2]; };
  static __device__ __forceinline__ void load(const T* p, Raw& r) {
    if constexpr (VW == 8) {
      const uint4 x = *reinterpret_cast<const uint4*>(p);
      r.w[0] = x.x; r.w[1] = x.y; r.w[2] = x.z; r.w[3] = x.w;
    } else {
      const uint2 x = *reinterpret_cast<const uint2*>(p);
      r.w[0] = x.x; r.w[1] = x.y;
    }
  }
  static __device__ __forceinline__ void clear(Raw& r) {
#pragma unroll
    for (int i = 0; i < VW / 2; ++i) r.w[i] = 0u;
  }
  static __device__ __forceinline__ void widen(const Raw& r, float (&v)[VW]) {
#pragma unroll
    for (int i = 0; i < VW / 2; ++i) {
      const float2 a = Pair<T>::get(r.w[i]);
      v[2 * i] = a.x; v[2 * i + 1] = a.y;
    }
  }
  static __device__ __forceinline__ void load(const T* p, float (&v)[VW]) {
    Raw r;
    load(p, r);
    widen(r, v);
  }
  static __device__ __forceinline__ void store(T* p, const float (&v)[VW]) {
    if constexpr (VW == 8)
      *reinterpret_cast<uint4*>(p) = make_uint4(Pair<T>::put(v[0], v[1]), Pair<T>::put(v[2], v[3]), Pair<T>::put(v[4], v[5]),
                                                Pair<T>::put(v[6], v[7]));
    else *reinterpret_cast<uint2*>(p) = make_uint2(Pair<T>::put(v[0], v[1]), Pair<T>::put(v[2], v[3]));
  }
};
template <int VW> struct Vec<__nv_bfloat16, VW> : HalfVec<__nv_bfloat16, VW> {};
template <int VW> struct Vec<__half, VW> : HalfVec<__half, VW> {};

// The hardware's exp2 and reciprocal units, one instruction each: the arguments here never need range scaling
// (results below 2^-126 flush to zero, 1 / infinity is 0).
__device__ __forceinline__ float exp_unit(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
  return y;
}
__device__ __forceinline__ float rcp_unit(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// EXACT: CUDA's division and log1pf.  For results that are kept in fp32, where what the units and the polynomial below leave
// (2e-7) shows: gates and norms of fp32 tensors were 1 - 5 % further from fp64 with them.
template <bool EXACT> __device__ __forceinline__ float reciprocal(float x) { return EXACT ? 1.f / x : rcp_unit(x); }
template <bool EXACT> __device__ __forceinline__ float exponential(float x) { return EXACT ? __expf(x) : exp_unit(x); }
template <bool EXACT> __device__ __forceinline__ float sigmoidf(float x) { return reciprocal<EXACT>(1.f + exponential<EXACT>(-x)); }
// log(1 + t) for 0 <= t <= 1 as t times a polynomial, a Chebyshev fit of log(1 + t) / t on [0, 1]: relative error
// below 2e-7 in fp32, no cancellation for small t, no division
__device__ __forceinline__ float log1p_unit(float t) {
  float p = 0.00525345793f;
  p = fmaf(p, t, -0.0295885075f);
  p = fmaf(p, t, 0.0783616677f);
  p = fmaf(p, t, -0.136747703f);
  p = fmaf(p, t, 0.191114306f);
  p = fmaf(p, t, -0.248443693f);
  p = fmaf(p, t, 0.333192706f);
  p = fmaf(p, t, -0.499995023f);
  p = fmaf(p, t, 1.f);
  return p * t;
}
// with t = exp(-|x|): softplus(x) = max(x, 0) + log(1 + t), sigmoid(x) = 1 / (1 + t) or t / (1 + t)
template <bool EXACT> __device__ __forceinline__ float softplusf(float x) {
  const float t = exponential<EXACT>(-fabsf(x));
  return fmaxf(x, 0.f) + (EXACT ? log1pf(t) : log1p_unit(t));
}
template <bool EXACT> __device__ __forceinline__ void softplus_sigmoid(float x, float& sp, float& sg) {
  const float t = exponential<EXACT>(-fabsf(x)), i1 = reciprocal<EXACT>(1.f + t);
  sp = fmaxf(x, 0.f) + (EXACT ? log1pf(t) : log1p_unit(t));
  sg = EXACT ? sigmoidf<true>(x) : x >= 0.f ? i1 : t * i1;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
// sum of a thread's products; fp32 tensors: in two halves, whose rounding is what four elements at a time had
template <class T, int VW>
__device__ __forceinline__ float sum_products(const float (&v)[VW], const float (&w)[VW]) {
  constexpr int N = std::is_same<T, float>::value && VW == 8 ? 4 : VW;
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < VW; c += N) {
    float h = 0.f;
#pragma unroll
    for (int t = c; t < c + N; ++t) h = fmaf(v[t], w[t], h);
    s += h;
  }
  return s;
}
// sum over the 2^LG neighbouring lanes that share a row
template <int LG>   // log2 of the lanes
__device__ __forceinline__ float row_sum(float x) {
#pragma unroll
  for (int o = (1 << LG) >> 1; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// ---------------------------------------------------------------------------
// gate activations
// ---------------------------------------------------------------------------
// A thread owns VW columns of the H*K and walks rows, so that a column's bias and exp(A_log) stay in registers.
// Block (x: row lanes x column threads, blockIdx.y: groups of 256 column threads).
struct GateConst {
  const float* A_log;    // [H] (KDA kinds)
  const float* dt_bias;  // [H*K] or null
  float lower_bound, normalizer, inv_normalizer, clamp_min;
  int has_clamp;
};
struct GateThread { int col; size_t row, step; bool on; };
template <int VW>
__device__ __forceinline__ GateThread gate_thread(int HK) {
  const int cv = HK / VW, per = cv < 256 ? cv : 256, lanes = 256 / per;
  GateThread t;
  const int rl = threadIdx.x / per, c = blockIdx.y * per + threadIdx.x - rl * per;
  t.on = rl < lanes && c < cv;
  t.col = c * VW;
  t.row = (size_t)blockIdx.x * lanes + rl;
  t.step = (size_t)gridDim.x * lanes;
  return t;
}

template <class TI, class TO, int KIND, int VW>
__global__ void __launch_bounds__(256) k_gate_fwd(const TI* __restrict__ g, TO* __restrict__ out, size_t rows, int H, int K,
                                                  GateConst c) {
  constexpr int U = 4;
  constexpr bool EXACT = std::is_same<TO, float>::value;
  const int HK = H * K;
  const GateThread th = gate_thread<VW>(HK);
  if (!th.on) return;
  float bias[VW], eA = 0.f;
#pragma unroll
  for (int t = 0; t < VW; ++t) bias[t] = 0.f;
  if (KIND != TOPS_GATE_ACT_LOG_SIGMOID) {
    eA = __expf(c.A_log[th.col / K]);
    if (c.dt_bias) Vec<float, VW>::load(c.dt_bias + th.col, bias);
  }
  for (size_t r0 = th.row; r0 < rows; r0 += th.step * U) {
    typename Vec<TI, VW>::Raw raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (r0 + u * th.step < rows) Vec<TI, VW>::load(g + (r0 + u * th.step) * HK + th.col, raw[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (r0 + u * th.step >= rows) break;
      float x[VW], y[VW];
      Vec<TI, VW>::widen(raw[u], x);
#pragma unroll
      for (int t = 0; t < VW; ++t) {
        const float xb = x[t] + bias[t];
        if (KIND == TOPS_GATE_ACT_KDA) y[t] = -eA * softplusf<EXACT>(xb);
        else if (KIND == TOPS_GATE_ACT_KDA_LOWER_BOUND) y[t] = c.lower_bound * sigmoidf<EXACT>(eA * xb);
        else {
          y[t] = EXACT ? -softplusf<true>(-xb) / c.normalizer : -softplusf<false>(-xb) * c.inv_normalizer;   // log_sigmoid(x) = -softplus(-x)
          if (c.has_clamp && y[t] < c.clamp_min) y[t] = c.clamp_min;
        }
      }
      Vec<TO, VW>::store(out + (r0 + u * th.step) * HK + th.col, y);
    }
  }
}

// Backward: dg per element; per block and column, the sums that become d dt_bias (sum of dg) and dA_log (sum of
// dy * y, or of dg * x for the lower-bound form).
template <class TI, class TD, int KIND, int VW>
__global__ void __launch_bounds__(256) k_gate_bwd(const TI* __restrict__ g, const TD* __restrict__ dy, TI* __restrict__ dg,
                                                  size_t rows, int H, int K, GateConst c, float* __restrict__ part_bias,
                                                  float* __restrict__ part_A) {
  // rows in flight, measured on [8, 4096, 16, 128] bf16: the KDA law 87 us with four and 104 with two, log-sigmoid 67
  // with two and 77 with four
  constexpr int U = KIND == TOPS_GATE_ACT_LOG_SIGMOID ? 2 : 4;
  // (the lower-bound law's dA_log is a small rest of large terms)
  constexpr bool EXACT = std::is_same<TI, float>::value || KIND == TOPS_GATE_ACT_KDA_LOWER_BOUND;
  const int HK = H * K;
  const GateThread th = gate_thread<VW>(HK);
  float bias[VW], sb[VW], sa[VW], eA = 0.f;
#pragma unroll
  for (int t = 0; t < VW; ++t) bias[t] = sb[t] = sa[t] = 0.f;
  if (th.on) {
    if (KIND != TOPS_GATE_ACT_LOG_SIGMOID) {
      eA = __expf(c.A_log[th.col / K]);
      if (c.dt_bias) Vec<float, VW>::load(c.dt_bias + th.col, bias);
    }
    for (size_t r0 = th.row; r0 < rows; r0 += th.step * U) {
      typename Vec<TI, VW>::Raw rx[U];
      typename Vec<TD, VW>::Raw rd[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (r0 + u * th.step < rows) {
          Vec<TI, VW>::load(g + (r0 + u * th.step) * HK + th.col, rx[u]);
          Vec<TD, VW>::load(dy + (r0 + u * th.step) * HK + th.col, rd[u]);
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (r0 + u * th.step >= rows) break;
        float x[VW], d[VW], o[VW];
        Vec<TI, VW>::widen(rx[u], x);
        Vec<TD, VW>::widen(rd[u], d);
#pragma unroll
        for (int t = 0; t < VW; ++t) {
          const float xb = x[t] + bias[t];
          if (KIND == TOPS_GATE_ACT_KDA) {
            float sp, sg;
            softplus_sigmoid<EXACT>(xb, sp, sg);
            const float ed = -eA * d[t];
            o[t] = ed * sg;
            sa[t] = fmaf(ed, sp, sa[t]);
          } else if (KIND == TOPS_GATE_ACT_KDA_LOWER_BOUND) {
            const float s = sigmoidf<EXACT>(eA * xb);
            o[t] = d[t] * c.lower_bound * s * (1.f - s) * eA;
            sa[t] = fmaf(o[t], xb, sa[t]);
          } else {
            float sp, sg;
            softplus_sigmoid<EXACT>(-xb, sp, sg);   // log_sigmoid(x) = -softplus(-x), 1 - sigmoid(x) = sigmoid(-x)
            o[t] = (c.has_clamp && -sp * c.inv_normalizer < c.clamp_min) ? 0.f : d[t] * sg * c.inv_normalizer;
          }
          sb[t] += o[t];
        }
        Vec<TI, VW>::store(dg + (r0 + u * th.step) * HK + th.col, o);
      }
    }
  }
  // the row lanes of a block that share columns are added in order
  const int cv = HK / VW, per = cv < 256 ? cv : 256, lanes = 256 / per;
  if (lanes > 1) {
    __shared__ float sm[256][VW + 1];
    for (int pass = 0; pass < 2; ++pass) {
      if (!(pass ? part_A : part_bias)) continue;   // uniform over the block
#pragma unroll
      for (int t = 0; t < VW; ++t) sm[threadIdx.x][t] = pass ? sa[t] : sb[t];
      __syncthreads();
      if ((int)threadIdx.x < per) {
        float s[VW];
#pragma unroll
        for (int t = 0; t < VW; ++t) s[t] = 0.f;
        for (int l = 0; l < lanes; ++l)
#pragma unroll
          for (int t = 0; t < VW; ++t) s[t] += sm[l * per + threadIdx.x][t];
        if (th.on) Vec<float, VW>::store((pass ? part_A : part_bias) + (size_t)blockIdx.x * HK + th.col, s);
      }
      __syncthreads();
    }
    return;
  }
  if (!th.on) return;
  if (part_bias) Vec<float, VW>::store(part_bias + (size_t)blockIdx.x * HK + th.col, sb);
  if (part_A) Vec<float, VW>::store(part_A + (size_t)blockIdx.x * HK + th.col, sa);
}

// out[col] = sum over row blocks of part[blk][col]: 32 columns x 32 row lanes per block, every lane walks its
// rows in order and the 32 lane sums are added in order, so the result does not depend on scheduling
__global__ void __launch_bounds__(1024) k_sum_blocks(const float* __restrict__ part, int nblk, int ncol,
                                                     float* __restrict__ out) {
  __shared__ float sm[32][33];
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + cx;
  float s = 0.f;
  if (col < ncol)
    for (int b = ry; b < nblk; b += 32) s += part[(size_t)b * ncol + col];
  sm[ry][cx] = s;
  __syncthreads();
  if (ry == 0 && col < ncol) {
    float t = 0.f;
#pragma unroll
    for (int r = 0; r < 32; ++r) t += sm[r][cx];
    out[col] = t;
  }
}
// dA[h] = sum over row blocks and the K columns of head h; one block of 32 warps per head, warp w takes the
// row blocks w, w + 32, ...
__global__ void __launch_bounds__(1024) k_sum_heads(const float* __restrict__ part, int nblk, int H, int K,
                                                    float* __restrict__ out) {
  __shared__ float sm[32];
  const int h = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float s = 0.f;
  for (int b = w; b < nblk; b += 32)
    for (int k = lane; k < K; k += 32) s += part[((size_t)b * H + h) * K + k];
  s = warp_sum(s);
  if (lane == 0) sm[w] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) t += sm[i];
    out[h] = t;
  }
}


// ---------------------------------------------------------------------------
// Row kernels (D <= 1024, D % 4 == 0): LPR = 2^LG neighbouring lanes share a row, lane j of them holds the vectors
// j, j + LPR, ... (NV of them); a block of 256 threads takes U x 256 / LPR rows at a time.
// ---------------------------------------------------------------------------
// rows a thread has in flight: kernels of one and of two input tensors
template <int NV> constexpr int rows_in_flight() { return NV == 1 ? 4 : NV == 2 ? 2 : 1; }
template <int NV> constexpr int rows_in_flight2() { return NV == 1 ? 2 : 1; }

template <class T, int VW, int NV, int LG>
__global__ void __launch_bounds__(256) k_l2norm_fwd(const T* __restrict__ x, T* __restrict__ y, float* __restrict__ rstd,
                                                    size_t rows, int D, float eps) {
  constexpr int U = rows_in_flight<NV>();
  constexpr int LPR = 1 << LG, per = 256 / LPR;
  const int lr = threadIdx.x & (LPR - 1);
  const size_t r0 = (size_t)blockIdx.x * per * U + threadIdx.x / LPR;
  typename Vec<T, VW>::Raw raw[U][NV];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int c = (n * LPR + lr) * VW;
      Vec<T, VW>::clear(raw[u][n]);
      if (r0 + u * per < rows && c < D) Vec<T, VW>::load(x + (r0 + u * per) * D + c, raw[u][n]);
    }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    float ss = 0.f, v[NV][VW];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      Vec<T, VW>::widen(raw[u][n], v[n]);
      ss += sum_products<T>(v[n], v[n]);
    }
    ss = row_sum<LG>(ss);
    const float r = rsqrtf(ss + eps);
    const size_t row = r0 + u * per;
    if (row < rows) {
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        const int c = (n * LPR + lr) * VW;
        float o[VW];
#pragma unroll
        for (int t = 0; t < VW; ++t) o[t] = v[n][t] * r;
        if (c < D) Vec<T, VW>::store(y + row * D + c, o);
      }
      if (rstd && lr == 0) rstd[row] = r;
    }
  }
}

// dx = r (dy - y (dy . y)) with y = x r
template <class T, int VW, int NV, int LG>
__global__ void __launch_bounds__(256) k_l2norm_bwd(const T* __restrict__ x, const T* __restrict__ dy, T* __restrict__ dx,
                                                    size_t rows, int D, float eps) {
  constexpr int U = rows_in_flight2<NV>();
  constexpr int LPR = 1 << LG, per = 256 / LPR;
  const int lr = threadIdx.x & (LPR - 1);
  const size_t r0 = (size_t)blockIdx.x * per * U + threadIdx.x / LPR;
  typename Vec<T, VW>::Raw rx[U][NV], rd[U][NV];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int c = (n * LPR + lr) * VW;
      Vec<T, VW>::clear(rx[u][n]);
      Vec<T, VW>::clear(rd[u][n]);
      if (r0 + u * per < rows && c < D) {
        Vec<T, VW>::load(x + (r0 + u * per) * D + c, rx[u][n]);
        Vec<T, VW>::load(dy + (r0 + u * per) * D + c, rd[u][n]);
      }
    }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    float ss = 0.f, dot = 0.f, v[NV][VW], d[NV][VW];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      Vec<T, VW>::widen(rx[u][n], v[n]);
      Vec<T, VW>::widen(rd[u][n], d[n]);
      ss += sum_products<T>(v[n], v[n]);
      dot += sum_products<T>(v[n], d[n]);
    }
    ss = row_sum<LG>(ss);
    dot = row_sum<LG>(dot);
    const float r = rsqrtf(ss + eps);
    const float k = dot * r * r;   // (dy . y) r = (dy . x) r^2
    const size_t row = r0 + u * per;
    if (row < rows) {
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        const int c = (n * LPR + lr) * VW;
        float o[VW];
#pragma unroll
        for (int t = 0; t < VW; ++t) o[t] = r * (d[n][t] - v[n][t] * k);
        if (c < D) Vec<T, VW>::store(dx + row * D + c, o);
      }
    }
  }
}

// the gate's rows: contiguous (pitch 0), or heads of tokens `pitch` elements apart
struct RowPitch {
  long long pitch;
  int heads;
  __device__ __forceinline__ size_t at(size_t row, int D) const {
    if (!pitch) return row * D;
    const unsigned r = (unsigned)row, tok = r / (unsigned)heads;
    return (size_t)tok * pitch + (size_t)(r - tok * heads) * D;
  }
};
struct NormWeight {
  const void* p;
  int dtype;
  template <int VW> __device__ __forceinline__ void load(int c, float (&v)[VW]) const {
    if (dtype == TOPS_F32) Vec<float, VW>::load(reinterpret_cast<const float*>(p) + c, v);
    else
#pragma unroll
      for (int t = 0; t < VW; ++t) v[t] = load_any(p, dtype, c + t);
  }
};

// gated RMS norm: y = x rsqrt(mean(x^2) + eps) w silu(g)
template <class T, int VW, int NV, int LG>
__global__ void __launch_bounds__(256) k_rmsnorm_gated_fwd(const T* __restrict__ x, const T* __restrict__ g,
                                                           NormWeight w, T* __restrict__ y, size_t rows, int D, float eps,
                                                           RowPitch gp) {
  constexpr int U = rows_in_flight2<NV>();
  constexpr int LPR = 1 << LG, per = 256 / LPR;
  const int lr = threadIdx.x & (LPR - 1);
  const size_t r0 = (size_t)blockIdx.x * per * U + threadIdx.x / LPR;
  typename Vec<T, VW>::Raw rx[U][NV], rg[U][NV];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int c = (n * LPR + lr) * VW;
      Vec<T, VW>::clear(rx[u][n]);
      if (r0 + u * per < rows && c < D) {
        Vec<T, VW>::load(x + (r0 + u * per) * D + c, rx[u][n]);
        Vec<T, VW>::load(g + gp.at(r0 + u * per, D) + c, rg[u][n]);
      }
    }
  const float invD = 1.f / (float)D;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    float ss = 0.f, v[NV][VW];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      Vec<T, VW>::widen(rx[u][n], v[n]);
      ss += sum_products<T>(v[n], v[n]);
    }
    ss = row_sum<LG>(ss);
    const float r = rsqrtf(fmaf(ss, invD, eps));
    const size_t row = r0 + u * per;
    if (row < rows) {
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        const int c = (n * LPR + lr) * VW;
        if (c < D) {
          float wv[VW], o[VW], gv[VW];
          Vec<T, VW>::widen(rg[u][n], gv);
#pragma unroll
          for (int t = 0; t < VW; ++t) wv[t] = 1.f;
          if (w.p) w.load<VW>(c, wv);
#pragma unroll
          for (int t = 0; t < VW; ++t) o[t] = v[n][t] * r * wv[t] * (gv[t] * sigmoidf<std::is_same<T, float>::value>(gv[t]));
          Vec<T, VW>::store(y + row * D + c, o);
        }
      }
    }
  }
}

// The blocks walk the rows with the grid's stride; a thread keeps the weight gradient of its columns in registers,
// a block adds its threads' in order and leaves one partial row in part_w[block][D].
template <class T, int VW, int NV, int LG>
__global__ void __launch_bounds__(256) k_rmsnorm_gated_bwd(const T* __restrict__ x, const T* __restrict__ g,
                                                           NormWeight w, const T* __restrict__ dy, T* __restrict__ dx,
                                                           T* __restrict__ dg, float* __restrict__ part_w, size_t rows, int D,
                                                           float eps, RowPitch gp, RowPitch dgp) {
  extern __shared__ float dw_sm[];   // [256 / LPR][D]
  constexpr int LPR = 1 << LG, per = 256 / LPR;
  const int lr = threadIdx.x & (LPR - 1), grp = threadIdx.x / LPR;
  const float invD = 1.f / (float)D;
  float dw[NV][VW];
#pragma unroll
  for (int n = 0; n < NV; ++n)
#pragma unroll
    for (int t = 0; t < VW; ++t) dw[n][t] = 0.f;
  // (every lane of a warp makes the same number of steps: the row sums are warp shuffles)
  for (size_t rb = (size_t)blockIdx.x * per; rb < rows; rb += (size_t)gridDim.x * per) {
    const size_t row = rb + grp;
    typename Vec<T, VW>::Raw rx[NV], rg[NV], rd[NV];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int c = (n * LPR + lr) * VW;
      Vec<T, VW>::clear(rx[n]);
      Vec<T, VW>::clear(rg[n]);
      Vec<T, VW>::clear(rd[n]);
      if (row < rows && c < D) {
        Vec<T, VW>::load(x + row * D + c, rx[n]);
        Vec<T, VW>::load(g + gp.at(row, D) + c, rg[n]);
        Vec<T, VW>::load(dy + row * D + c, rd[n]);
      }
    }
    float ss = 0.f, v[NV][VW], dv[NV][VW];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      Vec<T, VW>::widen(rx[n], v[n]);
      Vec<T, VW>::widen(rd[n], dv[n]);
      ss += sum_products<T>(v[n], v[n]);
    }
    ss = row_sum<LG>(ss);
    const float r = rsqrtf(fmaf(ss, invD, eps));
    float dot = 0.f;
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int c = (n * LPR + lr) * VW;
      float wv[VW], og[VW], gv[VW];
      Vec<T, VW>::widen(rg[n], gv);
#pragma unroll
      for (int t = 0; t < VW; ++t) wv[t] = 1.f;
      if (w.p && c < D) w.load<VW>(c, wv);
#pragma unroll
      for (int t = 0; t < VW; ++t) {
        const float gg = gv[t], s = sigmoidf<std::is_same<T, float>::value>(gg), silu = gg * s, xn = v[n][t] * r, dwv = dv[n][t] * wv[t];
        og[t] = dwv * xn * (s * (1.f + gg * (1.f - s)));   // d silu / dg = s (1 + g (1 - s))
        dw[n][t] += dv[n][t] * xn * silu;
        dv[n][t] = dwv * silu;                              // d(normalised x)
        dot = fmaf(dv[n][t], xn, dot);
      }
      if (row < rows && c < D) Vec<T, VW>::store(dg + dgp.at(row, D) + c, og);
    }
    dot = row_sum<LG>(dot) * invD;
    if (row < rows) {
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        const int c = (n * LPR + lr) * VW;
        float o[VW];
#pragma unroll
        for (int t = 0; t < VW; ++t) o[t] = r * (dv[n][t] - v[n][t] * r * dot);
        if (c < D) Vec<T, VW>::store(dx + row * D + c, o);
      }
    }
  }
  if (part_w) {
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int c = (n * LPR + lr) * VW;
      if (c < D) Vec<float, VW>::store(dw_sm + (size_t)grp * D + c, dw[n]);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < D; c += 256) {
      float s = 0.f;
      for (int i = 0; i < per; ++i) s += dw_sm[(size_t)i * D + c];
      part_w[(size_t)blockIdx.x * D + c] = s;
    }
  }
}

template <class F>
int dispatch(int dtype, F f) {
  if (dtype == TOPS_F32) return f((float*)nullptr);
  if (dtype == TOPS_BF16) return f((__nv_bfloat16*)nullptr);
  if (dtype == TOPS_F16) return f((__half*)nullptr);
  return TOPS_E_BAD_DTYPE;
}

GateConst gate_const(const tops_gate_act_params& p) {
  GateConst c;
  c.A_log = p.A_log; c.dt_bias = p.dt_bias; c.lower_bound = p.lower_bound; c.normalizer = p.normalizer; c.inv_normalizer = 1.f / p.normalizer;
  c.clamp_min = p.clamp_min; c.has_clamp = p.has_clamp_min;
  return c;
}
template <class F>
int dispatch_kind(int kind, F f) {
  if (kind == TOPS_GATE_ACT_KDA) return f(std::integral_constant<int, TOPS_GATE_ACT_KDA>());
  if (kind == TOPS_GATE_ACT_KDA_LOWER_BOUND) return f(std::integral_constant<int, TOPS_GATE_ACT_KDA_LOWER_BOUND>());
  return f(std::integral_constant<int, TOPS_GATE_ACT_LOG_SIGMOID>());
}
// Eight columns of a thread belong to one head when K is a multiple of 8; otherwise four do (K % 4 == 0 is required).
// Blocks: two waves of four per SM walk the rows; fewer when there are not that many rows.  The backward takes half of
// that: each of its blocks leaves a partial row per parameter.
struct GateGrid { int vw; dim3 grid; };
GateGrid gate_grid(int HK, int K, size_t rows, int waves) {
  GateGrid g;
  g.vw = K % 8 == 0 ? 8 : 4;
  const int cv = HK / g.vw, per = cv < 256 ? cv : 256, lanes = 256 / per, gy = (cv + per - 1) / per;
  const size_t need = (rows + lanes - 1) / lanes, most = (size_t)(148 * 4 * waves + gy - 1) / gy;
  g.grid = dim3((unsigned)(need < most ? need : most), gy);
  return g;
}
// log2 of the lanes per row, vectors per lane of the row kernels
struct RowShape { int vw, lg, nv; };
RowShape row_shape(int D) {
  RowShape r;
  r.vw = D % 8 == 0 ? 8 : 4;
  const int n = D / r.vw;
  r.lg = 0;
  while ((1 << r.lg) < n && r.lg < 5) ++r.lg;
  const int need = (n + 31) / 32;
  r.nv = need <= 1 ? 1 : need <= 2 ? 2 : need <= 4 ? 4 : 8;
  return r;
}
template <int V> using Int = std::integral_constant<int, V>;
template <class VW, class F>
int dispatch_lanes(const RowShape& r, VW vw, F f) {
  if (r.nv == 1) {
    switch (r.lg) {
      case 0: return f(vw, Int<1>(), Int<0>());
      case 1: return f(vw, Int<1>(), Int<1>());
      case 2: return f(vw, Int<1>(), Int<2>());
      case 3: return f(vw, Int<1>(), Int<3>());
      case 4: return f(vw, Int<1>(), Int<4>());
      default: return f(vw, Int<1>(), Int<5>());
    }
  }
  if (r.nv == 2) return f(vw, Int<2>(), Int<5>());
  if (r.nv == 4) return f(vw, Int<4>(), Int<5>());
  return f(vw, Int<VW::value == 8 ? 4 : 8>(), Int<5>());   // (D <= 1024: vectors of eight need at most four per lane)
}
template <class F>
int dispatch_row(const RowShape& r, F f) {
  return r.vw == 8 ? dispatch_lanes(r, Int<8>(), f) : dispatch_lanes(r, Int<4>(), f);
}
unsigned row_blocks(size_t rows, int lg, int u) {
  const size_t per = (size_t)(256 >> lg) * u;
  return (unsigned)((rows + per - 1) / per);
}
unsigned norm_bwd_blocks(size_t rows, int lg) {
  const unsigned n = row_blocks(rows, lg, 1);
  return n < 148 * 4 ? n : 148 * 4;
}

}  // namespace

int gate_check(const tops_gate_act_params& p) {
  if (p.rows < 1 || p.H < 1 || p.K < 1 || p.K % 4 != 0) return TOPS_E_BAD_SHAPE;
  if (p.kind < TOPS_GATE_ACT_KDA || p.kind > TOPS_GATE_ACT_LOG_SIGMOID) return TOPS_E_BAD_SHAPE;
  if (p.kind != TOPS_GATE_ACT_LOG_SIGMOID && !p.A_log) return TOPS_E_NULL;
  if (p.kind == TOPS_GATE_ACT_LOG_SIGMOID && !(p.normalizer != 0.f)) return TOPS_E_BAD_SHAPE;
  if (!aligned16(p.g) || !aligned16(p.out) || !aligned16(p.dt_bias)) return TOPS_E_ALIGN;
  return TOPS_OK;
}

int gate_fwd(const tops_gate_act_params& p, cudaStream_t st) {
  const GateConst c = gate_const(p);
  const GateGrid gg = gate_grid(p.H * p.K, p.K, (size_t)p.rows, 2);
  KernelScope ks("gate_act_fwd", st);
  int rc = dispatch(p.dtype, [&](auto* ti) {
    using TI = std::remove_pointer_t<decltype(ti)>;
    return dispatch(p.out_dtype, [&](auto* to) {
      using TO = std::remove_pointer_t<decltype(to)>;
      return dispatch_kind(p.kind, [&](auto kind) {
        constexpr int KIND = decltype(kind)::value;
        auto* g = reinterpret_cast<const TI*>(p.g);
        auto* o = reinterpret_cast<TO*>(p.out);
        if (gg.vw == 8) k_gate_fwd<TI, TO, KIND, 8><<<gg.grid, 256, 0, st>>>(g, o, (size_t)p.rows, p.H, p.K, c);
        else k_gate_fwd<TI, TO, KIND, 4><<<gg.grid, 256, 0, st>>>(g, o, (size_t)p.rows, p.H, p.K, c);
        return TOPS_OK;
      });
    });
  });
  return rc ? rc : post_launch();
}

size_t gate_bwd_workspace_bytes(const tops_gate_act_bwd_params& p) {
  const GateGrid gg = gate_grid(p.fwd.H * p.fwd.K, p.fwd.K, (size_t)p.fwd.rows, 1);
  return align_up((size_t)gg.grid.x * p.fwd.H * p.fwd.K * sizeof(float)) * 2 + 256;
}

int gate_bwd(const tops_gate_act_bwd_params& p, void* ws, cudaStream_t st) {
  const tops_gate_act_params& f = p.fwd;
  if (!aligned16(p.dy) || !aligned16(p.dg) || !aligned16(ws)) return TOPS_E_ALIGN;
  const int HK = f.H * f.K;
  const GateGrid gg = gate_grid(HK, f.K, (size_t)f.rows, 1);
  const int nblk = gg.grid.x;
  const bool kda = f.kind != TOPS_GATE_ACT_LOG_SIGMOID;
  float* part_bias = p.dbias ? reinterpret_cast<float*>(ws) : nullptr;
  float* part_A = (kda && p.dA_log) ? reinterpret_cast<float*>(reinterpret_cast<char*>(ws) + align_up((size_t)nblk * HK * sizeof(float)))
                                    : nullptr;
  const GateConst c = gate_const(f);
  {
    KernelScope ks("gate_act_bwd", st);
    int rc = dispatch(f.dtype, [&](auto* ti) {
      using TI = std::remove_pointer_t<decltype(ti)>;
      return dispatch(p.dy_dtype, [&](auto* td) {
        using TD = std::remove_pointer_t<decltype(td)>;
        return dispatch_kind(f.kind, [&](auto kind) {
          constexpr int KIND = decltype(kind)::value;
          auto* g = reinterpret_cast<const TI*>(f.g);
          auto* d = reinterpret_cast<const TD*>(p.dy);
          auto* o = reinterpret_cast<TI*>(p.dg);
          if (gg.vw == 8) k_gate_bwd<TI, TD, KIND, 8><<<gg.grid, 256, 0, st>>>(g, d, o, (size_t)f.rows, f.H, f.K, c, part_bias, part_A);
          else k_gate_bwd<TI, TD, KIND, 4><<<gg.grid, 256, 0, st>>>(g, d, o, (size_t)f.rows, f.H, f.K, c, part_bias, part_A);
          return TOPS_OK;
        });
      });
    });
    if (rc) return rc;
    if ((rc = post_launch())) return rc;
  }
  if (part_bias) {
    KernelScope ks("gate_act_bwd_sum", st);
    k_sum_blocks<<<(HK + 31) / 32, 1024, 0, st>>>(part_bias, nblk, HK, p.dbias);
    int rc = post_launch();
    if (rc) return rc;
  }
  if (part_A) {
    KernelScope ks("gate_act_bwd_sum", st);
    k_sum_heads<<<f.H, 1024, 0, st>>>(part_A, nblk, f.H, f.K, p.dA_log);
    return post_launch();
  }
  return TOPS_OK;
}

// A block owns 512 columns, two per thread, and walks the tokens, eight at a time through shared memory; with R = 16
// (the layer's rank) a thread's two rows of W stay in registers.  8192 tokens, N = 512: 10 us (16 MB written).
template <class T, int R_>   // R_: the rank, or 0: any multiple of 8 up to 64
__global__ void __launch_bounds__(256) k_lowrank_gate(tops_lowrank_gate_params p) {
  constexpr int TOK = 8;
  __shared__ __align__(16) float lo[64][TOK];
  const int R = R_ ? R_ : p.R, n = blockIdx.y * 512 + threadIdx.x * 2;
  const bool on = n < p.N;   // (N is a multiple of 8)
  const T *low = reinterpret_cast<const T*>(p.low), *W = reinterpret_cast<const T*>(p.W);
  const float inv = 1.f / p.normalizer;
  float bias[2] = {0.f, 0.f}, w[2][R_ ? R_ : 8];
  if (on) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      bias[j] = to_f(reinterpret_cast<const T*>(p.bias)[n + j]);
      if (R_) {
#pragma unroll
        for (int c = 0; c < R_; c += 8) {
          float t[8];
          Vec<T, 8>::load(W + (size_t)(n + j) * R + c, t);
#pragma unroll
          for (int i = 0; i < 8; ++i) w[j][c + i] = t[i];
        }
      }
    }
  }
  for (size_t r0 = (size_t)blockIdx.x * TOK; r0 < (size_t)p.rows; r0 += (size_t)gridDim.x * TOK) {
    for (int i = threadIdx.x; i < TOK * R; i += 256) {
      const int t = i / R, c = i - t * R;
      lo[c][t] = r0 + t < (size_t)p.rows ? to_f(low[(r0 + t) * p.low_pitch + c]) : 0.f;
    }
    __syncthreads();
    if (on) {
      float acc[2][TOK];
#pragma unroll
      for (int t = 0; t < TOK; ++t) { acc[0][t] = bias[0]; acc[1][t] = bias[1]; }
      auto eight = [&](int c) {   // channels c .. c + 7
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 x = *reinterpret_cast<const float4*>(&lo[c + i][0]), y = *reinterpret_cast<const float4*>(&lo[c + i][4]);
          const float l[TOK] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int t = 0; t < TOK; ++t) acc[j][t] = fmaf(l[t], w[j][R_ ? c + i : i], acc[j][t]);
        }
      };
      if (R_) {
#pragma unroll
        for (int c = 0; c < R_; c += 8) eight(c);
      } else {
        for (int c = 0; c < R; c += 8) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            float t[8];
            Vec<T, 8>::load(W + (size_t)(n + j) * R + c, t);
#pragma unroll
            for (int i = 0; i < 8; ++i) w[j][i] = t[i];
          }
          eight(c);
        }
      }
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        if (r0 + t >= (size_t)p.rows) break;
        T xr[2], yr[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          xr[j] = from_f<T>(acc[j][t]);
          float y = -softplusf<std::is_same<T, float>::value>(-to_f(xr[j])) * inv;
          if (p.has_clamp_min && y < p.clamp_min) y = p.clamp_min;
          yr[j] = from_f<T>(y);
        }
        const size_t o = (r0 + t) * p.N + n;
        struct __align__(2 * sizeof(T)) Two { T a, b; };
        if (p.x) *reinterpret_cast<Two*>(reinterpret_cast<T*>(p.x) + o) = Two{xr[0], xr[1]};
        *reinterpret_cast<Two*>(reinterpret_cast<T*>(p.y) + o) = Two{yr[0], yr[1]};
      }
    }
    __syncthreads();
  }
}

int lowrank_gate_fwd(const tops_lowrank_gate_params& p, cudaStream_t st) {
  if (p.rows < 1 || p.R < 8 || p.R > 64 || p.R % 8 != 0 || p.N < 8 || p.N % 8 != 0 || p.low_pitch < p.R || !(p.normalizer != 0.f))
    return TOPS_E_BAD_SHAPE;
  if (!aligned16(p.W) || !aligned16(p.x) || !aligned16(p.y)) return TOPS_E_ALIGN;
  const size_t need = ((size_t)p.rows + 7) / 8;
  const dim3 grid((unsigned)(need < 148 * 4 ? need : 148 * 4), (p.N + 511) / 512);
  KernelScope ks("lowrank_gate_fwd", st);
  int rc = dispatch(p.dtype, [&](auto* t) {
    using T = std::remove_pointer_t<decltype(t)>;
    if (p.R == 16) k_lowrank_gate<T, 16><<<grid, 256, 0, st>>>(p);
    else k_lowrank_gate<T, 0><<<grid, 256, 0, st>>>(p);
    return TOPS_OK;
  });
  return rc ? rc : post_launch();
}

int norm_check(const tops_norm_params& p) {
  if ((p.gate_pitch || p.dgate_pitch) && (p.heads < 1 || p.rows > 0xffffffffll || p.gate_pitch % 8 || p.dgate_pitch % 8))
    return TOPS_E_BAD_SHAPE;
  if (p.rows < 1 || p.D < 4 || p.D > 1024 || p.D % 4 != 0) return TOPS_E_BAD_SHAPE;
  if (!p.x || !p.y) return TOPS_E_NULL;
  if (!aligned16(p.x) || !aligned16(p.y) || !aligned16(p.gate) || !aligned16(p.weight) || !aligned16(p.dy) ||
      !aligned16(p.dx) || !aligned16(p.dgate))
    return TOPS_E_ALIGN;
  return TOPS_OK;
}

int l2norm_fwd(const tops_norm_params& p, cudaStream_t st) {
  const RowShape rs = row_shape(p.D);
  KernelScope ks("l2norm_fwd", st);
  int rc = dispatch(p.dtype, [&](auto* t) {
    using T = std::remove_pointer_t<decltype(t)>;
    return dispatch_row(rs, [&](auto vw, auto nv, auto lg) {
      constexpr int VW = decltype(vw)::value, NV = decltype(nv)::value, LG = decltype(lg)::value;
      k_l2norm_fwd<T, VW, NV, LG><<<row_blocks(p.rows, rs.lg, rows_in_flight<NV>()), 256, 0, st>>>(
          reinterpret_cast<const T*>(p.x), reinterpret_cast<T*>(p.y), p.rstd, (size_t)p.rows, p.D, p.eps);
      return TOPS_OK;
    });
  });
  return rc ? rc : post_launch();
}

int l2norm_bwd(const tops_norm_params& p, cudaStream_t st) {
  if (!p.dy || !p.dx) return TOPS_E_NULL;
  const RowShape rs = row_shape(p.D);
  KernelScope ks("l2norm_bwd", st);
  int rc = dispatch(p.dtype, [&](auto* t) {
    using T = std::remove_pointer_t<decltype(t)>;
    return dispatch_row(rs, [&](auto vw, auto nv, auto lg) {
      constexpr int VW = decltype(vw)::value, NV = decltype(nv)::value, LG = decltype(lg)::value;
      k_l2norm_bwd<T, VW, NV, LG><<<row_blocks(p.rows, rs.lg, rows_in_flight2<NV>()), 256, 0, st>>>(
          reinterpret_cast<const T*>(p.x), reinterpret_cast<const T*>(p.dy), reinterpret_cast<T*>(p.dx), (size_t)p.rows, p.D,
          p.eps);
      return TOPS_OK;
    });
  });
  return rc ? rc : post_launch();
}

int rmsnorm_gated_fwd(const tops_norm_params& p, cudaStream_t st) {
  if (!p.gate) return TOPS_E_NULL;
  const RowShape rs = row_shape(p.D);
  KernelScope ks("rmsnorm_gated_fwd", st);
  int rc = dispatch(p.dtype, [&](auto* t) {
    using T = std::remove_pointer_t<decltype(t)>;
    return dispatch_row(rs, [&](auto vw, auto nv, auto lg) {
      constexpr int VW = decltype(vw)::value, NV = decltype(nv)::value, LG = decltype(lg)::value;
      k_rmsnorm_gated_fwd<T, VW, NV, LG><<<row_blocks(p.rows, rs.lg, rows_in_flight2<NV>()), 256, 0, st>>>(
          reinterpret_cast<const T*>(p.x), reinterpret_cast<const T*>(p.gate), NormWeight{p.weight, p.weight_dtype},
          reinterpret_cast<T*>(p.y), (size_t)p.rows, p.D, p.eps, RowPitch{p.gate_pitch, p.heads});
      return TOPS_OK;
    });
  });
  return rc ? rc : post_launch();
}

size_t rmsnorm_gated_bwd_workspace_bytes(const tops_norm_params& p) {
  return align_up((size_t)norm_bwd_blocks((size_t)p.rows, row_shape(p.D).lg) * p.D * sizeof(float)) + 256;
}

int rmsnorm_gated_bwd(const tops_norm_params& p, void* ws, cudaStream_t st) {
  if (!p.gate || !p.dy || !p.dx || !p.dgate) return TOPS_E_NULL;
  if (!aligned16(ws)) return TOPS_E_ALIGN;
  const RowShape rs = row_shape(p.D);
  const unsigned blocks = norm_bwd_blocks((size_t)p.rows, rs.lg);
  const size_t smem = (size_t)(256 >> rs.lg) * p.D * sizeof(float);   // at most 32 KB
  float* part = p.dweight ? reinterpret_cast<float*>(ws) : nullptr;
  {
    KernelScope ks("rmsnorm_gated_bwd", st);
    int rc = dispatch(p.dtype, [&](auto* t) {
      using T = std::remove_pointer_t<decltype(t)>;
      return dispatch_row(rs, [&](auto vw, auto nv, auto lg) {
        constexpr int VW = decltype(vw)::value, NV = decltype(nv)::value, LG = decltype(lg)::value;
        k_rmsnorm_gated_bwd<T, VW, NV, LG><<<blocks, 256, smem, st>>>(
            reinterpret_cast<const T*>(p.x), reinterpret_cast<const T*>(p.gate), NormWeight{p.weight, p.weight_dtype},
            reinterpret_cast<const T*>(p.dy), reinterpret_cast<T*>(p.dx), reinterpret_cast<T*>(p.dgate), part, (size_t)p.rows,
            p.D, p.eps, RowPitch{p.gate_pitch, p.heads}, RowPitch{p.dgate_pitch, p.heads});
        return TOPS_OK;
      });
    });
    if (rc) return rc;
    if ((rc = post_launch())) return rc;
  }
  if (part) {
    KernelScope ks("rmsnorm_gated_bwd_sum", st);
    k_sum_blocks<<<(p.D + 31) / 32, 1024, 0, st>>>(part, (int)blocks, p.D, p.dweight);
    return post_launch();
  }
  return TOPS_OK;
}

}  // namespace elementwise
}  // namespace tops
