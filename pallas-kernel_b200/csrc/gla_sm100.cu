// Chunked GLA on the 5th-generation tensor cores (sm_100a): bf16 operands staged
// in shared memory by TMA, contractions issued with tcgen05.mma into tensor
// memory, fp32 accumulation, gates and state kept in fp32.
//
// Shapes taken here: bf16 q/k/v/g, chunk 64.  The plain form of the kernels: K = V = 128, T a
// multiple of 64, dense batch, per-channel or scalar gates.  The general form: packed batches, any T,
// 32 <= K <= 128, 32 <= V <= 1024 (multiples of 8), also constant or no gates.  Everything else runs on
// the generic kernels.
//
// Data layout.  Activations stay in the caller's [B,T,H,D] layout; a chunk of
// one head is a 64 x 128 tile whose rows are H*D elements apart, fetched as two
// 64 x 64 TMA boxes (SWIZZLE_128B) straight into the tile format UMMA
// descriptors read (sm100_prims.cuh).  Chunk-start states and their gradients
// are kept as bf16 [B,NT,H,K,V] scratch in HBM, pre-multiplied by the
// per-channel factors their consumers need (h' = h exp(mid) scale,
// dh' = dh exp(G_n - mid)): they are only ever used as bf16 tensor-core
// operands; the running state itself is fp32 in registers of the scan kernels.
//
// Kernels
//   k_scan<false>  h'_c,  h <- h * exp(G_n) + (k exp(G_n - G))^T v       (forward scan)
//   k_scan<true>   dh'_c, dh <- dh * exp(G_n) + (q scale exp(G))^T do    (reverse scan)
//   k_fwd_o        A = tril(q~ k~^T) scale;  o = q~ h'_c + A v            (chunk-parallel outputs)
//   k_fwd_fused    the forward scan and the outputs in one pass, state kept on chip
//   k_bwd_main     dA, dv, dq, dk, dg of one chunk from q, k, v, g, do, h'_c, dh'_c
//   k_join_segments  chains the time segments a sequence is cut into when there are few sequences
// A forward is k_fwd_fused when there are enough (batch, head, segment) blocks to fill the GPU (always in the general
// form), else k_scan<false> + k_fwd_o; a backward is k_scan<true> + k_bwd_main (and k_scan<false> first
// when the caller did not keep the forward's states).
// G is the chunk-local cumulative gate and q~ = q exp(G - mid),
// k~ = k exp(mid - G), mid = (G_0 + G_n) / 2 per channel.  The cumulative
// gates themselves are tensor-core products of the gate tile with constant
// 0 / 1 / +-1/2 patterns, so the exponents arrive in tensor memory in the
// layout the gating or the write-out needs.
//
// Thread layout (scans, k_fwd_o, k_fwd_fused, write-out warps of k_bwd_main): 16 compute warps.
// Thread (col, seg) with col = (warp & 3) * 32 + lane and seg = warp >> 2:
// a warp may only touch the 32 tensor-memory lanes (warp & 3) * 32 .. + 31, so
// the thread owns accumulator row `col` and splits the accumulator columns
// with the three other warps of its lane quarter by `seg`.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <vector>

#include "gla_sm100.cuh"
#include "sm100_host.cuh"
#include "sm100_tiles.cuh"

namespace tops {
namespace sm100 {


namespace {

// ===========================================================================
// Where the chunks of a call live
// ===========================================================================
// Every kernel exists in two forms.  The plain one (GEN = false) takes dense batches of whole chunks with
// K = V = 128.  The general one (GEN = true) takes packed batches, sequences of any length, K <= 128 and any V
// (multiples of 8):
//   * the last chunk of a sequence may be short.  Its tile fetch reads on into the next sequence (or past the end
//     of the tensor, where TMA fills zeros); the rows that are not its own are overwritten with zeros in shared
//     memory before a product reads them, so nothing of another sequence, not even an infinity, gets in: zero
//     gates repeat the last cumulative gate, zero q, k, v, do add nothing.  Only short chunks pay for it.
//   * the diagonal of the intra-chunk matrix, q_i . k_i, has no gates in it and is summed in fp32 from the raw q and k
//     while they are gated (the products of the gated bf16 operands lose about 2^-9 |q| |k|, which is all there is of a
//     diagonal entry where q_i and k_i are nearly orthogonal; the output of a sequence's first token is that entry
//     times v, and an output norm divides by it).
//   * q~, k~, A and dA are two bf16 halves each (hi + lo, 16 bits) and a product of two of them is hi hi + hi lo + lo hi,
//     as is the gated x of a summary scan: the CUDA-core kernels these calls ran on before keep A and dA in fp32, and
//     with single halves o was 3.23e-3 from the fp64 result where it had been 2.82e-3 (now 1.87e-3; dq 2.87e-3, 2.28e-3,
//     1.77e-3).  The second halves take the room of the second h' tile (forward) and of the second q, k slot and the
//     consumed gate tile (backward), so a chunk is gated after the one before has been written out: 16384 tokens in 13
//     documents, H = 16, forward 125 -> 181 us, chunk gradients 314 -> 350 us.  Not where K = V = 128 and all chunks are
//     whole: those calls have had single halves all along.
//   * the gated operands stay in range whatever the gates: see kSpan below.
//   * channels beyond K or V are zero-filled by TMA; the state tiles in scratch are always 128 x 128.
//   * V > 128 runs as VS slices of 128 value channels that share q, k and g.
//   * packed batches find their segments and chunks in tables that k_plan writes.
struct __align__(16) SegEntry {   // a run of chunks of one sequence, walked by one block (per head and value slice)
  int row, end;      // first token of the run; end of its sequence (token rows of the flattened [B*T] axis)
  int slot, nch;     // index of its first chunk among all chunks; number of chunks
  int id;            // index of the run in sequence order (the table itself is sorted by length, longest first)
  int seq, cnt, pad; // its sequence; number of runs that sequence is cut into
};
struct ChunkEntry { int row, end; };
struct Geo {
  const SegEntry* segs;       // packed batches; null: dense, cps chunks per segment
  const ChunkEntry* chunks;   // packed batches; null: dense
  int K, V, VS;
  int cps, nseg;              // dense: chunks per segment, segments per sequence
  int NTseq;                  // dense: chunks per sequence
};
// the block's position: blocks are numbered (segment, head, value slice), slice fastest
// cnt: runs its sequence is cut into.  A sequence of one run starts from and ends in the caller's states (index
// seqh); the runs of a longer one start from the states that k_join_segments_gen leaves (index sidx).
struct BlockPos { int h, vs, row, end, slot, nch, cnt; size_t sidx, seqh; };
__device__ __forceinline__ BlockPos block_pos(const Geo& g, int T, int H, int blk) {
  BlockPos q;
  q.vs = blk % g.VS;
  const int sh = blk / g.VS;
  q.h = sh % H;
  const int s = sh / H;
  int id;
  if (g.segs) {
    const SegEntry e = g.segs[s];
    q.row = e.row; q.end = e.end; q.slot = e.slot; q.nch = e.nch; id = e.id;
    q.cnt = e.cnt; q.seqh = (size_t)e.seq * H + q.h;
  } else {
    const int b = s / g.nseg, sg = s - b * g.nseg;
    q.row = b * T + sg * g.cps * C; q.end = (b + 1) * T;
    q.slot = b * g.NTseq + sg * g.cps;
    q.nch = min(g.cps, g.NTseq - sg * g.cps);
    q.cnt = g.nseg; q.seqh = (size_t)b * H + q.h;
    id = s;
  }
  q.sidx = (size_t)id * H + q.h;
  return q;
}
// overwrites rows [len, 64) of a 64 x 128 tile with zeros (threads t0, t0 + nt, ...)
__device__ __forceinline__ void zero_rows(uint8_t* tile, int len, int t0, int nt) {
  for (int i = t0; i < (64 - len) * 16; i += nt) {
    const int r = len + (i >> 4), piece = i & 15;
    *reinterpret_cast<uint4*>(tile + (piece >> 3) * SLAB64 + r * 128 + (piece & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
  }
}
// the part of q_i . k_i of 16 channels (two packed vectors of 8 of each)
__device__ __forceinline__ float dot8(uint4 a, uint4 b, float s) {
  const __nv_bfloat162 *x = reinterpret_cast<const __nv_bfloat162*>(&a), *y = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const float2 u = __bfloat1622float2(x[t]), v = __bfloat1622float2(y[t]);
    s = fmaf(u.x, v.x, s);
    s = fmaf(u.y, v.y, s);
  }
  return s;
}
// puts the sum of `n` partial dot products part[.][i] into a[j], j = i - j0 (row i's diagonal entry)
__device__ __forceinline__ void set_diagonal(float (&a)[16], const float* part, int n, int i, int j) {
  float d = 0.f;
  for (int c = 0; c < n; ++c) d += part[c * C + i];
#pragma unroll
  for (int t = 0; t < 16; ++t) a[t] = t == j ? d : a[t];
}
// 32 values of row `row` of a state [.., K, V], columns c0 .. c0 + 31 (zero outside K x V)
__device__ __forceinline__ void load_state32(float (&S)[32], const float* base, int row, int c0, int K, int V) {
#pragma unroll
  for (int j = 0; j < 32; j += 4) {
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (base && row < K && c0 + j < V) x = *reinterpret_cast<const float4*>(base + (size_t)row * V + c0 + j);
    S[j] = x.x; S[j + 1] = x.y; S[j + 2] = x.z; S[j + 3] = x.w;
  }
}
__device__ __forceinline__ void store_state32(float* base, const float (&S)[32], int row, int c0, int K, int V) {
#pragma unroll
  for (int j = 0; j < 32; j += 4)
    if (row < K && c0 + j < V)
      *reinterpret_cast<float4*>(base + (size_t)row * V + c0 + j) = make_float4(S[j], S[j + 1], S[j + 2], S[j + 3]);
}

// ---------------------------------------------------------------------------
// Strong gates (general form)
// ---------------------------------------------------------------------------
// exp(G - mid) and exp(mid - G) leave fp32 once a channel's gates sum to some -176 over a chunk (-2.8 a token); every
// result is finite all the same.  So the per-channel references of the stored tiles are kept within kSpan of zero,
//     h' = h exp(ref) scale,  dh' = dh exp(refd),   ref = clamp(mid), refd = clamp(G_n - mid)
// (the clamps are continuous: two kernels that see a mid on either side of the limit still agree), and a chunk in which
// a clamp takes effect, a "wide" one, is gated as
//     q~ = q exp(G - ref),  k~ = k exp(G_n - G - refd)
// whose exponents are at most kSpan for gates that do not grow.  These k~ and q~ no longer make the intra-chunk matrix:
// a wide chunk's A, dq_intra and dk_intra are summed pair by pair on the CUDA cores, with exp(G_i - G_j) as a product of
// the gates between.  All of it starts from the caller's q, k and gates (in L2).  kSpan = 64 leaves operands of any
// magnitude that fits bf16 activations a factor of 1e10 before fp32 ends.
// Kept out of the narrow chunks' way: a forward block that meets a wide chunk walks its run once more (fused_walk), the
// backward does the wide ones in a launch of their own (launch_bwd_main); where there are none that costs the forward 1 %
// and the backward about 5 us.  With every chunk wide: 13 documents in T = 16384, H = 16 forward + backward 0.74 -> 12.9 ms
// (16.8 on the CUDA-core kernels at chunk 16, which hold gates down to -11.8 a token), prompt of T = 3001 67 -> 600 us (1637).
constexpr float kSpan = 64.f;
// The backward takes a chunk as wide too when a channel's gates fall below -2 a token: the shares of the pairs (i, i) in
// q dq - k dk cancel, and what the products leave of them (2^-17) is no longer small beside dg, which is e^g of them.
__device__ __forceinline__ bool wide_span(float mid, float half, int len) {   // half: G_n - mid
  return fabsf(mid) > kSpan || fabsf(half) > kSpan || fabsf(mid + half) > 2.f * len;
}
__device__ __forceinline__ float clamp_span(float x) { return fminf(fmaxf(x, -kSpan), kSpan); }
// a chunk of one head as it lies in the caller's tensors
struct RawChunk {
  const __nv_bfloat16 *q, *k;   // first token, first channel
  const __nv_bfloat16* g;       // the same; scalar gates: the first token's; null: gconst at every token
  long long pitch, gstep;       // elements between tokens
  float gconst;
  int K, len;
};
template <bool SCALAR>
__device__ __forceinline__ float raw_gate(const RawChunk& r, int i, int c) {
  if (SCALAR) return r.g ? __bfloat162float(r.g[i * r.gstep]) : r.gconst;
  return __bfloat162float(r.g[i * r.gstep + c]);
}
// tril(A) scale of a wide chunk as hi + lo tiles: 16 warps, warp w columns w, w + 16, w + 32, w + 48, a lane four channels
template <bool SCALAR>
__device__ __forceinline__ void wide_matrix(const RawChunk r, uint8_t* hi, uint8_t* lo, float scale, int warp, int lane) {
  const int c0 = 4 * lane;
  const bool on = c0 < r.K;   // (K is a multiple of 8)
  float k[4][4], w[4][4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int j = warp + 16 * m;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      k[m][c] = on && j < r.len ? __bfloat162float(r.k[j * r.pitch + c0 + c]) * scale : 0.f;
      w[m][c] = 1.f;
    }
  }
#pragma unroll 1
  for (int i = 0; i < C; ++i) {
    const bool in = on && i < r.len;
    float q[4], eg[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      q[c] = in ? __bfloat162float(r.q[i * r.pitch + c0 + c]) : 0.f;
      eg[c] = in ? fast_exp(raw_gate<SCALAR>(r, i, c0 + c)) : 1.f;
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int j = warp + 16 * m;
      float a = 0.f;
      if (i > j) {
#pragma unroll
        for (int c = 0; c < 4; ++c) w[m][c] *= eg[c];
      }
      if (i >= j) {
#pragma unroll
        for (int c = 0; c < 4; ++c) a = fmaf(q[c] * k[m][c], w[m][c], a);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if (lane == m) {
        const __nv_bfloat16 top = __float2bfloat16_rn(a);
        const float f = __bfloat162float(top);
        *reinterpret_cast<__nv_bfloat16*>(hi + slab_off(i, j)) = top;
        *reinterpret_cast<__nv_bfloat16*>(lo + slab_off(i, j)) = __float2bfloat16_rn(fabsf(f) <= 3.4e38f ? a - f : 0.f);
      }
    }
  }
}
// summed gates of channel c: before token i0, and of the whole chunk; the first token's
struct WideSums { float before, total, first; };
template <bool SCALAR>
__device__ __forceinline__ WideSums wide_sums(const RawChunk& r, int c, int i0) {
  WideSums s{0.f, 0.f, 0.f};
#pragma unroll 1
  for (int i = 0; i < r.len; ++i) {
    if (i == i0) s.before = s.total;
    s.total += raw_gate<SCALAR>(r, i, c);
    if (i == 0) s.first = s.total;
  }
  return s;
}
// gates a wide chunk again: thread (channel, 16 time steps).  q~ only where a product needs it (qs null: not).
template <bool SCALAR>
__device__ __forceinline__ void wide_operands(const RawChunk r, uint8_t* qs, uint8_t* ks, uint8_t* klo, int col, int seg) {
  const ColAddr ca = col_prep(64, col);
  if (col >= r.K) {   // channels that do not exist: a scalar gate's infinity times their zeros is no zero
    for (int i = seg * SEG; i < seg * SEG + SEG; ++i) {
      *reinterpret_cast<unsigned short*>(ks + ca.at(i)) = *reinterpret_cast<unsigned short*>(klo + ca.at(i)) = 0;
      if (qs) *reinterpret_cast<unsigned short*>(qs + ca.at(i)) = 0;
    }
    return;
  }
  const WideSums s = wide_sums<SCALAR>(r, col, seg * SEG);
  const float mid = 0.5f * (s.first + s.total), ref = clamp_span(mid), refd = clamp_span(s.total - mid);
  float G = s.before;
#pragma unroll 1
  for (int t = 0; t < SEG; ++t) {
    const int i = seg * SEG + t;
    if (i >= r.len) break;
    G += raw_gate<SCALAR>(r, i, col);
    const float k = __bfloat162float(r.k[i * r.pitch + col]) * fast_exp(s.total - G - refd);
    const __nv_bfloat16 kh = __float2bfloat16_rn(k);
    *reinterpret_cast<__nv_bfloat16*>(ks + ca.at(i)) = kh;
    *reinterpret_cast<__nv_bfloat16*>(klo + ca.at(i)) = __float2bfloat16_rn(k - __bfloat162float(kh));
    if (qs) *reinterpret_cast<__nv_bfloat16*>(qs + ca.at(i)) = __float2bfloat16_rn(__bfloat162float(r.q[i * r.pitch + col]) * fast_exp(G - ref));
  }
}

// ===========================================================================
// State scans
// ===========================================================================
struct ScanParams {
  CUtensorMap mx, mg, my;  // x: k (fwd) / q (bwd); y: v / do
  CUtensorMap mst;         // the states tensor as [B*NT*H*128, 128] (TMA stores)
  const float* s0;         // state each block starts from: [B,H,nseg,K,V] or null (zero)
  const float* s0_seg;     // GEN: the same for the runs of a sequence that is cut into several
  __nv_bfloat16* states;   // h' / dh'  [B,T/64,H,K,V]; null: keep no chunk-start states (summary pass)
  float* s_final;          // state each block ends with: [B,H,nseg,K,V] or null
  float* gsum;             // summed log-gates of each block's chunks [B,H,nseg,K] or null
  int T, H, NT;            // T: tokens per sequence; NT: chunks per block (T / 64 / nseg)
  int nseg;                // time segments per sequence, one block each
  float scale;
  const __nv_bfloat16* gscalar;   // scalar gates [B,T,H] (SCALAR kernels; mg is unused then)
  const float* gamma;      // constant gates [H] (SCALAR GEN kernels; gscalar is null then; both null: no gate)
  Geo geo;                 // GEN kernels
  uint8_t* wide;           // GEN reverse scan: [chunk][H][4], one byte per quarter of the channels: the chunk is wide
  int skip_xy;             // test hook: the x/y tile load of this chunk is never issued (-1: none), so that the
                           // bounded wait for it runs out and the kernel leaves through its error path
};

// One block per (batch, head): 16 compute warps and two issuing warps.  The whole K x V state lives in
// registers of the compute warps (thread (q4, lane, seg): row k = 32 q4 + lane, columns 32 seg .. + 31).
// Software pipeline over the chunks p (in scan order), one block-wide barrier per chunk:
//   compute warps, iteration p:  stage h'_p for its TMA store;  gate x(p+1) in place (its exponents
//       were put in tensor memory two iterations ago);  barrier;  wait for the state product of
//       chunk p;  state <- state * exp(G_n(p)) + D(p).
//   product thread, iteration p:  barrier;  state product of chunk p+1 -> accumulator (p+1)&1;  exponent
//       product of chunk p+3 -> exponent slot (p+1)&1.
//   copy thread, iteration p:  barrier;  TMA store of h'_p;  TMA loads of g of chunk p+4 and, once the state
//       product of chunk p has completed, of x, y of chunk p+3.
// No compute warp ever blocks on the issue of a product or a copy.  x/y and g tiles: 3 stages each;
// state staging: 2 tiles.
constexpr int SCAN_THREADS = NTHREADS + 64;    // 16 compute warps, a warp that issues the products, a warp that issues the copies
constexpr int FUSED_THREADS = NTHREADS + 32;   // 16 compute warps and one driver warp (splitting it made this kernel slower)
struct ScanShared {
  uint64_t fullg[3], fullxy[5], ebar[2], sbar[2];
  uint32_t tmem_slot;
  int abort_flag;
  float gn[2][D], e0[2][D];   // row 63 (G_n) and row 0 of the exponent tile, per channel
};

// SCALAR: one gate per head and time step (simple_gla).  No gate tile is fetched and no exponent product is
// issued: every compute warp keeps the 64 gates of the next chunk in registers and cumulates them with
// shuffles (warp_cumulate), so a thread gates its 16 channels of x with one factor.
// SUM (summary pass: no chunk-start states, zero start): only the state after the block's chunks is wanted,
//     S = sum_c [prod_{c' after c} exp(G_n(c'))] D(c),
// so the decay of all later chunks is folded into the gating of x (exponent + R, R the summed gates of the chunks
// already done) and every state product accumulates into ONE tensor-memory tile: nothing of a chunk depends on
// the chunk before it but the running sum R, the chain product -> register update -> next product is gone and a
// chunk costs its gating and its products.  The chunks are walked from the far end (forward scan: last chunk
// first; reverse scan: first chunk first), so that R is known when a chunk is gated.
template <bool BWD, bool SCALAR, bool SUM, bool GEN>
__global__ void __launch_bounds__(SCAN_THREADS, 1) k_scan(const __grid_constant__ ScanParams p) {
  // every shared object is carved from the dynamic allocation, whose start is 1024-byte aligned when the
  // kernel has no static shared memory (checked below: the swizzled tiles need that alignment)
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* xs = smem;                       // 3 x (64 x 128): x, gated in place
  uint8_t* ys = xs + 3 * TILE64;            // 3 x (64 x 128): y
  uint8_t* gs = ys + 3 * TILE64;            // 3 x (64 x 128): g
  uint8_t* mt = gs + 3 * TILE64;            // exponent pattern, rows repeated to 128
  uint8_t* hst = mt + 2 * SLAB64;           // 2 x (128 x 128) bf16: chunk-start states on their way to HBM
  ScanShared& sh = *reinterpret_cast<ScanShared*>(hst + 2 * TILE128);
  volatile int* abort_flag = &sh.abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool driver = warp >= 16;   // warp 16 issues the products, warp 17 the copies
  const int q4 = warp & 3, seg = (warp >> 2) & 3, col = q4 * 32 + lane;
  BlockPos bp;
  if constexpr (GEN) {
    bp = block_pos(p.geo, p.T, p.H, blockIdx.x);
  } else {
    const int sg = blockIdx.x % p.nseg, bh = blockIdx.x / p.nseg, b = bh / p.H;
    bp.h = bh % p.H; bp.vs = 0; bp.row = b * p.T + sg * p.NT * C; bp.end = (b + 1) * p.T;
    bp.slot = b * (p.T / C) + sg * p.NT; bp.nch = p.NT; bp.sidx = bp.seqh = blockIdx.x; bp.cnt = 1;
  }
  const int h = bp.h, NT = bp.nch;
  const int VS = GEN ? p.geo.VS : 1, K = GEN ? p.geo.K : D, V = GEN ? p.geo.V : D;
  const int yc = bp.vs * D;   // first value channel of this block's slice
  const float* const start_state = (GEN && !SUM && bp.cnt > 1) ? p.s0_seg + bp.sidx * K * V
                                                       : (p.s0 ? p.s0 + bp.seqh * K * V : nullptr);
  const bool keep_states = p.states != nullptr;
  if (GEN && SUM && p.geo.segs && bp.cnt == 1) return;   // a packed sequence that is not cut needs no summary
  // tensor-memory columns: two exponent tiles, two state-product accumulators
  constexpr uint32_t cE = 0, cS = 256;
  if ((smem_u32(smem) & 1023u) != 0) {   // uniform over the block
    if (tid == 0) fail(12);
    return;
  }

  // chunk pp of this block (in the order the block walks them) within its run of chunks
  auto chunk_of = [&](int pp) { return (BWD != SUM) ? NT - 1 - pp : pp; };
  // SUM: summed gates of the chunks already done, per channel (two copies, written for the next chunk while the
  // current one is read; in the place of e0, which a summary pass does not use) or, for scalar gates, in a
  // register of every thread
  float* const racc = &sh.e0[0][0];
  float racc_s = 0.f;
  // x / y stages: three; a summary pass, which is bound by how many bytes it keeps in flight, has two more in the
  // state staging tiles it does not use (GEN: one more, and two tiles for what bf16 leaves of the gated x: its sums end
  // up in the caller's fp32 state)
  constexpr bool SPLIT = SUM && GEN;
  constexpr int NXY = SPLIT ? 4 : SUM ? 5 : 3;
  auto x_low = [&](int pp) { return hst + TILE128 + (pp & 1) * TILE64; };   // (read by the product of chunk pp, gone before gating pp + 2)
  auto x_stage = [&](int pp) { const int st = pp % NXY; return st < 3 ? xs + st * TILE64 : hst + (st - 3) * 2 * TILE64; };
  auto y_stage = [&](int pp) { const int st = pp % NXY; return st < 3 ? ys + st * TILE64 : hst + (st - 3) * 2 * TILE64 + TILE64; };
  auto xy_bar = [&](int pp) { return &sh.fullxy[pp % NXY]; };
  auto xy_parity = [&](int pp) { return (uint32_t)((pp / NXY) & 1); };
  auto chunk_row = [&](int pp) { return bp.row + chunk_of(pp) * C; };
  auto chunk_len = [&](int pp) { return GEN ? min(C, bp.end - chunk_row(pp)) : C; };   // rows that are the sequence's own
  auto issue_g = [&](int pp) {
    uint8_t* dst = gs + (pp % 3) * TILE64;
    mbar_expect_tx(&sh.fullg[pp % 3], TILE64);
    tma_load_3d(dst, &p.mg, &sh.fullg[pp % 3], 0, h, chunk_row(pp));
    tma_load_3d(dst + SLAB64, &p.mg, &sh.fullg[pp % 3], 64, h, chunk_row(pp));
  };
  auto issue_xy = [&](int pp) {
    uint8_t *xd = x_stage(pp), *yd = y_stage(pp);
    uint64_t* bar = xy_bar(pp);
    mbar_expect_tx(bar, 2 * TILE64);
    tma_load_3d(xd, &p.mx, bar, 0, h, chunk_row(pp));
    tma_load_3d(xd + SLAB64, &p.mx, bar, 64, h, chunk_row(pp));
    tma_load_3d(yd, &p.my, bar, yc, h, chunk_row(pp));
    tma_load_3d(yd + SLAB64, &p.my, bar, yc + 64, h, chunk_row(pp));
  };
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&sh.fullg[i], 1);
    for (int i = 0; i < 5; ++i) mbar_init(&sh.fullxy[i], 1);
    mbar_init(&sh.ebar[0], 1); mbar_init(&sh.ebar[1], 1); mbar_init(&sh.sbar[0], 1); mbar_init(&sh.sbar[1], 1);
    fence_barrier_init();
    tma_prefetch_desc(&p.mx); tma_prefetch_desc(&p.my);
    if (!SCALAR) tma_prefetch_desc(&p.mg);
    if (p.states) tma_prefetch_desc(&p.mst);
    sh.abort_flag = 0;
    for (int c = 0; c < 3 && c < NT; ++c)
      if (!SCALAR) issue_g(c);
    for (int c = 0; c < NXY && c < NT; ++c) issue_xy(c);
  }
  __syncwarp();
  if (warp == 0) { tmem_alloc(&sh.tmem_slot, 512); tmem_relinquish(); }
  // SCALAR: the gates of the next chunks, fetched three chunks ahead into this warp's ring (see GateRing; the
  // rings take the place of the gate tiles, which scalar gates do not use)
  GateRing gring;
  const long long gidx0 = (long long)(chunk_row(0) + lane) * p.H + h;
  const long long gstep = (long long)(chunk_row(NT > 1 ? 1 : 0) - chunk_row(0)) * p.H;   // +-64 H elements per chunk
  auto gate_index = [&](int c) { return (size_t)(gidx0 + c * gstep); };
  const float gconst = (GEN && SCALAR && p.gamma) ? p.gamma[h] : 0.f;   // GEN: a constant decay, or none
  auto load_gates = [&](int c) {
    const int len = c < NT ? chunk_len(c) : 0;
    const bool stored = !GEN || p.gscalar;
    gring.prefetch(p.gscalar, stored && lane < len, stored && lane + 32 < len, c < NT ? gate_index(c) : 0, (size_t)32 * p.H, c,
                   lane);
  };
  if (SCALAR) {
    if (!driver) {
      gring.init(gs + warp * GateRing::kBytesPerWarp);
      load_gates(0);
      load_gates(1);
      load_gates(2);
    }
  } else {
    build_tri_tile(mt, 128, BWD ? TRI_INCL : TRI_REVN);
    if (SUM && tid < 2 * D) racc[tid] = 0.f;
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = sh.tmem_slot;
  const uint32_t lane_base = q4 * 32;

  // exponents E = pattern . g of chunk pp: [time (repeated to 128 lanes)][channel]; row 63 is G_n
  // (called by the whole product warp: a short chunk's foreign gate rows are zeroed first)
  auto issue_gate_mma = [&](int pp) {
    if (SCALAR) return;
    if (GEN && chunk_len(pp) < C) {
      if (!mbar_wait(&sh.fullg[pp % 3], (pp / 3) & 1)) { *abort_flag = 1; fail(1); }
      zero_rows(gs + (pp % 3) * TILE64, chunk_len(pp), lane, 32);
      fence_async_smem();
      __syncwarp();
    }
    if (lane != 0) return;
    if (!mbar_wait(&sh.fullg[pp % 3], (pp / 3) & 1)) { *abort_flag = 1; fail(1); }
    tc_fence_after();
    const uint32_t ga = smem_u32(gs + (pp % 3) * TILE64);
    const uint32_t ma = smem_u32(mt);
#pragma unroll
    for (int j0 = 0; j0 < C; j0 += 16)
      umma_bf16(tm + cE + (pp & 1) * 128, desc_kmajor(ma, 128, 0, j0), desc_mnmajor(ga, 64, j0, 0),
                umma_idesc(128, 128, 0, 1), j0 > 0);
    umma_commit(&sh.ebar[pp & 1]);
  };
  auto issue_state_mma = [&](int pp) {
    const uint32_t xa = smem_u32(x_stage(pp)), ya = smem_u32(y_stage(pp));
    tc_fence_after();
#pragma unroll
    for (int k0 = 0; k0 < C; k0 += 16)   // (SUM: every chunk accumulates into the first tile)
      umma_bf16(tm + cS + (SUM ? 0 : (pp & 1) * 128), desc_mnmajor(xa, 64, k0, 0), desc_mnmajor(ya, 64, k0, 0),
                umma_idesc(128, 128, 1, 1), k0 > 0 || (SUM && pp > 0));
    if (SPLIT) {
      const uint32_t xla = smem_u32(x_low(pp));
#pragma unroll
      for (int k0 = 0; k0 < C; k0 += 16)
        umma_bf16(tm + cS, desc_mnmajor(xla, 64, k0, 0), desc_mnmajor(ya, 64, k0, 0), umma_idesc(128, 128, 1, 1), 1);
    }
    umma_commit(&sh.sbar[pp & 1]);
  };
  // gate x of chunk pp in place and publish G_n (and G_n - G_0, or G_0) of its channels
  // (SCALAR: they are the same for every channel and stay in the registers gn_next, e0_next of every thread)
  float gn_next = 0.f, e0_next = 0.f;
  auto gate_chunk = [&](int pp) {
    if ((!SCALAR && !mbar_wait(&sh.ebar[pp & 1], (pp >> 1) & 1)) || !mbar_wait(xy_bar(pp), xy_parity(pp))) {
      *abort_flag = 1;
      fail(1);
    }
    tc_fence_after();
    const int i = (q4 * 32 + lane) & 63;          // time row of this thread
    const int cg = (q4 >> 1) * 4 + seg;           // its 16 channels
    const int len = chunk_len(pp);
    const bool mine = !GEN || i < len;            // (a short chunk's foreign rows become zero)
    if (GEN && !mine) {
      uint8_t* yt = y_stage(pp) + (uint32_t)(cg >> 2) * SLAB64 + (uint32_t)i * 128u;
#pragma unroll
      for (int u = 0; u < 2; ++u)
        *reinterpret_cast<uint4*>(yt + (((uint32_t)((cg & 3) * 2 + u) ^ (uint32_t)i) & 7u) * 16u) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (SCALAR) {
      float g_lo, g_hi;
      gring.take(gate_index(pp), pp, lane, g_lo, g_hi);
      if (GEN) {
        g_lo = lane < len ? (p.gscalar ? g_lo : gconst) : 0.f;
        g_hi = lane + 32 < len ? (p.gscalar ? g_hi : gconst) : 0.f;
      }
      const WarpGates w = warp_cumulate(g_lo, g_hi, lane);
      const float Gi = (q4 & 1) ? w.hi : w.lo;
      gn_next = w.gn;
      e0_next = BWD ? w.g0 : w.gn - w.g0;
      const float f = BWD ? fast_exp(Gi + racc_s) * p.scale : fast_exp(w.gn - Gi + racc_s);
      if (SUM) racc_s += w.gn;
      uint8_t* xt = x_stage(pp);
      const uint32_t rowoff = (uint32_t)(cg >> 2) * SLAB64 + (uint32_t)i * 128u;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t off = rowoff + (((uint32_t)((cg & 3) * 2 + u) ^ (uint32_t)i) & 7u) * 16u;
        if constexpr (SPLIT) {
          uint4 l;
          const uint4 hi = scale8_by_split(*reinterpret_cast<const uint4*>(xt + off), f, l);
          *reinterpret_cast<uint4*>(xt + off) = mine ? hi : make_uint4(0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(x_low(pp) + off) = mine ? l : make_uint4(0u, 0u, 0u, 0u);
        } else {
          *reinterpret_cast<uint4*>(xt + off) =
              mine ? scale8_by(*reinterpret_cast<const uint4*>(xt + off), f) : make_uint4(0u, 0u, 0u, 0u);
        }
      }
      fence_async_smem();
      tc_fence_before();
      return;
    }
    float e[16];
    tmem_ld16(tmem_addr(tm, lane_base, cE + (pp & 1) * 128 + cg * 16), e);
    if (i == 63) {
#pragma unroll
      for (int t = 0; t < 16; ++t) sh.gn[pp & 1][cg * 16 + t] = e[t];
      if (SUM) {
#pragma unroll
        for (int t = 0; t < 16; ++t) racc[((pp + 1) & 1) * D + cg * 16 + t] = racc[(pp & 1) * D + cg * 16 + t] + e[t];
      }
      if (!BWD) {
#pragma unroll
        for (int t = 0; t < 16; ++t) e[t] = 0.f;   // row 63 of TRI_REVN carries G_n, its own exponent is 0
      }
    }
    if (i == 0 && !SUM) {   // forward: G_n - G_0; reverse: G_0 (for the scale of the stored states)
#pragma unroll
      for (int t = 0; t < 16; ++t) sh.e0[pp & 1][cg * 16 + t] = e[t];
    }
    if (SUM) {
#pragma unroll
      for (int t = 0; t < 16; ++t) e[t] += racc[(pp & 1) * D + cg * 16 + t];
    }
#pragma unroll
    for (int t = 0; t < 16; ++t) e[t] = BWD ? fast_exp(e[t]) * p.scale : fast_exp(e[t]);
    uint8_t* xt = x_stage(pp);
    const uint32_t rowoff = (uint32_t)(cg >> 2) * SLAB64 + (uint32_t)i * 128u;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t off = rowoff + (((uint32_t)((cg & 3) * 2 + u) ^ (uint32_t)i) & 7u) * 16u;
      if constexpr (SPLIT) {
        uint4 l;
        const uint4 hi = scale8_split(*reinterpret_cast<const uint4*>(xt + off), e + 8 * u, l);
        *reinterpret_cast<uint4*>(xt + off) = mine ? hi : make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(x_low(pp) + off) = mine ? l : make_uint4(0u, 0u, 0u, 0u);
      } else {
        *reinterpret_cast<uint4*>(xt + off) =
            mine ? scale8(*reinterpret_cast<const uint4*>(xt + off), e + 8 * u) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
    fence_async_smem();
    tc_fence_before();
  };
  // forward states are stored as h * exp(mid) * scale, mid = (G_0 + G_n) / 2 = G_n - (G_n - G_0) / 2;
  // reverse states as dh * exp(G_n - mid) = dh * exp((G_n - G_0) / 2)
  auto gn_of = [&](int pp) { return SCALAR ? gn_next : sh.gn[pp & 1][col]; };   // (SCALAR: of the chunk gated last)
  auto state_scale = [&](int pp) {
    const float gnv = gn_of(pp), e0 = SCALAR ? e0_next : sh.e0[pp & 1][col];
    if (GEN && BWD && !SUM && seg == 0 && bp.vs == 0) {
      const unsigned any = __ballot_sync(0xffffffffu, wide_span(0.5f * (gnv + e0), 0.5f * (gnv - e0), chunk_len(pp)));
      if (lane == 0) p.wide[((size_t)(bp.slot + chunk_of(pp)) * p.H + h) * 4 + q4] = any != 0;
    }
    if (GEN) return BWD ? fast_exp(clamp_span(0.5f * (gnv - e0))) : fast_exp(clamp_span(gnv - 0.5f * e0)) * p.scale;
    return BWD ? fast_exp(0.5f * (gnv - e0)) : fast_exp(gnv - 0.5f * e0) * p.scale;
  };

  if (warp == 16) {
    // ------------------------------------------------------------------ products
    // The two issuing threads run the same barriers as the compute warps and never wait for one another: the
    // product thread's time is the tensor core's (an issue takes about as long as the product before it runs),
    // the copy thread's is spent waiting for products to release tiles.
    issue_gate_mma(0);
    if (NT > 1) issue_gate_mma(1);
    __syncwarp();
    bool ok = !__syncthreads_or(*abort_flag);   // chunk 0 is gated
    if (ok) {
      if (lane == 0) issue_state_mma(0);
      if (NT > 2) issue_gate_mma(2);
      __syncwarp();
    }
    for (int pp = 0; ok && pp < NT; ++pp) {
      // h'_pp is staged, chunk pp+1 is gated; every thread of the block sees the same verdict, so
      // all of them leave the loop at the same barrier
      if (__syncthreads_or(*abort_flag)) break;
      if (lane == 0 && pp + 1 < NT) issue_state_mma(pp + 1);
      if (pp + 3 < NT) issue_gate_mma(pp + 3);   // its exponent slot was read by the gating of chunk pp+1
      __syncwarp();
    }
  } else if (warp == 17) {
    // ------------------------------------------------------------------ copies
    bool ok = !__syncthreads_or(*abort_flag);
    if (ok && lane == 0 && !SCALAR && NT > 3) issue_g(3);    // into the stage of chunk 0, whose exponent product is complete
    for (int pp = 0; ok && pp < NT; ++pp) {
      // the store of chunk pp-1 has read its staging tile: after the barrier the compute warps may
      // overwrite it (with the state of chunk pp+1)
      if (lane == 0) tma_store_wait_read();
      if (__syncthreads_or(*abort_flag)) break;
      if (lane == 0) {
        if (keep_states) {
          const int hrow = (((bp.slot + chunk_of(pp)) * p.H + h) * VS + bp.vs) * D;
          tma_store_2d(&p.mst, hst + (pp & 1) * TILE128, 0, hrow);
          tma_store_2d(&p.mst, hst + (pp & 1) * TILE128 + TILE128 / 2, 64, hrow);
          tma_store_commit();
        }
        if (!SCALAR && pp + 4 < NT) issue_g(pp + 4);   // the stage of chunk pp+1, whose exponent product is complete
        if (pp + NXY < NT) {                       // the x/y stage of chunk pp is free once its state product is done
          if (!mbar_wait(&sh.sbar[pp & 1], (pp >> 1) & 1)) { *abort_flag = 1; fail(2); }
          if (pp + NXY != p.skip_xy) issue_xy(pp + NXY);
        }
      }
      __syncwarp();
    }
    if (lane == 0) tma_store_wait_all();
  } else {
    // ------------------------------------------------------------------ state in registers
    // fp32 state: row k = col, columns 32 seg .. + 31
    float S[32];
    load_state32(S, start_state, col, yc + seg * 32, K, V);
    float gtot = 0.f;   // summed log-gates of this thread's channel over the block's chunks
    gate_chunk(0);
    if (SCALAR) load_gates(3);
    bool ok = !__syncthreads_or(*abort_flag);
    float decay = 1.f, hscale = 1.f, gn_cur = 0.f;   // of the chunk whose state product comes next
    if (ok) {
      gn_cur = gn_of(0);
      decay = fast_exp(gn_cur);
      hscale = state_scale(0);
    }
    for (int pp = 0; ok && pp < NT; ++pp) {
      // the state this chunk starts from (bf16), in the form its consumers use: staged in shared
      // memory in the tile format of the states tensor map and written out by a TMA store
      gtot += gn_cur;   // (published by the gating of this chunk, one iteration ago)
      if (keep_states) {
        uint8_t* tile = hst + (pp & 1) * TILE128;
#pragma unroll
        for (int j = 0; j < 32; j += 8)
          *reinterpret_cast<uint4*>(tile + tile_off(128, col, seg * 32 + j)) =
              make_uint4(pack_bf16(S[j] * hscale, S[j + 1] * hscale), pack_bf16(S[j + 2] * hscale, S[j + 3] * hscale),
                         pack_bf16(S[j + 4] * hscale, S[j + 5] * hscale), pack_bf16(S[j + 6] * hscale, S[j + 7] * hscale));
        fence_async_smem();
      }
      if (pp + 1 < NT) gate_chunk(pp + 1);
      if (__syncthreads_or(*abort_flag)) { ok = false; break; }
      float decay_n = 1.f, hscale_n = 1.f, gn_n = 0.f;
      if (pp + 1 < NT) {
        gn_n = gn_of(pp + 1);
        decay_n = fast_exp(gn_n);
        hscale_n = state_scale(pp + 1);
      }
      if (SCALAR) load_gates(pp + 4);
      // (SUM: the wait only keeps this thread within one phase of the barrier; the product was issued a chunk ago)
      if (!mbar_wait(&sh.sbar[pp & 1], (pp >> 1) & 1)) { *abort_flag = 1; fail(2); }
      tc_fence_after();
      if (!SUM) {
        float d[32];
        tmem_ld32(tmem_addr(tm, lane_base, cS + (pp & 1) * 128 + seg * 32), d);
#pragma unroll
        for (int t = 0; t < 32; ++t) S[t] = fmaf(S[t], decay, d[t]);
      }
      tc_fence_before();
      decay = decay_n;
      hscale = hscale_n;
      gn_cur = gn_n;
    }
    if (SUM && ok) {   // every product has completed: the accumulated tile is the state after the block's chunks
      tc_fence_after();
      tmem_ld32(tmem_addr(tm, lane_base, cS + seg * 32), S);
      tc_fence_before();
    }
    // (SUM: what the join needs, per run; otherwise the join has written the final state of a sequence cut into runs)
    if (ok && p.s_final && (SUM || bp.cnt == 1))
      store_state32(p.s_final + (SUM ? bp.sidx : bp.seqh) * K * V, S, col, yc + seg * 32, K, V);
    if (ok && p.gsum && seg == 0 && bp.vs == 0) p.gsum[bp.sidx * D + col] = gtot;
    // (a loop left early may leave gate copies of this thread in flight: they land before the block ends)
    if (SCALAR) asm volatile("cp.async.wait_all;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 512);
  if (tid == 0 && sh.abort_flag) {
    if (p.states) poison(p.states + ((size_t)((bp.slot + chunk_of(0)) * p.H + h) * VS + bp.vs) * D * D);
    if (p.s_final && (SUM || bp.cnt == 1)) poison(p.s_final + (SUM ? bp.sidx : bp.seqh) * K * V + yc);
    if (p.gsum) poison(p.gsum + bp.sidx * D);
  }
}

// Joins the time segments of each (batch, head).  A segment acts on the state entering it as
// h_out = h_in * exp(P) + S, with P the summed log-gates of its chunks (per channel) and S its end
// state from a zero start.  Forward order for states, reverse order for state gradients.
//   first [BH,K,V] or null;  P [BH,nseg,K];  S [BH,nseg,K,V];  start [BH,nseg,K,V] (out);  last [BH,K,V] or null (out)
template <bool REVERSE>
__global__ void k_join_segments(const float* __restrict__ first, const float* __restrict__ P, const float* __restrict__ S,
                                float* __restrict__ start, float* __restrict__ last, int nseg) {
  // grid (batch x head, slices): a block chains one slice of the K x V elements of one (batch, head)
  // (the loads of a step do not depend on the chain: unrolled, they are all in flight together)
  const int bh = blockIdx.x;
  const int span = D * D / gridDim.y;
  for (int e = blockIdx.y * span + threadIdx.x * 4; e < (blockIdx.y + 1) * span; e += blockDim.x * 4) {
    const int k = e / D;
    float4 cur = first ? *reinterpret_cast<const float4*>(first + (size_t)bh * D * D + e) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int i = 0; i < nseg; ++i) {
      const int r = REVERSE ? nseg - 1 - i : i;
      const size_t sb = ((size_t)bh * nseg + r) * D * D + e;
      *reinterpret_cast<float4*>(start + sb) = cur;
      const float w = __expf(P[((size_t)bh * nseg + r) * D + k]);
      const float4 add = *reinterpret_cast<const float4*>(S + sb);
      cur = make_float4(fmaf(cur.x, w, add.x), fmaf(cur.y, w, add.y), fmaf(cur.z, w, add.z), fmaf(cur.w, w, add.w));
    }
    if (last) *reinterpret_cast<float4*>(last + (size_t)bh * D * D + e) = cur;
  }
}

// The same for the general form: states are [K, V] per (sequence, head), segments of sequence n are
// [seg0[n], seg0[n+1]) (packed) or n * nseg .. (dense).  Sequences of one segment need no join.
template <bool REVERSE>
__global__ void k_join_segments_gen(const float* __restrict__ first, const float* __restrict__ P, const float* __restrict__ S,
                                    float* __restrict__ start, float* __restrict__ last, const int* __restrict__ seg0, int nseg,
                                    int H, int K, int V) {
  const int n = blockIdx.x / H, h = blockIdx.x - n * H;
  const int s0 = seg0 ? seg0[n] : n * nseg, cnt = seg0 ? seg0[n + 1] - s0 : nseg;
  if (cnt == 1) return;
  const size_t KV = (size_t)K * V;
  for (size_t e = (blockIdx.y * blockDim.x + threadIdx.x) * 4; e < KV; e += (size_t)gridDim.y * blockDim.x * 4) {
    const int k = (int)(e / V);
    float4 cur = first ? *reinterpret_cast<const float4*>(first + (size_t)blockIdx.x * KV + e) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int i = 0; i < cnt; ++i) {
      const size_t r = (size_t)(s0 + (REVERSE ? cnt - 1 - i : i)) * H + h;
      *reinterpret_cast<float4*>(start + r * KV + e) = cur;
      const float w = __expf(P[r * D + k]);
      const float4 add = *reinterpret_cast<const float4*>(S + r * KV + e);
      cur = make_float4(fmaf(cur.x, w, add.x), fmaf(cur.y, w, add.y), fmaf(cur.z, w, add.z), fmaf(cur.w, w, add.w));
    }
    if (last) *reinterpret_cast<float4*>(last + (size_t)blockIdx.x * KV + e) = cur;
  }
}

// Tables of a packed batch, written from the kernel's own parameters: no host buffer has to outlive the call and
// nothing goes through the copy engine.  The words start with (first token, end, first chunk slot) of every
// sequence; when all of them are in this launch (N > 0) it also writes the chunk table.
template <int W> struct PlanWords { int w[W]; };
constexpr int kPlanSmall = 1000, kPlanLarge = 8000;   // kernel parameters hold 4 KB cheaply, 32764 bytes at most
__device__ __forceinline__ void plan_chunks(const int* seqs, int N, ChunkEntry* chunks) {
  for (int n = blockIdx.x; n < N; n += gridDim.x) {
    const int row = seqs[3 * n], end = seqs[3 * n + 1], slot = seqs[3 * n + 2];
    for (int c = threadIdx.x; row + c * C < end; c += blockDim.x) chunks[slot + c] = ChunkEntry{row + c * C, end};
  }
}
template <int W>
__global__ void k_plan(const __grid_constant__ PlanWords<W> src, int* dst, int n, int N, ChunkEntry* chunks) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src.w[i];
  plan_chunks(src.w, N, chunks);
}
__global__ void k_plan_chunks(const int* __restrict__ seqs, int N, ChunkEntry* __restrict__ chunks) {
  plan_chunks(seqs, N, chunks);
}

// ===========================================================================
// Forward output
// ===========================================================================
struct FwdOParams {
  CUtensorMap mq, mk, mg, mv, mh;
  const __nv_bfloat16* gscalar;   // scalar gates [B,T,H] (SCALAR kernel; mg is unused then)
  __nv_bfloat16* o;
  int T, H, NT;
  float scale;
};

// SCALAR: no gate tile and no exponent product; every warp cumulates the chunk's 64 gates in registers.
template <bool SCALAR>
__global__ void __launch_bounds__(NTHREADS, 2) k_fwd_o(const __grid_constant__ FwdOParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* qs = smem;                 // q -> q~ in place
  uint8_t* ks = qs + TILE64;          // k -> k~ in place
  uint8_t* gs = ks + TILE64;          // g; later the bf16 intra matrix (first 8 KB)
  uint8_t* vt = gs + TILE64;
  uint8_t* hs = vt + TILE64;          // h_c exp(mid) scale, 128 x 128 (scaled by the scan kernel)
  uint8_t* mt = hs + TILE128;         // TRI_MID pattern, 64 x 64
  __shared__ uint64_t bar_load, bar_e, bar_a, bar_o;
  __shared__ uint32_t tmem_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q4 = warp & 3, seg = warp >> 2;
  // heads vary fastest over the blocks in flight: together they read whole token rows of the
  // [B,T,H,D] activations (all heads of a time step are contiguous in memory)
  const int h = blockIdx.x, ci = blockIdx.y, b = blockIdx.z;
  const int row = b * p.T + ci * C;
  constexpr uint32_t cO = 0, cE = 0, cA = 128;   // E is consumed before O is produced

  if (tid == 0) {
    mbar_init(&bar_load, 1); mbar_init(&bar_e, 1); mbar_init(&bar_a, 1); mbar_init(&bar_o, 1);
    fence_barrier_init();
    mbar_expect_tx(&bar_load, (SCALAR ? 3 : 4) * TILE64 + TILE128);
    if (!SCALAR) { tma_load_3d(gs, &p.mg, &bar_load, 0, h, row); tma_load_3d(gs + SLAB64, &p.mg, &bar_load, 64, h, row); }
    tma_load_3d(qs, &p.mq, &bar_load, 0, h, row); tma_load_3d(qs + SLAB64, &p.mq, &bar_load, 64, h, row);
    tma_load_3d(ks, &p.mk, &bar_load, 0, h, row); tma_load_3d(ks + SLAB64, &p.mk, &bar_load, 64, h, row);
    tma_load_3d(vt, &p.mv, &bar_load, 0, h, row); tma_load_3d(vt + SLAB64, &p.mv, &bar_load, 64, h, row);
    const int hrow = ((b * p.NT + ci) * p.H + h) * D;
    tma_load_2d(hs, &p.mh, &bar_load, 0, hrow); tma_load_2d(hs + TILE128 / 2, &p.mh, &bar_load, 64, hrow);
  }
  __syncwarp();
  if (warp == 0) { tmem_alloc(&tmem_slot, 256); tmem_relinquish(); }
  __nv_bfloat16 greg_lo = __float2bfloat16(0.f), greg_hi = greg_lo;   // SCALAR: the gates of time steps lane and lane + 32
  if (SCALAR) {   // (one chunk per block: the loads have the whole tile fetch to land)
    const __nv_bfloat16* src = p.gscalar + (size_t)(row + lane) * p.H + h;
    greg_lo = src[0];
    greg_hi = src[(size_t)32 * p.H];
  } else {
    build_tri_tile(mt, 64, TRI_MID);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = tmem_slot;
  const uint32_t lane_base = q4 * 32;
  bool ok = __syncthreads_and(mbar_wait(&bar_load, 0));
  if (!ok) fail(3);
  if (!SCALAR && ok && tid == 0) {
    tc_fence_after();
    const uint32_t ga = smem_u32(gs), ma = smem_u32(mt);
#pragma unroll
    for (int j0 = 0; j0 < C; j0 += 16)   // E = G - mid, [time][channel]
      umma_bf16(tm + cE, desc_kmajor(ma, 64, 0, j0), desc_mnmajor(ga, 64, j0, 0), umma_idesc(64, 128, 0, 1), j0 > 0);
    umma_commit(&bar_e);
  }
  __syncwarp();
  if (!SCALAR && ok) {
    ok = __syncthreads_and(mbar_wait(&bar_e, 0));
    if (!ok) fail(9);
  }
  if (SCALAR && ok) {
    // thread (q4, lane < 16, seg) gates 32 channels of time row 16 q4 + lane, whose cumulative gate sits in
    // lane (16 q4 + lane) mod 32 of the warp
    const WarpGates w = warp_cumulate(__bfloat162float(greg_lo), __bfloat162float(greg_hi), lane);
    const int i = 16 * q4 + (lane & 15);
    const float E = __shfl_sync(0xffffffffu, (q4 >> 1) ? w.hi : w.lo, i & 31) - w.mid();
    const float f = fast_exp(E), r = fast_exp(-E);
    if (lane < 16) {
      const uint32_t rowoff = (uint32_t)(seg >> 1) * SLAB64 + (uint32_t)i * 128u;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t off = rowoff + (((uint32_t)((seg & 1) * 4 + u) ^ (uint32_t)i) & 7u) * 16u;
        const uint4 qr = *reinterpret_cast<const uint4*>(qs + off), kr = *reinterpret_cast<const uint4*>(ks + off);
        *reinterpret_cast<uint4*>(qs + off) = scale8_by(qr, f);
        *reinterpret_cast<uint4*>(ks + off) = scale8_by(kr, r);
      }
    }
    fence_async_smem();
    tc_fence_before();
  }
  if (!SCALAR && ok) {
    tc_fence_after();
    float e[32];
    tmem_ld32(tmem_addr(tm, lane_base, cE + seg * 32), e);
    if (lane < 16) {   // rows of an M = 64 accumulator sit in lanes 0..15 of each 32-lane quarter
      const int i = 16 * q4 + lane;
      const uint32_t rowoff = (uint32_t)(seg >> 1) * SLAB64 + (uint32_t)i * 128u;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t off = rowoff + (((uint32_t)((seg & 1) * 4 + u) ^ (uint32_t)i) & 7u) * 16u;
        float f[8], r[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) { f[t] = fast_exp(e[8 * u + t]); r[t] = fast_exp(-e[8 * u + t]); }
        const uint4 qr = *reinterpret_cast<const uint4*>(qs + off), kr = *reinterpret_cast<const uint4*>(ks + off);
        *reinterpret_cast<uint4*>(qs + off) = scale8(qr, f);
        *reinterpret_cast<uint4*>(ks + off) = scale8(kr, r);
      }
    }
    fence_async_smem();
    tc_fence_before();
  }
  __syncthreads();
  if (ok && tid == 0) {
    tc_fence_after();
    const uint32_t qa = smem_u32(qs), ka = smem_u32(ks), ha = smem_u32(hs);
#pragma unroll
    for (int k0 = 0; k0 < D; k0 += 16)   // A = q~ k~^T
      umma_bf16(tm + cA, desc_kmajor(qa, 64, 0, k0), desc_kmajor(ka, 64, 0, k0), umma_idesc(64, 64, 0, 0), k0 > 0);
    umma_commit(&bar_a);
#pragma unroll
    for (int k0 = 0; k0 < D; k0 += 16)   // o = q~ h'
      umma_bf16(tm + cO, desc_kmajor(qa, 64, 0, k0), desc_mnmajor(ha, 128, k0, 0), umma_idesc(64, 128, 0, 1), k0 > 0);
  }
  __syncwarp();
  if (ok) {
    ok = __syncthreads_and(mbar_wait(&bar_a, 0));
    if (!ok) fail(4);
  }
  if (ok) {
    tc_fence_after();
    const int i = 16 * q4 + lane;
    float a[16];
    tmem_ld16(tmem_addr(tm, lane_base, cA + seg * 16), a);
    if (lane < 16) store_tril16(gs, i, seg * 16, a, p.scale);
    fence_async_smem();
    tc_fence_before();
  }
  __syncthreads();
  if (ok && tid == 0) {
    tc_fence_after();
    const uint32_t pa = smem_u32(gs), va = smem_u32(vt);
#pragma unroll
    for (int k0 = 0; k0 < C; k0 += 16)   // o += A v
      umma_bf16(tm + cO, desc_kmajor(pa, 64, 0, k0), desc_mnmajor(va, 64, k0, 0), umma_idesc(64, 128, 0, 1), 1);
    umma_commit(&bar_o);
  }
  __syncwarp();
  if (ok) {
    ok = __syncthreads_and(mbar_wait(&bar_o, 0));
    if (!ok) fail(5);
  }
  if (ok) {
    tc_fence_after();
    const int i = 16 * q4 + lane;
    __nv_bfloat16* dst = p.o + ((size_t)(row + i) * p.H + h) * D + seg * 32;
    float a[32];
    tmem_ld32(tmem_addr(tm, lane_base, cO + seg * 32), a);
    if (lane < 16) {
#pragma unroll
      for (int t = 0; t < 32; t += 8)
        *reinterpret_cast<uint4*>(dst + t) = make_uint4(pack_bf16(a[t], a[t + 1]), pack_bf16(a[t + 2], a[t + 3]),
                                                        pack_bf16(a[t + 4], a[t + 5]), pack_bf16(a[t + 6], a[t + 7]));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 256);
  if (tid == 0 && !ok) poison(p.o + ((size_t)row * p.H + h) * D);
}

// ===========================================================================
// Fused forward: state scan and chunk outputs in one pass
// ===========================================================================
// One block per (batch, head) walks its chunks in order with the K x V state in registers, so the
// chunk-start state never has to come back from HBM: per chunk it is staged once in shared memory
// as the bf16 operand h' = h exp(mid) scale of the output product (and, when the caller keeps the
// states for a backward pass, written out from there by a TMA store).  q, k, g, v are read once.
//   exponents  E = G - mid   [time (repeated to 128 lanes)][channel]      (pattern TRI_MID)
//              W[channel][0] = G_n,  W[channel][1] = G_n - mid            (pattern rows: ones, TRI_MID row 63)
//   gating     q~ = q exp(E), k~ = k exp(-E) in place
//   products   A = q~ k~^T;  o = q~ h' + tril(A) scale v;  D = k~^T v
//   state      h <- h exp(G_n) + exp(G_n - mid) D      (k exp(G_n - G) = k~ exp(G_n - mid), per channel)
// 16 compute warps (thread (q4, lane, seg): state row k = 32 q4 + lane, columns 32 seg .. + 31) and a
// driver warp that issues every product and copy; two block-wide barriers per chunk.
struct FusedParams {
  CUtensorMap mq, mk, mg, mv;
  CUtensorMap mst;         // the states tensor as [B*NT*H*128, 128] (TMA stores); unused when states == nullptr
  const float* s0;         // state each block starts from: [B,H,nseg,K,V] or null (zero)
  const float* s0_seg;     // GEN: the same for the runs of a sequence that is cut into several
  __nv_bfloat16* states;   // h' [B,T/64,H,K,V] or null
  float* s_final;          // state each block ends with: [B,H,nseg,K,V] or null
  __nv_bfloat16* o;        // [B,T,H,V]
  const __nv_bfloat16* gscalar;   // scalar gates [B,T,H] (SCALAR kernel; mg is unused then)
  int T, H, NT;            // T: tokens per sequence; NT: chunks per block (T / 64 / nseg)
  int nseg;                // time segments per sequence, one block each
  float scale;
  const float* gamma;      // constant gates [H] (SCALAR GEN kernel)
  Geo geo;                 // GEN kernel
  const __nv_bfloat16 *q, *k, *g;   // GEN: what the tensor maps fetch, for wide chunks
  long long qk_pitch;               // GEN: elements between tokens of q and k
};
struct FusedShared {
  uint64_t fullin[2], ebar, abar, sbar, obar;
  uint32_t tmem_slot;
  int abort_flag;
  int wide_at[2];   // WIDE: the last wide chunk of either parity
};
constexpr uint32_t FUSED_STAGE = 4 * TILE64;   // q, k, g, v
constexpr size_t FUSED_SMEM = 2 * FUSED_STAGE + 2 * TILE128 + 2 * SLAB64 + 2048 + TILE64 + sizeof(FusedShared);

// SCALAR: no gate tile is fetched and no exponent product issued; every compute warp cumulates the chunk's 64
// gates in registers (warp_cumulate), which gives its threads E of their time row, G_n and mid directly.
// WIDE: the walk over the run once more, where it has wide chunks (see kSpan): the tiles go by clamped references, and a
// wide chunk's tril(A) and gated operands are formed by the CUDA cores.  Returns whether the run has to be walked again.
template <bool SCALAR, bool GEN, bool WIDE>
__device__ __forceinline__ bool fused_walk(const FusedParams& p, uint8_t* smem) {
  uint8_t* in = smem;                         // 2 stages x (q, k, g, v)
  uint8_t* hst = in + 2 * FUSED_STAGE;        // 2 x (128 x 128) bf16: h' of the current chunk
  uint8_t* qlo = hst + TILE128;               // GEN: one h' tile; what bf16 leaves of q~ (then of A) and of k~
  uint8_t* klo = qlo + TILE64;
  uint8_t* mt = hst + 2 * TILE128;            // TRI_MID pattern, rows repeated to 128
  uint8_t* wt = mt + 2 * SLAB64;              // 16 x 64 pattern for G_n and G_n - mid
  uint8_t* ost = wt + 2048;                   // 64 x 128 bf16: the outputs of a chunk, row-major, before they leave
  FusedShared& sh = *reinterpret_cast<FusedShared*>(ost + TILE64);
  volatile int* abort_flag = &sh.abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool driver = warp == 16;
  const int q4 = warp & 3, seg = (warp >> 2) & 3, col = q4 * 32 + lane;
  BlockPos bp;
  if constexpr (GEN) {
    bp = block_pos(p.geo, p.T, p.H, blockIdx.x);
  } else {
    const int sg = blockIdx.x % p.nseg, bh = blockIdx.x / p.nseg, b = bh / p.H;
    bp.h = bh % p.H; bp.vs = 0; bp.row = b * p.T + sg * p.NT * C; bp.end = (b + 1) * p.T;
    bp.slot = b * (p.T / C) + sg * p.NT; bp.nch = p.NT; bp.sidx = bp.seqh = blockIdx.x; bp.cnt = 1;
  }
  const int h = bp.h, NT = bp.nch;
  const int VS = GEN ? p.geo.VS : 1, K = GEN ? p.geo.K : D, V = GEN ? p.geo.V : D;
  const int yc = bp.vs * D;   // first value channel of this block's slice
  const float* const start_state = (GEN && bp.cnt > 1) ? p.s0_seg + bp.sidx * K * V
                                                       : (p.s0 ? p.s0 + bp.seqh * K * V : nullptr);
  auto chunk_len = [&](int pp) { return GEN ? min(C, bp.end - (bp.row + pp * C)) : C; };
  constexpr uint32_t cE = 0, cD = 128, cO = 256, cA = 384, cW = 448;
  auto issue_load = [&](int pp) {
    uint8_t* qs = in + (pp & 1) * FUSED_STAGE;
    uint8_t *ks = qs + TILE64, *gs = ks + TILE64, *vs = gs + TILE64;
    uint64_t* bar = &sh.fullin[pp & 1];
    const int row = bp.row + pp * C;
    mbar_expect_tx(bar, SCALAR ? 3 * TILE64 : FUSED_STAGE);
    if (!SCALAR) { tma_load_3d(gs, &p.mg, bar, 0, h, row); tma_load_3d(gs + SLAB64, &p.mg, bar, 64, h, row); }
    tma_load_3d(qs, &p.mq, bar, 0, h, row); tma_load_3d(qs + SLAB64, &p.mq, bar, 64, h, row);
    tma_load_3d(ks, &p.mk, bar, 0, h, row); tma_load_3d(ks + SLAB64, &p.mk, bar, 64, h, row);
    tma_load_3d(vs, &p.mv, bar, yc, h, row); tma_load_3d(vs + SLAB64, &p.mv, bar, yc + 64, h, row);
  };
  if (tid == 0) {
    if (WIDE)
      for (uint64_t* bar : {&sh.fullin[0], &sh.fullin[1], &sh.ebar, &sh.abar, &sh.sbar, &sh.obar}) mbar_inval(bar);
    mbar_init(&sh.fullin[0], 1); mbar_init(&sh.fullin[1], 1);
    mbar_init(&sh.ebar, 1); mbar_init(&sh.abar, 1); mbar_init(&sh.sbar, 1); mbar_init(&sh.obar, 1);
    fence_barrier_init();
    tma_prefetch_desc(&p.mq); tma_prefetch_desc(&p.mk); tma_prefetch_desc(&p.mv);
    if (!SCALAR) tma_prefetch_desc(&p.mg);
    sh.abort_flag = 0;
    if (WIDE) sh.wide_at[0] = sh.wide_at[1] = -1;
    issue_load(0);
    if (NT > 1) issue_load(1);
  }
  __syncwarp();
  if (!WIDE && warp == 0) { tmem_alloc(&sh.tmem_slot, 512); tmem_relinquish(); }
  // SCALAR: the gates of time steps lane and lane + 32 of the next chunk, in registers, loaded right after the
  // first barrier of the chunk before: a chunk is long enough here for the load to land before the loop's back
  // edge (where a register with a load in flight stalls the warp; the state scans, whose chunks are short, use
  // GateRing instead)
  __nv_bfloat16 greg_lo = __float2bfloat16(0.f), greg_hi = greg_lo;
  auto load_gates = [&](int c) {
    if (GEN && !p.gscalar) return;
    const __nv_bfloat16* src = p.gscalar + (size_t)(bp.row + c * C + lane) * p.H + h;
    if (!GEN || lane < chunk_len(c)) greg_lo = src[0];
    if (!GEN || lane + 32 < chunk_len(c)) greg_hi = src[(size_t)32 * p.H];
  };
  const float gconst = (GEN && SCALAR && p.gamma) ? p.gamma[h] : 0.f;   // GEN: a constant decay, or none
  if (SCALAR) {
    if (!driver) load_gates(0);
  } else {
    build_tri_tile(mt, 128, TRI_MID);
    build_w_tile(wt);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = sh.tmem_slot;
  const uint32_t lane_base = q4 * 32;
  bool wide_any = false;   // GEN: this thread has seen a wide chunk
  // (known after B1)
  auto wide_chunk = [&](int pp) { return WIDE && *reinterpret_cast<volatile int*>(&sh.wide_at[pp & 1]) == pp; };

  if (driver) {
    // ------------------------------------------------------------------ products and copies
    // (called by the whole driver warp: a short chunk's foreign gate rows are zeroed first)
    auto issue_exponents = [&](int pp) {
      if (SCALAR) return;
      if (GEN && chunk_len(pp) < C) {
        if (!mbar_wait(&sh.fullin[pp & 1], (pp >> 1) & 1)) { *abort_flag = 1; fail(3); }
        zero_rows(in + (pp & 1) * FUSED_STAGE + 2 * TILE64, chunk_len(pp), lane, 32);
        fence_async_smem();
        __syncwarp();
      }
      if (lane != 0) return;
      if (!mbar_wait(&sh.fullin[pp & 1], (pp >> 1) & 1)) { *abort_flag = 1; fail(3); }
      tc_fence_after();
      const uint32_t ga = smem_u32(in + (pp & 1) * FUSED_STAGE + 2 * TILE64), ma = smem_u32(mt), wa = smem_u32(wt);
#pragma unroll
      for (int j0 = 0; j0 < C; j0 += 16)   // E: [time (repeated)][channel]
        umma_bf16(tm + cE, desc_kmajor(ma, 128, 0, j0), desc_mnmajor(ga, 64, j0, 0), umma_idesc(128, 128, 0, 1), j0 > 0);
#pragma unroll
      for (int j0 = 0; j0 < C; j0 += 16)   // W: [channel][G_n, G_n - mid, 0 ...]
        umma_bf16(tm + cW, desc_mnmajor(ga, 64, j0, 0), desc_kmajor(wa, 16, 0, j0), umma_idesc(128, 16, 1, 0), j0 > 0);
      umma_commit(&sh.ebar);
    };
    issue_exponents(0);
    __syncwarp();
    for (int pp = 0; pp < NT; ++pp) {
      const uint32_t ph = pp & 1;
      uint8_t* qs = in + (pp & 1) * FUSED_STAGE;
      uint8_t *ks = qs + TILE64, *gs = ks + TILE64, *vs = gs + TILE64;
      uint8_t* ht = GEN ? hst : hst + (pp & 1) * TILE128;
      // the state store of chunk pp-1 has read its staging tile, which the compute warps refill after
      // the next barrier (with the state of chunk pp+1)
      if (lane == 0) tma_store_wait_read();
      // B1: q~, k~ and h' of chunk pp are in shared memory, E and W have been read
      if (__syncthreads_or(*abort_flag)) break;
      const bool wide = wide_chunk(pp);
      if (wide && __syncthreads_or(*abort_flag)) break;   // q~, k~ once more, tril(A) scale
      if (lane == 0) {
        tc_fence_after();
        const uint32_t qa = smem_u32(qs), ka = smem_u32(ks), va = smem_u32(vs), ha = smem_u32(ht);
        if (!wide) {
#pragma unroll
          for (int k0 = 0; k0 < D; k0 += 16)   // A = q~ k~^T
            umma_bf16(tm + cA, desc_kmajor(qa, 64, 0, k0), desc_kmajor(ka, 64, 0, k0), umma_idesc(64, 64, 0, 0), k0 > 0);
        }
        if (GEN && !wide) {
          const uint32_t qla = smem_u32(qlo), kla = smem_u32(klo);
#pragma unroll
          for (int k0 = 0; k0 < D; k0 += 16)
            umma_bf16(tm + cA, desc_kmajor(qa, 64, 0, k0), desc_kmajor(kla, 64, 0, k0), umma_idesc(64, 64, 0, 0), 1);
#pragma unroll
          for (int k0 = 0; k0 < D; k0 += 16)
            umma_bf16(tm + cA, desc_kmajor(qla, 64, 0, k0), desc_kmajor(ka, 64, 0, k0), umma_idesc(64, 64, 0, 0), 1);
        }
        umma_commit(&sh.abar);
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)   // D[k][v] = sum_j k~[j][k] v[j][v]
          umma_bf16(tm + cD, desc_mnmajor(ka, 64, k0, 0), desc_mnmajor(va, 64, k0, 0), umma_idesc(128, 128, 1, 1), k0 > 0);
        if (GEN) {
          const uint32_t kla = smem_u32(klo);
#pragma unroll
          for (int k0 = 0; k0 < C; k0 += 16)
            umma_bf16(tm + cD, desc_mnmajor(kla, 64, k0, 0), desc_mnmajor(va, 64, k0, 0), umma_idesc(128, 128, 1, 1), 1);
        }
        umma_commit(&sh.sbar);
#pragma unroll
        for (int k0 = 0; k0 < D; k0 += 16)   // o = q~ h'
          umma_bf16(tm + cO, desc_kmajor(qa, 64, 0, k0), desc_mnmajor(ha, 128, k0, 0), umma_idesc(64, 128, 0, 1), k0 > 0);
        if (p.states) {
          const int hrow = (((bp.slot + pp) * p.H + h) * VS + bp.vs) * D;
          tma_store_2d(&p.mst, ht, 0, hrow);
          tma_store_2d(&p.mst, ht + TILE128 / 2, 64, hrow);
          tma_store_commit();
          if (GEN) tma_store_wait_read();   // (the one h' tile is refilled after B2)
        }
      }
      // B2: tril(A) scale is in shared memory (in the gate tile of this stage)
      if (__syncthreads_or(*abort_flag)) break;
      if (lane == 0) {
        tc_fence_after();
        const uint32_t pa = smem_u32(gs), va = smem_u32(vs);
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)   // o += tril(A) scale v
          umma_bf16(tm + cO, desc_kmajor(pa, 64, 0, k0), desc_mnmajor(va, 64, k0, 0), umma_idesc(64, 128, 0, 1), 1);
        if (GEN) {
          const uint32_t pla = smem_u32(qlo);
#pragma unroll
          for (int k0 = 0; k0 < C; k0 += 16)
            umma_bf16(tm + cO, desc_kmajor(pla, 64, 0, k0), desc_mnmajor(va, 64, k0, 0), umma_idesc(64, 128, 0, 1), 1);
        }
        umma_commit(&sh.obar);
      }
      // exponents of the next chunk (E and W of this one were read before B1)
      if (pp + 1 < NT) issue_exponents(pp + 1);
      // every tile of this stage is dead once its products are complete
      if (lane == 0 && pp + 2 < NT) {
        if (!mbar_wait(&sh.obar, ph)) { *abort_flag = 1; fail(5); }
        issue_load(pp + 2);
      }
      __syncwarp();
    }
    __syncthreads();   // (the compute warps copy the last outputs after this barrier)
    if (lane == 0) tma_store_wait_all();
  } else {
    // ------------------------------------------------------------------ state in registers
    float S[32];
    load_state32(S, start_state, col, yc + seg * 32, K, V);
    // Outputs leave in two steps: the accumulator rows (an M = 64 accumulator keeps 16 rows in the first
    // 16 lanes of each warp) are packed to bf16 in a shared tile; after the next block-wide barrier every
    // thread copies 32 contiguous bytes of it, so that a warp writes whole 256-byte rows.
    auto copy_out = [&](int pp) {
      const int r = tid >> 3, piece = tid & 7;   // 64 rows x 8 pieces of 16 channels
      // 16-byte pieces of a row are stored XOR-permuted by the row number (bank conflicts of the writers)
      const uint8_t* rowp = ost + r * 256;
      uint4* dst = reinterpret_cast<uint4*>(p.o + ((size_t)(bp.row + pp * C + r) * p.H + h) * V + yc + piece * 16);
      const uint4 x = *reinterpret_cast<const uint4*>(rowp + (((2 * piece) ^ r) & 15) * 16);
      const uint4 y = *reinterpret_cast<const uint4*>(rowp + (((2 * piece + 1) ^ r) & 15) * 16);
      if (GEN && r >= chunk_len(pp)) return;
      if (!GEN || yc + piece * 16 < V) __stcs(dst, x);
      if (!GEN || yc + piece * 16 + 8 < V) __stcs(dst + 1, y);
    };
    bool ok = true;
    for (int pp = 0; ok && pp < NT; ++pp) {
      const uint32_t ph = pp & 1;
      uint8_t* qs = in + (pp & 1) * FUSED_STAGE;
      uint8_t *ks = qs + TILE64, *gs = ks + TILE64;
      uint8_t* ht = GEN ? hst : hst + (pp & 1) * TILE128;
      float* diag = reinterpret_cast<float*>(gs + SLAB64);   // GEN: partial q_i . k_i [8][64], in the consumed gate tile
      if (!mbar_wait(&sh.fullin[pp & 1], (pp >> 1) & 1) || (!SCALAR && !mbar_wait(&sh.ebar, ph))) { *abort_flag = 1; fail(9); }
      tc_fence_after();
      const int len = chunk_len(pp);
      WarpGates wg;
      if (SCALAR) {
        float g_lo = __bfloat162float(greg_lo), g_hi = __bfloat162float(greg_hi);
        if (GEN) {
          g_lo = lane < len ? (p.gscalar ? g_lo : gconst) : 0.f;
          g_hi = lane + 32 < len ? (p.gscalar ? g_hi : gconst) : 0.f;
        }
        wg = warp_cumulate(g_lo, g_hi, lane);
      }
      // per-channel factors of this thread's state row
      float decay, c2;
      float em[16];
      bool wide_here = false;
      {
        float w[8];
        if (SCALAR) {
          w[0] = wg.gn;
          w[1] = wg.gn - wg.mid();
        } else {
          tmem_ld8(tmem_addr(tm, lane_base, cW), w);
          // (the exponents of the gating below are fetched now: their exponentials interleave with the staging)
          tmem_ld16(tmem_addr(tm, lane_base, cE + ((q4 >> 1) * 4 + seg) * 16), em);
        }
        decay = fast_exp(w[0]);                    // exp(G_n)
        float mid = w[0] - w[1];
        if (GEN) wide_here = fabsf(mid) > kSpan || fabsf(w[1]) > kSpan;
        if (WIDE) {
          mid = clamp_span(mid);
          w[1] = clamp_span(w[1]);
        } else {
          wide_any |= wide_here;
        }
        c2 = fast_exp(w[1]);                       // exp(G_n - mid)
        const float hscale = fast_exp(mid) * p.scale;   // exp(mid) scale
#pragma unroll
        for (int j = 0; j < 32; j += 8)
          *reinterpret_cast<uint4*>(ht + tile_off(128, col, seg * 32 + j)) =
              make_uint4(pack_bf16(S[j] * hscale, S[j + 1] * hscale), pack_bf16(S[j + 2] * hscale, S[j + 3] * hscale),
                         pack_bf16(S[j + 4] * hscale, S[j + 5] * hscale), pack_bf16(S[j + 6] * hscale, S[j + 7] * hscale));
      }
      // gate q, k: thread (q4, lane, seg) owns time row (32 q4 + lane) mod 64 and 16 channels
      if (GEN && ((q4 * 32 + lane) & 63) >= len) {   // a short chunk's foreign rows of q, k, v become zero
        const int i = (q4 * 32 + lane) & 63, cg = (q4 >> 1) * 4 + seg;
        const uint32_t rowoff = (uint32_t)(cg >> 2) * SLAB64 + (uint32_t)i * 128u;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint32_t off = rowoff + (((uint32_t)((cg & 3) * 2 + u) ^ (uint32_t)i) & 7u) * 16u;
          *reinterpret_cast<uint4*>(qs + off) = make_uint4(0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(ks + off) = make_uint4(0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(qlo + off) = make_uint4(0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(klo + off) = make_uint4(0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(gs + TILE64 + off) = make_uint4(0u, 0u, 0u, 0u);   // v
        }
      } else if (SCALAR) {
        const int i = (q4 * 32 + lane) & 63;
        const int cg = (q4 >> 1) * 4 + seg;
        const float E = ((q4 & 1) ? wg.hi : wg.lo) - wg.mid();
        const float f = fast_exp(E), r = fast_exp(-E);
        float dot = 0.f;
        const uint32_t rowoff = (uint32_t)(cg >> 2) * SLAB64 + (uint32_t)i * 128u;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint32_t off = rowoff + (((uint32_t)((cg & 3) * 2 + u) ^ (uint32_t)i) & 7u) * 16u;
          const uint4 qr = *reinterpret_cast<const uint4*>(qs + off), kr = *reinterpret_cast<const uint4*>(ks + off);
          if constexpr (GEN) {
            uint4 l;
            dot = dot8(qr, kr, dot);
            *reinterpret_cast<uint4*>(qs + off) = scale8_by_split(qr, f, l);
            *reinterpret_cast<uint4*>(qlo + off) = l;
            *reinterpret_cast<uint4*>(ks + off) = scale8_by_split(kr, r, l);
            *reinterpret_cast<uint4*>(klo + off) = l;
          } else {
            *reinterpret_cast<uint4*>(qs + off) = scale8_by(qr, f);
            *reinterpret_cast<uint4*>(ks + off) = scale8_by(kr, r);
          }
        }
        if (GEN) diag[cg * C + i] = dot;
      } else {
        float dot = 0.f;
        const int i = (q4 * 32 + lane) & 63;
        const int cg = (q4 >> 1) * 4 + seg;
        const uint32_t rowoff = (uint32_t)(cg >> 2) * SLAB64 + (uint32_t)i * 128u;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint32_t off = rowoff + (((uint32_t)((cg & 3) * 2 + u) ^ (uint32_t)i) & 7u) * 16u;
          float f[8], r[8];
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            f[t] = fast_exp(em[8 * u + t]);
            r[t] = fast_exp(-em[8 * u + t]);
          }
          const uint4 qr = *reinterpret_cast<const uint4*>(qs + off), kr = *reinterpret_cast<const uint4*>(ks + off);
          if constexpr (GEN) {
            uint4 l;
            dot = dot8(qr, kr, dot);
            *reinterpret_cast<uint4*>(qs + off) = scale8_split(qr, f, l);
            *reinterpret_cast<uint4*>(qlo + off) = l;
            *reinterpret_cast<uint4*>(ks + off) = scale8_split(kr, r, l);
            *reinterpret_cast<uint4*>(klo + off) = l;
          } else {
            *reinterpret_cast<uint4*>(qs + off) = scale8(qr, f);
            *reinterpret_cast<uint4*>(ks + off) = scale8(kr, r);
          }
        }
        if (GEN) diag[cg * C + i] = dot;
      }
      if (WIDE && wide_here) sh.wide_at[ph] = pp;
      fence_async_smem();
      tc_fence_before();
      if (__syncthreads_or(*abort_flag)) { ok = false; break; }   // B1
      if (pp > 0) copy_out(pp - 1);   // staged before the barrier; the products of this chunk run meanwhile
      if (SCALAR && pp + 1 < NT) load_gates(pp + 1);
      // tril(A) scale -> bf16 operand in the (dead) gate tile
      if (wide_chunk(pp)) {
        if constexpr (WIDE) {
          const size_t row = (size_t)bp.row + pp * C;
          RawChunk raw{p.q + row * p.qk_pitch + (size_t)h * K, p.k + row * p.qk_pitch + (size_t)h * K, nullptr, p.qk_pitch, 0, gconst, K, len};
          if (!SCALAR) { raw.g = p.g + (row * p.H + h) * K; raw.gstep = (long long)p.H * K; }
          else if (p.gscalar) { raw.g = p.gscalar + row * p.H + h; raw.gstep = p.H; }
          wide_operands<SCALAR>(raw, qs, ks, klo, col, seg);
          wide_matrix<SCALAR>(raw, gs, qlo, p.scale, warp, lane);
        }
        fence_async_smem();
        if (__syncthreads_or(*abort_flag)) { ok = false; break; }
      } else {
        if (!mbar_wait(&sh.abar, ph)) { *abort_flag = 1; fail(4); }
        tc_fence_after();
        const int i = 16 * q4 + lane;   // rows of an M = 64 accumulator sit in lanes 0..15 of each quarter
        float a[16];
        tmem_ld16(tmem_addr(tm, lane_base, cA + seg * 16), a);
        if (GEN && lane < 16 && seg == q4) set_diagonal(a, diag, 8, i, lane);
        if (lane < 16) {
          if (GEN) store_tril16_split(gs, qlo, i, seg * 16, a, p.scale);   // (q~'s lower half has been read)
          else store_tril16(gs, i, seg * 16, a, p.scale);
        }
      }
      fence_async_smem();
      tc_fence_before();
      if (__syncthreads_or(*abort_flag)) { ok = false; break; }   // B2
      // state update while the last output product runs
      if (!mbar_wait(&sh.sbar, ph)) { *abort_flag = 1; fail(2); }
      tc_fence_after();
      {
        float d[32];
        tmem_ld32(tmem_addr(tm, lane_base, cD + seg * 32), d);
#pragma unroll
        for (int t = 0; t < 32; ++t) S[t] = fmaf(S[t], decay, c2 * d[t]);
      }
      if (!mbar_wait(&sh.obar, ph)) { *abort_flag = 1; fail(5); }
      tc_fence_after();
      {
        const int i = 16 * q4 + lane;
        float a[32];
        tmem_ld32(tmem_addr(tm, lane_base, cO + seg * 32), a);
        if (lane < 16) {
#pragma unroll
          for (int t = 0; t < 32; t += 8)
            *reinterpret_cast<uint4*>(ost + i * 256 + (((seg * 4 + t / 8) ^ i) & 15) * 16) =
                make_uint4(pack_bf16(a[t], a[t + 1]), pack_bf16(a[t + 2], a[t + 3]), pack_bf16(a[t + 4], a[t + 5]),
                           pack_bf16(a[t + 6], a[t + 7]));
        }
      }
      tc_fence_before();
    }
    __syncthreads();   // the outputs of the last chunk are staged
    if (ok) copy_out(NT - 1);
    if (ok && p.s_final && bp.cnt == 1) store_state32(p.s_final + bp.seqh * K * V, S, col, yc + seg * 32, K, V);
  }
  tc_fence_before();
  const bool again = __syncthreads_or(wide_any) != 0;
  if (tid == 0 && sh.abort_flag) {
    poison(p.o + ((size_t)bp.row * p.H + h) * V + yc);
    if (p.s_final && bp.cnt == 1) poison(p.s_final + bp.seqh * K * V + yc);
  }
  return again && !sh.abort_flag;
}
// (a function of its own, so that the walk above has its registers to itself: with wide chunks taken care of inside it the
// kernel took 193 us where it takes 184, T = 16384 in 13 documents, H = 16)
template <bool SCALAR>
__device__ __noinline__ void fused_walk_wide(const FusedParams& p, uint8_t* smem) { fused_walk<SCALAR, true, true>(p, smem); }

template <bool SCALAR, bool GEN>
__global__ void __launch_bounds__(FUSED_THREADS) k_fwd_fused(const __grid_constant__ FusedParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0) {   // uniform over the block
    if (threadIdx.x == 0) fail(12);
    return;
  }
  const bool again = fused_walk<SCALAR, GEN, false>(p, smem);
  if constexpr (GEN) {
    if (again) fused_walk_wide<SCALAR>(p, smem);   // (o, states and final state are written once more)
  }
  if (threadIdx.x < 32) tmem_dealloc(reinterpret_cast<FusedShared*>(smem + FUSED_SMEM - sizeof(FusedShared))->tmem_slot, 512);
}

// ===========================================================================
// Backward of the chunks (persistent: each block walks chunks blockIdx.x,
// blockIdx.x + gridDim.x, ... and fetches the next chunk's tiles while the
// tensor core and the epilogue of the current one are still busy)
// ===========================================================================
struct BwdParams {
  CUtensorMap mq, mk, mg, mv, mdo, mh, mdh;
  void *dq, *dk, *dg;    // [B,T,H,K] fp32 or bf16 (dg may be null)
  __nv_bfloat16* dv;     // [B,T,H,V]
  const __nv_bfloat16* gscalar;   // scalar gates [B,T,H] (SCALAR kernels; mg is unused then)
  int T, H, NT, total;   // total = B * H * NT chunks
  float scale;
  const float* gamma;    // constant gates [H] (SCALAR GEN kernels)
  Geo geo;               // GEN kernels
  // GEN, V > 128: one launch per value slice.  dq, dk and dg are sums over the slices: every launch but the last
  // writes fp32 partial sums, every launch but the first adds the partial sums of the one before.
  int vs;
  const float *add_dq, *add_dk, *add_dg;   // null: nothing to add
  long long dqk_pitch, dv_pitch;           // GEN: elements between tokens of dq and dk, and of dv
  const __nv_bfloat16 *q, *k, *g;          // WIDE: what the tensor maps fetch
  long long qk_pitch;                      // WIDE: elements between tokens of q and k
  const int* wide;                         // WIDE: [chunk][H], not zero for the chunks to do
};
// chunks a block of a WIDE launch looks through at most
constexpr int kWideList = 512;

// The gradients of a wide chunk (see kSpan) for one channel and 16 time steps: what narrow chunks read from the products of
// q~, k~ and dA is summed here over the pairs of the chunk, from the caller's q, k and gates and the dA tiles (hi + lo).
// Leaves at scratch[time][channel] the 16 time steps' share of dg: the sum of q dq - k dk_intra from that step on and of
// k dk_inter before it.  (Narrow chunks add k dk_inter of all steps and take away that of the later ones; where the gates
// are strong both are larger than dg by more than fp32 holds.)
// run, tail: the two sums over all 16 steps; h_scale: exp(G_n - ref - refd), which sum_v h' dh' lacks
struct WideResult { float run, tail, h_scale; };
struct WideChannel {
  const float *add_dq, *add_dk;   // partial sums at the chunk's first token and this channel, or null
  void *dq, *dk;                  // outputs, likewise
  __nv_bfloat16* dv;              // null: no such value channel
  long long add_step, dqk_step, dv_step;
};
template <typename TG, bool SCALAR>
__device__ __noinline__ WideResult wide_gradients(const RawChunk r, const WideChannel out, uint32_t acc_dq, uint32_t acc_dk, uint32_t acc_dv,
                                                  const uint8_t* dA_hi, const uint8_t* dA_lo, float* scratch, int col, int seg) {
  const bool on = col < r.K;
  WideResult res{0.f, 0.f, 0.f};
  WideSums s{0.f, 0.f, 0.f};
  if (on) s = wide_sums<SCALAR>(r, col, seg * SEG);
  const float mid = 0.5f * (s.first + s.total), ref = clamp_span(mid), refd = clamp_span(s.total - mid);
  res.h_scale = fast_exp(s.total - ref - refd);
  float kdk[SEG];   // k dk_inter
#pragma unroll
  for (int t = 0; t < SEG; ++t) kdk[t] = 0.f;
  auto dA = [&](int i, int j) { return ld_bf16(dA_hi, slab_off(i, j)) + ld_bf16(dA_lo, slab_off(i, j)); };
  float G = s.before;   // of time step seg * SEG + 15
  if (on)
    for (int i = seg * SEG; i < seg * SEG + SEG && i < r.len; ++i) G += raw_gate<SCALAR>(r, i, col);
#pragma unroll
  for (int blk = 1; blk >= 0; --blk) {
    float dq[8], dk[8], dv[8];   // inter-chunk: with respect to q~ and k~
    const uint32_t c0 = seg * SEG + blk * 8;
    tmem_ld8(acc_dq + c0, dq);
    tmem_ld8(acc_dk + c0, dk);
    tmem_ld8(acc_dv + c0, dv);
#pragma unroll
    for (int u = 7; u >= 0; --u) {
      const int i = (int)c0 + u;
      if (i < r.len) {
        if (out.dv) st_out(out.dv, (size_t)(i * out.dv_step), dv[u]);
        if (on) {
          const float q = __bfloat162float(r.q[i * r.pitch + col]), k = __bfloat162float(r.k[i * r.pitch + col]);
          float gq = fast_exp(G - ref) * dq[u];
          const float inter = fast_exp(s.total - G - refd) * dk[u];
          float gk = 0.f;
          const float ei = fast_exp(raw_gate<SCALAR>(r, i, col));
          float w = ei;
          for (int j = i - 1; j >= 0 && w != 0.f; --j) {
            gq = fmaf(dA(i, j) * w, __bfloat162float(r.k[j * r.pitch + col]), gq);
            w *= fast_exp(raw_gate<SCALAR>(r, j, col));
          }
          w = 1.f;
          for (int j = i + 1; j < r.len && w != 0.f; ++j) {
            w *= fast_exp(raw_gate<SCALAR>(r, j, col));
            gk = fmaf(dA(j, i) * w, __bfloat162float(r.q[j * r.pitch + col]), gk);
          }
          // the pair (i, i) has no gate in it: its shares of q dq and k dk cancel, and under strong gates they are
          // larger than all else by more than fp32 holds
          res.run += q * gq - k * gk;
          const float dii = dA(i, i);
          gq = fmaf(dii, k, gq);
          gk = fmaf(dii, q, gk) + inter;
          kdk[blk * 8 + u] = k * inter;
          G -= raw_gate<SCALAR>(r, i, col);
          if (out.add_dq) {
            gq += out.add_dq[i * out.add_step];
            gk += out.add_dk[i * out.add_step];
          }
          st_out(reinterpret_cast<TG*>(out.dq), (size_t)(i * out.dqk_step), gq);
          st_out(reinterpret_cast<TG*>(out.dk), (size_t)(i * out.dqk_step), gk);
        }
      }
      scratch[i * D + col] = res.run;
    }
  }
#pragma unroll
  for (int t = 0; t < SEG; ++t) {
    scratch[(seg * SEG + t) * D + col] += res.tail;
    res.tail += kdk[t];
  }
  return res;
}

// Warp roles: warps 0-15 gate q and k of the next chunk and write the gradients of a chunk out of
// tensor memory (thread = one channel, 16 time steps); warps 16-19 convert A and dA to bf16 operands
// and reduce sum_v h' dh'; one thread of warp 20 issues every tensor-core product, one thread of warp 21
// every TMA load.
// The roles meet only through mbarriers, so the gradient write-out of chunk n runs while the
// exponent product, the gating and the A / dA products of chunk n+1 are under way; the six
// gradient products of chunk n+1 start as soon as chunk n has left tensor memory.
constexpr int BWD_THREADS = 704;
constexpr int BWD_EPI_THREADS = 512, BWD_GATE_THREADS = 128;

// TG: type of dq and dk; TD: type of dg.
// SCALAR: the gate is one value per head and time step; no gate tile is fetched and no exponent product
// issued: every write-out warp cumulates the 64 gates of a chunk in registers (warp_cumulate) and hands the
// factors exp(+-(G - mid)) of the time steps around by shuffles.  dg is summed over the key channels inside
// the kernel and written as fp32 [B,T,H] (the scalar gate's gradient is the sum of the channels').
template <typename TG, typename TD, bool SCALAR, bool GEN, bool WIDE>
__global__ void __launch_bounds__(BWD_THREADS, 1) k_bwd_main(const __grid_constant__ BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* qs = smem;                 // 2 x: q -> q exp(G - mid) in place (GEN: one, and what bf16 leaves of it)
  uint8_t* ks = qs + 2 * TILE64;      // 2 x: k -> k exp(mid - G) in place (GEN: likewise)
  uint8_t* gs = ks + 2 * TILE64;      // g (GEN: then what bf16 leaves of tril(A) scale and tril(dA) scale)
  uint8_t* vs = gs + TILE64;
  uint8_t* dos = vs + TILE64;
  uint8_t* hs = dos + TILE64;         // h_c exp(mid) scale, 128 x 128
  uint8_t* dhs = hs + TILE128;        // dh_c exp(G_n - mid), 128 x 128
  uint8_t* Ps = dhs + TILE128;        // tril(A) scale, bf16 64 x 64
  uint8_t* dAs = Ps + SLAB64;         // tril(dA) scale, bf16 64 x 64
  uint8_t* mtm = dAs + SLAB64;        // TRI_MID pattern, rows repeated to 128
  // single-slot barriers complete once per chunk (parity it & 1); two-slot ones are indexed by it & 1
  // and complete every other chunk (parity (it >> 1) & 1)
  __shared__ uint64_t full_g, full_qk[2], full_hdo, full_dhv, bar_gate, bar_A, bar_r1, bar_r2, bar_main, gated, conv_done,
      hdh_done[2], e_done[2];
  __shared__ uint32_t tmem_slot;
  __shared__ float sufsum[2][4][D];   // per-segment totals of the dg suffix sums
  __shared__ float tails[2][4][D];    // per-segment sum_i dk_inter k
  __shared__ float hdh_s[2][D];       // sum_v h' dh'
  __shared__ float dgk_s[2][C];       // SCALAR: dg of a chunk summed over the channels
  __shared__ float diag[1][GEN ? 8 * C : 1];   // GEN: partial q_i . k_i [8][64] of a chunk
  __shared__ volatile int abort_flag;
  __shared__ int wide_list[WIDE ? kWideList : 1], wide_count;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // tensor-memory columns: the exponent tile E_mid is consumed by the gating before A and dA take its place
  constexpr uint32_t cEm = 0, cA = 0, cET = 128, cdq = 256, cdk1 = 320, cdk2 = 384, cdv = 448;
  constexpr uint32_t cdA = GEN ? cdk1 : 64;
  int nit = (p.total - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  if constexpr (WIDE) {   // the wide ones of this block's chunks (the order does not matter), mostly none
    asm volatile("griddepcontrol.wait;" ::: "memory");   // the launch before this one is over, its writes are visible
    if (tid == 0) wide_count = 0;
    __syncthreads();
    for (int n = tid; n < nit; n += BWD_THREADS)
      if (p.wide[blockIdx.x + n * gridDim.x]) wide_list[atomicAdd(&wide_count, 1)] = blockIdx.x + n * gridDim.x;
    __syncthreads();
    nit = wide_count;
    if (nit == 0) return;
  }

  const int K = GEN ? p.geo.K : D, V = GEN ? p.geo.V : D;
  const int yc = GEN ? p.vs * D : 0;   // first value channel of this launch's slice
  // returns how many of the chunk's rows are the sequence's own
  auto chunk_rows = [&](int it, int& h, int& row, int& hrow) -> int {
    // heads vary fastest over the chunks in flight: together the blocks read and write whole
    // token rows of the [B,T,H,D] activations
    const int cid = WIDE ? wide_list[it] : blockIdx.x + it * gridDim.x;
    h = cid % p.H;
    if constexpr (GEN) {
      const int slot = cid / p.H;
      hrow = (cid * p.geo.VS + p.vs) * D;
      int end;
      if (p.geo.chunks) {
        const ChunkEntry e = p.geo.chunks[slot];
        row = e.row; end = e.end;
      } else {
        const int b = slot / p.NT;
        row = b * p.T + (slot - b * p.NT) * C; end = (b + 1) * p.T;
      }
      return min(C, end - row);
    } else {
      const int ci = (cid / p.H) % p.NT, b = cid / (p.H * p.NT);
      row = b * p.T + ci * C;
      hrow = ((b * p.NT + ci) * p.H + h) * D;
      return C;
    }
  };
  // bounded wait that also gives up when another role has failed
  auto wait = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
      if (mbar_try_wait(bar, parity)) return true;
      if ((i & 255u) == 255u && abort_flag) return false;
    }
    abort_flag = 1;
    fail(code);
    return false;
  };

  if (tid == 0) {
    mbar_init(&full_g, 1);
    mbar_init(&full_qk[0], 1); mbar_init(&full_qk[1], 1); mbar_init(&full_hdo, 1);
    mbar_init(&full_dhv, 1); mbar_init(&bar_gate, 1); mbar_init(&bar_A, 1); mbar_init(&bar_r1, 1); mbar_init(&bar_r2, 1);
    mbar_init(&bar_main, 1);
    mbar_init(&gated, BWD_EPI_THREADS); mbar_init(&conv_done, GEN ? BWD_EPI_THREADS : BWD_GATE_THREADS);
    mbar_init(&hdh_done[0], BWD_GATE_THREADS); mbar_init(&hdh_done[1], BWD_GATE_THREADS);
    mbar_init(&e_done[0], BWD_EPI_THREADS); mbar_init(&e_done[1], BWD_EPI_THREADS);
    fence_barrier_init();
    abort_flag = 0;
  }
  if (tid < 2 * C) dgk_s[tid >> 6][tid & 63] = 0.f;
  if (warp == 0) { tmem_alloc(&tmem_slot, 512); tmem_relinquish(); }
  if (!SCALAR) build_tri_tile(mtm, 128, TRI_MID);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = tmem_slot;

  if (warp < 16) {
    // ------------------------------------------------------------------ gradient write-out
    const int q4 = warp & 3, seg = warp >> 2, col = q4 * 32 + lane;
    const uint32_t lane_base = q4 * 32;
    const ColAddr ca = col_prep(64, col);
    const size_t ostride = (size_t)p.H * K, vstride = GEN ? (size_t)p.dv_pitch : ostride;
    const bool has_k = !GEN || col < K, has_v = !GEN || yc + col < V;
    TG* const dq_out = reinterpret_cast<TG*>(p.dq);
    TG* const dk_out = reinterpret_cast<TG*>(p.dk);
    TD* const dg_out = reinterpret_cast<TD*>(p.dg);
    // q -> q exp(G - mid), k -> k exp(mid - G) in place: thread (q4, lane, seg) owns time row
    // (32 q4 + lane) mod 64 and 16 channels
    // SCALAR: the gates of time steps lane and lane + 32 of the next chunk to be gated, and the factors
    // exp(G - mid), exp(mid - G) of time step (16 seg + lane) mod 32 + 32 (seg / 2) of the chunk gated last
    // (in registers, loaded a chunk ahead: see the note in k_fwd_fused)
    __nv_bfloat16 greg_lo = __float2bfloat16(0.f), greg_hi = greg_lo;
    float fw_next = 1.f, rw_next = 1.f;
    float gconst = 0.f;
    int glen = C;
    auto load_gates = [&](int it) {
      int h, row, hrow;
      glen = chunk_rows(it, h, row, hrow);
      if (GEN && !p.gscalar) {
        gconst = p.gamma ? p.gamma[h] : 0.f;
        return;
      }
      const __nv_bfloat16* src = p.gscalar + (size_t)(row + lane) * p.H + h;
      if (!GEN || lane < glen) greg_lo = src[0];
      if (!GEN || lane + 32 < glen) greg_hi = src[(size_t)32 * p.H];
    };
    if (SCALAR && nit > 0) load_gates(0);
    auto store_gated = [&](uint32_t off, bool mine, uint4 qh, uint4 ql, uint4 kh, uint4 kl) {   // GEN
      const uint4 none = make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(qs + off) = mine ? qh : none;
      *reinterpret_cast<uint4*>(qs + TILE64 + off) = mine ? ql : none;
      *reinterpret_cast<uint4*>(ks + off) = mine ? kh : none;
      *reinterpret_cast<uint4*>(ks + TILE64 + off) = mine ? kl : none;
    };
    auto raw_chunk = [&](int it) {   // GEN
      int h, row, hrow;
      const int len = chunk_rows(it, h, row, hrow);
      const size_t at = (size_t)row * p.qk_pitch + (size_t)h * K;
      RawChunk r{p.q + at, p.k + at, nullptr, p.qk_pitch, 0, p.gamma ? p.gamma[h] : 0.f, K, len};
      if (!SCALAR) { r.g = p.g + ((size_t)row * p.H + h) * K; r.gstep = (long long)p.H * K; }
      else if (p.gscalar) { r.g = p.gscalar + (size_t)row * p.H + h; r.gstep = p.H; }
      return r;
    };
    // GEN: A and dA -> masked hi + lo operands, 16 columns of both per thread (rows of an M = 64 accumulator sit in
    // lanes 0..15 of each quarter)
    auto convert = [&](int it) -> bool {
      if (!__all_sync(0xffffffffu, wait(&bar_A, it & 1, 7))) return false;
      tc_fence_after();
      const int ri = 16 * q4 + lane;
      float a[16], da[16];
      if (!WIDE) tmem_ld16(tmem_addr(tm, lane_base, cA + seg * 16), a);
      tmem_ld16(tmem_addr(tm, lane_base, cdA + seg * 16), da);
      if (lane < 16) {
        if (!WIDE) {
          if (seg == q4) set_diagonal(a, diag[0], 8, ri, lane);
          store_tril16_split(Ps, gs, ri, seg * 16, a, p.scale);
        }
        store_tril16_split(dAs, gs + SLAB64, ri, seg * 16, da, p.scale);
      }
      if constexpr (WIDE) {
        const RawChunk raw = raw_chunk(it);
        wide_operands<SCALAR>(raw, nullptr, ks, ks + TILE64, col, seg);
        wide_matrix<SCALAR>(raw, Ps, gs, p.scale, warp, lane);
      }
      fence_async_smem();
      tc_fence_before();
      mbar_arrive(&conv_done);
      return true;
    };
    auto gate_chunk = [&](int it) -> bool {
      const int sl = GEN ? 0 : it & 1;
      bool landed = (SCALAR || wait(&bar_gate, it & 1, 9)) && wait(&full_qk[sl], GEN ? it & 1 : (it >> 1) & 1, 6);
      if (SCALAR) landed = __all_sync(0xffffffffu, landed);   // (shuffles follow: the whole warp takes one path)
      if (!landed) return false;
      tc_fence_after();
      const int i = (q4 * 32 + lane) & 63;
      const int cg = (q4 >> 1) * 4 + seg;
      float dot = 0.f;
      bool mine = true;   // GEN: a short chunk's foreign rows become zero
      if (GEN) {
        int h_, row_, hrow_;
        mine = i < chunk_rows(it, h_, row_, hrow_);
      }
      if (SCALAR) {
        float g_lo = __bfloat162float(greg_lo), g_hi = __bfloat162float(greg_hi);
        if (GEN) {
          g_lo = lane < glen ? (p.gscalar ? g_lo : gconst) : 0.f;
          g_hi = lane + 32 < glen ? (p.gscalar ? g_hi : gconst) : 0.f;
        }
        const WarpGates w = warp_cumulate(g_lo, g_hi, lane);
        const float mid = w.mid();
        const float f_lo = fast_exp(w.lo - mid), r_lo = fast_exp(mid - w.lo);
        const float f_hi = fast_exp(w.hi - mid), r_hi = fast_exp(mid - w.hi);
        fw_next = (seg >> 1) ? f_hi : f_lo;
        rw_next = (seg >> 1) ? r_hi : r_lo;
        const float f = (q4 & 1) ? f_hi : f_lo, r = (q4 & 1) ? r_hi : r_lo;
        const uint32_t rowoff = (uint32_t)sl * TILE64 + (uint32_t)(cg >> 2) * SLAB64 + (uint32_t)i * 128u;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint32_t off = rowoff + (((uint32_t)((cg & 3) * 2 + u) ^ (uint32_t)i) & 7u) * 16u;
          const uint4 qr = *reinterpret_cast<const uint4*>(qs + off), kr = *reinterpret_cast<const uint4*>(ks + off);
          if constexpr (GEN) {
            uint4 ql, kl;
            dot = dot8(qr, kr, dot);
            const uint4 qh = scale8_by_split(qr, f, ql), kh = scale8_by_split(kr, r, kl);
            store_gated(off, mine, qh, ql, kh, kl);
          } else {
            *reinterpret_cast<uint4*>(qs + off) = scale8_by(qr, f);
            *reinterpret_cast<uint4*>(ks + off) = scale8_by(kr, r);
          }
        }
        if (GEN) diag[0][cg * C + i] = mine ? dot : 0.f;
        fence_async_smem();
        tc_fence_before();
        mbar_arrive(&gated);
        return true;
      }
      float em[16];
      tmem_ld16(tmem_addr(tm, lane_base, cEm + cg * 16), em);
      const uint32_t rowoff = (uint32_t)sl * TILE64 + (uint32_t)(cg >> 2) * SLAB64 + (uint32_t)i * 128u;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t off = rowoff + (((uint32_t)((cg & 3) * 2 + u) ^ (uint32_t)i) & 7u) * 16u;
        float f[8], r[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          f[t] = fast_exp(em[8 * u + t]);
          r[t] = fast_exp(-em[8 * u + t]);
        }
        const uint4 qr = *reinterpret_cast<const uint4*>(qs + off), kr = *reinterpret_cast<const uint4*>(ks + off);
        if constexpr (GEN) {
          uint4 ql, kl;
          dot = dot8(qr, kr, dot);
          const uint4 qh = scale8_split(qr, f, ql), kh = scale8_split(kr, r, kl);
          store_gated(off, mine, qh, ql, kh, kl);
        } else {
          *reinterpret_cast<uint4*>(qs + off) = scale8(qr, f);
          *reinterpret_cast<uint4*>(ks + off) = scale8(kr, r);
        }
      }
      if (GEN) diag[0][cg * C + i] = mine ? dot : 0.f;
      fence_async_smem();
      tc_fence_before();
      mbar_arrive(&gated);
      return true;
    };
    bool live = nit > 0 && (GEN || gate_chunk(0));
    if (SCALAR && !GEN && nit > 1) load_gates(1);
    for (int it = 0; live && it < nit; ++it) {
      const int sl = it & 1;
      int h, row, hrow;
      const int len = chunk_rows(it, h, row, hrow);
      if (GEN && !gate_chunk(it)) break;
      const float fw = fw_next, rw = rw_next;   // (SCALAR) of this chunk
      if constexpr (GEN) {
        if (SCALAR && it + 1 < nit) load_gates(it + 1);
        if (!convert(it)) break;
      } else {
        // the next chunk's gating runs while the tensor core works on this chunk's gradient products
        if (it + 1 < nit && !gate_chunk(it + 1)) break;
        if (SCALAR && it + 2 < nit) load_gates(it + 2);   // fetched where the thread waits anyway
      }
      bool done = wait(&bar_main, it & 1, 8) && wait(&hdh_done[sl], (it >> 1) & 1, 11);
      if (SCALAR) done = __all_sync(0xffffffffu, done);   // (shuffles follow: the whole warp takes one path)
      if (!done) break;
      tc_fence_after();
      const uint8_t* qt = qs + (GEN ? 0 : sl) * TILE64;
      const uint8_t* kt = ks + (GEN ? 0 : sl) * TILE64;
      const size_t obase = ((size_t)(row + seg * SEG) * p.H + h) * K + col;
      size_t vbase = obase;
      if (GEN) vbase = (size_t)(row + seg * SEG) * vstride + (size_t)h * V + yc + col;
      const size_t obase4 = obase - (lane & 3) + (size_t)(lane & 3) * ostride;   // channel group, own time row
      float dgl[SEG];
      float run = 0.f, tail = 0.f, h_scale = 1.f;
      float* const wide_sums_at = reinterpret_cast<float*>(qs);   // (q~ is of no use in a wide chunk)
      if constexpr (WIDE) {
          if (!wait(&conv_done, it & 1, 13)) break;   // (long done: this thread reads what the others converted)
          const size_t first = (size_t)row * p.H * K + (size_t)h * K + col, at = (size_t)row * p.dqk_pitch + (size_t)h * K + col;
          const WideChannel out{p.add_dq ? p.add_dq + first : nullptr, p.add_dk ? p.add_dk + first : nullptr, dq_out + at, dk_out + at,
                                has_v ? p.dv + (size_t)row * vstride + (size_t)h * V + yc + col : nullptr, (long long)ostride, p.dqk_pitch,
                                (long long)vstride};
          const WideResult res = wide_gradients<TG, SCALAR>(raw_chunk(it), out, tmem_addr(tm, lane_base, cdq), tmem_addr(tm, lane_base, cdk2),
                                                            tmem_addr(tm, lane_base, cdv), dAs, gs + SLAB64, wide_sums_at, col, seg);
          run = res.run; tail = res.tail; h_scale = res.h_scale;
      }
#pragma unroll
      for (int blk = WIDE ? -1 : 1; blk >= 0; --blk) {
        float et[8] = {}, dq[8], dk1[8], dk2[8], dv[8];
        const uint32_t c0 = seg * SEG + blk * 8;
        if (!SCALAR) tmem_ld8(tmem_addr(tm, lane_base, cET + 64 * sl + c0), et);
        tmem_ld8(tmem_addr(tm, lane_base, cdq + c0), dq);
        tmem_ld8(tmem_addr(tm, lane_base, cdk1 + c0), dk1);
        tmem_ld8(tmem_addr(tm, lane_base, cdk2 + c0), dk2);
        tmem_ld8(tmem_addr(tm, lane_base, cdv + c0), dv);
#pragma unroll
        for (int u = 7; u >= 0; --u) {
          const int t = blk * 8 + u;
          const uint32_t off = ca.at(seg * SEG + t);
          float qv = ld_bf16(qt, off), kv = ld_bf16(kt, off);   // q~, k~
          if (GEN) {
            qv += ld_bf16(qt + TILE64, off);
            kv += ld_bf16(kt + TILE64, off);
          }
          // exp(G - mid), exp(mid - G) of time step 16 seg + t
          const float e = SCALAR ? __shfl_sync(0xffffffffu, fw, (seg * SEG + t) & 31) : fast_exp(et[u]);
          const float r = SCALAR ? __shfl_sync(0xffffffffu, rw, (seg * SEG + t) & 31) : fast_exp(-et[u]);
          const float dqs = dq[u];                        // dq exp(mid - G)
          const float dki = dk2[u];                       // dk_inter exp(G - mid)
          const float dks = dk1[u] + dki;                 // dk exp(G - mid)
          run += qv * dqs - kv * dks;                     // q dq - k dk
          tail = fmaf(dki, kv, tail);                     // dk_inter k
          dgl[t] = run;
          if constexpr (GEN) {
            if (seg * SEG + t < len) {
              if (has_v) st_out(p.dv, vbase + t * vstride, dv[u]);
              if (has_k) {
                float gq = e * dqs, gk = r * dks;
                if (p.add_dq) {
                  gq += p.add_dq[obase + t * ostride];
                  gk += p.add_dk[obase + t * ostride];
                }
                const size_t o = (size_t)(row + seg * SEG + t) * p.dqk_pitch + (size_t)h * K + col;
                st_out(dq_out, o, gq);
                st_out(dk_out, o, gk);
              }
            }
          } else {
            st_out(p.dv, vbase + t * vstride, dv[u]);
            st_out(dq_out, obase + t * ostride, e * dqs);
            st_out(dk_out, obase + t * ostride, r * dks);
          }
        }
      }
      sufsum[sl][seg][col] = run;
      tails[sl][seg][col] = tail;
      tc_fence_before();
      asm volatile("bar.sync 1, %0;" ::"n"(BWD_EPI_THREADS) : "memory");
      const float later = (seg < 1 ? sufsum[sl][1][col] : 0.f) + (seg < 2 ? sufsum[sl][2][col] : 0.f) +
                          (seg < 3 ? sufsum[sl][3][col] : 0.f);
      // (of a wide chunk the steps of the earlier segments only, see wide_gradients)
      float cst;
      if (WIDE) cst = later + (seg > 0 ? tails[sl][0][col] : 0.f) + (seg > 1 ? tails[sl][1][col] : 0.f) + (seg > 2 ? tails[sl][2][col] : 0.f) +
                      hdh_s[sl][col] / p.scale * h_scale;
      else cst = later + tails[sl][0][col] + tails[sl][1][col] + tails[sl][2][col] + tails[sl][3][col] + hdh_s[sl][col] / p.scale;
      // (exp(G_n) sum_v h dh = sum_v h' dh' / scale)
      if (WIDE) {
#pragma unroll
        for (int t = 0; t < SEG; ++t) dgl[t] = wide_sums_at[(seg * SEG + t) * D + col];
        fence_async_smem();
      }
      mbar_arrive(&e_done[sl]);   // tensor memory, the q~ / k~ tiles and hdh_s of this chunk are free
      if constexpr (SCALAR) {
        // sum over the 128 channels: the lanes of a warp by a shuffle butterfly (lane t keeps the total of time
        // step t), then the four warps that share this segment through shared memory
#pragma unroll
        for (int t = 0; t < SEG; ++t) dgl[t] += cst;
        const float mine = warp_sum16(dgl, lane);
        if (lane < SEG) atomicAdd(&dgk_s[sl][seg * SEG + lane], mine);
        asm volatile("bar.sync 1, %0;" ::"n"(BWD_EPI_THREADS) : "memory");
        if (tid < C) {
          if (p.dg && (!GEN || tid < len)) {
            const size_t o = (size_t)(row + tid) * p.H + h;
            reinterpret_cast<float*>(p.dg)[o] = dgk_s[sl][tid] + ((GEN && p.add_dg) ? p.add_dg[o] : 0.f);
          }
          dgk_s[sl][tid] = 0.f;   // (this slot is used again two chunks on, two barriers later)
        }
      } else if (p.dg) {
        // after the accumulators are released: four time steps x four channels change hands inside each
        // group of four lanes, so that every store writes four neighbouring channels of one time step
#pragma unroll
        for (int t = 0; t < SEG; t += 4) {
          float w[4] = {dgl[t] + cst, dgl[t + 1] + cst, dgl[t + 2] + cst, dgl[t + 3] + cst};
          if constexpr (GEN) {
            // (every lane takes part in the exchange; K is a multiple of 8, so a group of four is inside or outside)
            const bool in = has_k && seg * SEG + t + (lane & 3) < len;
            if (p.add_dg) {
#pragma unroll
              for (int u = 0; u < 4; ++u)
                if (has_k && seg * SEG + t + u < len) w[u] += p.add_dg[obase + (t + u) * ostride];
            }
            st_transposed4(dg_out, obase4 + t * ostride, w, lane, in);
          } else {
            st_transposed4(dg_out, obase4 + t * ostride, w, lane);
          }
        }
      }
    }
  } else if (warp < 20) {
    // ------------------------------------------------------------------ A / dA -> masked bf16 operands
    const int g4 = warp & 3;
    const uint32_t lane_base = g4 * 32;
    for (int it = 0; it < nit; ++it) {
      if constexpr (!GEN) {
        // rows of the M = 64 accumulators sit in lanes 0..15 of each quarter
        if (!wait(&bar_A, it & 1, 7)) break;
        tc_fence_after();
        const int ri = 16 * g4 + lane;
#pragma unroll
        for (int sg = 0; sg < 4; ++sg) {
          float a[16];
          tmem_ld16(tmem_addr(tm, lane_base, cA + sg * 16), a);
          if (lane < 16) store_tril16(Ps, ri, sg * 16, a, p.scale);
          tmem_ld16(tmem_addr(tm, lane_base, cdA + sg * 16), a);
          if (lane < 16) store_tril16(dAs, ri, sg * 16, a, p.scale);
        }
        fence_async_smem();
        tc_fence_before();
        mbar_arrive(&conv_done);
      }
      // sum_v h'[k][v] dh'[k][v] for k = this thread, while the gradient products read the same tiles
      if (!wait(&full_hdo, it & 1, 6) || !wait(&full_dhv, it & 1, 6)) break;
      {
        const int gt = g4 * 32 + lane;
        float hd = 0.f;
#pragma unroll 4
        for (int c8 = 0; c8 < D; c8 += 8) {
          const uint32_t off = tile_off(128, gt, c8);
          const uint4 a = *reinterpret_cast<const uint4*>(hs + off), d = *reinterpret_cast<const uint4*>(dhs + off);
          const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a);
          const __nv_bfloat162* pd = reinterpret_cast<const __nv_bfloat162*>(&d);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 fa = __bfloat1622float2(pa[t]), fd = __bfloat1622float2(pd[t]);
            hd = fmaf(fa.x, fd.x, hd);
            hd = fmaf(fa.y, fd.y, hd);
          }
        }
        hdh_s[it & 1][gt] = hd;
      }
      mbar_arrive(&hdh_done[it & 1]);   // h' and dh' of this chunk are no longer read by threads
    }
  } else if (warp == 20) {
    // ------------------------------------------------------------------ tensor-core issue
    // GEN: the whole warp walks the chunks, because a short chunk's foreign rows of g, v, do are zeroed here before
    // a product reads them; products are issued by one thread
    if (GEN || lane == 0) {
      const uint32_t ga = smem_u32(gs), mma = smem_u32(mtm), va = smem_u32(vs), doa = smem_u32(dos), ha = smem_u32(hs),
                     dha = smem_u32(dhs), pa = smem_u32(Ps), daa = smem_u32(dAs);
      auto zero_foreign = [&](int it, uint8_t* t0, uint8_t* t1) {
        int h_, row_, hrow_;
        const int len = chunk_rows(it, h_, row_, hrow_);
        if (len == C) return;
        zero_rows(t0, len, lane, 32);
        if (t1) zero_rows(t1, len, lane, 32);
        fence_async_smem();
        __syncwarp();
      };
      auto issue_gate = [&](int it) {
        if (GEN) {
          zero_foreign(it, gs, nullptr);
          if (lane != 0) return;
        }
#pragma unroll
        for (int j0 = 0; j0 < C; j0 += 16)   // G - mid, [time (repeated)][channel]
          umma_bf16(tm + cEm, desc_kmajor(mma, 128, 0, j0), desc_mnmajor(ga, 64, j0, 0), umma_idesc(128, 128, 0, 1), j0 > 0);
#pragma unroll
        for (int j0 = 0; j0 < C; j0 += 16)   // G - mid, [channel][time]
          umma_bf16(tm + cET + 64 * (it & 1), desc_mnmajor(ga, 64, j0, 0), desc_kmajor(mma, 64, 0, j0),
                    umma_idesc(128, 64, 1, 0), j0 > 0);
        umma_commit(&bar_gate);
      };
      auto issue_A = [&](int it) {
        const uint32_t qta = smem_u32(qs + (it & 1) * TILE64), kta = smem_u32(ks + (it & 1) * TILE64);
#pragma unroll
        for (int k0 = 0; k0 < D; k0 += 16)   // A[i][j] = q~ k~^T
          umma_bf16(tm + cA, desc_kmajor(qta, 64, 0, k0), desc_kmajor(kta, 64, 0, k0), umma_idesc(64, 64, 0, 0), k0 > 0);
      };
      auto issue_dA = [&](int it) {
#pragma unroll
        for (int k0 = 0; k0 < D; k0 += 16)   // dA[i][j] = do v^T
          umma_bf16(tm + cdA, desc_kmajor(doa, 64, 0, k0), desc_kmajor(va, 64, 0, k0), umma_idesc(64, 64, 0, 0), k0 > 0);
        umma_commit(&bar_A);
      };
      // The gradient products in two groups.  The first needs neither A nor dA, so it starts as soon as
      // the chunk's tiles have landed, while the conversion warps still work on A and dA; after it dh'
      // and v are dead and the next chunk's are fetched.  The second group needs the converted operands.
      auto issue_inter = [&](int it) {
        const uint32_t kta = smem_u32(ks + (it & 1) * TILE64);
#pragma unroll
        for (int k0 = 0; k0 < D; k0 += 16)   // dq_inter^T[k][i] = h' do^T
          umma_bf16(tm + cdq, desc_kmajor(ha, 128, 0, k0), desc_kmajor(doa, 64, 0, k0), umma_idesc(128, 64, 0, 0), k0 > 0);
#pragma unroll
        for (int k0 = 0; k0 < D; k0 += 16)   // (dk_inter exp(G - mid))^T[k][j] = dh' v^T
          umma_bf16(tm + cdk2, desc_kmajor(dha, 128, 0, k0), desc_kmajor(va, 64, 0, k0), umma_idesc(128, 64, 0, 0), k0 > 0);
#pragma unroll
        for (int k0 = 0; k0 < D; k0 += 16)   // dv^T[v][j] = dh'^T k~^T
          umma_bf16(tm + cdv, desc_mnmajor(dha, 128, k0, 0), desc_kmajor(kta, 64, 0, k0), umma_idesc(128, 64, 1, 0), k0 > 0);
        umma_commit(&bar_r2);
      };
      auto issue_intra = [&](int it) {
        const uint32_t qta = smem_u32(qs + (it & 1) * TILE64), kta = smem_u32(ks + (it & 1) * TILE64);
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)   // dv^T[v][j] += sum_i do[i][v] A[i][j]
          umma_bf16(tm + cdv, desc_mnmajor(doa, 64, k0, 0), desc_mnmajor(pa, 64, k0, 0), umma_idesc(128, 64, 1, 1), 1);
        umma_commit(&bar_r1);                // h' and do are dead
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)   // dq^T[k][i] += sum_j k~[j][k] dA[i][j]
          umma_bf16(tm + cdq, desc_mnmajor(kta, 64, k0, 0), desc_kmajor(daa, 64, 0, k0), umma_idesc(128, 64, 1, 0), 1);
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)   // dk_intra^T[k][j] = sum_i q~[i][k] dA[i][j]
          umma_bf16(tm + cdk1, desc_mnmajor(qta, 64, k0, 0), desc_mnmajor(daa, 64, k0, 0), umma_idesc(128, 64, 1, 1), k0 > 0);
        umma_commit(&bar_main);
      };
      // (GEN: all lanes take the same path, also when a wait gives up)
      auto waitw = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
        const bool r = wait(bar, parity, code);
        return GEN ? (bool)__all_sync(0xffffffffu, r) : r;
      };
      if constexpr (GEN) {
        // q~, k~, A and dA are hi + lo: the products of two of them are hi hi + hi lo + lo hi.
        auto issue_before_gating = [&]() {   // dA, dq_inter, dk_inter: everything without q~ or k~
#pragma unroll
          for (int k0 = 0; k0 < D; k0 += 16)
            umma_bf16(tm + cdA, desc_kmajor(doa, 64, 0, k0), desc_kmajor(va, 64, 0, k0), umma_idesc(64, 64, 0, 0), k0 > 0);
#pragma unroll
          for (int k0 = 0; k0 < D; k0 += 16)
            umma_bf16(tm + cdq, desc_kmajor(ha, 128, 0, k0), desc_kmajor(doa, 64, 0, k0), umma_idesc(128, 64, 0, 0), k0 > 0);
#pragma unroll
          for (int k0 = 0; k0 < D; k0 += 16)
            umma_bf16(tm + cdk2, desc_kmajor(dha, 128, 0, k0), desc_kmajor(va, 64, 0, k0), umma_idesc(128, 64, 0, 0), k0 > 0);
        };
        const uint32_t qta = smem_u32(qs), kta = smem_u32(ks), qla = qta + TILE64, kla = kta + TILE64;
        const uint32_t pla = ga, dala = ga + SLAB64;
        auto mul_A = [&](uint32_t x, uint32_t y, uint32_t acc) {
#pragma unroll
          for (int k0 = 0; k0 < D; k0 += 16)
            umma_bf16(tm + cA, desc_kmajor(x, 64, 0, k0), desc_kmajor(y, 64, 0, k0), umma_idesc(64, 64, 0, 0), acc | (k0 > 0));
        };
        auto mul_dv = [&](uint32_t a) {    // dv^T[v][j] += sum_i do[i][v] A[i][j]
#pragma unroll
          for (int k0 = 0; k0 < C; k0 += 16)
            umma_bf16(tm + cdv, desc_mnmajor(doa, 64, k0, 0), desc_mnmajor(a, 64, k0, 0), umma_idesc(128, 64, 1, 1), 1);
        };
        auto mul_dq = [&](uint32_t k, uint32_t da) {   // dq^T[k][i] += sum_j k~[j][k] dA[i][j]
#pragma unroll
          for (int k0 = 0; k0 < C; k0 += 16)
            umma_bf16(tm + cdq, desc_mnmajor(k, 64, k0, 0), desc_kmajor(da, 64, 0, k0), umma_idesc(128, 64, 1, 0), 1);
        };
        auto mul_dk = [&](uint32_t q, uint32_t da, uint32_t acc) {   // dk_intra^T[k][j] = sum_i q~[i][k] dA[i][j]
#pragma unroll
          for (int k0 = 0; k0 < C; k0 += 16)
            umma_bf16(tm + cdk1, desc_mnmajor(q, 64, k0, 0), desc_mnmajor(da, 64, k0, 0), umma_idesc(128, 64, 1, 1), acc | (k0 > 0));
        };
        for (int it = 0; it < nit; ++it) {
          if (!SCALAR) {
            if (!waitw(&full_g, it & 1, 6)) break;
            tc_fence_after();
            issue_gate(it);
            __syncwarp();
          }
          // the tiles have landed, the previous chunk has left tensor memory
          if (!waitw(&full_hdo, it & 1, 6) || !waitw(&full_dhv, it & 1, 6)) break;
          zero_foreign(it, vs, dos);
          if (it >= 1 && !waitw(&e_done[(it - 1) & 1], ((it - 1) >> 1) & 1, 14)) break;
          tc_fence_after();
          if (lane == 0) issue_before_gating();
          __syncwarp();
          if (!waitw(&gated, it & 1, 12)) break;
          tc_fence_after();
          // (WIDE: k~ comes with the converted operands, A, dq_intra, dk_intra are no products)
          auto mul_dv_inter = [&]() {
#pragma unroll
            for (int k0 = 0; k0 < D; k0 += 16)   // dv^T[v][j] = dh'^T k~^T
              umma_bf16(tm + cdv, desc_mnmajor(dha, 128, k0, 0), desc_kmajor(kta, 64, 0, k0), umma_idesc(128, 64, 1, 0), k0 > 0);
            if (WIDE) {
#pragma unroll
              for (int k0 = 0; k0 < D; k0 += 16)
                umma_bf16(tm + cdv, desc_mnmajor(dha, 128, k0, 0), desc_kmajor(kla, 64, 0, k0), umma_idesc(128, 64, 1, 0), 1);
            }
            umma_commit(&bar_r2);   // dh' and v are dead
          };
          if (lane == 0) {
            if (!WIDE) { mul_A(qta, kta, 0); mul_A(qta, kla, 1); mul_A(qla, kta, 1); }
            umma_commit(&bar_A);
            if (!WIDE) mul_dv_inter();
          }
          __syncwarp();
          if (!waitw(&conv_done, it & 1, 13)) break;
          tc_fence_after();
          if (lane == 0) {
            if (WIDE) mul_dv_inter();
            mul_dv(pa); mul_dv(pla);
            umma_commit(&bar_r1);   // h' and do are dead
            if (!WIDE) {
              mul_dq(kta, daa); mul_dq(kta, dala); mul_dq(kla, daa);
              mul_dk(qta, daa, 0); mul_dk(qta, dala, 1); mul_dk(qla, daa, 1);
            }
            umma_commit(&bar_main);
          }
          __syncwarp();
        }
      } else {
        bool ok = SCALAR || waitw(&full_g, 0, 6);
        if (ok) {
          tc_fence_after();
          if (!SCALAR) issue_gate(0);
          ok = waitw(&gated, 0, 12);
        }
        if (ok) {
          tc_fence_after();
          issue_A(0);
          ok = waitw(&full_hdo, 0, 6) && waitw(&full_dhv, 0, 6);
        }
        if (ok) issue_dA(0);
        for (int it = 0; ok && it < nit; ++it) {
          // A and dA of this chunk are issued; the previous chunk has left tensor memory
          if (it >= 1 && !waitw(&e_done[(it - 1) & 1], ((it - 1) >> 1) & 1, 14)) break;
          tc_fence_after();
          issue_inter(it);
          if (!waitw(&conv_done, it & 1, 13)) break;   // A and dA of this chunk are in shared memory
          tc_fence_after();
          const bool more = it + 1 < nit;
          if (more && !SCALAR) {   // the next chunk's exponents take the place of A and dA in tensor memory
            if (!waitw(&full_g, (it + 1) & 1, 6)) break;
            issue_gate(it + 1);
          }
          issue_intra(it);
          if (more) {
            if (!waitw(&gated, (it + 1) & 1, 12)) break;
            tc_fence_after();
            issue_A(it + 1);
            if (!waitw(&full_hdo, (it + 1) & 1, 6) || !waitw(&full_dhv, (it + 1) & 1, 6)) break;
            issue_dA(it + 1);
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ TMA loads
    if (lane == 0) {
      auto load_g = [&](int it) {
        int h, row, hrow;
        chunk_rows(it, h, row, hrow);
        mbar_expect_tx(&full_g, TILE64);
        tma_load_3d(gs, &p.mg, &full_g, 0, h, row); tma_load_3d(gs + SLAB64, &p.mg, &full_g, 64, h, row);
      };
      auto load_qk = [&](int it) {
        int h, row, hrow;
        chunk_rows(it, h, row, hrow);
        const int sl = GEN ? 0 : it & 1;
        uint64_t* bar = &full_qk[sl];
        uint8_t* qd = qs + sl * TILE64;
        uint8_t* kd = ks + sl * TILE64;
        mbar_expect_tx(bar, 2 * TILE64);
        tma_load_3d(qd, &p.mq, bar, 0, h, row); tma_load_3d(qd + SLAB64, &p.mq, bar, 64, h, row);
        tma_load_3d(kd, &p.mk, bar, 0, h, row); tma_load_3d(kd + SLAB64, &p.mk, bar, 64, h, row);
      };
      auto load_hdo = [&](int it) {
        int h, row, hrow;
        chunk_rows(it, h, row, hrow);
        mbar_expect_tx(&full_hdo, TILE128 + TILE64);
        tma_load_3d(dos, &p.mdo, &full_hdo, yc, h, row); tma_load_3d(dos + SLAB64, &p.mdo, &full_hdo, yc + 64, h, row);
        tma_load_2d(hs, &p.mh, &full_hdo, 0, hrow); tma_load_2d(hs + TILE128 / 2, &p.mh, &full_hdo, 64, hrow);
      };
      auto load_dhv = [&](int it) {
        int h, row, hrow;
        chunk_rows(it, h, row, hrow);
        mbar_expect_tx(&full_dhv, TILE128 + TILE64);
        tma_load_3d(vs, &p.mv, &full_dhv, yc, h, row); tma_load_3d(vs + SLAB64, &p.mv, &full_dhv, yc + 64, h, row);
        tma_load_2d(dhs, &p.mdh, &full_dhv, 0, hrow); tma_load_2d(dhs + TILE128 / 2, &p.mdh, &full_dhv, 64, hrow);
      };
      if (!SCALAR) load_g(0);
      load_qk(0);
      load_hdo(0);
      load_dhv(0);
      bool ok = true;
      if (GEN) {   // one slot of q and k: refilled when the write-out has read them (from L2, fetched ahead)
        for (int it = 0; it + 1 < nit; ++it) {
          int h, row, hrow;
          chunk_rows(it + 1, h, row, hrow);
          tma_prefetch_l2_3d(&p.mq, 0, h, row); tma_prefetch_l2_3d(&p.mq, 64, h, row);
          tma_prefetch_l2_3d(&p.mk, 0, h, row); tma_prefetch_l2_3d(&p.mk, 64, h, row);
          if (!wait(&bar_r2, it & 1, 8) || !wait(&hdh_done[it & 1], (it >> 1) & 1, 11)) break;
          load_dhv(it + 1);
          if (!wait(&bar_r1, it & 1, 8)) break;
          load_hdo(it + 1);
          if (!SCALAR) {   // (the gate tile held the lower halves of A and dA; WIDE: the write-out reads dA)
            if (!wait(&bar_main, it & 1, 8) || (WIDE && !wait(&e_done[it & 1], (it >> 1) & 1, 14))) break;
            load_g(it + 1);
          }
          if (!wait(&e_done[it & 1], (it >> 1) & 1, 14)) break;
          load_qk(it + 1);
        }
        ok = false;   // (the loop below is the plain form's)
      } else if (nit > 1) {
        load_qk(1);
        if (!SCALAR) {
          ok = wait(&bar_gate, 0, 9);   // the exponent products of chunk 0 have read its gates
          if (ok) load_g(1);
        }
      }
      for (int it = 0; ok && it + 1 < nit; ++it) {
        // dh' and v are dead after the first group of products (and the h' dh' reduction), h' and do
        // after the first product of the second group
        if (!wait(&bar_r2, it & 1, 8) || !wait(&hdh_done[it & 1], (it >> 1) & 1, 11)) break;
        load_dhv(it + 1);
        if (!wait(&bar_r1, it & 1, 8)) break;
        load_hdo(it + 1);
        if (it + 2 < nit) {
          if (!wait(&e_done[it & 1], (it >> 1) & 1, 14)) break;
          load_qk(it + 2);
          if (!SCALAR) {
            if (!wait(&bar_gate, (it + 1) & 1, 9)) break;
            load_g(it + 2);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 512);
  if (tid == 0 && abort_flag && nit > 0) {
    int h, row, hrow;
    chunk_rows(0, h, row, hrow);
    poison(reinterpret_cast<TG*>(p.dq) + (GEN ? (size_t)row * p.dqk_pitch : (size_t)row * p.H * K) + (size_t)h * K);
    poison(p.dv + (GEN ? (size_t)row * p.dv_pitch : (size_t)row * p.H * V) + (size_t)h * V + yc);
  }
}

// ===========================================================================
// host side
// ===========================================================================
constexpr size_t SCAN_SMEM = 9 * TILE64 + 2 * SLAB64 + 2 * TILE128 + sizeof(ScanShared);
constexpr size_t FWD_O_SMEM = 4 * TILE64 + TILE128 + SLAB64 + 1024;
constexpr size_t BWD_SMEM = 7 * TILE64 + 2 * TILE128 + 2 * SLAB64 + 2 * SLAB64 + 1024;

// from this many (batch, head) pairs on, the forward runs as one fused pass (one block per pair)
// instead of a state scan followed by a chunk-parallel output kernel
constexpr int kFusedMinBlocks = 48;

std::atomic<int> g_test_skip_load{-1};

// One launch of the scan kernel over `nseg` time segments per (batch, head).  states == nullptr keeps
// no chunk-start states (a summary pass: end states and summed gates only).
int run_scan(bool bwd, const tops_chunk_problem& pb, int nseg, const void* x, const void* g, const void* y,
             const float* s0, void* states, float* s_final, float* gsum, cudaStream_t st) {
  ScanParams sp;
  const int BT = pb.B * pb.T;
  const bool scalar = pb.gate_kind == TOPS_GATE_SCALAR;
  int rc;
  if ((rc = act_map(&sp.mx, x, BT, pb.H)) || (rc = act_map(&sp.my, y, BT, pb.H))) return rc;
  if (!scalar && (rc = act_map(&sp.mg, g, BT, pb.H))) return rc;
  sp.gscalar = reinterpret_cast<const __nv_bfloat16*>(g);
  if (states && (rc = state_map(&sp.mst, states, (size_t)pb.B * (pb.T / C) * pb.H * D))) return rc;
  sp.s0 = s0; sp.states = reinterpret_cast<__nv_bfloat16*>(states); sp.s_final = s_final; sp.gsum = gsum;
  sp.T = pb.T; sp.H = pb.H; sp.NT = pb.T / C / nseg; sp.nseg = nseg; sp.scale = pb.scale;
  sp.skip_xy = g_test_skip_load.exchange(-1);   // one launch only
  dim3 grid(pb.B * pb.H * nseg);
  auto launch = [&](auto kernel, const char* label) {
    if ((rc = opt_in_smem(kernel, SCAN_SMEM))) return rc;
    KernelScope ks(label, st);
    kernel<<<grid, SCAN_THREADS, SCAN_SMEM, st>>>(sp);
    return post_launch();
  };
  // no chunk-start states and a zero start: the summary form of the kernel
  const bool sum = !states && !s0;
  if (bwd) {
    const char* label = states ? "sm100_bwd_dh" : "sm100_bwd_dh_summary";
    if (sum) return scalar ? launch(k_scan<true, true, true, false>, label) : launch(k_scan<true, false, true, false>, label);
    return scalar ? launch(k_scan<true, true, false, false>, label) : launch(k_scan<true, false, false, false>, label);
  }
  const char* label = states ? "sm100_fwd_h" : "sm100_fwd_h_summary";
  if (sum) return scalar ? launch(k_scan<false, true, true, false>, label) : launch(k_scan<false, false, true, false>, label);
  return scalar ? launch(k_scan<false, true, false, false>, label) : launch(k_scan<false, false, false, false>, label);
}

// Time segments per sequence.  The scans walk a sequence chunk by chunk with one block; when there are
// too few (batch, head) pairs to fill the GPU, each sequence is cut into segments that run as blocks of
// their own: a first pass finds what every segment does to the state entering it (end state from a zero
// start and summed gates), a small kernel chains the segments, and the real pass starts every segment
// from its true state.  At least four chunks per segment.
int pick_segments(const tops_chunk_problem& pb) {
  const int bh = pb.B * pb.H, nt = pb.T / C;
  if (2 * bh > sm_count()) return 1;
  int best = 1;
  for (int n = 2; n * bh <= sm_count() && n * 4 <= nt; ++n)
    if (nt % n == 0) best = n;
  return best;
}
// fp32 scratch of a segmented scan: end states, entry states (nseg x [B,H,K,V] each) and summed gates
size_t segment_floats(const tops_chunk_problem& pb, int nseg) {
  return nseg > 1 ? (size_t)pb.B * pb.H * nseg * (2 * D * D + D) : 0;
}
struct SegmentScratch {
  float *ends, *starts, *gsum;
  SegmentScratch(float* base, const tops_chunk_problem& pb, int nseg) {
    const size_t n = (size_t)pb.B * pb.H * nseg * D * D;
    ends = base; starts = base + n; gsum = base + 2 * n;
  }
};
// summary pass + join: leaves the state entering every segment in sc.starts and the state after the last
// (forward) / before the first (reverse) segment in `last` (may be null)
// With `have_summary` the scratch already holds the segments' end states and summed gates (a shard summary
// made by state_summary() for the same problem) and only the join runs.
int segment_starts(bool bwd, const tops_chunk_problem& pb, int nseg, const void* x, const void* g, const void* y,
                   const float* first, float* last, const SegmentScratch& sc, cudaStream_t st, bool have_summary = false) {
  int rc = have_summary ? TOPS_OK : run_scan(bwd, pb, nseg, x, g, y, nullptr, nullptr, sc.ends, sc.gsum, st);
  if (rc) return rc;
  KernelScope ks("sm100_join_segments", st);
  const dim3 grid(pb.B * pb.H, 16);   // 16 slices of 1024 elements: 256 threads x float4
  if (bwd) k_join_segments<true><<<grid, 256, 0, st>>>(first, sc.gsum, sc.ends, sc.starts, last, nseg);
  else k_join_segments<false><<<grid, 256, 0, st>>>(first, sc.gsum, sc.ends, sc.starts, last, nseg);
  return post_launch();
}

}  // namespace

bool supported(const tops_chunk_problem& pb) {
  if (pb.dtype != TOPS_BF16 || pb.gate_dtype != TOPS_BF16) return false;
  if (pb.gate_kind != TOPS_GATE_PER_CHANNEL && pb.gate_kind != TOPS_GATE_SCALAR) return false;
  if (pb.K != D || pb.V != D || pb.chunk != C || pb.T % C != 0 || pb.cu_seqlens || pb.cu_seqlens_host) return false;
  if (!(pb.scale > 0.f) || !(pb.scale < 1e30f)) return false;   // states are stored multiplied by scale
  if ((size_t)pb.B * pb.T >= (1u << 31)) return false;
  return device_is_sm100() && encode_fn() != nullptr;
}

static size_t state_bytes(const tops_chunk_problem& pb) {
  return align_up((size_t)pb.B * (pb.T / C) * pb.H * D * D * 2);
}

// The fused one-pass forward keeps the chunk-start states on chip: only the two-kernel form (too few
// blocks for one per (batch, head, segment)) needs them in scratch, and only when the caller does not
// keep them itself.
static bool fwd_is_fused(const tops_chunk_problem& pb, int nseg) { return pb.B * pb.H * nseg >= kFusedMinBlocks; }

size_t fwd_workspace_bytes(const tops_chunk_fwd_params& p) {
  const int nseg = pick_segments(p.pb);
  const bool states_in_ws = !p.saved_out && !fwd_is_fused(p.pb, nseg);
  return (states_in_ws ? state_bytes(p.pb) : 0) + segment_floats(p.pb, nseg) * sizeof(float) + 256;
}

int chunk_fwd(const tops_chunk_fwd_params& p, void* ws, size_t, cudaStream_t st) {
  const tops_chunk_problem& pb = p.pb;
  if (p.g_cumsum_out || p.A_out || p.h_out) return TOPS_E_UNSUPPORTED;
  if (!aligned16(p.q) || !aligned16(p.k) || !aligned16(p.v) || !aligned16(p.g) || !aligned16(p.o) ||
      !aligned16(p.h0) || !aligned16(p.ht) || !aligned16(p.saved_out) || !aligned16(ws))
    return TOPS_E_ALIGN;
  const int BT = pb.B * pb.T, NT = pb.T / C;
  const int nseg = pick_segments(pb);
  const bool scalar = pb.gate_kind == TOPS_GATE_SCALAR;
  // workspace: [chunk-start states unless the caller keeps them] [segment scratch]
  char* wsp = reinterpret_cast<char*>(ws);
  void* h = p.saved_out ? p.saved_out : wsp;
  const bool fused = fwd_is_fused(pb, nseg);
  if (!aligned16(p.segments)) return TOPS_E_ALIGN;
  const SegmentScratch sc(p.segments ? reinterpret_cast<float*>(p.segments)
                                     : reinterpret_cast<float*>(wsp + ((p.saved_out || fused) ? 0 : state_bytes(pb))),
                          pb, nseg);
  int rc;
  const float* start = p.h0;
  float* last = p.ht;
  if (nseg > 1) {
    if ((rc = segment_starts(false, pb, nseg, p.k, p.g, p.v, p.h0, p.ht, sc, st, p.segments != nullptr))) return rc;
    start = sc.starts;
    last = nullptr;   // the join kernel has written the final state
  }
  if (fused) {
    // enough blocks to fill the GPU with one per (batch, head, segment): one pass over q, k, g, v
    FusedParams up;
    if ((rc = act_map(&up.mq, p.q, BT, pb.H)) || (rc = act_map(&up.mk, p.k, BT, pb.H)) ||
        (rc = act_map(&up.mv, p.v, BT, pb.H)))
      return rc;
    if (!scalar && (rc = act_map(&up.mg, p.g, BT, pb.H))) return rc;
    up.gscalar = reinterpret_cast<const __nv_bfloat16*>(p.g);
    up.states = nullptr;
    if (p.saved_out) {   // only a caller that keeps the states for its backward pass needs them in HBM
      if ((rc = state_map(&up.mst, p.saved_out, (size_t)pb.B * NT * pb.H * D))) return rc;
      up.states = reinterpret_cast<__nv_bfloat16*>(p.saved_out);
    }
    up.s0 = start; up.s_final = last; up.o = reinterpret_cast<__nv_bfloat16*>(p.o);
    up.T = pb.T; up.H = pb.H; up.NT = NT / nseg; up.nseg = nseg; up.scale = pb.scale;
    if ((rc = opt_in_smem(k_fwd_fused<true, false>, FUSED_SMEM)) || (rc = opt_in_smem(k_fwd_fused<false, false>, FUSED_SMEM))) return rc;
    KernelScope ks("sm100_fwd_fused", st);
    if (scalar) k_fwd_fused<true, false><<<pb.B * pb.H * nseg, FUSED_THREADS, FUSED_SMEM, st>>>(up);
    else k_fwd_fused<false, false><<<pb.B * pb.H * nseg, FUSED_THREADS, FUSED_SMEM, st>>>(up);
    return post_launch();
  }
  rc = run_scan(false, pb, nseg, p.k, p.g, p.v, start, h, last, nullptr, st);
  if (rc) return rc;
  FwdOParams fp;
  if ((rc = act_map(&fp.mq, p.q, BT, pb.H)) || (rc = act_map(&fp.mk, p.k, BT, pb.H)) ||
      (rc = act_map(&fp.mv, p.v, BT, pb.H)) || (rc = state_map(&fp.mh, h, (size_t)pb.B * NT * pb.H * D)))
    return rc;
  if (!scalar && (rc = act_map(&fp.mg, p.g, BT, pb.H))) return rc;
  fp.gscalar = reinterpret_cast<const __nv_bfloat16*>(p.g);
  fp.o = reinterpret_cast<__nv_bfloat16*>(p.o); fp.T = pb.T; fp.H = pb.H; fp.NT = NT; fp.scale = pb.scale;
  if ((rc = opt_in_smem(k_fwd_o<true>, FWD_O_SMEM)) || (rc = opt_in_smem(k_fwd_o<false>, FWD_O_SMEM))) return rc;
  KernelScope ks("sm100_fwd_o", st);
  if (scalar) k_fwd_o<true><<<dim3(pb.H, NT, pb.B), NTHREADS, FWD_O_SMEM, st>>>(fp);
  else k_fwd_o<false><<<dim3(pb.H, NT, pb.B), NTHREADS, FWD_O_SMEM, st>>>(fp);
  return post_launch();
}

size_t bwd_workspace_bytes(const tops_chunk_bwd_params& p) {
  return (p.h_saved ? 1 : 2) * state_bytes(p.pb) + segment_floats(p.pb, pick_segments(p.pb)) * sizeof(float) + 256;
}

bool bwd_dtypes_ok(const tops_chunk_bwd_params& p) {
  if (p.pb.gate_kind != TOPS_GATE_PER_CHANNEL)   // dg is the scalar gate's gradient, fp32 [B,T,H]
    return (p.grad_dtype == TOPS_F32 || p.grad_dtype == TOPS_BF16) && p.dg_dtype == TOPS_F32;
  return (p.grad_dtype == TOPS_F32 && p.dg_dtype == TOPS_F32) ||
         (p.grad_dtype == TOPS_BF16 && (p.dg_dtype == TOPS_F32 || p.dg_dtype == TOPS_BF16));
}

template <typename TG, typename TD, bool SCALAR = false, bool GEN = false>
int launch_bwd_main(const BwdParams& bp, cudaStream_t st) {
  int rc = opt_in_smem(k_bwd_main<TG, TD, SCALAR, GEN, false>, BWD_SMEM);
  if (rc) return rc;
  const int grid = bp.total < sm_count() ? bp.total : sm_count();
  {
    KernelScope ks("sm100_bwd_main", st);
    k_bwd_main<TG, TD, SCALAR, GEN, false><<<grid, BWD_THREADS, BWD_SMEM, st>>>(bp);
    if ((rc = post_launch())) return rc;
  }
  if constexpr (GEN) {
    if (!bp.gscalar && !bp.gamma && SCALAR) return TOPS_OK;   // no gate
    // What the launch above left of wide chunks is written again.  A launch of its own: it finds nothing to do as a rule,
    // and taken care of in the kernel above wide chunks cost the narrow ones registers, 354 -> 407 us at T = 16384 in 13
    // documents, H = 16 (364 us as a function called at the kernel's end).  It may be scheduled while the launch before it
    // drains (see the wait in the kernel).
    if ((rc = opt_in_smem(k_bwd_main<TG, TD, SCALAR, GEN, true>, BWD_SMEM))) return rc;
    const int blocks = cdiv(bp.total, kWideList);
    KernelScope ks("sm100_bwd_wide", st);
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid > blocks ? grid : blocks); cfg.blockDim = dim3(BWD_THREADS); cfg.dynamicSmemBytes = BWD_SMEM; cfg.stream = st;
    cfg.attrs = &early; cfg.numAttrs = 1;
    TOPS_CUDA_OK(cudaLaunchKernelEx(&cfg, k_bwd_main<TG, TD, SCALAR, GEN, true>, bp));
    return post_launch();
  }
  return TOPS_OK;
}

int chunk_bwd(const tops_chunk_bwd_params& p, void* ws, size_t, cudaStream_t st) {
  const tops_chunk_problem& pb = p.pb;
  if (!bwd_dtypes_ok(p)) return TOPS_E_UNSUPPORTED;
  if (!aligned16(p.q) || !aligned16(p.k) || !aligned16(p.v) || !aligned16(p.g) || !aligned16(p.do_) ||
      !aligned16(p.h0) || !aligned16(p.dht) || !aligned16(p.dh0) || !aligned16(p.dq) || !aligned16(p.dk) ||
      !aligned16(p.dv) || !aligned16(p.dg) || !aligned16(p.h_saved) || !aligned16(p.rev_segments) || !aligned16(ws))
    return TOPS_E_ALIGN;
  // workspace: [dh'] [h' unless the forward kept it] [segment scratch]
  const int nseg = pick_segments(pb);
  const char* h = reinterpret_cast<const char*>(p.h_saved);
  char* dh = reinterpret_cast<char*>(ws);
  const SegmentScratch sc(reinterpret_cast<float*>(dh + (h ? 1 : 2) * state_bytes(pb)), pb, nseg);
  int rc = TOPS_OK;
  if (!h) {
    char* hw = dh + state_bytes(pb);
    const float* start = p.h0;
    if (nseg > 1) {
      if ((rc = segment_starts(false, pb, nseg, p.k, p.g, p.v, p.h0, nullptr, sc, st))) return rc;
      start = sc.starts;
    }
    if ((rc = run_scan(false, pb, nseg, p.k, p.g, p.v, start, hw, nullptr, nullptr, st))) return rc;
    h = hw;
  }
  {
    const float* start = p.dht;
    float* last = p.dh0;
    if (nseg > 1) {
      const SegmentScratch rsc(p.rev_segments ? reinterpret_cast<float*>(p.rev_segments) : sc.ends, pb, nseg);
      if ((rc = segment_starts(true, pb, nseg, p.q, p.g, p.do_, p.dht, p.dh0, rsc, st, p.rev_segments != nullptr))) return rc;
      start = rsc.starts;
      last = nullptr;   // the join kernel has written dh0
    }
    if ((rc = run_scan(true, pb, nseg, p.q, p.g, p.do_, start, dh, last, nullptr, st))) return rc;
  }
  BwdParams bp;
  const int BT = pb.B * pb.T, NT = pb.T / C;
  const size_t rows = (size_t)pb.B * NT * pb.H * D;
  const bool scalar = pb.gate_kind == TOPS_GATE_SCALAR;
  if ((rc = act_map(&bp.mq, p.q, BT, pb.H)) || (rc = act_map(&bp.mk, p.k, BT, pb.H)) ||
      (rc = act_map(&bp.mv, p.v, BT, pb.H)) ||
      (rc = act_map(&bp.mdo, p.do_, BT, pb.H)) || (rc = state_map(&bp.mh, h, rows)) ||
      (rc = state_map(&bp.mdh, dh, rows)))
    return rc;
  if (!scalar && (rc = act_map(&bp.mg, p.g, BT, pb.H))) return rc;
  bp.gscalar = reinterpret_cast<const __nv_bfloat16*>(p.g);
  bp.dq = p.dq; bp.dk = p.dk; bp.dg = p.dg;
  bp.dv = reinterpret_cast<__nv_bfloat16*>(p.dv); bp.T = pb.T; bp.H = pb.H; bp.NT = NT; bp.scale = pb.scale;
  bp.total = NT * pb.B * pb.H;
  if (scalar)
    return p.grad_dtype == TOPS_F32 ? launch_bwd_main<float, float, true>(bp, st)
                                    : launch_bwd_main<__nv_bfloat16, float, true>(bp, st);
  if (p.grad_dtype == TOPS_F32) return launch_bwd_main<float, float>(bp, st);
  if (p.dg_dtype == TOPS_F32) return launch_bwd_main<__nv_bfloat16, float>(bp, st);
  return launch_bwd_main<__nv_bfloat16, __nv_bfloat16>(bp, st);
}

// ---------------------------------------------------------------------------
// the general form: packed batches, any T, K <= 128, V in slices of 128, constant or no gate
// ---------------------------------------------------------------------------
namespace {

// Time (us) of a pass over runs of chunks, one block per SM: a block costs `fixed` (its first loads, tensor memory, the
// states in and out) plus `per` a chunk; when there are more blocks than SMs they follow one another, longest first,
// and the last ones to finish leave some imbalance.  The constants are those of operands in single halves (fused forward
// 28 us for runs of 6 chunks, 212 us for 64; summary scan 18 us for 6, 1.1 us a chunk).  With two halves they are 11 + 4.7
// a chunk and 8.5 + 1.75, but all passes grew alike: plans made with those, and with the scan's own in the backward, were
// no faster (13 documents, H = 16: scans and fused forward 357 -> 364 us; 30 documents, H = 4: forward 84 -> 89 us).
struct RunCost { long long chunks = 0; int blocks = 0, longest = 0; };
double pass_time(const RunCost& r, int sms, double fixed, double per) {
  if (!r.blocks) return 0.0;
  const double longest = fixed + per * r.longest;
  if (r.blocks <= sms) return longest;
  const double even = (fixed * r.blocks + per * r.chunks) / sms + 0.3 * longest;
  return longest > even ? longest : even;
}

// Everything the launches of one call need to know about where chunks live.
struct GenPlan {
  Geo geo{};
  int N = 0, HV = 0, total_chunks = 0, runs = 0;
  bool cut = false;             // some sequence is walked as several runs
  std::vector<int> nch;         // packed: chunks per sequence
  int cps = 0;

  explicit GenPlan(const tops_chunk_problem& pb) {
    geo.K = pb.K; geo.V = pb.V; geo.VS = cdiv(pb.V, D);
    HV = pb.H * geo.VS;
    int longest = 0;
    if (pb.cu_seqlens_host) {
      N = pb.N;
      nch.resize(N);
      for (int n = 0; n < N; ++n) {
        nch[n] = cdiv(pb.cu_seqlens_host[n + 1] - pb.cu_seqlens_host[n], C);
        total_chunks += nch[n];
        longest = nch[n] > longest ? nch[n] : longest;
      }
    } else {
      N = pb.B;
      longest = geo.NTseq = cdiv(pb.T, C);
      total_chunks = N * longest;
    }
    // Cutting sequences into runs costs a summary pass and a join (which moves three states per run); it pays when whole
    // sequences would leave SMs idle.  Every candidate length is priced.
    const int sms = sm_count();
    cps = longest;
    double best = 1e30;
    for (int c = longest; c >= 4; c = c > 64 ? c * 3 / 4 : c - (c > 16 ? 2 : 1)) {
      RunCost all, sum;
      for (int n = 0; n < (nch.empty() ? 1 : N); ++n) {
        const int k = nch.empty() ? longest : nch[n], cnt = cdiv(k, c), mult = (nch.empty() ? N : 1) * HV;
        const int len = cdiv(k, cnt);
        all.chunks += (long long)k * mult; all.blocks += cnt * mult;
        if (len > all.longest) all.longest = len;
        if (cnt > 1) {
          sum.chunks += (long long)k * mult; sum.blocks += cnt * mult;
          if (len > sum.longest) sum.longest = len;
        }
      }
      const double join = sum.blocks ? 8.0 + 12.0 * sum.blocks / geo.VS * pb.K * pb.V / 4e6 : 0.0;
      const double t = pass_time(all, sms, 9.0, 3.2) + pass_time(sum, sms, 11.0, 1.1) + join;
      if (t < best - 1e-9) { best = t; cps = c; }
    }
    if (nch.empty()) {
      geo.nseg = cdiv(longest, cps);
      geo.cps = cdiv(longest, geo.nseg);
      geo.nseg = cdiv(longest, geo.cps);
      runs = N * geo.nseg;
      cut = geo.nseg > 1;
    } else {
      geo.nseg = 1; geo.cps = longest;
      for (int n = 0; n < N; ++n) { const int c = count(n); runs += c; cut = cut || c > 1; }
    }
  }
  // runs of sequence n (packed): as even as whole chunks allow, none empty
  int run_len(int n) const { return cdiv(nch[n], cdiv(nch[n], cps)); }
  int count(int n) const { return cdiv(nch[n], run_len(n)); }
  int blocks() const { return runs * HV; }
  size_t words() const { return nch.empty() ? 0 : 3 * (size_t)N + (size_t)align_up(N + 1, 4) + (3 * (size_t)N % 4 ? 4 - 3 * (size_t)N % 4 : 0) + 8 * (size_t)runs; }
  size_t table_bytes() const { return nch.empty() ? 0 : align_up(words() * 4) + align_up((size_t)total_chunks * sizeof(ChunkEntry)); }
  size_t state_bytes() const { return align_up((size_t)total_chunks * HV * D * D * 2); }
  size_t wide_bytes() const { return align_up((size_t)total_chunks * (HV / geo.VS) * 4); }
  size_t seg_state() const { return (size_t)runs * (HV / geo.VS) * geo.K * geo.V; }
  // end states, entry states, summed gates of the runs
  size_t seg_bytes() const { return cut ? align_up((2 * seg_state() + (size_t)runs * (HV / geo.VS) * D) * sizeof(float)) : 0; }

  const int* seg0 = nullptr;   // device: first run of every sequence
  // writes the tables into `ws` (table_bytes() of it)
  int upload(const tops_chunk_problem& pb, void* ws, cudaStream_t st) {
    if (nch.empty()) return TOPS_OK;
    int* dst = reinterpret_cast<int*>(ws);
    ChunkEntry* chunks = reinterpret_cast<ChunkEntry*>(reinterpret_cast<char*>(ws) + align_up(words() * 4));
    std::vector<int> w(words(), 0);
    const size_t seg0_at = align_up(3 * (size_t)N, 4), seg_at = seg0_at + align_up(N + 1, 4);
    std::vector<SegEntry> e;
    e.reserve(runs);
    int slot = 0, id = 0;
    for (int n = 0; n < N; ++n) {
      const int row = pb.cu_seqlens_host[n], end = pb.cu_seqlens_host[n + 1], len = run_len(n), cnt = count(n);
      w[3 * n] = row; w[3 * n + 1] = end; w[3 * n + 2] = slot;
      w[seg0_at + n] = id;
      for (int i = 0; i < cnt; ++i, ++id) {
        const int c0 = i * len;
        e.push_back(SegEntry{row + c0 * C, end, slot + c0, nch[n] - c0 < len ? nch[n] - c0 : len, id, n, cnt, 0});
      }
      slot += nch[n];
    }
    w[seg0_at + N] = id;
    std::stable_sort(e.begin(), e.end(), [](const SegEntry& a, const SegEntry& b) { return a.nch > b.nch; });
    memcpy(w.data() + seg_at, e.data(), e.size() * sizeof(SegEntry));
    geo.segs = reinterpret_cast<const SegEntry*>(dst + seg_at);
    geo.chunks = chunks;
    seg0 = dst + seg0_at;
    KernelScope ks("sm100_plan", st);
    if (w.size() <= kPlanSmall) {
      PlanWords<kPlanSmall> pw;
      memcpy(pw.w, w.data(), w.size() * 4);
      k_plan<kPlanSmall><<<N < 64 ? N : 64, 128, 0, st>>>(pw, dst, (int)w.size(), N, chunks);
      return post_launch();
    }
    static_assert(sizeof(PlanWords<kPlanLarge>) + 64 <= 32764, "kernel parameter space");
    for (size_t at = 0; at < w.size(); at += kPlanLarge) {
      PlanWords<kPlanLarge> pw;
      const size_t n = w.size() - at < kPlanLarge ? w.size() - at : kPlanLarge;
      memcpy(pw.w, w.data() + at, n * 4);
      k_plan<kPlanLarge><<<32, 128, 0, st>>>(pw, dst + at, (int)n, 0, chunks);
      const int rc = post_launch();
      if (rc) return rc;
    }
    k_plan_chunks<<<N < 512 ? N : 512, 128, 0, st>>>(dst, N, chunks);
    return post_launch();
  }
};
struct GenSegs {
  float *ends, *starts, *gsum;
  GenSegs(void* base, const GenPlan& g) {
    ends = reinterpret_cast<float*>(base); starts = ends + g.seg_state(); gsum = starts + g.seg_state();
  }
};
bool scalar_kind(int kind) { return kind != TOPS_GATE_PER_CHANNEL; }

// pitch: of x and y where they are q, k or v (x_pitch 0 and y_pitch 0: contiguous)
struct XYPitch { int64_t x = 0, y = 0; };
int run_scan_gen(bool bwd, bool sum, const tops_chunk_problem& pb, const GenPlan& g, const void* x, const void* gate, const void* y,
                 XYPitch pitch, const float* s0, const float* s0_seg, void* states, float* s_final, float* gsum, cudaStream_t st,
                 void* wide = nullptr) {
  ScanParams sp;
  const int BT = pb.B * pb.T;
  const bool scalar = scalar_kind(pb.gate_kind);
  int rc;
  if ((rc = act_map(&sp.mx, x, BT, pb.H, pb.K, pitch.x)) || (rc = act_map(&sp.my, y, BT, pb.H, pb.V, pitch.y))) return rc;
  if (!scalar && (rc = act_map(&sp.mg, gate, BT, pb.H, pb.K))) return rc;
  sp.gscalar = pb.gate_kind == TOPS_GATE_SCALAR ? reinterpret_cast<const __nv_bfloat16*>(gate) : nullptr;
  sp.gamma = pb.gate_kind == TOPS_GATE_GAMMA ? reinterpret_cast<const float*>(gate) : nullptr;
  if (states && (rc = state_map(&sp.mst, states, (size_t)g.total_chunks * g.HV * D))) return rc;
  sp.s0 = s0; sp.s0_seg = s0_seg; sp.states = reinterpret_cast<__nv_bfloat16*>(states); sp.s_final = s_final; sp.gsum = gsum;
  sp.T = pb.T; sp.H = pb.H; sp.NT = 0; sp.nseg = 1; sp.scale = pb.scale; sp.geo = g.geo; sp.skip_xy = -1;
  sp.wide = reinterpret_cast<uint8_t*>(wide);
  auto launch = [&](auto kernel, const char* label) {
    if ((rc = opt_in_smem(kernel, SCAN_SMEM))) return rc;
    KernelScope ks(label, st);
    kernel<<<g.blocks(), SCAN_THREADS, SCAN_SMEM, st>>>(sp);
    return post_launch();
  };
  if (bwd) {
    const char* label = sum ? "sm100_bwd_dh_summary" : "sm100_bwd_dh";
    if (sum) return scalar ? launch(k_scan<true, true, true, true>, label) : launch(k_scan<true, false, true, true>, label);
    return scalar ? launch(k_scan<true, true, false, true>, label) : launch(k_scan<true, false, false, true>, label);
  }
  const char* label = sum ? "sm100_fwd_h_summary" : "sm100_fwd_h";
  if (sum) return scalar ? launch(k_scan<false, true, true, true>, label) : launch(k_scan<false, false, true, true>, label);
  return scalar ? launch(k_scan<false, true, false, true>, label) : launch(k_scan<false, false, false, true>, label);
}

// summary pass + join for the sequences that are cut into runs
int gen_starts(bool bwd, const tops_chunk_problem& pb, const GenPlan& g, const void* x, const void* gate, const void* y,
               XYPitch pitch, const float* first, float* last, const GenSegs& sc, cudaStream_t st) {
  if (!g.cut) return TOPS_OK;
  int rc = run_scan_gen(bwd, true, pb, g, x, gate, y, pitch, nullptr, nullptr, nullptr, sc.ends, sc.gsum, st);
  if (rc) return rc;
  KernelScope ks("sm100_join_segments", st);
  const int slices = cdiv(pb.K * pb.V, 1024);
  const dim3 grid(g.N * pb.H, slices < 16 ? slices : 16);
  if (bwd) k_join_segments_gen<true><<<grid, 256, 0, st>>>(first, sc.gsum, sc.ends, sc.starts, last, g.seg0, g.geo.nseg, pb.H, pb.K, pb.V);
  else k_join_segments_gen<false><<<grid, 256, 0, st>>>(first, sc.gsum, sc.ends, sc.starts, last, g.seg0, g.geo.nseg, pb.H, pb.K, pb.V);
  return post_launch();
}
}  // namespace

// What TOPS_IMPL_AUTO gives to the general form.  K, V below 32 leave most of a 128-wide tile empty: those stay on
// the CUDA-core kernels.  An odd number of scalar gates would make a 4-byte gate fetch straddle the tensor's end.
bool supported_gen(const tops_chunk_problem& pb) {
  if (pb.dtype != TOPS_BF16 || pb.chunk != C) return false;
  const bool stored_gate = pb.gate_kind == TOPS_GATE_PER_CHANNEL || pb.gate_kind == TOPS_GATE_SCALAR;
  if (stored_gate && pb.gate_dtype != TOPS_BF16) return false;
  if (pb.K < 32 || pb.K > D || pb.K % 8 != 0 || pb.V < 32 || pb.V > 8 * D || pb.V % 8 != 0) return false;
  if (!(pb.scale > 0.f) || !(pb.scale < 1e30f)) return false;
  if (pb.gate_kind == TOPS_GATE_SCALAR && ((size_t)pb.B * pb.T * pb.H) % 2 != 0) return false;
  if ((size_t)pb.B * pb.T >= (1u << 31) - 64) return false;
  const size_t chunk_rows = ((size_t)pb.B * pb.T / C + pb.B + (pb.cu_seqlens_host ? pb.N : 0)) * pb.H * cdiv(pb.V, D);
  if (chunk_rows * D >= (1u << 31)) return false;   // rows of the state map are 32-bit coordinates
  return device_is_sm100() && encode_fn() != nullptr;
}

// The plain form cuts a sequence only where whole runs of equal length come out; with few (batch, head) pairs and an
// awkward chunk count (a prime, say) it would leave most SMs idle where the general form does not.
bool prefer_gen(const tops_chunk_problem& pb) {
  if (!supported(pb)) return supported_gen(pb);
  const int nseg = pick_segments(pb), bh = pb.B * pb.H, nt = pb.T / C;
  if (2 * bh > sm_count() || nt < 8) return false;
  const int want = sm_count() / bh < nt / 4 ? sm_count() / bh : nt / 4;
  return 4 * nseg < 3 * want && supported_gen(pb);
}

size_t gen_saved_bytes(const tops_chunk_problem& pb) { return GenPlan(pb).state_bytes(); }

size_t gen_fwd_workspace_bytes(const tops_chunk_fwd_params& p) {
  const GenPlan g(p.pb);
  return g.table_bytes() + g.seg_bytes() + 256;
}

int gen_chunk_fwd(const tops_chunk_fwd_params& p, void* ws, cudaStream_t st) {
  const tops_chunk_problem& pb = p.pb;
  const bool scalar = scalar_kind(pb.gate_kind);
  if (!aligned16(p.q) || !aligned16(p.k) || !aligned16(p.v) || (pb.gate_kind != TOPS_GATE_GAMMA && !aligned16(p.g)) ||
      !aligned16(p.o) || !aligned16(p.h0) || !aligned16(p.ht) || !aligned16(p.saved_out) || !aligned16(ws))
    return TOPS_E_ALIGN;
  if (p.pitch % 8 != 0) return TOPS_E_ALIGN;
  GenPlan g(pb);
  char* wsp = reinterpret_cast<char*>(ws);
  int rc = g.upload(pb, wsp, st);
  if (rc) return rc;
  wsp += g.table_bytes();
  void* h = p.saved_out;
  const GenSegs sc(wsp, g);
  const XYPitch kv{p.pitch, p.pitch};
  if ((rc = gen_starts(false, pb, g, p.k, p.g, p.v, kv, p.h0, p.ht, sc, st))) return rc;
  const int BT = pb.B * pb.T;
  const __nv_bfloat16* gs = pb.gate_kind == TOPS_GATE_SCALAR ? reinterpret_cast<const __nv_bfloat16*>(p.g) : nullptr;
  const float* gamma = pb.gate_kind == TOPS_GATE_GAMMA ? reinterpret_cast<const float*>(p.g) : nullptr;
  const size_t state_rows = (size_t)g.total_chunks * g.HV * D;
  FusedParams up;
  if ((rc = act_map(&up.mq, p.q, BT, pb.H, pb.K, p.pitch)) || (rc = act_map(&up.mk, p.k, BT, pb.H, pb.K, p.pitch)) ||
      (rc = act_map(&up.mv, p.v, BT, pb.H, pb.V, p.pitch)))
    return rc;
  if (!scalar && (rc = act_map(&up.mg, p.g, BT, pb.H, pb.K))) return rc;
  up.gscalar = gs; up.gamma = gamma; up.states = nullptr;
  if (h) {
    if ((rc = state_map(&up.mst, h, state_rows))) return rc;
    up.states = reinterpret_cast<__nv_bfloat16*>(h);
  }
  up.s0 = p.h0; up.s0_seg = sc.starts; up.s_final = p.ht; up.o = reinterpret_cast<__nv_bfloat16*>(p.o);
  up.T = pb.T; up.H = pb.H; up.NT = 0; up.nseg = 1; up.scale = pb.scale; up.geo = g.geo;
  up.q = reinterpret_cast<const __nv_bfloat16*>(p.q); up.k = reinterpret_cast<const __nv_bfloat16*>(p.k);
  up.g = reinterpret_cast<const __nv_bfloat16*>(p.g); up.qk_pitch = p.pitch ? p.pitch : (long long)pb.H * pb.K;
  if ((rc = opt_in_smem(k_fwd_fused<true, true>, FUSED_SMEM)) || (rc = opt_in_smem(k_fwd_fused<false, true>, FUSED_SMEM))) return rc;
  KernelScope ks("sm100_fwd_fused", st);
  if (scalar) k_fwd_fused<true, true><<<g.blocks(), FUSED_THREADS, FUSED_SMEM, st>>>(up);
  else k_fwd_fused<false, true><<<g.blocks(), FUSED_THREADS, FUSED_SMEM, st>>>(up);
  return post_launch();
}

// fp32 partial sums of dq, dk and dg over the value slices
static size_t gen_partial_floats(const tops_chunk_bwd_params& p) {
  if (p.pb.V <= D) return 0;
  const size_t n = (size_t)p.pb.B * p.pb.T * p.pb.H;
  return n * p.pb.K * 2 + (p.dg ? n * (scalar_kind(p.pb.gate_kind) ? 1 : p.pb.K) : 0);
}

size_t gen_bwd_workspace_bytes(const tops_chunk_bwd_params& p) {
  const GenPlan g(p.pb);
  return g.table_bytes() + (p.h_saved ? 1 : 2) * g.state_bytes() + g.seg_bytes() + g.wide_bytes() +
         align_up(gen_partial_floats(p) * sizeof(float)) + 256;
}

int gen_chunk_bwd(const tops_chunk_bwd_params& p, void* ws, cudaStream_t st) {
  const tops_chunk_problem& pb = p.pb;
  if (!bwd_dtypes_ok(p)) return TOPS_E_UNSUPPORTED;
  if (!aligned16(p.q) || !aligned16(p.k) || !aligned16(p.v) || (pb.gate_kind != TOPS_GATE_GAMMA && !aligned16(p.g)) ||
      !aligned16(p.do_) || !aligned16(p.h0) || !aligned16(p.dht) || !aligned16(p.dh0) || !aligned16(p.dq) || !aligned16(p.dk) ||
      !aligned16(p.dv) || !aligned16(p.dg) || !aligned16(p.h_saved) || !aligned16(ws))
    return TOPS_E_ALIGN;
  if (p.pitch % 8 != 0 || p.grad_pitch % 8 != 0) return TOPS_E_ALIGN;
  GenPlan g(pb);
  char* wsp = reinterpret_cast<char*>(ws);
  int rc = g.upload(pb, wsp, st);
  if (rc) return rc;
  wsp += g.table_bytes();
  char* dh = wsp; wsp += g.state_bytes();
  const char* h = reinterpret_cast<const char*>(p.h_saved);
  char* hw = nullptr;
  if (!h) { hw = wsp; wsp += g.state_bytes(); }
  const GenSegs sc(wsp, g); wsp += g.seg_bytes();
  char* wide = wsp; wsp += g.wide_bytes();
  float* part = reinterpret_cast<float*>(wsp);
  if (!h) {
    const XYPitch kv{p.pitch, p.pitch};
    if ((rc = gen_starts(false, pb, g, p.k, p.g, p.v, kv, p.h0, nullptr, sc, st))) return rc;
    if ((rc = run_scan_gen(false, false, pb, g, p.k, p.g, p.v, kv, p.h0, sc.starts, hw, nullptr, nullptr, st))) return rc;
    h = hw;
  }
  const XYPitch qdo{p.pitch, 0};
  if ((rc = gen_starts(true, pb, g, p.q, p.g, p.do_, qdo, p.dht, p.dh0, sc, st))) return rc;
  if ((rc = run_scan_gen(true, false, pb, g, p.q, p.g, p.do_, qdo, p.dht, sc.starts, dh, p.dh0, nullptr, st, wide))) return rc;
  BwdParams bp;
  const int BT = pb.B * pb.T;
  const size_t rows = (size_t)g.total_chunks * g.HV * D;
  const bool scalar = scalar_kind(pb.gate_kind);
  if ((rc = act_map(&bp.mq, p.q, BT, pb.H, pb.K, p.pitch)) || (rc = act_map(&bp.mk, p.k, BT, pb.H, pb.K, p.pitch)) ||
      (rc = act_map(&bp.mv, p.v, BT, pb.H, pb.V, p.pitch)) || (rc = act_map(&bp.mdo, p.do_, BT, pb.H, pb.V)) ||
      (rc = state_map(&bp.mh, h, rows)) || (rc = state_map(&bp.mdh, dh, rows)))
    return rc;
  if (!scalar && (rc = act_map(&bp.mg, p.g, BT, pb.H, pb.K))) return rc;
  bp.gscalar = pb.gate_kind == TOPS_GATE_SCALAR ? reinterpret_cast<const __nv_bfloat16*>(p.g) : nullptr;
  bp.gamma = pb.gate_kind == TOPS_GATE_GAMMA ? reinterpret_cast<const float*>(p.g) : nullptr;
  bp.dv = reinterpret_cast<__nv_bfloat16*>(p.dv);
  bp.q = reinterpret_cast<const __nv_bfloat16*>(p.q); bp.k = reinterpret_cast<const __nv_bfloat16*>(p.k);
  bp.g = reinterpret_cast<const __nv_bfloat16*>(p.g); bp.qk_pitch = p.pitch ? p.pitch : (long long)pb.H * pb.K;
  bp.wide = reinterpret_cast<const int*>(wide);
  bp.T = pb.T; bp.H = pb.H; bp.NT = g.nch.empty() ? g.geo.NTseq : g.total_chunks; bp.scale = pb.scale; bp.geo = g.geo;
  bp.total = g.total_chunks * pb.H;
  const size_t n = (size_t)BT * pb.H;
  float *pdq = part, *pdk = part + n * pb.K, *pdg = p.dg ? part + 2 * n * pb.K : nullptr;
  for (int vs = 0; vs < g.geo.VS; ++vs) {
    const bool last = vs == g.geo.VS - 1;
    bp.vs = vs;
    bp.dqk_pitch = last && p.grad_pitch ? p.grad_pitch : (long long)pb.H * pb.K;
    bp.dv_pitch = p.grad_pitch ? p.grad_pitch : (long long)pb.H * pb.V;
    bp.dq = last ? p.dq : pdq; bp.dk = last ? p.dk : pdk; bp.dg = last ? p.dg : pdg;
    bp.add_dq = vs ? pdq : nullptr; bp.add_dk = vs ? pdk : nullptr; bp.add_dg = vs ? pdg : nullptr;
    if (scalar) rc = (!last || p.grad_dtype == TOPS_F32) ? launch_bwd_main<float, float, true, true>(bp, st)
                                                         : launch_bwd_main<__nv_bfloat16, float, true, true>(bp, st);
    else if (!last || p.grad_dtype == TOPS_F32) rc = launch_bwd_main<float, float, false, true>(bp, st);
    else if (p.dg_dtype == TOPS_F32) rc = launch_bwd_main<__nv_bfloat16, float, false, true>(bp, st);
    else rc = launch_bwd_main<__nv_bfloat16, __nv_bfloat16, false, true>(bp, st);
    if (rc) return rc;
  }
  return TOPS_OK;
}

// The summary of one time shard for the state exchange between ranks: the state after the shard from a
// zero start (forward: x = k, y = v) or the state gradient before the shard for a zero gradient after it
// (reverse: x = q, y = do).  Uses the time-segmented summary scan when there are few (batch, head) pairs.
size_t summary_workspace_bytes(const tops_chunk_problem& pb) {
  return segment_floats(pb, pick_segments(pb)) * sizeof(float) + 256;
}

int state_summary(const tops_chunk_problem& pb, bool reverse, const void* x, const void* g, const void* y,
                  float* state_out, void* ws, cudaStream_t st) {
  if (!aligned16(x) || !aligned16(g) || !aligned16(y) || !aligned16(state_out) || !aligned16(ws)) return TOPS_E_ALIGN;
  const int nseg = pick_segments(pb);
  if (nseg == 1) return run_scan(reverse, pb, 1, x, g, y, nullptr, nullptr, state_out, nullptr, st);
  const SegmentScratch sc(reinterpret_cast<float*>(ws), pb, nseg);
  return segment_starts(reverse, pb, nseg, x, g, y, nullptr, state_out, sc, st);
}

int device_error(int* out) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_error, sizeof(int)) != cudaSuccess) return TOPS_E_CUDA;
  *out = v;
  return TOPS_OK;
}

void test_skip_load(int chunk) { g_test_skip_load.store(chunk); }

int device_error_set(int code) {
  return cudaMemcpyToSymbol(g_error, &code, sizeof(int)) == cudaSuccess ? TOPS_OK : TOPS_E_CUDA;
}

}  // namespace sm100
}  // namespace tops
