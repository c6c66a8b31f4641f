// Chunked KDA (gated delta rule, WY / UT-transform form) on the 5th-generation tensor cores.
//
// Shapes taken here: bf16 q/k/v/g/beta, K = V = 128, chunk 64, T a multiple of 64, dense batch.
// Everything else runs on the token-serial kernels of kda.cu.
//
// Per chunk of one head, with G the chunk-local cumulative gate (natural log), mid = (G_0 + G_n) / 2
// per channel, E = G - mid, and the chunk-start state kept as h' = h exp(mid):
//     q~ = q exp(E) scale      k^ = k exp(E)      k~ = k exp(-E)
//     Aqk = tril(q~ k~^T)                                  (the scale rides on q~)
//     L   = stril(diag(beta) k^ k~^T)        T = (I + L)^-1          (unit lower triangular, 64 x 64)
//     T'  = T diag(beta)        w = T' k^
//     v'  = T' v - w h'
//     o   = q~ h' + Aqk v'
//     h  <- h exp(G_n) + exp(G_n - mid) (k~^T v')
// Everything down to w is a chunk's own business: k_kda_prep computes it for all chunks at once.  What is left to walk
// from chunk to chunk (k_kda_scan_fwd) is two dependent products, w h' and k~^T v'; the reverse scan of the state
// gradient (k_kda_scan_bwd) has the same shape, k~ dh^ and w^T dv', and reads the same tiles.  The rest of the backward
// is chunk-parallel again (k_kda_bwd_intra, k_kda_bwd_out).
// The cumulative gates are a tensor-core product of the gate tile with a constant 0 / +-1/2 / 1 pattern
// (sm100_tiles.cuh), every contraction is a tcgen05.mma on bf16 tiles in shared memory with fp32
// accumulators in tensor memory, the running state is fp32 in registers, and the 64 x 64 triangular
// inverse is computed in fp32 on the CUDA cores: 16 x 16 diagonal blocks by forward substitution, the
// off-diagonal blocks by two levels of T_lo,hi = -T_lo,lo (L_lo,hi T_hi,hi) block products.
#include "kda_sm100.cuh"
#include "sm100_host.cuh"
#include "sm100_tiles.cuh"

namespace tops {
namespace sm100 {
namespace {

// What k_kda_prep leaves of a chunk of one head, in the order and the (swizzled) form the scans' shared memory wants it,
// so that one untiled bulk copy brings it in: T' | k~ | -w | q~ | Aqk | (G_n, mid) per channel | T.
constexpr uint32_t PREP_TB = 0, PREP_K = SLAB64, PREP_W = PREP_K + TILE64, PREP_Q = PREP_W + TILE64, PREP_A = PREP_Q + TILE64,
                   PREP_F = PREP_A + SLAB64, PREP_T = PREP_F + D * 8, PREP_BYTES = PREP_T + SLAB64;
constexpr uint32_t PREP_FWD = PREP_T;            // the forward scan reads all but T
constexpr uint32_t PREP_BWD = PREP_T - PREP_K;   // the reverse scan k~ .. (G_n, mid)

__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory"); }

// sum_k a[k] b[S k] over N entries of a row (read 16 bytes at a time) and a column
template <int N, int S>
__device__ __forceinline__ float dot_row_col(const float* __restrict__ a, const float* __restrict__ b) {
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < N; k += 4) {
    const float4 x = *reinterpret_cast<const float4*>(a + k);
    s = fmaf(x.x, b[k * S], s);
    s = fmaf(x.y, b[(k + 1) * S], s);
    s = fmaf(x.z, b[(k + 2) * S], s);
    s = fmaf(x.w, b[(k + 3) * S], s);
  }
  return s;
}
// the same for the rows a and a + step of 32 entries, which share the column: 6 shared-memory loads for 8 multiply-adds
// where one row at a time takes 16 (two resident blocks saturate the load path: k_kda_prep 808 -> 770 us at B = 4,
// T = 8192, H = 32)
__device__ __forceinline__ float2 dot_rows_col32(const float* __restrict__ a, int step, const float* __restrict__ b, int bstride) {
  float2 s = make_float2(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(a + step + k);
    const float b0 = b[k * bstride], b1 = b[(k + 1) * bstride], b2 = b[(k + 2) * bstride], b3 = b[(k + 3) * bstride];
    s.x = fmaf(x.x, b0, s.x); s.y = fmaf(y.x, b0, s.y);
    s.x = fmaf(x.y, b1, s.x); s.y = fmaf(y.y, b1, s.y);
    s.x = fmaf(x.z, b2, s.x); s.y = fmaf(y.z, b2, s.y);
    s.x = fmaf(x.w, b3, s.x); s.y = fmaf(y.w, b3, s.y);
  }
  return s;
}

// T = (I + L)^-1 for a strictly lower triangular 64 x 64 L, fp32, row-major with row stride 64, by the
// 512 compute threads.  W: 1024 floats of scratch.
__device__ __forceinline__ void invert_unit_lower(const float* __restrict__ Lm, float* __restrict__ Tm,
                                                  float* __restrict__ W, int tid) {
  for (int idx = tid; idx < C * C / 4; idx += NTHREADS) {
    const int i = idx >> 4, j = (idx & 15) * 4;
    if ((j >> 4) > (i >> 4)) *reinterpret_cast<float4*>(Tm + i * C + j) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (tid < 64) {   // 16 x 16 diagonal blocks: column c of block b by forward substitution
    const int b = tid >> 4, c = tid & 15;
    const float* Lb = Lm + (16 * b) * C + 16 * b;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s = i == c ? 1.f : 0.f;
#pragma unroll
      for (int j0 = 0; j0 < i; j0 += 4) {
        const float4 l = *reinterpret_cast<const float4*>(Lb + i * C + j0);
        s = fmaf(-l.x, x[j0], s);
        if (j0 + 1 < i) s = fmaf(-l.y, x[j0 + 1], s);
        if (j0 + 2 < i) s = fmaf(-l.z, x[j0 + 2], s);
        if (j0 + 3 < i) s = fmaf(-l.w, x[j0 + 3], s);
      }
      x[i] = s;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) Tm[(16 * b + i) * C + 16 * b + c] = x[i];
  }
  compute_sync();
  {   // 32 x 32 diagonal blocks: T_10 = -T_11 (L_10 T_00), T_32 = -T_33 (L_32 T_22)
    const int p = tid >> 8, i = (tid >> 4) & 15, j = tid & 15, o = 32 * p;
    W[tid] = dot_row_col<16, C>(Lm + (o + 16 + i) * C + o, Tm + o * C + o + j);
    compute_sync();
    Tm[(o + 16 + i) * C + o + j] = -dot_row_col<16, 16>(Tm + (o + 16 + i) * C + o + 16, W + p * 256 + j);
  }
  compute_sync();
  {   // the 32 x 32 block below the diagonal: T_lo = -T_hh (L_lo T_00')
    const int i = tid >> 5, j = tid & 31;   // rows i and i + 16
    const float2 s = dot_rows_col32(Lm + (32 + i) * C, 16 * C, Tm + j, C);
    W[i * 32 + j] = s.x;
    W[(16 + i) * 32 + j] = s.y;
    compute_sync();
    const float2 t = dot_rows_col32(Tm + (32 + i) * C + 32, 16 * C, W + j, 32);
    Tm[(32 + i) * C + j] = -t.x;
    Tm[(48 + i) * C + j] = -t.y;
  }
  compute_sync();
}

// ===========================================================================
// Chunk-parallel part of the forward
// ===========================================================================
struct KdaPrepParams {
  CUtensorMap mq, mk, mg;
  const __nv_bfloat16* beta;    // [B,T,H]
  uint8_t* prep;                // [B*NT*H] x PREP_BYTES
  int c0;                       // first chunk of the stretch
  float* Aqk_out;               // [B,T,H,64] fp32 or null
  float* Akk_out;               // [B,T,H,64] fp32 or null
  int T, H, NT, total;          // NT: chunks of the stretch; total = B * H * NT chunks
  float scale;
};
struct KdaPrepShared {
  uint64_t bar_load, bar_e, bar_a, bar_w;
  uint32_t tmem_slot;
  float a[D], g0[D];      // G_n - mid and G_0 per channel
  alignas(16) float2 f[D];   // (G_n, mid): the source of a bulk copy
  float beta[C];
};
constexpr size_t KDA_PREP_SMEM = 4 * TILE64 + 3 * SLAB64 + 2 * SLAB64 + sizeof(KdaPrepShared) + 1024;

// Persistent, two blocks per SM (104 KB of shared memory, 256 tensor-memory columns each): a chunk is a chain of short
// dependent steps (exponents, gating, two products, the inversion, w), and the other block's chunk fills the waits.
__global__ void __launch_bounds__(NTHREADS, 2) k_kda_prep(const __grid_constant__ KdaPrepParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* qs = smem;                 // q -> q~ in place; then T in fp32 during the inversion
  uint8_t* ks = qs + TILE64;          // k -> k~ in place
  uint8_t* gs = ks + TILE64;          // g; then L in fp32
  uint8_t* khs = gs + TILE64;         // k^; then -w
  uint8_t* tb = khs + TILE64;         // T' (bf16); scratch of the inversion before that
  uint8_t* ts = tb + SLAB64;          // T (bf16)
  uint8_t* at = ts + SLAB64;          // Aqk (bf16)
  uint8_t* mt = at + SLAB64;          // TRI_MID pattern, rows repeated to 128
  KdaPrepShared& sh = *reinterpret_cast<KdaPrepShared*>(mt + 2 * SLAB64);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q4 = warp & 3, seg = warp >> 2;
  constexpr uint32_t cE = 0, cA = 128, cK = 192;   // cE later holds w
  if (tid == 0) {
    mbar_init(&sh.bar_load, 1); mbar_init(&sh.bar_e, 1); mbar_init(&sh.bar_a, 1); mbar_init(&sh.bar_w, 1);
    fence_barrier_init();
    tma_prefetch_desc(&p.mq); tma_prefetch_desc(&p.mk); tma_prefetch_desc(&p.mg);
  }
  __syncwarp();
  if (warp == 0) { tmem_alloc(&sh.tmem_slot, 256); tmem_relinquish(); }
  build_tri_tile(mt, 128, TRI_MID);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = sh.tmem_slot, lane_base = q4 * 32;
  const int ri = 16 * q4 + lane;   // row of an M = 64 accumulator held by lanes 0..15 of each quarter
  const uint32_t qa = smem_u32(qs), ka = smem_u32(ks), kha = smem_u32(khs), ga = smem_u32(gs), ma = smem_u32(mt), tba = smem_u32(tb);
  auto chunk_row = [&](int cid) {   // its first token
    const int bc = cid / p.H, b = bc / p.NT;
    return b * p.T + (p.c0 + bc - b * p.NT) * C;
  };
  bool ok = true;
  int it = 0;
  for (int cid = blockIdx.x; cid < p.total; cid += gridDim.x, ++it) {
    const uint32_t ph = it & 1;
    const int h = cid % p.H, row = chunk_row(cid);   // chunks are numbered (batch, chunk, head)
    uint8_t* out = p.prep + (size_t)cid * PREP_BYTES;
    if (tid == 32 && cid + gridDim.x < p.total) {   // the tiles of this block's next chunk, on their way to L2
      const int nc = cid + gridDim.x, nh = nc % p.H, nrow = chunk_row(nc);
      tma_prefetch_l2_3d(&p.mg, 0, nh, nrow); tma_prefetch_l2_3d(&p.mg, 64, nh, nrow);
      tma_prefetch_l2_3d(&p.mq, 0, nh, nrow); tma_prefetch_l2_3d(&p.mq, 64, nh, nrow);
      tma_prefetch_l2_3d(&p.mk, 0, nh, nrow); tma_prefetch_l2_3d(&p.mk, 64, nh, nrow);
    }
    if (tid == 0) {
      tma_store_wait_read();   // the previous chunk's tiles have been read
      mbar_expect_tx(&sh.bar_load, 3 * TILE64);
      tma_load_3d(gs, &p.mg, &sh.bar_load, 0, h, row); tma_load_3d(gs + SLAB64, &p.mg, &sh.bar_load, 64, h, row);
      tma_load_3d(qs, &p.mq, &sh.bar_load, 0, h, row); tma_load_3d(qs + SLAB64, &p.mq, &sh.bar_load, 64, h, row);
      tma_load_3d(ks, &p.mk, &sh.bar_load, 0, h, row); tma_load_3d(ks + SLAB64, &p.mk, &sh.bar_load, 64, h, row);
    }
    if (tid < C) sh.beta[tid] = __bfloat162float(p.beta[(size_t)(row + tid) * p.H + h]);
    ok = __syncthreads_and(mbar_wait(&sh.bar_load, ph));
    if (!ok) { fail(3); break; }
    if (tid == 0) {
      tc_fence_after();
#pragma unroll
      for (int j0 = 0; j0 < C; j0 += 16)   // E = G - mid: [time (repeated to 128 lanes)][channel]
        umma_bf16(tm + cE, desc_kmajor(ma, 128, 0, j0), desc_mnmajor(ga, 64, j0, 0), umma_idesc(128, 128, 0, 1), j0 > 0);
      umma_commit(&sh.bar_e);
    }
    __syncwarp();
    ok = __syncthreads_and(mbar_wait(&sh.bar_e, ph));
    if (!ok) { fail(9); break; }
    tc_fence_after();
    {   // gate q and k: thread (q4, lane, seg) owns time row (32 q4 + lane) mod 64 and 16 channels
      const int i = (q4 * 32 + lane) & 63;
      const int cg = (q4 >> 1) * 4 + seg;
      float em[16];
      tmem_ld16(tmem_addr(tm, lane_base, cE + cg * 16), em);
      const uint32_t rowoff = (uint32_t)(cg >> 2) * SLAB64 + (uint32_t)i * 128u;
      if (i == 63) {
#pragma unroll
        for (int t = 0; t < 16; ++t) sh.a[cg * 16 + t] = em[t];
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t off = rowoff + (((uint32_t)((cg & 3) * 2 + u) ^ (uint32_t)i) & 7u) * 16u;
        if (i == 0) {   // G_0 = g_0
          const uint4 graw = *reinterpret_cast<const uint4*>(gs + off);
          const __nv_bfloat162* pg = reinterpret_cast<const __nv_bfloat162*>(&graw);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float2 x = __bfloat1622float2(pg[t]);
            sh.g0[cg * 16 + 8 * u + 2 * t] = x.x;
            sh.g0[cg * 16 + 8 * u + 2 * t + 1] = x.y;
          }
        }
        float f[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) f[t] = fast_exp(-em[8 * u + t]);
        const uint4 kraw = *reinterpret_cast<const uint4*>(ks + off);
        *reinterpret_cast<uint4*>(ks + off) = scale8(kraw, f);
#pragma unroll
        for (int t = 0; t < 8; ++t) f[t] = fast_exp(em[8 * u + t]);
        *reinterpret_cast<uint4*>(khs + off) = scale8(kraw, f);
#pragma unroll
        for (int t = 0; t < 8; ++t) f[t] *= p.scale;
        *reinterpret_cast<uint4*>(qs + off) = scale8(*reinterpret_cast<const uint4*>(qs + off), f);
      }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid < D) sh.f[tid] = make_float2(2.f * sh.a[tid] + sh.g0[tid], sh.a[tid] + sh.g0[tid]);
    if (tid == 0) {
      tc_fence_after();
#pragma unroll
      for (int k0 = 0; k0 < D; k0 += 16)   // k^ k~^T
        umma_bf16(tm + cK, desc_kmajor(kha, 64, 0, k0), desc_kmajor(ka, 64, 0, k0), umma_idesc(64, 64, 0, 0), k0 > 0);
#pragma unroll
      for (int k0 = 0; k0 < D; k0 += 16)   // Aqk = q~ k~^T
        umma_bf16(tm + cA, desc_kmajor(qa, 64, 0, k0), desc_kmajor(ka, 64, 0, k0), umma_idesc(64, 64, 0, 0), k0 > 0);
      umma_commit(&sh.bar_a);
      bulk_store(out + PREP_K, ks, TILE64);
      bulk_store(out + PREP_Q, qs, TILE64);
      tma_store_commit();
    }
    __syncwarp();
    ok = __syncthreads_and(mbar_wait(&sh.bar_a, ph));
    if (!ok) { fail(4); break; }
    tc_fence_after();
    float* Lm = reinterpret_cast<float*>(gs);
    float* Tm = reinterpret_cast<float*>(qs);
    {   // L = stril(beta k^ k~^T) in fp32 for the inversion; Aqk -> bf16
      float a[16];
      tmem_ld16(tmem_addr(tm, lane_base, cK + seg * 16), a);
      if (lane < 16) {
        const float bi = sh.beta[ri];
#pragma unroll
        for (int t = 0; t < 16; t += 4) {
          const int j = seg * 16 + t;
          *reinterpret_cast<float4*>(Lm + ri * C + j) =
              make_float4(j < ri ? bi * a[t] : 0.f, j + 1 < ri ? bi * a[t + 1] : 0.f, j + 2 < ri ? bi * a[t + 2] : 0.f,
                          j + 3 < ri ? bi * a[t + 3] : 0.f);
        }
      }
      tmem_ld16(tmem_addr(tm, lane_base, cA + seg * 16), a);
      if (lane < 16) {
        store_tril16(at, ri, seg * 16, a, 1.f);
        if (p.Aqk_out) {
          float* dst = p.Aqk_out + ((size_t)(row + ri) * p.H + h) * C + seg * 16;
#pragma unroll
          for (int t = 0; t < 16; t += 4) {
            const int j = seg * 16 + t;
            *reinterpret_cast<float4*>(dst + t) = make_float4(j <= ri ? a[t] : 0.f, j + 1 <= ri ? a[t + 1] : 0.f,
                                                              j + 2 <= ri ? a[t + 2] : 0.f, j + 3 <= ri ? a[t + 3] : 0.f);
          }
        }
      }
    }
    fence_async_smem();
    tc_fence_before();
    if (tid == 0) tma_store_wait_read();   // q~ has left: its tile holds T from here on
    __syncthreads();
    invert_unit_lower(Lm, Tm, reinterpret_cast<float*>(tb), tid);
    {
      const int i = tid >> 3, j0 = (tid & 7) * 8;
      const float4 x = *reinterpret_cast<const float4*>(Tm + i * C + j0);
      const float4 y = *reinterpret_cast<const float4*>(Tm + i * C + j0 + 4);
      const float* bj = sh.beta + j0;
      *reinterpret_cast<uint4*>(ts + slab_off(i, j0)) =
          make_uint4(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w), pack_bf16(y.x, y.y), pack_bf16(y.z, y.w));
      *reinterpret_cast<uint4*>(tb + slab_off(i, j0)) =
          make_uint4(pack_bf16(x.x * bj[0], x.y * bj[1]), pack_bf16(x.z * bj[2], x.w * bj[3]), pack_bf16(y.x * bj[4], y.y * bj[5]),
                     pack_bf16(y.z * bj[6], y.w * bj[7]));
      if (p.Akk_out) {
        float* dst = p.Akk_out + ((size_t)(row + i) * p.H + h) * C + j0;
        *reinterpret_cast<float4*>(dst) = x;
        *reinterpret_cast<float4*>(dst + 4) = y;
      }
    }
    fence_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
#pragma unroll
      for (int k0 = 0; k0 < C; k0 += 16)   // w[i][k] = sum_j T'[i][j] k^[j][k]
        umma_bf16(tm + cE, desc_kmajor(tba, 64, 0, k0), desc_mnmajor(kha, 64, k0, 0), umma_idesc(64, 128, 0, 1), k0 > 0);
      umma_commit(&sh.bar_w);
      bulk_store(out + PREP_TB, tb, SLAB64);
      bulk_store(out + PREP_A, at, SLAB64);
      bulk_store(out + PREP_F, sh.f, D * 8);
      bulk_store(out + PREP_T, ts, SLAB64);
      tma_store_commit();
    }
    __syncwarp();
    ok = __syncthreads_and(mbar_wait(&sh.bar_w, ph));
    if (!ok) { fail(5); break; }
    tc_fence_after();
    {
      float x[32];
      tmem_ld32(tmem_addr(tm, lane_base, cE + seg * 32), x);
      if (lane < 16) {
#pragma unroll
        for (int t = 0; t < 32; t += 8)
          *reinterpret_cast<uint4*>(khs + tile_off(64, ri, seg * 32 + t)) =
              make_uint4(pack_bf16(-x[t], -x[t + 1]), pack_bf16(-x[t + 2], -x[t + 3]), pack_bf16(-x[t + 4], -x[t + 5]),
                         pack_bf16(-x[t + 6], -x[t + 7]));
      }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      bulk_store(out + PREP_W, khs, TILE64);
      tma_store_commit();
    }
  }
  if (tid == 0) tma_store_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 256);
  if (tid == 0 && !ok) poison(reinterpret_cast<__nv_bfloat16*>(p.prep + (size_t)blockIdx.x * PREP_BYTES + PREP_W));
}

// ===========================================================================
// Forward scan and outputs
// ===========================================================================
// One block per (batch, head) walks its chunks.  The chain from one state to the next is
//     h' staged -> v' += (-w) h' -> v' to bf16 -> k~^T v' -> state update -> h' staged
// (T' v is in the accumulator before h' is there); the outputs q~ h' + Aqk v' run beside it and are written by warps of
// their own.  The roles meet only through mbarriers:
//   warps 0-15   state in registers: thread (q4, lane, seg) owns state row k = 32 q4 + lane, columns 32 seg .. + 31;
//                stage h', pack v', update the state
//   warps 16-19  write the outputs of a chunk
//   warp 20      one thread issues every product and the stores of h' and v' for a backward pass
//   warp 21      one thread issues the loads, two chunks ahead
// A form with everything of a chunk in one chain (four dependent product rounds and the inversion) took 10.4 us a
// chunk; this one takes 3.3.
struct KdaScanFwdParams {
  CUtensorMap mv, mvn, mst;     // v; v' [B*T,H,128] and h' [B*NT*H*128, 128] (TMA stores, only when kept)
  const uint8_t* prep;
  const float* s0;              // [B,H,K,V] or null (zero)
  float* s_final;               // [B,H,K,V] or null
  __nv_bfloat16* o;             // [B,T,H,V]
  int keep;                     // store h' and v'
  int T, H, NT, c0;             // NT, c0: chunks of the stretch, its first
};
struct KdaScanFwdShared {
  uint64_t full[2], hready, vbar, vready, sbar, obar[2], ofree[2];
  uint32_t tmem_slot;
  volatile int abort_flag;
};
constexpr int KDA_SF_THREADS = NTHREADS + 192;
constexpr uint32_t KDA_SF_STAGE = PREP_FWD + TILE64;   // + v
constexpr size_t KDA_SF_SMEM = 2 * KDA_SF_STAGE + TILE128 + TILE64 + sizeof(KdaScanFwdShared);

// bounded wait that also gives up when another role has failed
__device__ __forceinline__ bool role_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 255u && *abort_flag) return false;
  }
  *abort_flag = 1;
  fail(code);
  return false;
}

__global__ void __launch_bounds__(KDA_SF_THREADS, 1) k_kda_scan_fwd(const __grid_constant__ KdaScanFwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* hst = smem + 2 * KDA_SF_STAGE;   // h' (128 x 128)
  uint8_t* vts = hst + TILE128;             // v' (64 x 128)
  KdaScanFwdShared& sh = *reinterpret_cast<KdaScanFwdShared*>(vts + TILE64);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.x % p.H, b = blockIdx.x / p.H, NT = p.NT;
  constexpr uint32_t cV = 0, cD = 128, cO = 256;   // cO: two accumulators
  if ((smem_u32(smem) & 1023u) != 0) {   // uniform over the block
    if (tid == 0) fail(12);
    return;
  }
  auto stage = [&](int c) { return smem + (c & 1) * KDA_SF_STAGE; };
  auto slot = [&](int c) { return (size_t)(b * NT + c) * p.H + h; };
  auto wait = [&](uint64_t* bar, uint32_t parity, int code) { return role_wait(bar, parity, &sh.abort_flag, code); };
  if (tid == 0) {
    mbar_init(&sh.full[0], 1); mbar_init(&sh.full[1], 1); mbar_init(&sh.hready, NTHREADS); mbar_init(&sh.vready, NTHREADS);
    mbar_init(&sh.vbar, 1); mbar_init(&sh.sbar, 1); mbar_init(&sh.obar[0], 1); mbar_init(&sh.obar[1], 1);
    mbar_init(&sh.ofree[0], 128); mbar_init(&sh.ofree[1], 128);
    fence_barrier_init();
    sh.abort_flag = 0;
  }
  __syncwarp();
  if (warp == 0) { tmem_alloc(&sh.tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = sh.tmem_slot;

  if (warp < 16) {
    // ------------------------------------------------------------------ state
    const int q4 = warp & 3, seg = warp >> 2, col = q4 * 32 + lane, ri = 16 * q4 + lane;
    const uint32_t lane_base = q4 * 32;
    float S[32];
    {
      const float* src = p.s0 ? p.s0 + ((size_t)blockIdx.x * D + col) * D + seg * 32 : nullptr;
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        float4 x = src ? *reinterpret_cast<const float4*>(src + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        S[j] = x.x; S[j + 1] = x.y; S[j + 2] = x.z; S[j + 3] = x.w;
      }
    }
    auto factors = [&](int c) { return reinterpret_cast<const float2*>(stage(c) + PREP_F)[col]; };   // (G_n, mid)
    bool ok = wait(&sh.full[0], 0, 3);
    float2 f = ok ? factors(0) : make_float2(0.f, 0.f);
    for (int c = 0; ok && c < NT; ++c) {
      const float hscale = fast_exp(f.y), decay = fast_exp(f.x), c2 = fast_exp(f.x - f.y);
#pragma unroll
      for (int j = 0; j < 32; j += 8)
        *reinterpret_cast<uint4*>(hst + tile_off(128, col, seg * 32 + j)) =
            make_uint4(pack_bf16(S[j] * hscale, S[j + 1] * hscale), pack_bf16(S[j + 2] * hscale, S[j + 3] * hscale),
                       pack_bf16(S[j + 4] * hscale, S[j + 5] * hscale), pack_bf16(S[j + 6] * hscale, S[j + 7] * hscale));
      fence_async_smem();
      mbar_arrive(&sh.hready);
      if (!(ok = wait(&sh.vbar, c & 1, 7))) break;
      tc_fence_after();
      {
        float x[32];
        tmem_ld32(tmem_addr(tm, lane_base, cV + seg * 32), x);
        if (lane < 16) {
#pragma unroll
          for (int t = 0; t < 32; t += 8)
            *reinterpret_cast<uint4*>(vts + tile_off(64, ri, seg * 32 + t)) =
                make_uint4(pack_bf16(x[t], x[t + 1]), pack_bf16(x[t + 2], x[t + 3]), pack_bf16(x[t + 4], x[t + 5]),
                           pack_bf16(x[t + 6], x[t + 7]));
        }
      }
      fence_async_smem();
      tc_fence_before();
      mbar_arrive(&sh.vready);
      if (c + 1 < NT) {   // the next chunk's factors, while its product runs
        if (!(ok = wait(&sh.full[(c + 1) & 1], ((c + 1) >> 1) & 1, 3))) break;
        f = factors(c + 1);
      }
      if (!(ok = wait(&sh.sbar, c & 1, 2))) break;
      tc_fence_after();
      float d[32];
      tmem_ld32(tmem_addr(tm, lane_base, cD + seg * 32), d);
#pragma unroll
      for (int t = 0; t < 32; ++t) S[t] = fmaf(S[t], decay, c2 * d[t]);
      tc_fence_before();
    }
    if (ok && p.s_final) {
      float* dst = p.s_final + ((size_t)blockIdx.x * D + col) * D + seg * 32;
#pragma unroll
      for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(dst + j) = make_float4(S[j], S[j + 1], S[j + 2], S[j + 3]);
    }
  } else if (warp < 20) {
    // ------------------------------------------------------------------ outputs
    const int g4 = warp & 3;
    for (int c = 0; c < NT; ++c) {
      if (!wait(&sh.obar[c & 1], (c >> 1) & 1, 5)) break;
      tc_fence_after();
      __nv_bfloat16* dst = p.o + ((size_t)(b * p.T + (p.c0 + c) * C + 16 * g4 + lane) * p.H + h) * D;
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        float a[32];
        tmem_ld32(tmem_addr(tm, g4 * 32, cO + (c & 1) * 128 + s * 32), a);
        if (lane < 16) {
#pragma unroll
          for (int t = 0; t < 32; t += 8)
            __stcs(reinterpret_cast<uint4*>(dst + s * 32 + t),
                   make_uint4(pack_bf16(a[t], a[t + 1]), pack_bf16(a[t + 2], a[t + 3]), pack_bf16(a[t + 4], a[t + 5]),
                              pack_bf16(a[t + 6], a[t + 7])));
        }
      }
      tc_fence_before();
      mbar_arrive(&sh.ofree[c & 1]);
    }
  } else if (warp == 20) {
    // ------------------------------------------------------------------ products, stores of h' and v'
    if (lane == 0) {
      const uint32_t ha = smem_u32(hst), va = smem_u32(vts);
      auto issue_tv = [&](int c) {   // v' = T' v (to which -w h' is added)
        const uint32_t tba = smem_u32(stage(c) + PREP_TB), vraw = smem_u32(stage(c) + PREP_FWD);
        tc_fence_after();
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)
          umma_bf16(tm + cV, desc_kmajor(tba, 64, 0, k0), desc_mnmajor(vraw, 64, k0, 0), umma_idesc(64, 128, 0, 1), k0 > 0);
      };
      bool ok = wait(&sh.full[0], 0, 3);
      if (ok) issue_tv(0);
      for (int c = 0; ok && c < NT; ++c) {
        const uint32_t ka = smem_u32(stage(c) + PREP_K), wa = smem_u32(stage(c) + PREP_W), qa = smem_u32(stage(c) + PREP_Q),
                       aa = smem_u32(stage(c) + PREP_A);
        if (!wait(&sh.hready, c & 1, 8)) break;
        tc_fence_after();
        if (p.keep) tma_store_wait_read();   // v' of the chunk before has been read (its tile is refilled after vbar)
#pragma unroll
        for (int k0 = 0; k0 < D; k0 += 16)   // v' += (-w) h'
          umma_bf16(tm + cV, desc_kmajor(wa, 64, 0, k0), desc_mnmajor(ha, 128, k0, 0), umma_idesc(64, 128, 0, 1), 1);
        umma_commit(&sh.vbar);
        if (c >= 2 && !wait(&sh.ofree[c & 1], ((c - 2) >> 1) & 1, 10)) break;
        tc_fence_after();
#pragma unroll
        for (int k0 = 0; k0 < D; k0 += 16)   // o = q~ h'
          umma_bf16(tm + cO + (c & 1) * 128, desc_kmajor(qa, 64, 0, k0), desc_mnmajor(ha, 128, k0, 0), umma_idesc(64, 128, 0, 1), k0 > 0);
        if (p.keep) {
          const int hrow = (int)slot(c) * D;
          tma_store_2d(&p.mst, hst, 0, hrow);
          tma_store_2d(&p.mst, hst + TILE128 / 2, 64, hrow);
          tma_store_commit();
        }
        if (!wait(&sh.vready, c & 1, 11)) break;
        tc_fence_after();
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)   // D[k][v] = sum_j k~[j][k] v'[j][v]
          umma_bf16(tm + cD, desc_mnmajor(ka, 64, k0, 0), desc_mnmajor(va, 64, k0, 0), umma_idesc(128, 128, 1, 1), k0 > 0);
        if (p.keep) {   // (then there is one stretch, c0 = 0)
          const int row = b * p.T + c * C;
          tma_store_3d(&p.mvn, vts, 0, h, row);
          tma_store_3d(&p.mvn, vts + SLAB64, 64, h, row);
          tma_store_commit();
          tma_store_wait_read1();   // h' has been read: the state warps refill its tile after sbar
        }
        umma_commit(&sh.sbar);
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)   // o += Aqk v'
          umma_bf16(tm + cO + (c & 1) * 128, desc_kmajor(aa, 64, 0, k0), desc_mnmajor(va, 64, k0, 0), umma_idesc(64, 128, 0, 1), 1);
        umma_commit(&sh.obar[c & 1]);        // and the stage is free
        if (c + 1 < NT) {
          if (!wait(&sh.full[(c + 1) & 1], ((c + 1) >> 1) & 1, 3)) break;
          issue_tv(c + 1);                   // (v' has left tensor memory)
        }
      }
      tma_store_wait_all();
    }
  } else {
    // ------------------------------------------------------------------ loads
    if (lane == 0) {
      for (int c = 0; c < NT; ++c) {
        if (c >= 2 && !wait(&sh.obar[c & 1], ((c - 2) >> 1) & 1, 5)) break;
        uint64_t* bar = &sh.full[c & 1];
        uint8_t* dst = stage(c);
        const int row = b * p.T + (p.c0 + c) * C;
        mbar_expect_tx(bar, KDA_SF_STAGE);
        bulk_load(dst, p.prep + slot(c) * PREP_BYTES, PREP_FWD, bar);
        tma_load_3d(dst + PREP_FWD, &p.mv, bar, 0, h, row);
        tma_load_3d(dst + PREP_FWD + SLAB64, &p.mv, bar, 64, h, row);
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 512);
  if (tid == 0 && sh.abort_flag) {
    poison(p.o + ((size_t)(b * p.T + p.c0 * C) * p.H + h) * D);
    if (p.s_final) poison(p.s_final + (size_t)blockIdx.x * D * D);
  }
}

// ===========================================================================
// Backward, part A: the reverse scan of the state gradient
// ===========================================================================
// dh is the gradient with respect to the state a chunk hands on (h_next); per chunk, right to left, with
// dh^ = exp(G_n - mid) dh (per key channel):
//     dv'  = Aqk^T do + k~ dh^                         gradient of the delta-corrected values
//     D    = q~^T do - w^T dv'                         gradient with respect to h' = h exp(mid)
//     dh  <- dh exp(G_n) + exp(mid) D
// Aqk^T do and q~^T do are in their accumulators before the chunk's dh^ is there, so the chain is two products as in
// the forward scan: dh^ staged -> k~ dh^ -> dv' to bf16 -> w^T dv' -> update.  dh^ (bf16, [B,NT,H,K,V]) and dv' (bf16,
// [B,T,H,V]) are kept for the chunk-parallel kernels.  Roles as above, without the output warps.
struct KdaScanBwdParams {
  CUtensorMap mdo, mdvn, mst;        // do; dv' and dh^ (TMA stores)
  const uint8_t* prep;
  const float* dht;                  // [B,H,K,V] or null (zero)
  float* dh0;                        // [B,H,K,V] or null
  __nv_bfloat16* dvn;                // dv' (for the poison of a failed block)
  int T, H, NT;
};
struct KdaScanBwdShared {
  uint64_t full[2], free[2], hready, vbar, vready, sbar;
  uint32_t tmem_slot;
  volatile int abort_flag;
};
constexpr int KDA_SB_THREADS = NTHREADS + 64;
constexpr uint32_t KDA_SB_STAGE = PREP_BWD + TILE64;   // + do
constexpr size_t KDA_SB_SMEM = 2 * KDA_SB_STAGE + TILE128 + TILE64 + sizeof(KdaScanBwdShared);

__global__ void __launch_bounds__(KDA_SB_THREADS, 1) k_kda_scan_bwd(const __grid_constant__ KdaScanBwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* dhst = smem + 2 * KDA_SB_STAGE;   // dh^ (128 x 128)
  uint8_t* dvs = dhst + TILE128;             // dv' (64 x 128)
  KdaScanBwdShared& sh = *reinterpret_cast<KdaScanBwdShared*>(dvs + TILE64);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.x % p.H, b = blockIdx.x / p.H, NT = p.NT;
  constexpr uint32_t cV = 0, cD = 128;   // cD: two accumulators
  if ((smem_u32(smem) & 1023u) != 0) {
    if (tid == 0) fail(12);
    return;
  }
  // (the stage holds the chunk's tiles from PREP_K on)
  auto stage = [&](int c) { return smem + (c & 1) * KDA_SB_STAGE; };
  auto chunk_of = [&](int c) { return NT - 1 - c; };
  auto slot = [&](int c) { return (size_t)(b * NT + chunk_of(c)) * p.H + h; };
  auto wait = [&](uint64_t* bar, uint32_t parity, int code) { return role_wait(bar, parity, &sh.abort_flag, code); };
  if (tid == 0) {
    mbar_init(&sh.full[0], 1); mbar_init(&sh.full[1], 1); mbar_init(&sh.free[0], 1); mbar_init(&sh.free[1], 1);
    mbar_init(&sh.hready, NTHREADS); mbar_init(&sh.vready, NTHREADS); mbar_init(&sh.vbar, 1); mbar_init(&sh.sbar, 1);
    fence_barrier_init();
    sh.abort_flag = 0;
  }
  __syncwarp();
  if (warp == 0) { tmem_alloc(&sh.tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = sh.tmem_slot;

  if (warp < 16) {
    const int q4 = warp & 3, seg = warp >> 2, col = q4 * 32 + lane, ri = 16 * q4 + lane;
    const uint32_t lane_base = q4 * 32;
    float S[32];   // dh: row k = col, columns 32 seg .. + 31
    {
      const float* src = p.dht ? p.dht + ((size_t)blockIdx.x * D + col) * D + seg * 32 : nullptr;
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        float4 x = src ? *reinterpret_cast<const float4*>(src + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        S[j] = x.x; S[j + 1] = x.y; S[j + 2] = x.z; S[j + 3] = x.w;
      }
    }
    auto factors = [&](int c) { return reinterpret_cast<const float2*>(stage(c) + PREP_F - PREP_K)[col]; };   // (G_n, mid)
    bool ok = wait(&sh.full[0], 0, 3);
    float2 f = ok ? factors(0) : make_float2(0.f, 0.f);
    for (int c = 0; ok && c < NT; ++c) {
      const float cmid = fast_exp(f.y), decay = fast_exp(f.x), c2 = fast_exp(f.x - f.y);
#pragma unroll
      for (int j = 0; j < 32; j += 8)
        *reinterpret_cast<uint4*>(dhst + tile_off(128, col, seg * 32 + j)) =
            make_uint4(pack_bf16(S[j] * c2, S[j + 1] * c2), pack_bf16(S[j + 2] * c2, S[j + 3] * c2),
                       pack_bf16(S[j + 4] * c2, S[j + 5] * c2), pack_bf16(S[j + 6] * c2, S[j + 7] * c2));
      fence_async_smem();
      mbar_arrive(&sh.hready);
      if (!(ok = wait(&sh.vbar, c & 1, 7))) break;
      tc_fence_after();
      {
        float x[32];
        tmem_ld32(tmem_addr(tm, lane_base, cV + seg * 32), x);
        if (lane < 16) {
#pragma unroll
          for (int t = 0; t < 32; t += 8)
            *reinterpret_cast<uint4*>(dvs + tile_off(64, ri, seg * 32 + t)) =
                make_uint4(pack_bf16(x[t], x[t + 1]), pack_bf16(x[t + 2], x[t + 3]), pack_bf16(x[t + 4], x[t + 5]),
                           pack_bf16(x[t + 6], x[t + 7]));
        }
      }
      fence_async_smem();
      tc_fence_before();
      mbar_arrive(&sh.vready);
      if (c + 1 < NT) {
        if (!(ok = wait(&sh.full[(c + 1) & 1], ((c + 1) >> 1) & 1, 3))) break;
        f = factors(c + 1);
      }
      if (!(ok = wait(&sh.sbar, c & 1, 2))) break;
      tc_fence_after();
      float d[32];
      tmem_ld32(tmem_addr(tm, lane_base, cD + (c & 1) * 128 + seg * 32), d);
#pragma unroll
      for (int t = 0; t < 32; ++t) S[t] = fmaf(S[t], decay, cmid * d[t]);
      tc_fence_before();
    }
    if (ok && p.dh0) {
      float* dst = p.dh0 + ((size_t)blockIdx.x * D + col) * D + seg * 32;
#pragma unroll
      for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(dst + j) = make_float4(S[j], S[j + 1], S[j + 2], S[j + 3]);
    }
  } else if (warp == 16) {
    // ------------------------------------------------------------------ products, stores of dh^ and dv'
    if (lane == 0) {
      const uint32_t dha = smem_u32(dhst), dva = smem_u32(dvs);
      auto issue_do = [&](int c) {
        const uint32_t qa = smem_u32(stage(c) + PREP_Q - PREP_K), aa = smem_u32(stage(c) + PREP_A - PREP_K),
                       doa = smem_u32(stage(c) + PREP_BWD);
        tc_fence_after();
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)   // dv'[j][v] = sum_i Aqk[i][j] do[i][v]
          umma_bf16(tm + cV, desc_mnmajor(aa, 64, k0, 0), desc_mnmajor(doa, 64, k0, 0), umma_idesc(64, 128, 1, 1), k0 > 0);
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)   // D[k][v] = sum_i q~[i][k] do[i][v]
          umma_bf16(tm + cD + (c & 1) * 128, desc_mnmajor(qa, 64, k0, 0), desc_mnmajor(doa, 64, k0, 0), umma_idesc(128, 128, 1, 1), k0 > 0);
      };
      bool ok = wait(&sh.full[0], 0, 3);
      if (ok) issue_do(0);
      for (int c = 0; ok && c < NT; ++c) {
        const uint32_t ka = smem_u32(stage(c)), wa = smem_u32(stage(c) + PREP_W - PREP_K);
        if (!wait(&sh.hready, c & 1, 8)) break;
        tc_fence_after();
        tma_store_wait_read();   // dv' of the chunk before has been read
#pragma unroll
        for (int k0 = 0; k0 < D; k0 += 16)   // dv' += k~ dh^
          umma_bf16(tm + cV, desc_kmajor(ka, 64, 0, k0), desc_mnmajor(dha, 128, k0, 0), umma_idesc(64, 128, 0, 1), 1);
        umma_commit(&sh.vbar);
        {
          const int hrow = (int)slot(c) * D;
          tma_store_2d(&p.mst, dhst, 0, hrow);
          tma_store_2d(&p.mst, dhst + TILE128 / 2, 64, hrow);
          tma_store_commit();
        }
        if (!wait(&sh.vready, c & 1, 11)) break;
        tc_fence_after();
#pragma unroll
        for (int k0 = 0; k0 < C; k0 += 16)   // D += (-w)^T dv'
          umma_bf16(tm + cD + (c & 1) * 128, desc_mnmajor(wa, 64, k0, 0), desc_mnmajor(dva, 64, k0, 0), umma_idesc(128, 128, 1, 1), 1);
        const int row = b * p.T + chunk_of(c) * C;
        tma_store_3d(&p.mdvn, dvs, 0, h, row);
        tma_store_3d(&p.mdvn, dvs + SLAB64, 64, h, row);
        tma_store_commit();
        tma_store_wait_read1();   // dh^ has been read: its tile is refilled after sbar
        umma_commit(&sh.sbar);
        umma_commit(&sh.free[c & 1]);
        if (c + 1 < NT) {
          if (!wait(&sh.full[(c + 1) & 1], ((c + 1) >> 1) & 1, 3)) break;
          issue_do(c + 1);        // (dv' has left tensor memory)
        }
      }
      tma_store_wait_all();
    }
  } else {
    // ------------------------------------------------------------------ loads
    if (lane == 0) {
      for (int c = 0; c < NT; ++c) {
        if (c >= 2 && !wait(&sh.free[c & 1], ((c - 2) >> 1) & 1, 5)) break;
        uint64_t* bar = &sh.full[c & 1];
        uint8_t* dst = stage(c);
        const int row = b * p.T + chunk_of(c) * C;
        mbar_expect_tx(bar, KDA_SB_STAGE);
        bulk_load(dst, p.prep + slot(c) * PREP_BYTES + PREP_K, PREP_BWD, bar);
        tma_load_3d(dst + PREP_BWD, &p.mdo, bar, 0, h, row);
        tma_load_3d(dst + PREP_BWD + SLAB64, &p.mdo, bar, 64, h, row);
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 512);
  if (tid == 0 && sh.abort_flag) {
    poison(p.dvn + ((size_t)b * p.T * p.H + h) * D);
    if (p.dh0) poison(p.dh0 + (size_t)blockIdx.x * D * D);
  }
}

// ===========================================================================
// Backward, part B1: gradients of the two per-chunk matrices and of the solve's right-hand side (one block per chunk
// and head)
// ===========================================================================
//     dR = T^T dv'                 gradient of R in v' = T R, R = beta (v - k^ h')
//     dv = beta dR (output)        dbeta1 = sum_v dR v        (the h' part of dbeta comes with dk^b below)
//     dS = tril(do v'^T)           gradient of q~ k~^T (the scale rides on q~)
//     dL = -stril(dR v'^T)         gradient of L = stril(beta k^ k~^T) through T = (I + L)^-1: dT = dv' R^T and
//                                  dL = -T^T dT T^T = -(T^T dv') (T R)^T
// -dR (bf16 [B,T,H,V]), dS and dL (bf16 [B,T,H,64], row i of a chunk at token i) are scratch for part B2.
struct KdaIntraParams {
  CUtensorMap mdo, mvn, mdvn, mv;
  const uint8_t* prep;
  const __nv_bfloat16* beta;
  __nv_bfloat16 *dS, *dL, *ndr, *dv;
  float* dbeta1;
  int T, H, NT;
};

__global__ void __launch_bounds__(NTHREADS, 2) k_kda_bwd_intra(const __grid_constant__ KdaIntraParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* dos = smem;                 // do
  uint8_t* vns = dos + TILE64;         // v'
  uint8_t* dvs = vns + TILE64;         // dv'
  uint8_t* vs = dvs + TILE64;          // v
  uint8_t* nrs = vs + TILE64;          // -dR
  uint8_t* ts = nrs + TILE64;          // T (64 x 64)
  __shared__ uint64_t bar_r, bar_s, bar_1, bar_2;
  __shared__ uint32_t tmem_slot;
  __shared__ float db_s[C];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q4 = warp & 3, seg = warp >> 2;
  const int h = blockIdx.x, ci = blockIdx.y, b = blockIdx.z;
  const int row = b * p.T + ci * C;
  constexpr uint32_t cS = 0, cL = 64, cR = 128;
  if (tid == 0) {
    mbar_init(&bar_r, 1); mbar_init(&bar_s, 1); mbar_init(&bar_1, 1); mbar_init(&bar_2, 1);
    fence_barrier_init();
    mbar_expect_tx(&bar_r, 2 * TILE64 + SLAB64);   // what the longer chain needs first
    tma_load_3d(dvs, &p.mdvn, &bar_r, 0, h, row); tma_load_3d(dvs + SLAB64, &p.mdvn, &bar_r, 64, h, row);
    bulk_load(ts, p.prep + ((size_t)(b * p.NT + ci) * p.H + h) * PREP_BYTES + PREP_T, SLAB64, &bar_r);
    tma_load_3d(vs, &p.mv, &bar_r, 0, h, row); tma_load_3d(vs + SLAB64, &p.mv, &bar_r, 64, h, row);
    mbar_expect_tx(&bar_s, 2 * TILE64);
    tma_load_3d(vns, &p.mvn, &bar_s, 0, h, row); tma_load_3d(vns + SLAB64, &p.mvn, &bar_s, 64, h, row);
    tma_load_3d(dos, &p.mdo, &bar_s, 0, h, row); tma_load_3d(dos + SLAB64, &p.mdo, &bar_s, 64, h, row);
  }
  __syncwarp();
  if (warp == 0) { tmem_alloc(&tmem_slot, 256); tmem_relinquish(); }
  if (tid < C) db_s[tid] = 0.f;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = tmem_slot;
  const uint32_t lane_base = q4 * 32;
  const int ri = 16 * q4 + lane;   // rows of an M = 64 accumulator sit in lanes 0..15 of each quarter
  const size_t orow = ((size_t)(row + ri) * p.H + h) * C + seg * 16;
  const float bi = lane < 16 ? __bfloat162float(p.beta[(size_t)(row + ri) * p.H + h]) : 0.f;
  bool ok = __syncthreads_and(mbar_wait(&bar_r, 0) && mbar_wait(&bar_s, 0));
  if (!ok) fail(3);
  if (ok && tid == 0) {
    tc_fence_after();
    const uint32_t doa = smem_u32(dos), vna = smem_u32(vns), dva = smem_u32(dvs), ta = smem_u32(ts);
#pragma unroll
    for (int k0 = 0; k0 < C; k0 += 16)   // dR[j][v] = sum_i T[i][j] dv'[i][v]
      umma_bf16(tm + cR, desc_mnmajor(ta, 64, k0, 0), desc_mnmajor(dva, 64, k0, 0), umma_idesc(64, 128, 1, 1), k0 > 0);
    umma_commit(&bar_1);
#pragma unroll
    for (int k0 = 0; k0 < D; k0 += 16)   // dS[i][j] = do v'^T
      umma_bf16(tm + cS, desc_kmajor(doa, 64, 0, k0), desc_kmajor(vna, 64, 0, k0), umma_idesc(64, 64, 0, 0), k0 > 0);
  }
  __syncwarp();
  if (ok) { ok = __syncthreads_and(mbar_wait(&bar_1, 0)); if (!ok) fail(4); }
  if (ok) {
    tc_fence_after();
    float x[32];
    tmem_ld32(tmem_addr(tm, lane_base, cR + seg * 32), x);
    if (lane < 16) {
      const size_t g0i = ((size_t)(row + ri) * p.H + h) * D + seg * 32;
      float dot = 0.f;
#pragma unroll
      for (int t = 0; t < 32; t += 8) {
        const uint32_t off = tile_off(64, ri, seg * 32 + t);
        const uint4 vraw = *reinterpret_cast<const uint4*>(vs + off);
        const __nv_bfloat162* pv = reinterpret_cast<const __nv_bfloat162*>(&vraw);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2 vv = __bfloat1622float2(pv[u]);
          dot = fmaf(x[t + 2 * u], vv.x, dot);
          dot = fmaf(x[t + 2 * u + 1], vv.y, dot);
        }
        const uint4 neg = make_uint4(pack_bf16(-x[t], -x[t + 1]), pack_bf16(-x[t + 2], -x[t + 3]),
                                     pack_bf16(-x[t + 4], -x[t + 5]), pack_bf16(-x[t + 6], -x[t + 7]));
        *reinterpret_cast<uint4*>(nrs + off) = neg;
        *reinterpret_cast<uint4*>(p.ndr + g0i + t) = neg;
        __stcs(reinterpret_cast<uint4*>(p.dv + g0i + t),
               make_uint4(pack_bf16(bi * x[t], bi * x[t + 1]), pack_bf16(bi * x[t + 2], bi * x[t + 3]),
                          pack_bf16(bi * x[t + 4], bi * x[t + 5]), pack_bf16(bi * x[t + 6], bi * x[t + 7])));
      }
      atomicAdd(&db_s[ri], dot);
    }
    fence_async_smem();
    tc_fence_before();
  }
  __syncthreads();
  if (ok && tid == 0) {
    tc_fence_after();
    const uint32_t nra = smem_u32(nrs), vna = smem_u32(vns);
#pragma unroll
    for (int k0 = 0; k0 < D; k0 += 16)   // dL[i][j] = -dR v'^T
      umma_bf16(tm + cL, desc_kmajor(nra, 64, 0, k0), desc_kmajor(vna, 64, 0, k0), umma_idesc(64, 64, 0, 0), k0 > 0);
    umma_commit(&bar_2);
  }
  if (ok && tid < C) p.dbeta1[(size_t)(row + tid) * p.H + h] = db_s[tid];
  __syncwarp();
  if (ok) { ok = __syncthreads_and(mbar_wait(&bar_2, 0)); if (!ok) fail(6); }
  if (ok) {
    tc_fence_after();
    float a[16], l[16];
    tmem_ld16(tmem_addr(tm, lane_base, cS + seg * 16), a);
    tmem_ld16(tmem_addr(tm, lane_base, cL + seg * 16), l);
    if (lane < 16) {
      uint32_t w[8], x[8];
#pragma unroll
      for (int t = 0; t < 16; t += 2) {
        const int j = seg * 16 + t;
        w[t >> 1] = pack_bf16(j <= ri ? a[t] : 0.f, j + 1 <= ri ? a[t + 1] : 0.f);
        x[t >> 1] = pack_bf16(j < ri ? l[t] : 0.f, j + 1 < ri ? l[t + 1] : 0.f);
      }
      *reinterpret_cast<uint4*>(p.dS + orow) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4*>(p.dS + orow + 8) = make_uint4(w[4], w[5], w[6], w[7]);
      *reinterpret_cast<uint4*>(p.dL + orow) = make_uint4(x[0], x[1], x[2], x[3]);
      *reinterpret_cast<uint4*>(p.dL + orow + 8) = make_uint4(x[4], x[5], x[6], x[7]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 256);
  if (tid == 0 && !ok) {
    poison(p.dL + ((size_t)row * p.H + h) * C);
    poison(p.dv + ((size_t)row * p.H + h) * D);
  }
}
constexpr size_t KDA_INTRA_SMEM = 5 * TILE64 + SLAB64 + 1024;

// ===========================================================================
// Backward, part B2: dq, dk, dg, dbeta of a chunk (one block per chunk and head)
// ===========================================================================
// Accumulators are channel-major (row = key channel, column = time step), so that a thread owns one channel
// over 16 time steps and the reverse cumulative sum of dg stays in registers:
//     dq~^T  = h' do^T + k~^T dS^T
//     dk~^T  = dh^ v'^T  (kept apart: its product with k~ is part of dg)  +  q~^T dS + (beta k^)^T dL
//     dk^b^T = h' (-dR)^T + k~^T dL^T                      gradient of beta k^ (= beta k exp(E))
//     dq = dq~ exp(E) scale      dk = dk~ exp(-E) + dk^b beta exp(E)      dbeta = dbeta1 + sum_k k exp(E) dk^b
//     dg = reverse cumsum over the chunk of (q~ dq~ + beta k^ dk^b - k~ dk~)
//          + sum_v h' dh^ + sum_i k~ dk~_inter          (the exp(G_n) dependence of the state update)
struct KdaBwdOutParams {
  CUtensorMap mq, mk, mg, mdo, mvn, mndr, mh, mdh, mdS, mdL;
  const __nv_bfloat16* beta;
  const float* dbeta1;
  void *dq, *dk, *dg;     // [B,T,H,K] fp32 or bf16
  void* dbeta;            // [B,T,H]   fp32 or bf16
  int T, H, NT, total;    // total = B * H * NT chunks
  float scale;
};
constexpr size_t KDA_OUT_SMEM = 7 * TILE64 + 2 * TILE128 + 2 * SLAB64 + 2 * SLAB64 + 1024;

// Persistent: block x walks chunks x, x + gridDim.x, ... (heads fastest, so the blocks in flight read whole
// token rows).  Everything of a chunk but q and k is dead once its products have completed, so the next
// chunk's g, do, v', -dR, h', dh^, dS, dL are fetched while the threads write the gradients of this one out;
// q and k (gated in place, read by the write-out) are brought into L2 meanwhile and fetched after it.
template <typename TG>
__global__ void __launch_bounds__(NTHREADS, 1) k_kda_bwd_out(const __grid_constant__ KdaBwdOutParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* qs = smem;                  // q -> q~ in place
  uint8_t* ks = qs + TILE64;           // k -> k~ in place
  uint8_t* gs = ks + TILE64;           // g
  uint8_t* khs = gs + TILE64;          // beta k^
  uint8_t* drs = khs + TILE64;         // do and -dR as one tile of 128 rows: they meet the same h'
  uint8_t* vns = drs + 2 * TILE64;     // v'
  uint8_t* hs = vns + TILE64;          // h' (128 x 128)
  uint8_t* dhs = hs + TILE128;         // dh^ (128 x 128)
  uint8_t* dSs = dhs + TILE128;        // dS (64 x 64) and below it dL: a slab of 128 rows that meets the same k~
  uint8_t* dLs = dSs + SLAB64;
  uint8_t* mtm = dLs + SLAB64;         // TRI_MID pattern, rows repeated to 128
  // every barrier completes once per chunk (parity it & 1)
  __shared__ uint64_t bar_g, bar_qk, bar_rest, bar_e, bar_main;
  __shared__ uint32_t tmem_slot;
  __shared__ float sufsum[4][D], tails[4][D], hdh_s[D], beta_s[C], db_s[C];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q4 = warp & 3, seg = warp >> 2, col = q4 * 32 + lane;
  const int nit = (p.total - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  constexpr uint32_t cE = 0, cET = 128, cdq = 192, cdkb = 256, cdki = 320, cdkr = 384;   // dq~ and dk^b side by side
  auto chunk_rows = [&](int it, int& h, int& row, int& hrow) {
    const int cid = blockIdx.x + it * gridDim.x;
    const int ci = (cid / p.H) % p.NT, b = cid / (p.H * p.NT);
    h = cid % p.H;
    row = b * p.T + ci * C;
    hrow = ((b * p.NT + ci) * p.H + h) * D;
  };
  auto load_g = [&](int it) {
    int h, row, hrow;
    chunk_rows(it, h, row, hrow);
    mbar_expect_tx(&bar_g, TILE64);
    tma_load_3d(gs, &p.mg, &bar_g, 0, h, row); tma_load_3d(gs + SLAB64, &p.mg, &bar_g, 64, h, row);
  };
  auto load_qk = [&](int it) {
    int h, row, hrow;
    chunk_rows(it, h, row, hrow);
    mbar_expect_tx(&bar_qk, 2 * TILE64);
    tma_load_3d(qs, &p.mq, &bar_qk, 0, h, row); tma_load_3d(qs + SLAB64, &p.mq, &bar_qk, 64, h, row);
    tma_load_3d(ks, &p.mk, &bar_qk, 0, h, row); tma_load_3d(ks + SLAB64, &p.mk, &bar_qk, 64, h, row);
  };
  auto prefetch_qk = [&](int it) {
    int h, row, hrow;
    chunk_rows(it, h, row, hrow);
    tma_prefetch_l2_3d(&p.mq, 0, h, row); tma_prefetch_l2_3d(&p.mq, 64, h, row);
    tma_prefetch_l2_3d(&p.mk, 0, h, row); tma_prefetch_l2_3d(&p.mk, 64, h, row);
  };
  auto load_rest = [&](int it) {
    int h, row, hrow;
    chunk_rows(it, h, row, hrow);
    mbar_expect_tx(&bar_rest, 3 * TILE64 + 2 * TILE128 + 2 * SLAB64);
    tma_load_3d(drs, &p.mdo, &bar_rest, 0, h, row); tma_load_3d(drs + 2 * SLAB64, &p.mdo, &bar_rest, 64, h, row);
    tma_load_3d(vns, &p.mvn, &bar_rest, 0, h, row); tma_load_3d(vns + SLAB64, &p.mvn, &bar_rest, 64, h, row);
    tma_load_3d(drs + SLAB64, &p.mndr, &bar_rest, 0, h, row); tma_load_3d(drs + 3 * SLAB64, &p.mndr, &bar_rest, 64, h, row);
    tma_load_2d(hs, &p.mh, &bar_rest, 0, hrow); tma_load_2d(hs + TILE128 / 2, &p.mh, &bar_rest, 64, hrow);
    tma_load_2d(dhs, &p.mdh, &bar_rest, 0, hrow); tma_load_2d(dhs + TILE128 / 2, &p.mdh, &bar_rest, 64, hrow);
    tma_load_3d(dSs, &p.mdS, &bar_rest, 0, h, row);
    tma_load_3d(dLs, &p.mdL, &bar_rest, 0, h, row);
  };
  auto beta_of = [&](int it) {   // threads 0..63
    int h, row, hrow;
    chunk_rows(it, h, row, hrow);
    return p.beta[((size_t)row + tid) * p.H + h];
  };
  if (tid == 0) {
    mbar_init(&bar_g, 1); mbar_init(&bar_qk, 1); mbar_init(&bar_rest, 1); mbar_init(&bar_e, 1); mbar_init(&bar_main, 1);
    fence_barrier_init();
    if (nit > 0) { load_g(0); load_qk(0); load_rest(0); }
  }
  __syncwarp();
  if (warp == 0) { tmem_alloc(&tmem_slot, 512); tmem_relinquish(); }
  __nv_bfloat16 beta_next = __float2bfloat16(0.f);   // threads 0..63: beta of the next chunk, as loaded
  if (tid < C && nit > 0) beta_next = beta_of(0);
  build_tri_tile(mtm, 128, TRI_MID);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = tmem_slot;
  const uint32_t lane_base = q4 * 32;
  TG* const dq_out = reinterpret_cast<TG*>(p.dq);
  TG* const dk_out = reinterpret_cast<TG*>(p.dk);
  TG* const dg_out = reinterpret_cast<TG*>(p.dg);
  const size_t ostride = (size_t)p.H * D;
  const ColAddr ca = col_prep(64, col);
  bool ok = true;
  // Every bounded wait sits at the start of a chunk's work, before any copy for the chunk after it is issued:
  // when one gives up, all copies in flight were issued before its spin began and have long landed.
  for (int it = 0; it < nit; ++it) {
    const uint32_t ph = it & 1;
    const bool more = it + 1 < nit;
    int h, row, hrow;
    chunk_rows(it, h, row, hrow);
    float db1 = 0.f;   // threads 0..63: the scan's part of dbeta (read here, used after the write-out)
    if (tid < C) {
      beta_s[tid] = __bfloat162float(beta_next);
      db_s[tid] = 0.f;
      db1 = p.dbeta1[((size_t)row + tid) * p.H + h];
    }
    ok = __syncthreads_and(mbar_wait(&bar_g, ph));
    if (!ok) { fail(3); break; }
    if (tid == 0) {
      tc_fence_after();
      const uint32_t ga = smem_u32(gs), mma = smem_u32(mtm);
#pragma unroll
      for (int j0 = 0; j0 < C; j0 += 16)   // G - mid, [time (repeated)][channel]
        umma_bf16(tm + cE, desc_kmajor(mma, 128, 0, j0), desc_mnmajor(ga, 64, j0, 0), umma_idesc(128, 128, 0, 1), j0 > 0);
#pragma unroll
      for (int j0 = 0; j0 < C; j0 += 16)   // G - mid, [channel][time]
        umma_bf16(tm + cET, desc_mnmajor(ga, 64, j0, 0), desc_kmajor(mma, 64, 0, j0), umma_idesc(128, 64, 1, 0), j0 > 0);
      umma_commit(&bar_e);
    }
    __syncwarp();
    ok = __syncthreads_and(mbar_wait(&bar_e, ph) && mbar_wait(&bar_qk, ph));
    if (!ok) { fail(9); break; }
    {   // gate: thread (q4, lane, seg) owns time row (32 q4 + lane) mod 64 and 16 channels
      tc_fence_after();
      const int i = (q4 * 32 + lane) & 63;
      const int cg = (q4 >> 1) * 4 + seg;
      float em[16];
      tmem_ld16(tmem_addr(tm, lane_base, cE + cg * 16), em);
      const uint32_t rowoff = (uint32_t)(cg >> 2) * SLAB64 + (uint32_t)i * 128u;
      const float bi = beta_s[i];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t off = rowoff + (((uint32_t)((cg & 3) * 2 + u) ^ (uint32_t)i) & 7u) * 16u;
        float fb[8], fs[8], r[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const float f = fast_exp(em[8 * u + t]);
          fb[t] = f * bi;
          fs[t] = f * p.scale;
          r[t] = fast_exp(-em[8 * u + t]);
        }
        const uint4 kraw = *reinterpret_cast<const uint4*>(ks + off);
        *reinterpret_cast<uint4*>(qs + off) = scale8(*reinterpret_cast<const uint4*>(qs + off), fs);
        *reinterpret_cast<uint4*>(khs + off) = scale8(kraw, fb);
        *reinterpret_cast<uint4*>(ks + off) = scale8(kraw, r);
      }
      fence_async_smem();
      tc_fence_before();
    }
    ok = __syncthreads_and(mbar_wait(&bar_rest, ph));
    if (!ok) { fail(6); break; }
    if (tid == 0) {
      tc_fence_after();
      const uint32_t qa = smem_u32(qs), ka = smem_u32(ks), kha = smem_u32(khs), dra = smem_u32(drs), vna = smem_u32(vns),
                     ha = smem_u32(hs), dha = smem_u32(dhs), dSa = smem_u32(dSs), dLa = smem_u32(dLs);
#pragma unroll
      for (int k0 = 0; k0 < D; k0 += 16)   // dq~^T[k][i] = h' do^T;  dk^b^T[k][j] = h' (-dR)^T
        umma_bf16(tm + cdq, desc_kmajor(ha, 128, 0, k0), desc_kmajor(dra, 128, 0, k0), umma_idesc(128, 128, 0, 0), k0 > 0);
#pragma unroll
      for (int k0 = 0; k0 < C; k0 += 16)   // dq~^T[k][i] += sum_j k~[j][k] dS[i][j];  dk^b^T[k][j] += sum_i k~[i][k] dL[j][i]
        umma_bf16(tm + cdq, desc_mnmajor(ka, 64, k0, 0), desc_kmajor(dSa, 128, 0, k0), umma_idesc(128, 128, 1, 0), 1);
#pragma unroll
      for (int k0 = 0; k0 < D; k0 += 16)   // dk~_inter^T[k][j] = dh^ v'^T
        umma_bf16(tm + cdki, desc_kmajor(dha, 128, 0, k0), desc_kmajor(vna, 64, 0, k0), umma_idesc(128, 64, 0, 0), k0 > 0);
#pragma unroll
      for (int k0 = 0; k0 < C; k0 += 16)   // dk~_rest^T[k][j] = sum_i q~[i][k] dS[i][j]
        umma_bf16(tm + cdkr, desc_mnmajor(qa, 64, k0, 0), desc_mnmajor(dSa, 64, k0, 0), umma_idesc(128, 64, 1, 1), k0 > 0);
#pragma unroll
      for (int k0 = 0; k0 < C; k0 += 16)   // dk~_rest^T[k][j] += sum_i (beta k^)[i][k] dL[i][j]
        umma_bf16(tm + cdkr, desc_mnmajor(kha, 64, k0, 0), desc_mnmajor(dLa, 64, k0, 0), umma_idesc(128, 64, 1, 1), 1);
      umma_commit(&bar_main);
    }
    __syncwarp();
    {   // sum_v h'[k][v] dh^[k][v] while the products run: thread = (channel, quarter of the columns)
      const int kk = tid >> 2, part = tid & 3;
      float hd = 0.f;
#pragma unroll
      for (int c8 = 0; c8 < 32; c8 += 8) {
        const uint32_t off = tile_off(128, kk, part * 32 + c8);
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
      hd += __shfl_xor_sync(0xffffffffu, hd, 1);
      hd += __shfl_xor_sync(0xffffffffu, hd, 2);
      if (part == 0) hdh_s[kk] = hd;
    }
    ok = __syncthreads_and(mbar_wait(&bar_main, ph));
    if (!ok) { fail(8); break; }
    // the products are complete and no thread reads h', dh^ any more: all of this chunk but q~, k~, beta k^
    // is dead, the next chunk's tiles take their place while the gradients are written out
    if (tid == 0 && more) {
      load_g(it + 1);
      load_rest(it + 1);
      prefetch_qk(it + 1);
    }
    if (tid < C && more) beta_next = beta_of(it + 1);
    const size_t obase = ((size_t)(row + seg * SEG) * p.H + h) * D + col;
    const size_t obase4 = obase - (lane & 3) + (size_t)(lane & 3) * ostride;
    float dgl[SEG], dbl[SEG];
    float run = 0.f, tail = 0.f;
    tc_fence_after();
#pragma unroll
    for (int blk = 1; blk >= 0; --blk) {
      float et[8], dq[8], dki[8], dkr[8], dkb[8];
      const uint32_t c0 = seg * SEG + blk * 8;
      tmem_ld8(tmem_addr(tm, lane_base, cET + c0), et);
      tmem_ld8(tmem_addr(tm, lane_base, cdq + c0), dq);
      tmem_ld8(tmem_addr(tm, lane_base, cdki + c0), dki);
      tmem_ld8(tmem_addr(tm, lane_base, cdkr + c0), dkr);
      tmem_ld8(tmem_addr(tm, lane_base, cdkb + c0), dkb);
#pragma unroll
      for (int u = 7; u >= 0; --u) {
        const int t = blk * 8 + u, ti = seg * SEG + t;
        const uint32_t off = ca.at(ti);
        const float qv = ld_bf16(qs, off), kv = ld_bf16(ks, off), kbv = ld_bf16(khs, off);   // q~, k~, beta k^
        const float e = fast_exp(et[u]), r = fast_exp(-et[u]);
        const float dkt = dki[u] + dkr[u];                 // dk~
        run += qv * dq[u] + kbv * dkb[u] - kv * dkt;
        tail = fmaf(dki[u], kv, tail);
        dgl[t] = run;
        st_out(dq_out, obase + t * ostride, e * p.scale * dq[u]);
        st_out(dk_out, obase + t * ostride, r * dkt + e * beta_s[ti] * dkb[u]);
        dbl[t] = kv * e * e * dkb[u];   // dbeta2[t] = sum_k k exp(E) dk^b = sum_k k~ e^2 dk^b
      }
    }
    {   // sum over the channels: the lanes of a warp by a shuffle butterfly, the four warps of a segment by atomics
      const float mine = warp_sum16(dbl, lane);
      if (lane < SEG) atomicAdd(&db_s[seg * SEG + lane], mine);
    }
    sufsum[seg][col] = run;
    tails[seg][col] = tail;
    tc_fence_before();
    __syncthreads();   // q~, k~, beta k^ and tensor memory have been read
    if (tid == 0 && more) load_qk(it + 1);
    {
      const float later = (seg < 1 ? sufsum[1][col] : 0.f) + (seg < 2 ? sufsum[2][col] : 0.f) + (seg < 3 ? sufsum[3][col] : 0.f);
      const float cst = later + tails[0][col] + tails[1][col] + tails[2][col] + tails[3][col] + hdh_s[col];
#pragma unroll
      for (int t = 0; t < SEG; t += 4) {
        float w[4] = {dgl[t] + cst, dgl[t + 1] + cst, dgl[t + 2] + cst, dgl[t + 3] + cst};
        st_transposed4(dg_out, obase4 + t * ostride, w, lane);
      }
      if (tid < C) st_out(reinterpret_cast<TG*>(p.dbeta), ((size_t)row + tid) * p.H + h, db_s[tid] + db1);
    }
    __syncthreads();   // sufsum, tails, hdh_s, db_s, beta_s are free for the next chunk
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tm, 512);
  if (tid == 0 && !ok) {
    int h, row, hrow;
    chunk_rows(0, h, row, hrow);
    poison(dq_out + ((size_t)row * p.H + h) * D);
  }
}

}  // namespace

bool kda_supported(const tops_chunk_kda_fwd_params& p) {
  if (p.dtype != TOPS_BF16 || p.gate_dtype != TOPS_BF16) return false;
  if (p.K != D || p.V != D || p.chunk != C || p.T % C != 0) return false;
  if (!(p.scale > 0.f) || !(p.scale < 1e30f)) return false;
  if ((size_t)p.B * p.T >= (1u << 31) || (size_t)p.B * p.T * p.H * 2 >= (1u << 31)) return false;   // (32-bit state rows)
  return device_is_sm100() && encode_fn() != nullptr;
}

// saved for a backward pass: [prep] [h'] [v']; without one only [prep] is needed, as scratch
static size_t prep_bytes(int B, int T, int H) { return align_up((size_t)B * (T / C) * H * PREP_BYTES); }
static size_t chunk_state_bytes(int B, int T, int H) { return align_up((size_t)B * (T / C) * H * D * D * 2); }
static size_t activation_bytes(int B, int T, int H) { return align_up((size_t)B * T * H * D * 2); }
size_t kda_chunk_saved_bytes(const tops_chunk_kda_fwd_params& p) {
  return prep_bytes(p.B, p.T, p.H) + chunk_state_bytes(p.B, p.T, p.H) + activation_bytes(p.B, p.T, p.H);
}
// Without one the sequences are walked in stretches whose tiles take a gigabyte at most (the state between them in fp32):
// the tiles are 4.5 times the size of q, and nothing but the scan that follows reads them.  Two stretches instead of one at
// B = 4, T = 8192, H = 32.
constexpr size_t kPrepScratch = 1ull << 30;
static int stretch_chunks(const tops_chunk_kda_fwd_params& p) {
  const int NT = p.T / C;
  const size_t per = (size_t)p.B * p.H * PREP_BYTES, fit = kPrepScratch / per;
  const int most = fit < 1 ? 1 : fit < (size_t)NT ? (int)fit : NT;
  return (NT + (NT + most - 1) / most - 1) / ((NT + most - 1) / most);   // (stretches of about equal length)
}
static size_t boundary_state_bytes(const tops_chunk_kda_fwd_params& p) {
  return stretch_chunks(p) < p.T / C ? align_up((size_t)p.B * p.H * D * D * 4) : 0;
}
size_t kda_chunk_fwd_workspace_bytes(const tops_chunk_kda_fwd_params& p) {
  return p.saved ? 0 : prep_bytes(p.B, stretch_chunks(p) * C, p.H) + boundary_state_bytes(p);
}

int kda_chunk_fwd(const tops_chunk_kda_fwd_params& p, cudaStream_t st) {
  if (!aligned16(p.q) || !aligned16(p.k) || !aligned16(p.v) || !aligned16(p.g) || !aligned16(p.o) || !aligned16(p.h0) ||
      !aligned16(p.ht) || !aligned16(p.saved) || !aligned16(p.workspace) || !aligned16(p.Aqk_out) || !aligned16(p.Akk_out))
    return TOPS_E_ALIGN;
  const int BT = p.B * p.T, NT = p.T / C;
  int rc;
  // a caller that passes no scratch gets it from the stream's memory pool for the length of the call
  void* own = nullptr;
  uint8_t* prep = reinterpret_cast<uint8_t*>(p.saved ? p.saved : p.workspace);
  if (!p.saved && p.workspace_bytes < kda_chunk_fwd_workspace_bytes(p)) {
    if (p.workspace) return TOPS_E_WORKSPACE;
    TOPS_CUDA_OK(cudaMallocAsync(&own, kda_chunk_fwd_workspace_bytes(p), st));
    prep = reinterpret_cast<uint8_t*>(own);
  }
  float* boundary = nullptr;   // the state between two stretches
  if (!p.saved && boundary_state_bytes(p)) boundary = reinterpret_cast<float*>(prep + prep_bytes(p.B, stretch_chunks(p) * C, p.H));
  auto run = [&](int c0, int nch) -> int {
    {
      KdaPrepParams pp;
      if ((rc = act_map(&pp.mq, p.q, BT, p.H)) || (rc = act_map(&pp.mk, p.k, BT, p.H)) || (rc = act_map(&pp.mg, p.g, BT, p.H))) return rc;
      pp.beta = reinterpret_cast<const __nv_bfloat16*>(p.beta);
      pp.prep = prep; pp.Aqk_out = p.Aqk_out; pp.Akk_out = p.Akk_out;
      pp.T = p.T; pp.H = p.H; pp.NT = nch; pp.c0 = c0; pp.total = p.B * nch * p.H; pp.scale = p.scale;
      if ((rc = opt_in_smem(k_kda_prep, KDA_PREP_SMEM))) return rc;
      const int grid = pp.total < 2 * sm_count() ? pp.total : 2 * sm_count();
      KernelScope ks("sm100_kda_prep", st);
      k_kda_prep<<<grid, NTHREADS, KDA_PREP_SMEM, st>>>(pp);
      if ((rc = post_launch())) return rc;
    }
    KdaScanFwdParams sp;
    if ((rc = act_map(&sp.mv, p.v, BT, p.H))) return rc;
    sp.keep = p.saved != nullptr;
    if (p.saved) {
      uint8_t* h = prep + prep_bytes(p.B, p.T, p.H);
      if ((rc = state_map(&sp.mst, h, (size_t)p.B * NT * p.H * D)) || (rc = act_map(&sp.mvn, h + chunk_state_bytes(p.B, p.T, p.H), BT, p.H)))
        return rc;
    }
    // (a block reads the state it starts from before it writes the one it ends with)
    sp.prep = prep; sp.s0 = c0 ? boundary : p.h0; sp.s_final = c0 + nch < NT ? boundary : p.ht; sp.o = reinterpret_cast<__nv_bfloat16*>(p.o);
    sp.T = p.T; sp.H = p.H; sp.NT = nch; sp.c0 = c0;
    if ((rc = opt_in_smem(k_kda_scan_fwd, KDA_SF_SMEM))) return rc;
    KernelScope ks("sm100_kda_scan_fwd", st);
    k_kda_scan_fwd<<<p.B * p.H, KDA_SF_THREADS, KDA_SF_SMEM, st>>>(sp);
    return post_launch();
  };
  const int stretch = p.saved ? NT : stretch_chunks(p);
  rc = TOPS_OK;
  for (int c0 = 0; rc == TOPS_OK && c0 < NT; c0 += stretch) rc = run(c0, NT - c0 < stretch ? NT - c0 : stretch);
  if (own && cudaFreeAsync(own, st) != cudaSuccess && rc == TOPS_OK) rc = TOPS_E_CUDA;
  return rc;
}

static size_t kda_mat_bytes(const tops_chunk_kda_bwd_params& p) { return align_up((size_t)p.B * p.T * p.H * C * 2); }
static size_t kda_beta_bytes(const tops_chunk_kda_bwd_params& p) { return align_up((size_t)p.B * p.T * p.H * 4); }

size_t kda_chunk_bwd_workspace_bytes(const tops_chunk_kda_bwd_params& p) {
  // [dh^] [dv'] [-dR] [dS] [dL] [dbeta1]
  return chunk_state_bytes(p.B, p.T, p.H) + 2 * activation_bytes(p.B, p.T, p.H) + 2 * kda_mat_bytes(p) + kda_beta_bytes(p) + 256;
}

bool kda_bwd_supported(const tops_chunk_kda_bwd_params& p) {
  tops_chunk_kda_fwd_params f{};
  f.B = p.B; f.T = p.T; f.H = p.H; f.K = p.K; f.V = p.V; f.chunk = p.chunk; f.dtype = p.dtype; f.gate_dtype = p.gate_dtype;
  f.scale = p.scale;
  return kda_supported(f) && (p.grad_dtype == TOPS_F32 || p.grad_dtype == TOPS_BF16);
}

int kda_chunk_bwd(const tops_chunk_kda_bwd_params& p, void* ws, cudaStream_t st) {
  const void* ptrs[] = {p.q, p.k, p.v, p.g, p.do_, p.dht, p.saved, p.dq, p.dk, p.dv, p.dg, p.dh0, ws};
  for (const void* x : ptrs)
    if (!aligned16(x)) return TOPS_E_ALIGN;
  const int BT = p.B * p.T, NT = p.T / C;
  const size_t rows = (size_t)p.B * NT * p.H * D;
  const uint8_t* prep = reinterpret_cast<const uint8_t*>(p.saved);
  const uint8_t* hsaved = prep + prep_bytes(p.B, p.T, p.H);
  const uint8_t* vnsaved = hsaved + chunk_state_bytes(p.B, p.T, p.H);
  char* w = reinterpret_cast<char*>(ws);
  __nv_bfloat16* dh = reinterpret_cast<__nv_bfloat16*>(w); w += chunk_state_bytes(p.B, p.T, p.H);
  __nv_bfloat16* dvn = reinterpret_cast<__nv_bfloat16*>(w); w += activation_bytes(p.B, p.T, p.H);
  __nv_bfloat16* ndr = reinterpret_cast<__nv_bfloat16*>(w); w += activation_bytes(p.B, p.T, p.H);
  __nv_bfloat16* dS = reinterpret_cast<__nv_bfloat16*>(w); w += kda_mat_bytes(p);
  __nv_bfloat16* dL = reinterpret_cast<__nv_bfloat16*>(w); w += kda_mat_bytes(p);
  float* dbeta1 = reinterpret_cast<float*>(w);
  int rc;
  {
    KdaScanBwdParams sp;
    if ((rc = act_map(&sp.mdo, p.do_, BT, p.H)) || (rc = act_map(&sp.mdvn, dvn, BT, p.H)) || (rc = state_map(&sp.mst, dh, rows))) return rc;
    sp.prep = prep; sp.dht = p.dht; sp.dh0 = p.dh0; sp.dvn = dvn;
    sp.T = p.T; sp.H = p.H; sp.NT = NT;
    if ((rc = opt_in_smem(k_kda_scan_bwd, KDA_SB_SMEM))) return rc;
    KernelScope ks("sm100_kda_bwd_scan", st);
    k_kda_scan_bwd<<<p.B * p.H, KDA_SB_THREADS, KDA_SB_SMEM, st>>>(sp);
    if ((rc = post_launch())) return rc;
  }
  const bool state_gradient_only = !p.dq && !p.dk && !p.dg && !p.dbeta;
  if (state_gradient_only && !p.dv) return TOPS_OK;
  {
    KdaIntraParams ip;
    if ((rc = act_map(&ip.mdo, p.do_, BT, p.H)) || (rc = act_map(&ip.mvn, vnsaved, BT, p.H)) ||
        (rc = act_map(&ip.mdvn, dvn, BT, p.H)) || (rc = act_map(&ip.mv, p.v, BT, p.H)))
      return rc;
    ip.prep = prep; ip.beta = reinterpret_cast<const __nv_bfloat16*>(p.beta);
    ip.dS = dS; ip.dL = dL; ip.ndr = ndr; ip.dv = reinterpret_cast<__nv_bfloat16*>(p.dv); ip.dbeta1 = dbeta1;
    ip.T = p.T; ip.H = p.H; ip.NT = NT;
    if ((rc = opt_in_smem(k_kda_bwd_intra, KDA_INTRA_SMEM))) return rc;
    KernelScope ks("sm100_kda_bwd_intra", st);
    k_kda_bwd_intra<<<dim3(p.H, NT, p.B), NTHREADS, KDA_INTRA_SMEM, st>>>(ip);
    if ((rc = post_launch())) return rc;
  }
  if (state_gradient_only) return TOPS_OK;   // (dv = beta T^T dv' is the kernel's above)
  {
    KdaBwdOutParams op;
    if ((rc = act_map(&op.mq, p.q, BT, p.H)) || (rc = act_map(&op.mk, p.k, BT, p.H)) ||
        (rc = act_map(&op.mg, p.g, BT, p.H)) || (rc = act_map(&op.mdo, p.do_, BT, p.H)) ||
        (rc = act_map(&op.mvn, vnsaved, BT, p.H)) || (rc = act_map(&op.mndr, ndr, BT, p.H)) ||
        (rc = state_map(&op.mh, hsaved, rows)) || (rc = state_map(&op.mdh, dh, rows)) ||
        (rc = mat_map(&op.mdS, dS, BT, p.H)) || (rc = mat_map(&op.mdL, dL, BT, p.H)))
      return rc;
    op.beta = reinterpret_cast<const __nv_bfloat16*>(p.beta);
    op.dbeta1 = dbeta1; op.dq = p.dq; op.dk = p.dk; op.dg = p.dg; op.dbeta = p.dbeta;
    op.T = p.T; op.H = p.H; op.NT = NT; op.scale = p.scale;
    op.total = p.B * p.H * NT;
    const int grid = op.total < sm_count() ? op.total : sm_count();
    KernelScope ks("sm100_kda_bwd_out", st);
    if (p.grad_dtype == TOPS_F32) {
      if ((rc = opt_in_smem(k_kda_bwd_out<float>, KDA_OUT_SMEM))) return rc;
      k_kda_bwd_out<float><<<grid, NTHREADS, KDA_OUT_SMEM, st>>>(op);
    } else {
      if ((rc = opt_in_smem(k_kda_bwd_out<__nv_bfloat16>, KDA_OUT_SMEM))) return rc;
      k_kda_bwd_out<__nv_bfloat16><<<grid, NTHREADS, KDA_OUT_SMEM, st>>>(op);
    }
    return post_launch();
  }
}

int kda_device_error(int* out) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_error, sizeof(int)) != cudaSuccess) return TOPS_E_CUDA;
  *out = v;
  return TOPS_OK;
}

int kda_device_error_set(int code) {
  return cudaMemcpyToSymbol(g_error, &code, sizeof(int)) == cudaSuccess ? TOPS_OK : TOPS_E_CUDA;
}

}  // namespace sm100
}  // namespace tops
