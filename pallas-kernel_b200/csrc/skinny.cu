// Linear projections of a few rows (a decode step's tokens): y_m = x W_m^T for several weight matrices at once.
//
// Bound by reading the weights once: 6.3 MB for the five input projections of a 1024-wide layer, about a microsecond of
// HBM or L2; the library's GEMMs take 4 us and a launch each.  A block owns 16 weight rows and its 8 warps split the
// contraction, so that every warp's loads (16 bytes per lane, two weight rows) are in flight at once and a small layer
// still gives every SM a block; the warps' fp32 tiles meet in shared memory and are added in warp order.  The products
// are mma.sync m16n8k16: with at most 64 rows of x a tcgen05 tile (M = 64 or 128) would be mostly padding, and the
// operands come straight from global memory in fragment order: the contraction is permuted, the same way for W and x,
// so that a lane's 16 contiguous bytes are its fragments of two consecutive products.
// 1024 -> 3088 (five matrices), 8 rows, and the output projection: 6.0 us for both launches against 26 us for seven.
#include "skinny.cuh"

namespace tops {
namespace skinny {
namespace {

constexpr int WARPS = 8;

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: groups of 8 rows of x
template <int NT>
__global__ void __launch_bounds__(WARPS * 32) k_skinny_linear(const __grid_constant__ tops_skinny_linear_params p) {
  __shared__ float part[WARPS][16][8 * NT + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  int tile = blockIdx.x, m = 0;
  while (tile >= (p.N[m] + 15) / 16) { tile -= (p.N[m] + 15) / 16; ++m; }   // (the grid is the sum of the tiles)
  const int n0 = tile * 16, N = p.N[m];
  const __nv_bfloat16* W = reinterpret_cast<const __nv_bfloat16*>(p.W[m]);
  const __nv_bfloat16* x = reinterpret_cast<const __nv_bfloat16*>(p.x);
  const bool lo = n0 + g < N, hi = n0 + g + 8 < N;
  const __nv_bfloat16 *wl = W + (size_t)(n0 + g) * p.K + 8 * t, *wh = wl + (size_t)8 * p.K;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  constexpr int U = NT <= 2 ? 4 : 2;   // blocks of 32 channels whose loads are in flight together
  for (int kb = warp; kb * 32 < p.K; kb += WARPS * U) {
    uint4 a[U], b[U], xr[U][NT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k0 = (kb + u * WARPS) * 32;
      const bool in = k0 < p.K;
      a[u] = in && lo ? __ldg(reinterpret_cast<const uint4*>(wl + k0)) : zero;
      b[u] = in && hi ? __ldg(reinterpret_cast<const uint4*>(wh + k0)) : zero;
#pragma unroll
      for (int i = 0; i < NT; ++i)
        xr[u][i] = in && 8 * i + g < p.rows ? __ldg(reinterpret_cast<const uint4*>(x + (size_t)(8 * i + g) * p.x_pitch + k0 + 8 * t)) : zero;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        mma_bf16(acc[i], a[u].x, b[u].x, a[u].y, b[u].y, xr[u][i].x, xr[u][i].y);
        mma_bf16(acc[i], a[u].z, b[u].z, a[u].w, b[u].w, xr[u][i].z, xr[u][i].w);
      }
  }
  // accumulator: rows g and g + 8 of the tile, columns (rows of x) 2 t and 2 t + 1 of each group
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    part[warp][g][8 * i + 2 * t] = acc[i][0];
    part[warp][g][8 * i + 2 * t + 1] = acc[i][1];
    part[warp][g + 8][8 * i + 2 * t] = acc[i][2];
    part[warp][g + 8][8 * i + 2 * t + 1] = acc[i][3];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 16 * p.rows; e += WARPS * 32) {
    const int r = e >> 4, n = e & 15;
    if (n0 + n >= N) continue;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) s += part[w][n][r];
    reinterpret_cast<__nv_bfloat16*>(p.y[m])[(size_t)r * p.y_pitch[m] + n0 + n] = __float2bfloat16_rn(s);
  }
}

}  // namespace

int linear(const tops_skinny_linear_params& p, cudaStream_t st) {
  if (p.rows < 1 || p.rows > 64 || p.count < 1 || p.count > TOPS_SKINNY_MAX || p.K < 32 || p.K % 32 != 0 || p.x_pitch < p.K ||
      p.x_pitch % 8 != 0)
    return TOPS_E_BAD_SHAPE;
  if (reinterpret_cast<uintptr_t>(p.x) & 15) return TOPS_E_ALIGN;
  int tiles = 0;
  for (int m = 0; m < p.count; ++m) {
    if (!p.W[m] || !p.y[m]) return TOPS_E_NULL;
    if (p.N[m] < 1 || p.y_pitch[m] < p.N[m]) return TOPS_E_BAD_SHAPE;
    if (reinterpret_cast<uintptr_t>(p.W[m]) & 15) return TOPS_E_ALIGN;
    tiles += cdiv(p.N[m], 16);
  }
  KernelScope ks("skinny_linear", st);
  if (p.rows <= 8) k_skinny_linear<1><<<tiles, WARPS * 32, 0, st>>>(p);
  else if (p.rows <= 16) k_skinny_linear<2><<<tiles, WARPS * 32, 0, st>>>(p);
  else if (p.rows <= 32) k_skinny_linear<4><<<tiles, WARPS * 32, 0, st>>>(p);
  else k_skinny_linear<8><<<tiles, WARPS * 32, 0, st>>>(p);
  return post_launch();
}

}  // namespace skinny
}  // namespace tops
