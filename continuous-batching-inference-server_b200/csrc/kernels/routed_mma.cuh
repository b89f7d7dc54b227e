// The products of the routed feed-forward over many rows without tcgen05 (CBIS_TCGEN05=0, and matrices of more rows than a
// tensor map's coordinates count): 128 x 64 tiles on mma.sync m16n8k16 with 32-bit sums.
#pragma once
#include "common.cuh"

namespace cbis {
namespace rt {

constexpr int MM_M = 128, MM_N = 64, MM_K = 32, MM_LD = MM_K + 8;      // shared rows padded to 80 bytes: no two of a load's eight rows share a bank

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((unsigned)__cvta_generic_to_shared(smem)));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The operands and the result of routed_tc5_kernel.  grid (max tiles, ceil(N / 64)), 256 threads: the eight warps own the eight
// 32 x 32 pieces of a 128 x 64 tile (of gate and of up columns with DUAL); the next 32 columns of the operands are fetched into
// registers while the tensor cores work on the ones in shared memory.
template <bool DUAL>
__global__ void __launch_bounds__(256)
routed_mma_kernel(const __nv_bfloat16* a, const __nv_bfloat16* __restrict__ b, const int* sorted, const float* weights,
                  const int* tile_expert, const int* tile_start, const int* tile_rows, const int* n_tiles, void* out, int N, int K,
                  int b_rows, int act, int weight_on_input, float limit, float beta, float shift) {
  constexpr int NB = DUAL ? 2 : 1;
  __shared__ __align__(16) __nv_bfloat16 As[MM_M][MM_LD];
  __shared__ __align__(16) __nv_bfloat16 Bs[NB][MM_N][MM_LD];
  pdl_trigger();
  pdl_wait();
  const int tile = blockIdx.x;
  if (tile >= *n_tiles) return;
  const int start = tile_start[tile], rows = tile_rows[tile], n0 = blockIdx.y * MM_N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;      // warps 4 down, 2 across
  const int piece_k = (threadIdx.x & 3) * 8, piece_r = threadIdx.x >> 2;      // rows piece_r and piece_r + 64 of A, piece_r of B
  const __nv_bfloat16* b_src = n0 + piece_r < N ? b + ((size_t)tile_expert[tile] * b_rows + n0 + piece_r) * K : nullptr;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 ra[2], rb[NB];
  auto fetch = [&](int k0) {
    const int k = k0 + piece_k;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = piece_r + i * 64;
      ra[i] = r < rows && k < K ? *reinterpret_cast<const uint4*>(a + (size_t)(start + r) * K + k) : zero;
    }
#pragma unroll
    for (int m = 0; m < NB; ++m) rb[m] = b_src && k < K ? *reinterpret_cast<const uint4*>(b_src + (size_t)m * N * K + k) : zero;
  };
  float acc[NB][2][4][4];      // [gate | up][16 rows of the warp's 32][8 columns of its 32][fragment]
#pragma unroll
  for (int m = 0; m < NB; ++m)
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[m][i >> 4][(i >> 2) & 3][i & 3] = 0.f;
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += MM_K) {
#pragma unroll
    for (int i = 0; i < 2; ++i) *reinterpret_cast<uint4*>(&As[piece_r + i * 64][piece_k]) = ra[i];
#pragma unroll
    for (int m = 0; m < NB; ++m) *reinterpret_cast<uint4*>(&Bs[m][piece_r][piece_k]) = rb[m];
    if (k0 + MM_K < K) fetch(k0 + MM_K);
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < MM_K; kk += 16) {
      uint32_t fa[2][4], fb[4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)      // rows (lane % 16), columns kk + 8 * (lane / 16): the four 8 x 8 quarters of A
        ldmatrix_x4(fa[mt], &As[wm + mt * 16 + (lane & 15)][kk + (lane >> 4) * 8]);
#pragma unroll
      for (int m = 0; m < NB; ++m)
#pragma unroll
        for (int jp = 0; jp < 2; ++jp) {      // two blocks of 8 columns a load: (n, k), (n, k + 8), (n + 8, k), (n + 8, k + 8)
          ldmatrix_x4(fb, &Bs[m][wn + jp * 16 + (lane & 7) + ((lane >> 4) << 3)][kk + ((lane >> 3) & 1) * 8]);
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            mma_bf16(acc[m][mt][jp * 2], fa[mt], fb[0], fb[1]);
            mma_bf16(acc[m][mt][jp * 2 + 1], fa[mt], fb[2], fb[3]);
          }
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int r = wm + mt * 16 + (lane >> 2) + half * 8;
      if (r >= rows) continue;
      const float w = weights[sorted[start + r]];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int n = n0 + wn + j * 8 + (lane & 3) * 2 + i;
          if (n >= N) continue;
          const size_t at = (size_t)(start + r) * N + n;
          const float v = acc[0][mt][j][half * 2 + i];
          if constexpr (DUAL) {
            const float s = weight_on_input ? w : 1.f;
            from_f32(static_cast<__nv_bfloat16*>(out)[at], gated_product(s * v, s * acc[1][mt][j][half * 2 + i], act, limit, beta, shift));
          } else {
            static_cast<float*>(out)[at] = weight_on_input ? v : w * v;
          }
        }
    }
}

}  // namespace rt
}  // namespace cbis
