// The state-space recurrence of state_space.cu over LONG segments of bfloat16 rows, 64 rows at a time, as matrix products.
//
// For the rows of a chunk, with a_t = -exp(A_log) dt_t, c_t = a_0 + ... + a_t (within the chunk) and S the state before it:
//   y_t = e^(c_t) C_t . S  +  sum over s <= t of e^(c_t - c_s) dt_s (C_t . B_s) x_s  +  D x_t
//   S'  = e^(c_last) S  +  sum over s of B_s (e^(c_last - c_s) dt_s x_s)^T
// which is what the row-by-row walk computes, in other groups of sums.  The walk is a chain of dependent steps (422 us for
// 1,500 rows of 64 heads of 64 x 128 on one prompt, a quarter of a microsecond a row, with most of the SM waiting); here
// the chain is one step per 64 rows, and the same prompt takes 110 us.  Against 64 bits the results are three times as close as
// the walk's (2.9e-7 of the largest value, the walk 8.8e-7, over segments of 33 to 700 rows).
//
// The products run on the tensor cores (mma.sync m16n8k16, 32-bit sums) without giving up 32-bit values: x, B and C are
// bfloat16 already and enter as they are; a factor that is 32-bit (the scores with their decays, the state, the weighted x)
// is cut into three bfloat16 parts whose sum is the value to 2^-25 of it, one product each.  The other factor of every such
// product is exact, so a product's error is that of its 32-bit sum.  The tensor cores cut a sum off where they do not
// round it: the first parts' products and the others' are summed apart, and every sum begins at zero and is added to what
// was there with a rounding of its own, so that few of these cuts fall on a large value.
//
// grid (P / 32, heads, segments), eight warps and one that works out the next chunk's step sizes and decays (a chain of logarithms,
// exponentials and shuffles in which the eight would wait: 128 us instead of 110, and 115 instead of 85 for 32 heads of 64 x 64): a block walks the chunks of one segment for 32 columns of one head's state,
// which stays in registers between chunks (the accumulators of its own update).  155 KB of shared memory at N = 128: one block
// an SM; the next chunk's rows arrive by cp.async while this one is worked on.
#include "common.cuh"
#include "mma_sync.cuh"

namespace cbis {
namespace ssm {

constexpr int Q = 64, PB = 32, WORKERS = 256, THREADS = WORKERS + 32;
constexpr int MP = Q + 8, XP = PB + 8;           // elements per shared row: 16 bytes more than the row, no bank met twice

template <int N> struct Shape {
  static constexpr int NP = N + 8;
  // in bfloat16 elements: two buffers of C, B, x; three parts of the scores, of the state, of the weighted x
  static constexpr int C0 = 0, B0 = C0 + 2 * Q * NP, X0 = B0 + 2 * Q * NP, M0 = X0 + 2 * Q * XP, S0 = M0 + 3 * Q * MP,
                       W0 = S0 + 3 * N * XP, END = W0 + 3 * Q * XP;
  // and two buffers of cum (64-bit), dt, e^cum, the rows' weights in the state, the state's decay over a chunk
  static constexpr int BYTES = END * 2 + 2 * (Q * 8 + 3 * Q * 4) + 2 * 4;
};

__device__ __forceinline__ unsigned s32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy16(void* smem, const void* gmem, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s32(smem)), "l"(gmem), "r"(valid ? 16 : 0) : "memory");
}
// All nine warps, from two places of the code: a barrier with its number of threads, since __syncthreads() has to be the same
// call for a whole block.
__device__ __forceinline__ void block_meets() { asm volatile("barrier.sync 1, %0;" ::"n"(THREADS) : "memory"); }
// Two neighbouring values into three bfloat16 parts each, `part` elements apart.  (What is infinite has rests that are no numbers: it
// stays not finite, and so does every sum it enters, which are those it enters in the walk row by row.)
__device__ __forceinline__ void store_parts(__nv_bfloat16* at, int part, float v0, float v1) {
  unsigned parts[3];
  cut3(v0, v1, parts);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<unsigned*>(at + i * part) = parts[i];
}
// Whether one of the eight bfloat16 of a fragment is infinite or no number: 0 times it is no number.
__device__ __forceinline__ bool not_finite(const uint32_t (&r)[4]) {
  const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
  __nv_bfloat162 s = zero;
#pragma unroll
  for (int i = 0; i < 4; ++i) s = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&r[i]), zero, s);
  return (*reinterpret_cast<const uint32_t*>(&s) & 0x7FFF7FFFu) != 0;
}

template <int N>
__global__ void __launch_bounds__(THREADS, 1)
ssm_chunks_kernel(const __nv_bfloat16* xbc, int xbc_ld, const __nv_bfloat16* proj, int proj_ld, int dt_off,
                  const float* __restrict__ dt_bias, const float* __restrict__ A_log, const float* __restrict__ Dskip, float* state,
                  long long slot_stride, const int* seg_slot, const int* cu_rows, float* y, int y_ld, int H, int P, int G,
                  int from_rows) {
  using T = Shape<N>;
  constexpr int NP = T::NP;
  constexpr int S_TILES = N == 128 ? 4 : 2;      // 8-column pieces of the state a warp holds (16 rows of it)
  extern __shared__ __align__(16) __nv_bfloat16 sm[];
  // [Q] each.  The sums of the a_t are 64-bit: with decays of e^-1 a row their 32-bit sum is 64 times as large as the
  // differences between neighbouring rows that matter, and their error would be ten times that of the row-by-row walk
  double* cum2 = reinterpret_cast<double*>(sm + T::END);
  float *dts2 = reinterpret_cast<float*>(cum2 + 2 * Q), *ecum2 = dts2 + 2 * Q, *weight2 = ecum2 + 2 * Q, *decay2 = weight2 + 2 * Q;
  pdl_trigger();
  const int h = blockIdx.y, s = blockIdx.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row0 = cu_rows[s], n_rows = cu_rows[s + 1] - row0;      // the step's tables: written before its first kernel
  pdl_wait();
  if (n_rows < from_rows) return;       // short segments are walked row by row (ssm_scan_kernel)
  const int g = lane >> 2, t4 = lane & 3;
  const int x_col = h * P + blockIdx.x * PB, b_col = H * P + (h / (H / G)) * N, c_col = b_col + G * N;
  const float neg_a = -expf(A_log[h]), bias = dt_bias[h], dskip = Dskip[h];
  const int n_chunks = (n_rows + Q - 1) / Q;

  auto load = [&](int c) {      // rows past the segment's end are zeros
    const int buf = c & 1;
    for (int i = threadIdx.x; i < Q * (N / 8); i += WORKERS) {
      const int r = i / (N / 8), k = (i % (N / 8)) * 8;
      const bool valid = c * Q + r < n_rows;
      const __nv_bfloat16* src = xbc + (size_t)(row0 + (valid ? c * Q + r : 0)) * xbc_ld;
      copy16(sm + T::C0 + (buf * Q + r) * NP + k, src + c_col + k, valid);
      copy16(sm + T::B0 + (buf * Q + r) * NP + k, src + b_col + k, valid);
    }
    for (int i = threadIdx.x; i < Q * (PB / 8); i += WORKERS) {
      const int r = i / (PB / 8), k = (i % (PB / 8)) * 8;
      const bool valid = c * Q + r < n_rows;
      copy16(sm + T::X0 + (buf * Q + r) * XP + k, xbc + (size_t)(row0 + (valid ? c * Q + r : 0)) * xbc_ld + x_col + k, valid);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the ninth warp's raw step sizes of a chunk, rows 2 lane and 2 lane + 1
  float raw[2];
  auto load_raw = [&](int c) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = c * Q + 2 * lane + i;
      raw[i] = r < n_rows ? to_f32(proj[(size_t)(row0 + r) * proj_ld + dt_off + h]) : 0.f;
    }
  };
  // the ninth warp: a chunk's step sizes, decays and weights, from the raw values that it holds
  auto scalars = [&](int c) {
    double* cum = cum2 + (c & 1) * Q;
    float *dts = dts2 + (c & 1) * Q, *ecum = ecum2 + (c & 1) * Q, *weight = weight2 + (c & 1) * Q;
    float dt[2];
    double a[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float z = raw[i] + bias;
      dt[i] = c * Q + 2 * lane + i < n_rows ? (z > 20.f ? z : log1pf(expf(z))) : 0.f;
      a[i] = (double)neg_a * (double)dt[i];
    }
    double up = a[0] + a[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, up, o);
      if (lane >= o) up += v;
    }
    const double last = __shfl_sync(0xffffffffu, up, 31), before = __shfl_up_sync(0xffffffffu, up, 1);
    const double cs[2] = {(lane ? before : 0.0) + a[0], up};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      cum[2 * lane + i] = cs[i];
      dts[2 * lane + i] = dt[i];
      ecum[2 * lane + i] = expf((float)cs[i]);
      weight[2 * lane + i] = expf((float)(last - cs[i])) * dt[i];
    }
    if (lane == 0) decay2[c & 1] = expm1f((float)last);      // (see ssm_scan_kernel: decays close to 1)
  };
  if (warp == WORKERS / 32) {
    load_raw(0);
    scalars(0);
    if (n_chunks > 1) load_raw(1);
    for (int c = 0; c < n_chunks; ++c) {      // the two meetings of every chunk, see below
      block_meets();
      if (c + 1 < n_chunks) scalars(c + 1);
      if (c + 2 < n_chunks) load_raw(c + 2);
      block_meets();
    }
    return;
  }
  load(0);

  // the state: rows n0 .. n0 + 15 of N, columns p0 .. p0 + 8 S_TILES - 1 of the block's 32, as accumulators (c0, c1: row
  // g, columns 2 t4 and 2 t4 + 1; c2, c3: row g + 8).  In memory a column's N values lie side by side.
  const int n0 = N == 128 ? 16 * warp : 16 * (warp & 3), p0 = N == 128 ? 0 : 16 * (warp >> 2);
  float* sp = state + (long long)seg_slot[s] * slot_stride + ((size_t)h * P + blockIdx.x * PB) * N;
  float S[S_TILES][4];
#pragma unroll
  for (int j = 0; j < S_TILES; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) S[j][e] = sp[(size_t)(p0 + 8 * j + 2 * t4 + (e & 1)) * N + n0 + g + 8 * (e >> 1)];

  // this warp's 16 rows of the chunk and which half of the columns: early rows have little below the diagonal, so that the two
  // warps of a quarter of the SM (w and w + 4) get an early and a late piece
  const int half = warp >> 2, t0 = 16 * (half ? 3 - (warp & 3) : warp & 3);
  for (int c = 0; c < n_chunks; ++c) {
    const __nv_bfloat16 *sC = sm + T::C0 + (c & 1) * Q * NP, *sB = sm + T::B0 + (c & 1) * Q * NP, *sX = sm + T::X0 + (c & 1) * Q * XP;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    block_meets();      // the chunk's rows and scalars are there; everyone is done with the chunk before
    if (c + 1 < n_chunks) load(c + 1);
    const double* cum = cum2 + (c & 1) * Q;
    const float *dts = dts2 + (c & 1) * Q, *ecum = ecum2 + (c & 1) * Q, *weight = weight2 + (c & 1) * Q;
    // the state in three parts, [part][n][p]
#pragma unroll
    for (int j = 0; j < S_TILES; ++j)
#pragma unroll
      for (int hi = 0; hi < 2; ++hi)
        store_parts(sm + T::S0 + (n0 + g + 8 * hi) * XP + p0 + 8 * j + 2 * t4, N * XP, S[j][2 * hi], S[j][2 * hi + 1]);
    // ---- scores C B^T of 16 rows and 32 columns, with their decays and step sizes, into [part][t][s]; 0 above the diagonal
    {
      float acc[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
      const int s0 = 32 * half;
      if (s0 <= t0 + 15) {
#pragma unroll
        for (int k = 0; k < N; k += 16) {
          uint32_t a[4], b0[4], b1[4];
          ldm4<false>(a, sC + (t0 + (lane & 15)) * NP + k + (lane >> 4) * 8);
          ldm4<false>(b0, sB + (s0 + (lane & 7) + ((lane >> 4) << 3)) * NP + k + ((lane >> 3) & 1) * 8);
          ldm4<false>(b1, sB + (s0 + 16 + (lane & 7) + ((lane >> 4) << 3)) * NP + k + ((lane >> 3) & 1) * 8);
          mma_16816(acc[0], a, b0[0], b0[1]);
          mma_16816(acc[1], a, b0[2], b0[3]);
          mma_16816(acc[2], a, b1[0], b1[1]);
          mma_16816(acc[3], a, b1[2], b1[3]);
        }
      }
#pragma unroll
      for (int hi = 0; hi < 2; ++hi) {
        const int t = t0 + g + 8 * hi;
        const double ct = cum[t];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int sc = s0 + 8 * j + 2 * t4;
          const float v0 = sc <= t ? acc[j][2 * hi] * (expf((float)(ct - cum[sc])) * dts[sc]) : 0.f;
          const float v1 = sc + 1 <= t ? acc[j][2 * hi + 1] * (expf((float)(ct - cum[sc + 1])) * dts[sc + 1]) : 0.f;
          store_parts(sm + T::M0 + t * MP + sc, Q * MP, v0, v1);
        }
      }
    }
    // ---- x weighted for the state, into [part][s][p]
    for (int i = threadIdx.x; i < Q * PB / 2; i += WORKERS) {
      const int r = i / (PB / 2), p = (i % (PB / 2)) * 2;
      const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sX + r * XP + p));
      store_parts(sm + T::W0 + r * XP + p, Q * XP, weight[r] * x.x, weight[r] * x.y);
    }
    block_meets();      // the parts of the scores, of the state and of the weighted x are there
    // ---- y of 16 rows and 16 columns: first C S from the state before the chunk, then its decay
    float yv[2][4], first[2][4], rest[2][4];
    auto zero = [&]() {
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) first[j][e] = rest[j][e] = 0.f;
    };
    zero();
    const int py = 16 * half;
#pragma unroll
    for (int k = 0; k < N; k += 16) {
      uint32_t a[4], b[4];
      ldm4<false>(a, sC + (t0 + (lane & 15)) * NP + k + (lane >> 4) * 8);
#pragma unroll
      for (int part = 0; part < 3; ++part) {
        ldm4<true>(b, sm + T::S0 + part * N * XP + (k + (lane & 7) + ((lane >> 3) & 1) * 8) * XP + py + (lane >> 4) * 8);
        mma_16816(part == 0 ? first[0] : rest[0], a, b[0], b[1]);
        mma_16816(part == 0 ? first[1] : rest[1], a, b[2], b[3]);
      }
    }
    {
      const float e0 = ecum[t0 + g], e1 = ecum[t0 + g + 8];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) yv[j][e] = (first[j][e] + rest[j][e]) * (e < 2 ? e0 : e1);
    }
    zero();
    const float decay_m1 = decay2[c & 1];
    // ---- ... then the chunk's own rows, up to the diagonal
    for (int k = 0; k <= t0; k += 16) {
      uint32_t a[4], b[4];
      ldm4<true>(b, sX + (k + (lane & 7) + ((lane >> 3) & 1) * 8) * XP + py + (lane >> 4) * 8);
      if (k == t0 && __any_sync(0xffffffffu, not_finite(b))) {
        // the zeros above the diagonal times an infinite x of a later row would be no number: these rows one by one, to their own
        for (int s1 = 0; s1 < 16; ++s1)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int r1 = g + 8 * (e >> 1);
            if (s1 > r1) continue;
            const __nv_bfloat16* m = sm + T::M0 + (t0 + r1) * MP + t0 + s1;
            const float w = to_f32(m[0]) + (to_f32(m[Q * MP]) + to_f32(m[2 * Q * MP]));
#pragma unroll
            for (int j = 0; j < 2; ++j) first[j][e] = fmaf(w, to_f32(sX[(t0 + s1) * XP + py + 8 * j + 2 * t4 + (e & 1)]), first[j][e]);
          }
        break;
      }
#pragma unroll
      for (int part = 0; part < 3; ++part) {
        ldm4<false>(a, sm + T::M0 + part * Q * MP + (t0 + (lane & 15)) * MP + k + (lane >> 4) * 8);
        mma_16816(part == 0 ? first[0] : rest[0], a, b[0], b[1]);
        mma_16816(part == 0 ? first[1] : rest[1], a, b[2], b[3]);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) yv[j][e] += first[j][e] + rest[j][e];
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const int t = t0 + g + 8 * hi;
      if (c * Q + t < n_rows) {
        float* dst = y + (size_t)(row0 + c * Q + t) * y_ld + x_col + py + 2 * t4;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sX + t * XP + py + 8 * j + 2 * t4));
          *reinterpret_cast<float2*>(dst + 8 * j) = make_float2(fmaf(dskip, x.x, yv[j][2 * hi]), fmaf(dskip, x.y, yv[j][2 * hi + 1]));
        }
      }
    }
    // ---- the state after the chunk
    float s_first[S_TILES][4], s_rest[S_TILES][4];
#pragma unroll
    for (int j = 0; j < S_TILES; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) s_first[j][e] = s_rest[j][e] = 0.f;
#pragma unroll
    for (int k = 0; k < Q; k += 16) {
      uint32_t a[4];      // B^T: rows of the state, from [s][n]
      ldm4<true>(a, sB + (k + (lane & 7) + (lane >> 4) * 8) * NP + n0 + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int part = 0; part < 3; ++part)
#pragma unroll
        for (int j = 0; j < S_TILES; j += 2) {
          uint32_t b[4];
          ldm4<true>(b, sm + T::W0 + part * Q * XP + (k + (lane & 7) + ((lane >> 3) & 1) * 8) * XP + p0 + 8 * j + (lane >> 4) * 8);
          mma_16816(part == 0 ? s_first[j] : s_rest[j], a, b[0], b[1]);
          mma_16816(part == 0 ? s_first[j + 1] : s_rest[j + 1], a, b[2], b[3]);
        }
    }
#pragma unroll
    for (int j = 0; j < S_TILES; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j][e] = fmaf(decay_m1, S[j][e], S[j][e] + (s_first[j][e] + s_rest[j][e]));
  }
#pragma unroll
  for (int j = 0; j < S_TILES; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) sp[(size_t)(p0 + 8 * j + 2 * t4 + (e & 1)) * N + n0 + g + 8 * (e >> 1)] = S[j][e];
}

}  // namespace ssm
}  // namespace cbis

using namespace cbis;

// The arguments of cbis_ssm_scan for bfloat16 rows; segments of `from_rows` rows and more are done, the others left alone.
// Takes N 64 or 128 and P a multiple of 32, x | B | C in rows of whole 16-byte pieces, y in even rows.
CBIS_EXPORT int cbis_ssm_chunks(const void* xbc, int xbc_ld, const void* proj, int proj_ld, int dt_off, const float* dt_bias,
                                const float* A_log, const float* D, float* state, long long slot_stride, const int* seg_slot,
                                const int* cu_rows, float* y, int y_ld, int n_segments, int H, int P, int N, int G, int from_rows,
                                void* stream) {
  if (n_segments <= 0) return CBIS_OK;
  if (H <= 0 || P <= 0 || P % ssm::PB || (N != 64 && N != 128) || G <= 0 || H % G || from_rows < 1) return CBIS_ERR_BAD_SIZE;
  if (xbc_ld % 8 || ((uintptr_t)xbc & 15) || y_ld % 2 || ((uintptr_t)y & 7)) return CBIS_ERR_ALIGNMENT;
  if (n_segments > 65535 || H > 65535) return CBIS_ERR_TOO_LARGE;
  auto kern = N == 128 ? ssm::ssm_chunks_kernel<128> : ssm::ssm_chunks_kernel<64>;
  const size_t smem = N == 128 ? ssm::Shape<128>::BYTES : ssm::Shape<64>::BYTES;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return (int)launch_pdl(kern, dim3(P / ssm::PB, H, n_segments), dim3(ssm::THREADS), smem, (cudaStream_t)stream,
                         (const __nv_bfloat16*)xbc, xbc_ld, (const __nv_bfloat16*)proj, proj_ld, dt_off, dt_bias, A_log, D, state,
                         slot_stride, seg_slot, cu_rows, y, y_ld, H, P, G, from_rows);
}
