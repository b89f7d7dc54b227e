// 32-bit matrix product on the FP32 units (FFMA only: no TF32, no tensor cores), with the
// bias and the activation applied to the 32-bit sum before it is stored.
//   C[M,N] = act(A[M,K] * W + bias)     W is [K,N] (GPT-2 Conv1D layout) or [N,K] (a token table as head)
// The reference calls cublasSgemm and adds the bias in a second kernel (kernels/linear.cu:15-34).
#include "common.cuh"

namespace cbis {

template <int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
linear_f32_kernel(const float* A, const float* __restrict__ W, const float* __restrict__ bias,
                  float* __restrict__ C, int M, int N, int K, int w_is_nk, int act, int lda, int ldc) {
  constexpr int THREADS = (BM / TM) * (BN / TN);
  __shared__ float As[BK][BM + 4];
  __shared__ float Bs[BK][BN + 4];
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // A tile: BM x BK, consecutive threads along k (rows of A are contiguous in k)
    for (int i = tid; i < BM * BK; i += THREADS) {
      const int mm = i / BK, kk = i % BK;
      const int m = m0 + mm, k = k0 + kk;
      As[kk][mm] = (m < M && k < K) ? A[(size_t)m * lda + k] : 0.f;
    }
    if (w_is_nk) {
      for (int i = tid; i < BN * BK; i += THREADS) {
        const int nn = i / BK, kk = i % BK;
        const int n = n0 + nn, k = k0 + kk;
        Bs[kk][nn] = (n < N && k < K) ? W[(size_t)n * K + k] : 0.f;
      }
    } else {
      for (int i = tid; i < BN * BK; i += THREADS) {
        const int kk = i / BN, nn = i % BN;
        const int n = n0 + nn, k = k0 + kk;
        Bs[kk][nn] = (n < N && k < K) ? W[(size_t)k * N + n] : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      C[(size_t)m * ldc + n] = activate(v, act);
    }
  }
}

// More than 16 rows with W stored [N, K] (both operands contiguous along k, 16-byte aligned): tiles of BM x BN
// outputs, k in pieces of 32 that arrive by 16-byte cp.async in a ring of buffers (the next pieces are on their way while
// this one is multiplied), operands kept [row][k] in shared memory so that the copy is straight and a thread reads
// four k of a row at once.  A thread owns TM x TN outputs, TY rows and TX columns apart, and walks k from left to right with
// one fused multiply-add per element: the order of the kernels above and below, hence the same bits.  The tile
// shrinks (64x64, 32x64, 32x32) until the grid fills the SMs: a 512 x 256 x 1024 product had 8 blocks of the
// 128 x 128 kernel above and took 190 us.
__device__ __forceinline__ void cp_async16_f32(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int bytes = valid ? 16 : 0;   // 0 bytes read: the 16 bytes in shared memory are filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
// Waits until at most N of the copies' groups are still on their way.
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// Five pieces are in the ring: a piece of a 32 x 32 tile is multiplied in 0.3 us, a trip to L2 takes 0.7, so with two
// buffers a block waited most of its time (the two products of 512 rows with 256 columns, K 256 and 1,024: 55 us on average; 29 with the ring, 14 with the blocks spread evenly as well).
// Four for the larger tiles, so that three blocks (of 64 x 64) or four fit on an SM: with five, 2048 x 6144 x 2048 took 1,426 us (with
// two buffers 1,410), 512 x 2048 x 2048 205; with four 1,352 and 151.
template <int TILE> constexpr int nk_stages = TILE > 32 * 32 ? 4 : 5;
// A thread owns TM x TN outputs: with more a load from shared memory serves more multiply-adds, with fewer a block has the
// warps to hide a load's trip.  32 x 64: 4 x 4 (512 x 768 x 256: 14.8 us, 2 x 4: 15.9); 32 x 32, a grid that gives an SM one block:
// 2 x 2 (512 x 256 x 1024: 20 us, 2 x 4: 28, 4 x 4: 39).
template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
linear_f32_nk_kernel(const float* A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
                     int M, int N, int K, int act, int lda, int ldc) {
  constexpr int NK_STAGES = nk_stages<BM * BN>, BK = 32, PITCH = BK + 4, TX = BN / TN, TY = BM / TM, THREADS = TX * TY;
  extern __shared__ __align__(16) float nk_smem[];
  float (*As)[BM][PITCH] = reinterpret_cast<float (*)[BM][PITCH]>(nk_smem);                              // [NK_STAGES][BM][PITCH]
  float (*Ws)[BN][PITCH] = reinterpret_cast<float (*)[BN][PITCH]>(nk_smem + NK_STAGES * BM * PITCH);     // [NK_STAGES][BN][PITCH]
  pdl_trigger();
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  auto load_w = [&](int k0, int stage) {
    for (int i = tid; i < BN * (BK / 4); i += THREADS) {
      const int r = i / (BK / 4), c = (i % (BK / 4)) * 4;
      const bool valid = n0 + r < N && k0 + c < K;
      cp_async16_f32(&Ws[stage][r][c], valid ? W + (size_t)(n0 + r) * K + k0 + c : W, valid);
    }
  };
  auto load_a = [&](int k0, int stage) {
    for (int i = tid; i < BM * (BK / 4); i += THREADS) {
      const int r = i / (BK / 4), c = (i % (BK / 4)) * 4;
      const bool valid = m0 + r < M && k0 + c < K;
      cp_async16_f32(&As[stage][r][c], valid ? A + (size_t)(m0 + r) * lda + k0 + c : A, valid);
    }
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  const int n_kt = (K + BK - 1) / BK;
  for (int kt = 0; kt < min(n_kt, NK_STAGES - 1); ++kt) load_w(kt * BK, kt);   // the weights do not come from the kernel before
  pdl_wait();
  for (int kt = 0; kt < NK_STAGES - 1; ++kt) {      // one group of copies a piece (the first holds the weights of all of these)
    if (kt < n_kt) load_a(kt * BK, kt);
    cp_async_commit();
  }
  for (int kt = 0; kt < n_kt; ++kt) {
    const int stage = kt % NK_STAGES;
    cp_async_wait<NK_STAGES - 2>();
    __syncthreads();      // the piece is there for everyone, and everyone is done with the piece before it, whose buffer is filled next
    if (kt + NK_STAGES - 1 < n_kt) {
      load_w((kt + NK_STAGES - 1) * BK, (kt + NK_STAGES - 1) % NK_STAGES);
      load_a((kt + NK_STAGES - 1) * BK, (kt + NK_STAGES - 1) % NK_STAGES);
    }
    cp_async_commit();
    const int kc = min(BK, K - kt * BK);   // a multiple of 4; the sum stops at K (0 * 0 could still flip the sign of a zero)
    auto four = [&](int kk) {
      float4 a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(&As[stage][ty + TY * i][kk]);
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(&Ws[stage][tx + TX * j][kk]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          float v = acc[i][j];
          v = fmaf(a[i].x, b[j].x, v);
          v = fmaf(a[i].y, b[j].y, v);
          v = fmaf(a[i].z, b[j].z, v);
          v = fmaf(a[i].w, b[j].w, v);
          acc[i][j] = v;
        }
    };
    if (kc == BK) {
#pragma unroll
      for (int kk = 0; kk < BK; kk += 4) four(kk);
    } else {
      for (int kk = 0; kk < kc; kk += 4) four(kk);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + TY * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + TX * j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      C[(size_t)m * ldc + n] = activate(v, act);
    }
  }
}

// Up to 16 rows (decoding) with W stored [N, K]: the tiled kernel above would run N / 64 blocks that walk K in
// steps of 16 with two barriers each: 62 us for a 16 x 768 x 256 product.  Here a block takes 16, 8 or 4 output columns
// and a thread owns ONE output (lane m of a half-warp: row m; the half-warp: one column).  K comes in pieces of
// 256: the block copies the piece of A (16 rows) and of W (its columns) into shared memory with coalesced 16-byte
// loads, all in flight at once, and every thread then walks its piece from left to right with one fused
// multiply-add per element: the same order as the tiled kernel, hence the same bits, so that a token decoded
// alone and the same token inside a prompt portion still agree exactly.
// With 16-byte aligned rows (STAGES > 0) up to STAGES pieces are on their way at once, the weights' since
// before the wait for the kernel ahead: piece by piece, each a trip to L2 with nothing else to do, the products of a
// 256-wide model's decode step took 6.7 us on average; 5.2 so, 4.8 with the blocks spread evenly (common.cuh).
// A walk is bound by its loads from shared memory (two of 16 bytes for four multiply-adds, all of a block's through one SM), so
// where N is small a block takes 8 or 4 columns instead of 16 and the same loads are spread over two or four times the SMs.  16 rows of 256 columns,
// K = 1,024: 9.4 us with 16 columns a block and a walk without the next loads on their way, 6.9 now; 768 columns, K = 256: 3.4 and 3.1; one
// row 3.2 and 2.6.
constexpr int FR_KC = 256, FR_PITCH = FR_KC + 4;
constexpr int fr_stage_bytes(int cols) { return (16 + cols) * FR_PITCH * (int)sizeof(float); }
// AHEAD: sixteen k at a time, the next sixteen's loads on their way meanwhile, where a block has few warps to hide a load's trip
// behind; not for pieces under 128, which end before that pays.
template <bool AHEAD>
__device__ __forceinline__ float few_rows_walk(const float* a, const float* w, int kc, float acc) {
  int k = 0;
  if (AHEAD && kc >= 128) {
    float4 av[2][4], wv[2][4];
    auto load = [&](float4 (&x)[4], float4 (&y)[4], int k) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = *reinterpret_cast<const float4*>(a + k + 4 * i);
        y[i] = *reinterpret_cast<const float4*>(w + k + 4 * i);
      }
    };
    auto add = [&](const float4 (&x)[4], const float4 (&y)[4]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc = fmaf(x[i].x, y[i].x, acc);
        acc = fmaf(x[i].y, y[i].y, acc);
        acc = fmaf(x[i].z, y[i].z, acc);
        acc = fmaf(x[i].w, y[i].w, acc);
      }
    };
    const int n = kc >> 4;
    load(av[0], wv[0], 0);
    int i = 0;
    for (; i + 1 < n; i += 2) {
      load(av[1], wv[1], 16 * (i + 1));
      add(av[0], wv[0]);
      if (i + 2 < n) load(av[0], wv[0], 16 * (i + 2));
      add(av[1], wv[1]);
    }
    if (i < n) add(av[0], wv[0]);
    k = 16 * n;
  }
#pragma unroll 8
  for (; k + 4 <= kc; k += 4) {
    const float4 av = *reinterpret_cast<const float4*>(a + k), wv = *reinterpret_cast<const float4*>(w + k);
    acc = fmaf(av.x, wv.x, acc);
    acc = fmaf(av.y, wv.y, acc);
    acc = fmaf(av.z, wv.z, acc);
    acc = fmaf(av.w, wv.w, acc);
  }
  for (; k < kc; ++k) acc = fmaf(a[k], w[k], acc);
  return acc;
}
template <int STAGES, int COLS, bool AHEAD>
__global__ void __launch_bounds__(16 * COLS)
linear_f32_few_rows_kernel(const float* A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
                           int M, int N, int K, int act, int lda, int ldc) {
  extern __shared__ __align__(16) float fr_smem[];      // [stages][16 + COLS][FR_PITCH]: A's piece, W's piece
  pdl_trigger();
  const int tid = threadIdx.x;
  const int m = tid & 15, c = tid >> 4, n0 = blockIdx.x * COLS, n = n0 + c;
  float acc = 0.f;
  if constexpr (STAGES > 0) {
    const int n_p = (K + FR_KC - 1) / FR_KC, stages = min(n_p, STAGES);
    auto a_of = [&](int p) { return fr_smem + (size_t)(p % stages) * (16 + COLS) * FR_PITCH; };
    auto load = [&](int p, const float* src, int ld, int n_rows, int rows, float* dst) {      // n_rows of 256: rows past the end are zeros
      for (int i = tid; i < n_rows * (FR_KC / 4); i += 16 * COLS) {
        const int r = i / (FR_KC / 4), k = (i % (FR_KC / 4)) * 4;
        const bool valid = r < rows && p * FR_KC + k < K;
        cp_async16_f32(dst + r * FR_PITCH + k, valid ? src + (size_t)r * ld + p * FR_KC + k : src, valid);
      }
    };
    const float* w0 = W + (size_t)n0 * K;
    for (int p = 0; p < stages; ++p) load(p, w0, K, COLS, N - n0, a_of(p) + 16 * FR_PITCH);
    const float b = bias && n < N ? bias[n] : 0.f;
    pdl_wait();  // A comes from the kernel before
    for (int p = 0; p < STAGES; ++p) {
      if (p < stages) load(p, A, lda, 16, M, a_of(p));
      cp_async_commit();
    }
    for (int p = 0; p < n_p; ++p) {
      cp_async_wait<STAGES - 1>();
      __syncthreads();
      const float* a = a_of(p);
      acc = few_rows_walk<AHEAD>(a + m * FR_PITCH, a + (16 + c) * FR_PITCH, min(FR_KC, K - p * FR_KC), acc);
      if (p + stages < n_p) {
        __syncthreads();
        load(p + stages, w0, K, COLS, N - n0, a_of(p) + 16 * FR_PITCH);
        load(p + stages, A, lda, 16, M, a_of(p));
      }
      cp_async_commit();
    }
    if (m < M && n < N) {
      if (bias) acc += b;
      C[(size_t)m * ldc + n] = activate(acc, act);
    }
    return;
  }
  float (*As)[FR_PITCH] = reinterpret_cast<float (*)[FR_PITCH]>(fr_smem);
  float (*Ws)[FR_PITCH] = reinterpret_cast<float (*)[FR_PITCH]>(fr_smem + 16 * FR_PITCH);
  pdl_wait();  // A comes from the kernel before
  for (int k0 = 0; k0 < K; k0 += FR_KC) {
    const int kc = min(FR_KC, K - k0);
#pragma unroll
    for (int i = tid; i < 16 * FR_KC; i += 256) {
      const int r = i / FR_KC, k = i % FR_KC;
      As[r][k] = (k < kc && r < M) ? A[(size_t)r * lda + k0 + k] : 0.f;
      Ws[r][k] = (k < kc && n0 + r < N) ? __ldg(W + (size_t)(n0 + r) * K + k0 + k) : 0.f;
    }
    __syncthreads();
    // (a piece shorter than 256 ends in zeros of A and W: adding 0 * 0 changes no bit of the sum... except the sign of
    // a zero sum, so the loop stops at the piece's end)
    acc = few_rows_walk<AHEAD>(As[m], Ws[c], kc, acc);
    __syncthreads();
  }
  if (m < M && n < N) {
    if (bias) acc += bias[n];
    C[(size_t)m * ldc + n] = activate(acc, act);
  }
}

}  // namespace cbis

using namespace cbis;

// lda / ldc: row strides of A and C in elements (>= K, >= N).
// variant: 0 the launcher's choice; 1 never the cp.async kernel (the older tiled kernels: all give the same bits).
CBIS_EXPORT int cbis_linear_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                                int w_is_nk, int act, int lda, int ldc, int variant, void* stream) {
  if (M <= 0 || N <= 0) return CBIS_OK;
  if (K <= 0 || lda < K || ldc < N) return CBIS_ERR_BAD_SIZE;
  cudaStream_t st = (cudaStream_t)stream;
  if (variant != 1 && w_is_nk && M > 16 && K % 4 == 0 && lda % 4 == 0 && !(((uintptr_t)A | (uintptr_t)W) & 15)) {
    // (a 128 x 128 tile, 8 x 8 outputs a thread, was measured too: 198 registers, one block per SM, no faster than 64 x 64)
    const long long b64 = (long long)((M + 63) / 64) * ((N + 63) / 64),
                    b32 = (long long)((M + 31) / 32) * ((N + 63) / 64);
#define CBIS_NK(BM_, BN_, TM_, TN_)                                                                                    \
  {                                                                                                                    \
    auto kern = linear_f32_nk_kernel<BM_, BN_, TM_, TN_>;                                                              \
    const dim3 grid((N + BN_ - 1) / BN_, (M + BM_ - 1) / BM_);                                                         \
    size_t smem;                                                                                                       \
    cudaError_t e = spread_evenly(kern, (long long)grid.x * grid.y, nk_stages<BM_ * BN_> * (BM_ + BN_) * 36 * sizeof(float), &smem); \
    if (e != cudaSuccess) return (int)e;                                                                               \
    return (int)launch_pdl(kern, grid, dim3((BM_ / TM_) * (BN_ / TN_)), smem, st, A, W, bias, C, M, N, K, act, lda, ldc); \
  }
    if (b64 >= 2 * 148) CBIS_NK(64, 64, 4, 4)
    if (b32 >= 148) CBIS_NK(32, 64, 4, 4)
    CBIS_NK(32, 32, 2, 2)
#undef CBIS_NK
  }
  if (M > 256) {
    dim3 grid((N + 127) / 128, (M + 127) / 128);
    return (int)launch_pdl(linear_f32_kernel<128, 128, 8, 8, 8>, grid, dim3(256), 0, st, A, W, bias, C, M, N, K, w_is_nk,
                           act, lda, ldc);
  }
  if (M > 16) {
    dim3 grid((N + 63) / 64, (M + 63) / 64);
    return (int)launch_pdl(linear_f32_kernel<64, 64, 16, 4, 4>, grid, dim3(256), 0, st, A, W, bias, C, M, N, K, w_is_nk,
                           act, lda, ldc);
  }
  if (w_is_nk) {   // decoding: one thread per output, 16 outputs (rows) x 2 columns per warp, a warp for every two columns of a block
    const bool aligned = K % 4 == 0 && lda % 4 == 0 && !(((uintptr_t)A | (uintptr_t)W) & 15);
    const int pieces = (K + FR_KC - 1) / FR_KC, per_sm = ((N + 15) / 16 + 147) / 148;
    // as long a ring as lets all of an SM's blocks (up to the six that one stage allows) run side by side: 16 rows, K = 2,048, four
    // stages -> this rule: N = 6,144 61 us -> 46, 50,257 442 -> 307; N = 2,304 with one stage 24, with two 21
    const int ring = per_sm <= 1 ? 4 : (per_sm <= 3 ? 2 : 1), stages = !aligned ? 1 : (pieces < ring ? pieces : ring);
    // 8 or 4 columns a block while that gives an SM no second block, and while the walk is long enough to pay for more blocks: not under
    // K = 128 (16 rows of 592 columns, K = 64: 2.2 -> 2.7 us), and under 256, but for a row or four, only up to half as many blocks
    // (16 rows, K = 128: 592 columns in 148 blocks 2.6 -> 2.8)
    const int most = K < 128 ? 0 : (K < FR_KC && M > 4 ? 74 : 148);
    const int cols = !aligned || N > 8 * most ? 16 : (N > 4 * most ? 8 : 4);
    // Loads ahead in the walk take registers: with them three blocks of 16 columns fit on an SM instead of six, and one alone has
    // warps enough without (16 rows, K = 2,048: N = 1,185 19.0 us without and 19.8 with, 3,072 32.7 and 31.2, 7,200 58.8 and 63.4)
    const bool ahead = ring == 2 && K >= 3 * FR_KC;
    auto kern = !aligned ? linear_f32_few_rows_kernel<0, 16, false> : (cols == 8 ? linear_f32_few_rows_kernel<4, 8, true>
                         : (cols == 4 ? linear_f32_few_rows_kernel<4, 4, true> : (ring == 4 ? linear_f32_few_rows_kernel<4, 16, false>
                         : (ring == 1 ? linear_f32_few_rows_kernel<1, 16, false> : (ahead ? linear_f32_few_rows_kernel<2, 16, true>
                         : linear_f32_few_rows_kernel<2, 16, false>)))));
    size_t smem;
    const int blocks = (N + cols - 1) / cols;
    cudaError_t e = spread_evenly(kern, blocks, (size_t)stages * fr_stage_bytes(cols), &smem);
    if (e != cudaSuccess) return (int)e;
    return (int)launch_pdl(kern, dim3(blocks), dim3(16 * cols), smem, st, A, W, bias, C, M, N, K, act, lda, ldc);
  }
  dim3 grid((N + 63) / 64, (M + 15) / 16);
  return (int)launch_pdl(linear_f32_kernel<16, 64, 16, 1, 4>, grid, dim3(256), 0, st, A, W, bias, C, M, N, K, w_is_nk,
                         act, lda, ldc);
}
