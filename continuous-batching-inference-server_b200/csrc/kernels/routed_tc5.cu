// A routed mixture of gated feed-forwards over many rows of bfloat16 on the 5th-generation tensor cores.
//   * routed_plan: the (row, choice) pairs sorted by expert on the device, an expert's pairs in tiles of 128 rows;
//   * routed_gather: the pairs' input rows, in that order, so that a tile of pairs is a run of rows that TMA can copy;
//   * routed_tc5 twice: gate and up products with the gated product in the epilogue, then the down product;
//   * routed_combine: a row's choices summed in their order.
// A pair's result depends on its own row alone: its place in a tile changes no sum's order.
//
// routed_tc5 is built like the dense product (gemm_tcgen05.cu): a block per SM walks over 128 x 256 tiles; one thread
// streams 64-column pieces of 128 rows of pairs and of 256 rows of the expert's matrix into a ring of four stages by TMA,
// one thread issues tcgen05.mma (128 x 256 x 16) into one of two accumulators in tensor memory, sixteen warps read the
// other.  For the gate and up products the 256 rows are 128 gate rows and the 128 up rows beside them, so that an
// accumulator holds both factors of 128 hidden columns.  Experts with few rows are bound by streaming their matrices (the
// ring keeps 192 KB an SM on its way), experts with many by the tensor cores.
// 1,500 rows, 2 of 16 experts of 1,408 at width 2,048: 56 us (gate and up; 58 with the activation chosen beside every value) and
// 33 us (down).  The mma.sync tiles that this
// replaces (128 x 64, rows gathered through the index list) took 229 and 141 us, a tenth of the tensor cores' rate.
//
// Every wait on an mbarrier is bounded: when one runs out the block sets *error, waits for its copies and products in
// flight, frees its tensor memory and returns.
#include "routed_mma.cuh"
#include "tc5_common.cuh"

namespace cbis {
namespace rt {

constexpr int TILE_M = 128, TILE_N = 256, STAGES = 4;
constexpr int A_BYTES = TILE_M * TC_BK * 2, B_BYTES = TILE_N * TC_BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int EPI_WARPS = 16, THREADS = 64 + 32 * EPI_WARPS;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;

// One block.  offsets [E + 1]; sorted [pairs]: the pairs expert by expert; place [pairs]: where a pair stands in `sorted`;
// per tile its expert, its first place in `sorted` and its rows; n_tiles [1].
__global__ void __launch_bounds__(1024)
routed_plan_kernel(const int* ids, int n_pairs, int E, int* offsets, int* sorted, int* place, int* tile_expert, int* tile_start,
                   int* tile_rows, int* n_tiles) {
  extern __shared__ int plan_smem[];
  int* count = plan_smem;          // E
  int* cursor = plan_smem + E;     // E
  pdl_trigger();
  pdl_wait();
  for (int e = threadIdx.x; e < E; e += blockDim.x) count[e] = cursor[e] = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
    const int e = ids[p];
    if (e >= 0 && e < E) atomicAdd(&count[e], 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0, t = 0;
    for (int e = 0; e < E; ++e) {
      offsets[e] = at;
      for (int r = 0; r < count[e]; r += TILE_M) {
        tile_expert[t] = e;
        tile_start[t] = at + r;
        tile_rows[t] = min(TILE_M, count[e] - r);
        ++t;
      }
      at += count[e];
    }
    offsets[E] = at;
    *n_tiles = t;
  }
  __syncthreads();
  for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
    const int e = ids[p];
    if (e >= 0 && e < E) {
      const int at = offsets[e] + atomicAdd(&cursor[e], 1);
      sorted[at] = p;
      place[p] = at;
    }
  }
}

// x[i] = h[sorted[i] / top] for the places that hold a pair; 16 bytes a thread, a block a place.
__global__ void __launch_bounds__(128)
routed_gather_kernel(const __nv_bfloat16* h, int h_ld, const int* offsets, const int* sorted, __nv_bfloat16* x, int W, int E,
                     int top) {
  pdl_trigger();
  pdl_wait();
  const int i = blockIdx.x;
  if (i >= offsets[E]) return;
  const __nv_bfloat16* src = h + (size_t)(sorted[i] / top) * h_ld;
  for (int c = threadIdx.x * 8; c < W; c += 128 * 8)
    *reinterpret_cast<uint4*>(x + (size_t)i * W + c) = *reinterpret_cast<const uint4*>(src + c);
}

// A: [places, K] rows in the plan's order.  B: all experts' matrices one below the other, b_rows rows an expert.
// DUAL: out[place, n] (bfloat16, N columns) = act(s g) * (s u), g and u the products with rows n and N + n of the expert's
// matrix, s the pair's weight where it multiplies the input.  Else: out[place, n] (32-bit) = the product with row n, times
// the pair's weight where it multiplies the output.  Rows of a tile past the expert's own, and columns past N, hold
// products of other experts' rows and are not stored.
template <bool DUAL>
__global__ void __launch_bounds__(THREADS, 1)
routed_tc5_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const int* sorted,
                  const float* weights, const int* tile_expert, const int* tile_start, const int* tile_rows, const int* n_tiles,
                  void* out, int N, int K, int b_rows, int act, int weight_on_input, float limit, float beta, float shift,
                  int* error) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned long long* full = reinterpret_cast<unsigned long long*>(tiles + STAGES * STAGE_BYTES);
  unsigned long long* empty = full + STAGES;
  unsigned long long* acc_full = empty + STAGES;       // [2]
  unsigned long long* acc_empty = acc_full + 2;         // [2]
  unsigned long long* drained = acc_empty + 2;
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(drained + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  constexpr int COLS = DUAL ? TILE_N / 2 : TILE_N;      // columns of the result a tile holds

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_kt = (K + TC_BK - 1) / TC_BK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], EPI_WARPS);
    }
    mbar_init(drained, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * TILE_N)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem_base = *tmem_slot;
  pdl_trigger();   // only now that this block holds its tensor memory (see gemm_tcgen05_kernel)
  pdl_wait();
  const int m_tiles = *n_tiles, num_tiles = m_tiles * ((N + COLS - 1) / COLS);

  if (warp == 0) {
    if (lane == 0) {
      unsigned it = 0;
      for (int tile = blockIdx.x; tile < num_tiles && !*abort_flag; tile += gridDim.x) {
        const int mt = tile % m_tiles, n0 = tile / m_tiles * COLS;
        const int m0 = tile_start[mt], b0 = tile_expert[mt] * b_rows + n0, b1 = b0 + (DUAL ? N : TILE_N / 2);
        for (int kt = 0; kt < n_kt; ++kt, ++it) {
          const unsigned s = it % STAGES, round = it / STAGES;
          if (round > 0 && !mbar_wait(&empty[s], (round - 1) & 1)) {
            *abort_flag = 1;
            atomicExch(error, 51);
            break;
          }
          if (*abort_flag) break;
          unsigned char* sa = tiles + s * STAGE_BYTES;
          mbar_expect_tx(&full[s], STAGE_BYTES);
          tma_load_2d(sa, &map_a, kt * TC_BK, m0, &full[s]);
          tma_load_2d(sa + A_BYTES, &map_b, kt * TC_BK, b0, &full[s]);
          tma_load_2d(sa + A_BYTES + B_BYTES / 2, &map_b, kt * TC_BK, b1, &full[s]);
        }
      }
      if (*abort_flag) {      // the copies requested last may still be on their way: the block must not leave before they land
        for (unsigned j = it > (unsigned)STAGES ? it - STAGES : 0; j < it; ++j)
          if (!mbar_wait(&full[j % STAGES], (j / STAGES) & 1)) atomicExch(error, 54);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr unsigned idesc = umma_idesc(TILE_M, TILE_N);
      unsigned it = 0, local = 0;
      for (int tile = blockIdx.x; tile < num_tiles && !*abort_flag; tile += gridDim.x, ++local) {
        const unsigned buf = local & 1, use = local >> 1;
        if (use > 0 && !mbar_wait(&acc_empty[buf], (use - 1) & 1)) {
          *abort_flag = 1;
          atomicExch(error, 52);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned tmem_d = tmem_base + buf * TILE_N;
        bool ok = true;
        for (int kt = 0; kt < n_kt; ++kt, ++it) {
          const unsigned s = it % STAGES, round = it / STAGES;
          if (!mbar_wait(&full[s], round & 1)) {
            *abort_flag = 1;
            atomicExch(error, 53);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned char* sa = tiles + s * STAGE_BYTES;
          const unsigned long long da = umma_desc(sa), db = umma_desc(sa + A_BYTES);
#pragma unroll
          for (int k = 0; k < TC_BK / 16; ++k)
            umma_bf16(tmem_d, da + (unsigned long long)(k * 2), db + (unsigned long long)(k * 2), idesc, (kt > 0 || k > 0) ? 1u : 0u);
          umma_commit(&empty[s]);
        }
        if (!ok) break;
        umma_commit(&acc_full[buf]);
      }
      if (*abort_flag) {      // tensor memory is freed only after the products issued so far have finished
        umma_commit(drained);
        if (!mbar_wait(drained, 0)) atomicExch(error, 55);
      }
    }
  } else {
    // the four warps of a quarter of tensor memory take the result's pieces of 16 columns in turn; a thread has a row
    const int quarter = warp & 3, turn = (warp - 2) >> 2;
    unsigned local = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++local) {
      const int mt = tile % m_tiles, n0 = tile / m_tiles * COLS;
      const int row = quarter * 32 + lane, rows = tile_rows[mt], at = tile_start[mt] + row;
      const unsigned buf = local & 1, use = local >> 1;
      const float weight = row < rows ? weights[sorted[at]] : 0.f;
      if (!mbar_wait(&acc_full[buf], use & 1)) {
        *abort_flag = 1;
        atomicExch(error, 56);
        break;
      }
      if (*abort_flag) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned acc = tmem_base + ((unsigned)(quarter * 32) << 16) + buf * TILE_N;
      for (int c0 = turn * 16; c0 < COLS; c0 += 16 * (EPI_WARPS / 4)) {
        const int n = n0 + c0;
        if (n >= N) break;
        float v[16];
        tmem_ld16(acc + (unsigned)c0, v);
        if constexpr (DUAL) {
          float u[16];
          tmem_ld16(acc + (unsigned)(TILE_N / 2 + c0), u);
          const float s = weight_on_input ? weight : 1.f;
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] *= s, u[i] *= s;
          gated_products(v, u, act, limit, beta, shift);
          __align__(16) __nv_bfloat162 pk[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) pk[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
          if (row < rows) {      // N is a multiple of 8: eight columns are all there or none is
            uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(out) + (size_t)at * N + n);
            dst[0] = *reinterpret_cast<uint4*>(&pk[0]);
            if (n + 8 < N) dst[1] = *reinterpret_cast<uint4*>(&pk[4]);
          }
        } else {
          const float s = weight_on_input ? 1.f : weight;
          if (row < rows) {
            float4* dst = reinterpret_cast<float4*>(static_cast<float*>(out) + (size_t)at * N + n);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (n + 4 * i < N) dst[i] = make_float4(s * v[4 * i], s * v[4 * i + 1], s * v[4 * i + 2], s * v[4 * i + 3]);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[buf])) : "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * TILE_N) : "memory");
  }
}

// out[row, n] (+)= the row's choices' results, in that order; 32-bit, four columns a thread.  A choice of E or above has no
// result: it adds weight * h[row, n].  y is in the plan's order.
__global__ void __launch_bounds__(256)
routed_combine_kernel(const float* y, const int* place, float* out, int out_ld, int W, int top, int accumulate, const int* ids,
                      const float* weights, int E, const __nv_bfloat16* h, int h_ld) {
  pdl_trigger();
  pdl_wait();
  const size_t r = blockIdx.x;
  for (int n = threadIdx.x * 4; n < W; n += 256 * 4) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < top; ++k) {
      const size_t pair = r * top + k;
      if (ids[pair] < E) {
        const float4 a = *reinterpret_cast<const float4*>(y + (size_t)place[pair] * W + n);
        v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
      } else {
        const float w = weights[pair];
        const __nv_bfloat16* hr = h + r * h_ld + n;
        v.x += w * to_f32(hr[0]); v.y += w * to_f32(hr[1]); v.z += w * to_f32(hr[2]); v.w += w * to_f32(hr[3]);
      }
    }
    float* o = out + r * out_ld + n;
    if (accumulate) {
      v.x += o[0]; v.y += o[1]; v.z += o[2]; v.w += o[3];
    }
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
}

template <bool DUAL>
static int launch(const void* a, int places, int K, const void* b, long long b_total, int b_rows, int N, const int* sorted,
                  const float* weights, const int* tile_expert, const int* tile_start, const int* tile_rows, const int* n_tiles,
                  int max_tiles, void* out, int act, int weight_on_input, float limit, float beta, float shift, int* error,
                  int tc5, cudaStream_t st) {
  if (!tc5)
    return (int)launch_pdl(routed_mma_kernel<DUAL>, dim3(max_tiles, (N + MM_N - 1) / MM_N), dim3(256), 0, st, (const __nv_bfloat16*)a,
                           (const __nv_bfloat16*)b, sorted, weights, tile_expert, tile_start, tile_rows, n_tiles, out, N, K, b_rows,
                           act, weight_on_input, limit, beta, shift);
  CUtensorMap map_a, map_b;
  int s = make_map(&map_a, a, places, K, K, TILE_M);
  if (s == CBIS_OK) s = make_map(&map_b, b, (int)b_total, K, K, TILE_N / 2);
  if (s != CBIS_OK) return s;
  auto kern = routed_tc5_kernel<DUAL>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  if (e != cudaSuccess) return (int)e;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int cols = DUAL ? TILE_N / 2 : TILE_N;
  const long long most = (long long)max_tiles * ((N + cols - 1) / cols);
  return (int)launch_pdl(kern, dim3((unsigned)(most < sms ? most : sms)), dim3(THREADS), (size_t)SMEM_BYTES, st, map_a, map_b,
                         sorted, weights, tile_expert, tile_start, tile_rows, n_tiles, out, N, K, b_rows, act, weight_on_input,
                         limit, beta, shift, error);
}

}  // namespace rt
}  // namespace cbis

using namespace cbis;

// ints of scratch the plan needs: offsets (E + 1), sorted and place (pairs each), three tables of max_tiles, n_tiles (1)
CBIS_EXPORT long long cbis_routed_plan_ints(int pairs, int E) {
  const long long max_tiles = (pairs + rt::TILE_M - 1) / rt::TILE_M + E;
  return (long long)E + 1 + 2ll * pairs + 3 * max_tiles + 1;
}

// The whole routed feed-forward for many rows of bfloat16.  plan: cbis_routed_plan_ints ints; x [pairs, W] and hid
// [pairs, F] bfloat16; y [pairs, W] 32-bit; out [rows, W] 32-bit, overwritten, or added to with `accumulate`.  W and F are
// multiples of 8.  tc5: the products on TMA + tcgen05 (or on mma.sync, which matrices with more rows than a coordinate counts take
// in any case); error: int on the device, set non-zero if a wait inside those kernels ran out.
CBIS_EXPORT int cbis_routed_tiles(const void* h, int h_ld, const void* gate_up, const void* down, const int* ids,
                                  const float* weights, int* plan, void* x, void* hid, float* y, float* out, int out_ld, int rows,
                                  int W, int F, int E, int top, int act, int weight_on_input, int accumulate,
                                  void* stream, float limit, float beta, float shift, int* error, int tc5) {
  if (rows <= 0) return CBIS_OK;
  if (W <= 0 || F <= 0 || E <= 0 || top <= 0) return CBIS_ERR_BAD_SIZE;
  if (W % 8 || F % 8 || h_ld % 8) return CBIS_ERR_ALIGNMENT;
  if (((uintptr_t)h | (uintptr_t)gate_up | (uintptr_t)down | (uintptr_t)x | (uintptr_t)hid | (uintptr_t)y) & 15) return CBIS_ERR_ALIGNMENT;
  if (E > 4096 || (long long)rows * top > 0x3fffffffLL) return CBIS_ERR_TOO_LARGE;
  tc5 = tc5 && 2ll * E * F <= 0x7fffffffLL && (long long)E * W <= 0x7fffffffLL;
  if (tc5 && error == nullptr) return CBIS_ERR_ALIGNMENT;
  cudaStream_t st = (cudaStream_t)stream;
  const int pairs = rows * top;
  const int max_tiles = (pairs + rt::TILE_M - 1) / rt::TILE_M + E;
  int* offsets = plan;
  int* sorted = offsets + E + 1;
  int* place = sorted + pairs;
  int* tile_expert = place + pairs;
  int* tile_start = tile_expert + max_tiles;
  int* tile_rows = tile_start + max_tiles;
  int* n_tiles = tile_rows + max_tiles;
  cudaError_t err = launch_pdl(rt::routed_plan_kernel, dim3(1), dim3(1024), (size_t)2 * E * sizeof(int), st, ids, pairs, E,
                               offsets, sorted, place, tile_expert, tile_start, tile_rows, n_tiles);
  if (err != cudaSuccess) return (int)err;
  err = launch_pdl(rt::routed_gather_kernel, dim3(pairs), dim3(128), 0, st, (const __nv_bfloat16*)h, h_ld, (const int*)offsets,
                   (const int*)sorted, (__nv_bfloat16*)x, W, E, top);
  if (err != cudaSuccess) return (int)err;
  int s = rt::launch<true>(x, pairs, W, gate_up, 2ll * E * F, 2 * F, F, sorted, weights, tile_expert, tile_start, tile_rows,
                           n_tiles, max_tiles, hid, act, weight_on_input, limit, beta, shift, error, tc5, st);
  if (s != CBIS_OK) return s;
  s = rt::launch<false>(hid, pairs, F, down, (long long)E * W, W, W, sorted, weights, tile_expert, tile_start, tile_rows,
                        n_tiles, max_tiles, y, act, weight_on_input, limit, beta, shift, error, tc5, st);
  if (s != CBIS_OK) return s;
  return (int)launch_pdl(rt::routed_combine_kernel, dim3(rows), dim3(256), 0, st, (const float*)y, (const int*)place, out, out_ld, W,
                         top, accumulate, ids, weights, E, (const __nv_bfloat16*)h, h_ld);
}
