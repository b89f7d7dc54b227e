// Prefill attention over the paged cache in true 32-bit (no tensor cores): the 32-bit path's counterpart of the
// tiled kernels.  The reference gives every (row, head) a warp that walks all keys of the prefix one by one, so a
// prefill re-reads the prefix once per row (kernels/attention.cu:57-98); the general kernel of this package does
// the same, and a 32,767-token prompt in portions of 512 took it 5.5 s at the reference's sizes.  Here a block
// takes 64 consecutive rows of one (segment, head): keys and values go through shared memory once per 64 rows, in
// tiles of 64 keys (32 above head size 64) gathered page by page through the block table by cp.async, the next tile on its
// way while this one is worked on, the tile after that already looked up in the block table.  Everything is 32-bit
// arithmetic; the softmax is the online form with running maximum and sum per row (kernels/attention.cu:74-95).
//
// The kernel is bound by the issue of multiply-adds and of loads from shared memory, so a thread works on a square of
// the tile: 4 rows x 8 keys of the scores (12 loads of 16 bytes for 128 multiply-adds) and 4 rows x HD / 8 dims of P V
// (8 loads for 64 at head size 32); the eight threads of a row combine maximum and sum with three shuffles, and P goes
// through shared memory inside a warp.  With 2 rows x 8 keys a thread and tiles of 32 fetched between two barriers the
// kernel ran at a quarter of the multiply-add rate (512 rows behind 8,192 keys, 8 heads of 32: 215 us a layer where
// the multiply-adds alone take 59); it now takes 156.
//
// A long context with few rows (a 512-token portion behind 30,000 cached tokens, 8 heads) gives too few blocks
// for 148 SMs, each with a thousand key tiles to walk: the keys are then cut into chunks of chunk_keys (absolute
// key indices, so a key's chunk does not depend on how the prompt was cut), a block takes (row tile, head, chunk)
// and leaves its unnormalised sum, maximum and denominator in scratch memory, and a second kernel merges the
// chunks of every row.
#include "attention_merge.cuh"

namespace cbis {

constexpr int F_THREADS = 128;
template <int HD> struct F32Tile {
  static constexpr int R = 4, BM = 16 * R;                   // rows of a thread and of a tile (8 at head size 32: two blocks an SM instead of three, 165 us against 156)
  static constexpr int BN = HD <= 64 ? 64 : 32;              // keys of a tile
  static constexpr int PITCH = HD + 4;                        // floats per row of Q, K, V: 16 bytes of padding spread the rows over the banks
  static constexpr int P_PITCH = BN + 8;                      // of P: the rows of a warp's four row groups 8 banks apart
  static constexpr int FLOATS = (BM + 4 * BN) * PITCH + BM * P_PITCH;      // Q, two buffers of keys and values, P
};

__device__ __forceinline__ void f32_copy16(float* smem, const float* gmem, bool valid) {
  const int bytes = valid ? 16 : 0;   // 0 bytes read: the 16 bytes in shared memory are filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(bytes));
}

// grid: (row tiles of the longest segment x chunks, heads, segments from seg0 on).
template <int HD>
__global__ void __launch_bounds__(F_THREADS)
paged_prefill_f32_kernel(const float* q, int q_ld, const float* kc, const float* vc, const int* block_table, int max_blocks,
                         const int* cu_rows, const int* seg_start, float* out, int out_ld, int seg0, int n_head, int n_kv_head,
                         int ps, float scale, int window, int n_chunks, int chunk_keys, float* partial, int row0) {
  using T = F32Tile<HD>;
  constexpr int BN = T::BN, PITCH = T::PITCH, P_PITCH = T::P_PITCH, R = T::R, F_BM = T::BM;
  constexpr int KU = BN / 8;                     // keys of a tile per thread: key group + 8 u
  constexpr int VW = HD % 32 == 0 ? 4 : 2;       // floats of a value row per load ...
  constexpr int NI = HD / (8 * VW);              // ... and loads: dims (key group) * VW + 8 VW i
  constexpr int COPIES = BN * (HD / 4) / F_THREADS;      // 16-byte copies of a tile's keys (or values) per thread
  static_assert(BN * (HD / 4) % F_THREADS == 0, "every thread copies alike");
  extern __shared__ __align__(16) float smem_f[];
  float* sQ = smem_f;                            // [F_BM][PITCH]
  float* sKV = sQ + F_BM * PITCH;                // [2][keys, values][BN][PITCH]
  float* sP = sKV + 4 * BN * PITCH;              // [F_BM][P_PITCH]
  pdl_trigger();
  // late row tiles have the most keys to walk: they are given out first
  const int seg = seg0 + blockIdx.z, h = blockIdx.y;
  const int chunk = blockIdx.x % n_chunks, tile = gridDim.x / n_chunks - 1 - blockIdx.x / n_chunks;
  const int r_begin = cu_rows[seg], n_rows = cu_rows[seg + 1] - r_begin;      // the step's tables: written before its first kernel
  if (tile * F_BM >= n_rows) {
    pdl_wait();
    return;
  }
  const int hk = h / (n_head / n_kv_head);
  const int pos0 = seg_start[seg] + tile * F_BM;
  const int rows_here = min(F_BM, n_rows - tile * F_BM);
  int kend = pos0 + rows_here;
  int kbegin = first_seen(pos0, window);
  if (n_chunks > 1) {   // this block's share of the keys; a chunk wholly outside the rows' range leaves nothing
    kbegin = max(kbegin, chunk * chunk_keys);
    kend = min(kend, (chunk + 1) * chunk_keys);
    if (kbegin >= kend) {
      pdl_wait();
      return;
    }
  }
  const int* bt = block_table + (size_t)seg * max_blocks;
  const int tid = threadIdx.x, lane = tid & 31, kg = lane & 7;
  const int rg = (tid >> 5) * 4 + (lane >> 3);   // this thread's rows: rg + 16 i; a warp's rows are its own throughout
  const int ps_shift = (ps & (ps - 1)) == 0 ? 31 - __clz(ps) : -1;
  const int kt_first = kbegin / BN, kt_last = (kend - 1) / BN;
  auto page_at = [&](int j) { return ps_shift >= 0 ? j >> ps_shift : j / ps; };

  // pages of this thread's rows of a tile, a tile before they are needed (keys before the window may lie in pages already
  // given back: they are not looked up)
  int page[COPIES];
  auto look_up = [&](int kt) {
#pragma unroll
    for (int n = 0; n < COPIES; ++n) {
      const int j = kt * BN + (tid + n * F_THREADS) / (HD / 4);
      page[n] = (j >= kbegin && j < kend) ? bt[page_at(j)] : 0;
    }
  };
  auto copy_tile = [&](int kt) {
    float* k_to = sKV + ((kt - kt_first) & 1) * 2 * BN * PITCH;
#pragma unroll
    for (int n = 0; n < COPIES; ++n) {
      const int i = tid + n * F_THREADS, rr = i / (HD / 4), c = (i % (HD / 4)) * 4, j = kt * BN + rr;
      const bool valid = j >= kbegin && j < kend;
      const size_t src = valid ? (((size_t)page[n] * n_kv_head + hk) * ps + (j - page_at(j) * ps)) * HD + c : 0;
      f32_copy16(k_to + rr * PITCH + c, kc + src, valid);
      f32_copy16(k_to + (BN + rr) * PITCH + c, vc + src, valid);
    }
  };
  look_up(kt_first);
  pdl_wait();
  for (int i = tid; i < F_BM * (HD / 4); i += F_THREADS) {
    const int rr = i / (HD / 4), c = (i % (HD / 4)) * 4;
    const bool valid = rr < rows_here;
    f32_copy16(sQ + rr * PITCH + c, valid ? q + (size_t)(r_begin + tile * F_BM + rr) * q_ld + h * HD + c : q, valid);
  }
  copy_tile(kt_first);
  asm volatile("cp.async.commit_group;\n" ::);
  look_up(kt_first + 1);

  float o[R][NI][VW], m[R], l[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int d = 0; d < NI; ++d)
#pragma unroll
      for (int e = 0; e < VW; ++e) o[i][d][e] = 0.f;
  }
  for (int kt = kt_first; kt <= kt_last; ++kt) {
    const int j0 = kt * BN;
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();      // this tile is there, and everyone is done with the one before it, whose buffer is filled next
    if (kt < kt_last) {
      copy_tile(kt + 1);
      asm volatile("cp.async.commit_group;\n" ::);
      look_up(kt + 2);
    }
    const float* sK = sKV + ((kt - kt_first) & 1) * 2 * BN * PITCH;
    const float* sV = sK + BN * PITCH;
    float s[R][KU];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int u = 0; u < KU; ++u) s[i][u] = 0.f;
#pragma unroll 2
    for (int c = 0; c < HD; c += 4) {
      float4 qa[R];
#pragma unroll
      for (int i = 0; i < R; ++i) qa[i] = *reinterpret_cast<const float4*>(sQ + (rg + 16 * i) * PITCH + c);
#pragma unroll
      for (int u = 0; u < KU; ++u) {
        const float4 kv = *reinterpret_cast<const float4*>(sK + (kg + 8 * u) * PITCH + c);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          s[i][u] = fmaf(qa[i].x, kv.x, s[i][u]);
          s[i][u] = fmaf(qa[i].y, kv.y, s[i][u]);
          s[i][u] = fmaf(qa[i].z, kv.z, s[i][u]);
          s[i][u] = fmaf(qa[i].w, kv.w, s[i][u]);
        }
      }
    }
    const bool edge = j0 < kbegin || j0 + BN > kend || j0 + BN - 1 > pos0 || (window != 0 && j0 < first_seen(pos0 + F_BM - 1, window));
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = rg + 16 * i, p = pos0 + r, lo = edge ? max(kbegin, first_seen(p, window)) : 0, hi = edge ? min(kend, p + 1) : j0 + BN;
      float mx = -INFINITY;
#pragma unroll
      for (int u = 0; u < KU; ++u) {
        const int j = j0 + kg + 8 * u;
        s[i][u] = (j >= lo && j < hi) ? s[i][u] * scale : -INFINITY;
        mx = fmaxf(mx, s[i][u]);
      }
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
      const float m_new = fmaxf(m[i], mx);
      const float base = m_new == -INFINITY ? 0.f : m_new;   // a row with no key in range yet
      const float corr = expf(m[i] - base);
      float psum = 0.f;
#pragma unroll
      for (int u = 0; u < KU; ++u) {
        const float e = expf(s[i][u] - base);
        psum += e;
        sP[r * P_PITCH + kg + 8 * u] = e;
      }
      psum += __shfl_xor_sync(0xffffffffu, psum, 1);
      psum += __shfl_xor_sync(0xffffffffu, psum, 2);
      psum += __shfl_xor_sync(0xffffffffu, psum, 4);
      l[i] = l[i] * corr + psum;
      m[i] = m_new;
#pragma unroll
      for (int d = 0; d < NI; ++d)
#pragma unroll
        for (int e = 0; e < VW; ++e) o[i][d][e] *= corr;
    }
    __syncwarp();   // the eight threads of a row are neighbours in one warp: P of the warp's rows is complete
#pragma unroll 2
    for (int j = 0; j < BN; j += 4) {
      float pv[R][4];
#pragma unroll
      for (int i = 0; i < R; ++i) *reinterpret_cast<float4*>(pv[i]) = *reinterpret_cast<const float4*>(sP + (rg + 16 * i) * P_PITCH + j);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        float vv[NI][VW];
#pragma unroll
        for (int d = 0; d < NI; ++d) {
          const float* at = sV + (j + jj) * PITCH + kg * VW + 8 * VW * d;
          if constexpr (VW == 4) *reinterpret_cast<float4*>(vv[d]) = *reinterpret_cast<const float4*>(at);
          else *reinterpret_cast<float2*>(vv[d]) = *reinterpret_cast<const float2*>(at);
        }
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int d = 0; d < NI; ++d)
#pragma unroll
            for (int e = 0; e < VW; ++e) o[i][d][e] = fmaf(pv[i][jj], vv[d][e], o[i][d][e]);
      }
    }
    __syncwarp();   // P is read before the next tile's is written
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int r = rg + 16 * i;
    if (r >= rows_here) continue;
    const size_t row = (size_t)(r_begin + tile * F_BM + r);
    float* dst;
    float f = 1.f;
    if (n_chunks > 1) {
      dst = partial + (((row - row0) * n_head + h) * n_chunks + chunk) * (HD + 4);
      if (kg == 0) *reinterpret_cast<float2*>(dst + HD) = make_float2(m[i], l[i]);
    } else {
      dst = out + row * out_ld + h * HD;
      f = 1.f / l[i];
    }
#pragma unroll
    for (int d = 0; d < NI; ++d) {
      float* at = dst + kg * VW + 8 * VW * d;
      if constexpr (VW == 4) *reinterpret_cast<float4*>(at) = make_float4(o[i][d][0] * f, o[i][d][1] * f, o[i][d][2] * f, o[i][d][3] * f);
      else *reinterpret_cast<float2*>(at) = make_float2(o[i][d][0] * f, o[i][d][1] * f);
    }
  }
}

}  // namespace cbis

using namespace cbis;

// Attention of the segments seg0 .. seg0+n_seg-1 of a step (each a run of rows, cu_rows) over their pages, in
// 32-bit.  Takes head sizes 16, 32, ... 128 (any page size); refuses anything else.  With chunk_keys > 0 (a
// multiple of 32) the keys are cut into n_chunks chunks of that many: partial then holds
// n_rows * n_head * n_chunks * (hd + 4) floats for the rows row0 .. row0+n_rows-1 (those of the segments), positions
// the position of every row of the step, and a second kernel merges the chunks of these rows.
CBIS_EXPORT int cbis_paged_prefill_f32(const float* q, int q_ld, const float* kc, const float* vc, const int* block_table,
                                       int max_blocks, const int* cu_rows, const int* seg_start, float* out, int out_ld,
                                       int seg0, int n_seg, int max_seg_rows, int n_head, int n_kv_head, int hd, int ps,
                                       float scale, int window, int n_chunks, int chunk_keys, float* partial,
                                       const int* positions, int row0, int n_rows, void* stream) {
  if (n_seg <= 0 || max_seg_rows <= 0) return CBIS_OK;
  if (n_chunks < 1 || (n_chunks > 1 && (chunk_keys <= 0 || chunk_keys % 32 || !partial || !positions || n_rows <= 0 ||
                                        ((uintptr_t)partial & 15))))
    return CBIS_ERR_BAD_SIZE;
  if (hd < 16 || hd > 128 || hd % 16 || ps <= 0 || n_head <= 0 || n_kv_head <= 0 || n_head % n_kv_head) return CBIS_ERR_BAD_SIZE;
  if (q_ld % 4 || out_ld % 4 || ((uintptr_t)q & 15) || ((uintptr_t)kc & 15) || ((uintptr_t)vc & 15) || ((uintptr_t)out & 15))
    return CBIS_ERR_ALIGNMENT;
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaErrorInvalidValue;
#define CBIS_PF32(HD_)                                                                                               \
  if (hd == HD_) {                                                                                                   \
    auto kern = paged_prefill_f32_kernel<HD_>;                                                                       \
    const dim3 grid(((max_seg_rows + F32Tile<HD_>::BM - 1) / F32Tile<HD_>::BM) * n_chunks, n_head, n_seg);           \
    const size_t smem = (size_t)F32Tile<HD_>::FLOATS * sizeof(float);                                                \
    if (smem > 48 * 1024) {                                                                                          \
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                        \
      if (e != cudaSuccess) return (int)e;                                                                           \
    }                                                                                                                \
    e = launch_pdl(kern, grid, dim3(F_THREADS), smem, st, q, q_ld, kc, vc, block_table, max_blocks, cu_rows, seg_start, out, \
                   out_ld, seg0, n_head, n_kv_head, ps, scale, window, n_chunks, chunk_keys, partial, row0);         \
  }
  CBIS_PF32(16) CBIS_PF32(32) CBIS_PF32(48) CBIS_PF32(64) CBIS_PF32(80) CBIS_PF32(96) CBIS_PF32(112) CBIS_PF32(128)
#undef CBIS_PF32
  if (e == cudaSuccess && n_chunks > 1)
    e = launch_pdl(prefill_merge_kernel<float, false>, dim3(n_rows), dim3(128), 0, st, (const float*)partial, positions, (const int*)nullptr, out, out_ld, row0,
                   n_head, hd, window, n_chunks, chunk_keys, (const float*)nullptr, 0);
  return (int)e;
}
