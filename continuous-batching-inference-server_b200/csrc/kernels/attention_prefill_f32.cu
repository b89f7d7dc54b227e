// Prefill attention over the paged cache of 32-bit values: the 32-bit path's counterpart of the tiled kernels; head sizes above
// 64 by 32-bit multiply-adds (the first kernel), up to 64 as products of bfloat16 parts on the tensor cores (the second).  The
// reference gives every (row, head) a warp that walks all keys of the prefix one by one, so a
// prefill re-reads the prefix once per row (kernels/attention.cu:57-98); the general kernel of this package does
// the same, and a 32,767-token prompt in portions of 512 took it 5.5 s at the reference's sizes.  Here a block
// takes 64 consecutive rows of one (segment, head): keys and values go through shared memory once per 64 rows, in
// tiles of 32 keys (the second kernel: 64) gathered page by page through the block table by cp.async, the next tile on its
// way while this one is worked on, the tile after that already looked up in the block table.  Maxima, weights and sums are
// 32-bit; the softmax is the online form with running maximum and sum per row (kernels/attention.cu:74-95).
//
// The first kernel is bound by the issue of multiply-adds and of loads from shared memory, so a thread works on a square of
// the tile: 4 rows x 4 keys of the scores and 4 rows x HD / 8 dims of P V; the eight threads of a row combine maximum and
// sum with three shuffles, and P goes through shared memory inside a warp.
//
// A long context with few rows (a 512-token portion behind 30,000 cached tokens, 8 heads) gives too few blocks
// for 148 SMs, each with a thousand key tiles to walk: the keys are then cut into chunks of chunk_keys (absolute
// key indices, so a key's chunk does not depend on how the prompt was cut), a block takes (row tile, head, chunk)
// and leaves its unnormalised sum, maximum and denominator in scratch memory, and a second kernel merges the
// chunks of every row.
#include "attention_merge.cuh"
#include "mma_sync.cuh"
#include "packed.cuh"

namespace cbis {

constexpr int F_THREADS = 128;
template <int HD> struct F32Tile {
  static constexpr int R = 4, BM = 16 * R;                   // rows of a thread and of a tile
  static constexpr int BN = 32;                              // keys of a tile
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

// ---- head sizes up to 64: the same tiles as products on the tensor cores, without giving up 32-bit values --------------
//
// q, k, v and P are cut into three bfloat16 parts each whose sum is the value to 2^-25 of it, and a product of two values is the
// six products of parts whose sizes are within 2^-16 of the largest (mma.sync m16n8k16, 32-bit sums); the three left out are
// below 2^-24 of it together.  The first parts' products and the other five are summed apart, every tile's sums begin at
// zero and are added to what was there with a rounding of their own, as in state_space_chunks.cu.
//
// A block takes 64 rows of one (segment, head), four warps of 16 rows; tiles of 64 keys come page by page by cp.async in
// 32 bits, are cut once per block into shared memory while the next tile is on its way, and P is cut in registers, where the
// scores' accumulators already lie as the next product's operand.  Bound by the tensor cores' legacy path (192 products a
// warp and tile at head size 32) beside the exponentials and the cutting.
// 512 rows behind 8,192 keys, 8 heads of 32, with the merge of the chunks: 125 us, where the first kernel took 173 and its
// multiply-adds alone take 59; behind 30,000 keys 453 and 643; one tile of 13 rows 5.1 and 5.4.  Head size 16 behind 8,192 keys 78 and
// 113, 48 197 and 262, 64 258 and 335.  Above 64 a block's copies and parts leave an SM room for one, and registers spill: head size
// 80 behind 8,192 keys 471, the first kernel 445, 96 582 and 502, 128 1,010 and 658.
// Three blocks an SM at head size 32: four, of 128 registers a thread, gain 3 % behind 8,192 keys and lose a third where there are few tiles.
// Against 64 bits (2-norm, 64 to 30,000 keys) it is 0.7e-7 to 5.7e-7 off, where sums of 32-bit products one by one are 1.0e-7 to 200e-7
// off; the tests hold it to 1.2 times their error + 3e-8.  Only with scores of twenty and more over few keys is it further off than
// they are (64 keys: 2.2e-7, they 1.3e-7 to 2.1e-7): the tensor cores cut the addends of a sum off where a multiply-add rounds.
//
// A value that is not finite has parts that are no numbers: a tile with one, or with one of 10^18 and more (a row tile, for q),
// is worked out value by value from the 32-bit copies instead, and the next tile is fetched only then.
// Values are cut at 2^60 times their size, and a tile's sums go back to theirs: as they are, values below 2^-109 or so would lose
// their third parts (1e-35: 3e-6 off instead of 2e-7), scaled no part of any 32-bit value is too small for bfloat16, and the sum of
// 64 weights of at most 1 times less than 10^18 stays below the largest number.
constexpr int M_BM = 64, M_BN = 64;
constexpr float V_UP = 1152921504606846976.f, V_DOWN = 1.f / V_UP;      // 2^60
template <int HD> struct F32MmaTile {
  static constexpr int PITCH = HD + 8;                                    // bfloat16 elements of a part's row: no bank met twice
  static constexpr int STAGE = 2 * M_BN * HD;                             // floats of a tile's keys and values as they come
  static constexpr int PARTS = 3 * M_BN * PITCH;                          // elements of the parts of keys, or of values
  static constexpr int BYTES = STAGE * 4 + M_BM * HD * 4 + 2 * PARTS * 2 + 16;
};

// Whether v can be cut: finite, and so far from the largest number that no sum of products of parts overflows.
__device__ __forceinline__ bool can_cut(float v) { return fabsf(v) < 1e18f; }
// The six products of parts: a1 b1 into `first`, the others, the smallest first, into `rest`.
__device__ __forceinline__ void mma_parts(float (&first)[4], float (&rest)[4], const unsigned (&a)[3][4], unsigned b1l, unsigned b1h,
                                          unsigned b2l, unsigned b2h, unsigned b3l, unsigned b3h) {
  mma_16816(rest, a[2], b1l, b1h);
  mma_16816(first, a[0], b1l, b1h);
  mma_16816(rest, a[1], b2l, b2h);
  mma_16816(rest, a[0], b3l, b3h);
  mma_16816(rest, a[1], b1l, b1h);
  mma_16816(rest, a[0], b2l, b2h);
}

// The grid and the arguments of paged_prefill_f32_kernel.
template <int HD>
__global__ void __launch_bounds__(128, HD <= 16 ? 4 : (HD <= 32 ? 3 : 2))
paged_prefill_f32_mma_kernel(const float* q, int q_ld, const float* kc, const float* vc, const int* block_table, int max_blocks,
                             const int* cu_rows, const int* seg_start, float* out, int out_ld, int seg0, int n_head,
                             int n_kv_head, int ps, float scale, int window, int n_chunks, int chunk_keys, float* partial, int row0) {
  using T = F32MmaTile<HD>;
  constexpr int PITCH = T::PITCH, KD = HD / 16, ND = HD / 8;
  constexpr int COPIES = M_BN * (HD / 4) / 128;      // 16-byte copies of a tile's keys (or values) per thread
  extern __shared__ __align__(16) float smem_f[];
  float* sQ = smem_f;                                                            // [64][HD]
  float* sStage = sQ + M_BM * HD;                                                // [keys, values][64][HD]
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(sStage + T::STAGE);   // [part][key][PITCH]
  __nv_bfloat16* sV = sK + T::PARTS;
  int* sBad = reinterpret_cast<int*>(sV + T::PARTS);                             // tiles (by parity) with a value that cannot be cut
  pdl_trigger();
  // late row tiles have the most keys to walk: they are given out first
  const int seg = seg0 + blockIdx.z, h = blockIdx.y;
  const int chunk = blockIdx.x % n_chunks, tile = gridDim.x / n_chunks - 1 - blockIdx.x / n_chunks;
  const int r_begin = cu_rows[seg], n_rows = cu_rows[seg + 1] - r_begin;      // the step's tables: written before its first kernel
  if (tile * M_BM >= n_rows) {
    pdl_wait();
    return;
  }
  const int hk = h / (n_head / n_kv_head);
  const int pos0 = seg_start[seg] + tile * M_BM;
  const int rows_here = min(M_BM, n_rows - tile * M_BM);
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
  const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t4 = lane & 3, wr = (tid >> 5) * 16;      // wr: the warp's first row
  const int ps_shift = (ps & (ps - 1)) == 0 ? 31 - __clz(ps) : -1;
  const int kt_first = kbegin / M_BN, kt_last = (kend - 1) / M_BN;
  auto page_at = [&](int j) { return ps_shift >= 0 ? j >> ps_shift : j / ps; };

  // pages of this thread's rows of a tile, a tile before they are needed (keys before the window may lie in pages already
  // given back: they are not looked up)
  int page[COPIES];
  auto look_up = [&](int kt) {
#pragma unroll
    for (int n = 0; n < COPIES; ++n) {
      const int j = kt * M_BN + (tid + n * 128) / (HD / 4);
      page[n] = (j >= kbegin && j < kend) ? bt[page_at(j)] : 0;
    }
  };
  auto copy_tile = [&](int kt) {
#pragma unroll
    for (int n = 0; n < COPIES; ++n) {
      const int i = tid + n * 128, rr = i / (HD / 4), c = (i % (HD / 4)) * 4, j = kt * M_BN + rr;
      const bool valid = j >= kbegin && j < kend;
      const size_t src = valid ? (((size_t)page[n] * n_kv_head + hk) * ps + (j - page_at(j) * ps)) * HD + c : 0;
      f32_copy16(sStage + rr * HD + c, kc + src, valid);
      f32_copy16(sStage + (M_BN + rr) * HD + c, vc + src, valid);
    }
  };
  if (tid < 2) sBad[tid] = 0;
  look_up(kt_first);
  pdl_wait();
  for (int i = tid; i < M_BM * (HD / 4); i += 128) {
    const int rr = i / (HD / 4), c = (i % (HD / 4)) * 4;
    const bool valid = rr < rows_here;
    f32_copy16(sQ + rr * HD + c, valid ? q + (size_t)(r_begin + tile * M_BM + rr) * q_ld + h * HD + c : q, valid);
  }
  asm volatile("cp.async.commit_group;\n" ::);
  copy_tile(kt_first);
  asm volatile("cp.async.commit_group;\n" ::);
  look_up(kt_first + 1);
  // this warp's rows of q, cut, as operands: rows g and g + 8, head dims 16 kd + 2 t4, + 1 and + 8, + 9
  asm volatile("cp.async.wait_group 1;\n" ::);
  __syncthreads();
  unsigned qa[KD][3][4];
  bool q_good = true;
#pragma unroll
  for (int kd = 0; kd < KD; ++kd)
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const float2 v = *reinterpret_cast<const float2*>(sQ + (wr + g + 8 * (f & 1)) * HD + 16 * kd + 8 * (f >> 1) + 2 * t4);
      q_good = q_good && can_cut(v.x) && can_cut(v.y);
      unsigned part[3];
      cut3(v.x, v.y, part);
#pragma unroll
      for (int i = 0; i < 3; ++i) qa[kd][i][f] = part[i];
    }
  q_good = __syncthreads_and(q_good);

  float o[ND][4], m[2], l[2];      // rows g (elements 0, 1) and g + 8 (2, 3); dims 8 n + 2 t4, + 1
#pragma unroll
  for (int hi = 0; hi < 2; ++hi) m[hi] = -INFINITY, l[hi] = 0.f;
#pragma unroll
  for (int n = 0; n < ND; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[n][e] = 0.f;

  for (int kt = kt_first; kt <= kt_last; ++kt) {
    const int j0 = kt * M_BN, par = (kt - kt_first) & 1;
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();      // this tile is there, and everyone is done with the parts of the one before it
    const float *fK = sStage, *fV = fK + M_BN * HD;
    if (tid == 0) sBad[par ^ 1] = 0;      // (last read before the barrier above, set again after the next tile's)
    bool good = true;
#pragma unroll
    for (int n = 0; n < 2 * COPIES; ++n) {
      const int i = tid + n * 128, rr = i / (HD / 4), c = (i % (HD / 4)) * 4;      // keys, then values: rows 64 on
      float4 v = *reinterpret_cast<const float4*>(fK + rr * HD + c);
      good = good && can_cut(v.x) && can_cut(v.y) && can_cut(v.z) && can_cut(v.w);
      if (n >= COPIES) {
        const unsigned long long up = pack2(V_UP, V_UP);
        unpack2(mul2(pack2(v.x, v.y), up), v.x, v.y);
        unpack2(mul2(pack2(v.z, v.w), up), v.z, v.w);
      }
      unsigned lo[3], hi[3];
      cut3(v.x, v.y, lo);
      cut3(v.z, v.w, hi);
      __nv_bfloat16* to = (n < COPIES ? sK + rr * PITCH : sV + (rr - M_BN) * PITCH) + c;
#pragma unroll
      for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(to + p * M_BN * PITCH) = make_uint2(lo[p], hi[p]);
    }
    if (!good) sBad[par] = 1;
    __syncthreads();      // the parts are there, and the copy is free for the next tile
    const bool by_parts = q_good && sBad[par] == 0;      // the whole block alike
    auto fetch_next = [&]() {
      if (kt < kt_last) {
        copy_tile(kt + 1);
        asm volatile("cp.async.commit_group;\n" ::);
        look_up(kt + 2);
      }
    };
    if (by_parts) fetch_next();
    float s[8][4];
    if (by_parts) {
#pragma unroll
      for (int np = 0; np < 4; ++np) {      // 16 keys
        float first[2][4], rest[2][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) first[0][e] = first[1][e] = rest[0][e] = rest[1][e] = 0.f;
#pragma unroll
        for (int kd = 0; kd < KD; ++kd) {
          unsigned b[3][4];
#pragma unroll
          for (int p = 0; p < 3; ++p)
            ldm4<false>(b[p], sK + (p * M_BN + 16 * np + (lane & 7) + ((lane >> 4) << 3)) * PITCH + 16 * kd + ((lane >> 3) & 1) * 8);
          mma_parts(first[0], rest[0], qa[kd], b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
          mma_parts(first[1], rest[1], qa[kd], b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if constexpr (HD < 64) {      // two sums an instruction (at 64 the pairs of registers would spill)
            if (e % 2) continue;
#pragma unroll
            for (int i = 0; i < 2; ++i)
              unpack2(add2(pack2(first[i][e], first[i][e + 1]), pack2(rest[i][e], rest[i][e + 1])), s[2 * np + i][e], s[2 * np + i][e + 1]);
          } else {
            s[2 * np][e] = first[0][e] + rest[0][e];
            s[2 * np + 1][e] = first[1][e] + rest[1][e];
          }
        }
      }
    } else {
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float *qr = sQ + (wr + g + 8 * (e >> 1)) * HD, *kr = fK + (8 * n + 2 * t4 + (e & 1)) * HD;
          float a = 0.f;
#pragma unroll 1
          for (int c = 0; c < HD; ++c) a = fmaf(qr[c], kr[c], a);
          s[n][e] = a;
        }
    }
    const bool edge = j0 < kbegin || j0 + M_BN > kend || j0 + M_BN - 1 > pos0 || (window != 0 && j0 < first_seen(pos0 + M_BM - 1, window));
    float corr[2];
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      if (edge) {      // the keys this row sees: [lo, up) of the tile; a tile that all rows see whole is not compared (131 -> 126 us)
        const int p = pos0 + wr + g + 8 * hi, lo = max(kbegin, first_seen(p, window)) - j0, up = min(kend, p + 1) - j0;
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = 8 * n + 2 * t4 + e;
            s[n][2 * hi + e] = j >= lo && j < up ? s[n][2 * hi + e] * scale : -INFINITY;
          }
      } else {
#pragma unroll
        for (int n = 0; n < 8; ++n)
          unpack2(mul2(pack2(s[n][2 * hi], s[n][2 * hi + 1]), pack2(scale, scale)), s[n][2 * hi], s[n][2 * hi + 1]);
      }
      float mx = -INFINITY;
#pragma unroll
      for (int n = 0; n < 8; ++n) mx = fmaxf(mx, fmaxf(s[n][2 * hi], s[n][2 * hi + 1]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_new = fmaxf(m[hi], mx);
      const float base = m_new == -INFINITY ? 0.f : m_new;   // a row with no key in range yet
      corr[hi] = expf(m[hi] - base);
      float psum = 0.f;
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float& v = s[n][2 * hi + e];
          v = expf(v - base);
          psum += v;
        }
      psum += __shfl_xor_sync(0xffffffffu, psum, 1);
      psum += __shfl_xor_sync(0xffffffffu, psum, 2);
      l[hi] = l[hi] * corr[hi] + psum;
      m[hi] = m_new;
    }
    if (by_parts) {
      float first[ND][4], rest[ND][4];
#pragma unroll
      for (int n = 0; n < ND; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) first[n][e] = rest[n][e] = 0.f;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {      // 16 keys: the scores' accumulators lie as the operand's registers do
        unsigned pa[3][4];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          unsigned part[3];
          cut3(s[2 * kk + (f >> 1)][2 * (f & 1)], s[2 * kk + (f >> 1)][2 * (f & 1) + 1], part);
#pragma unroll
          for (int i = 0; i < 3; ++i) pa[i][f] = part[i];
        }
#pragma unroll
        for (int nd = 0; nd < ND; nd += 2) {
          unsigned b[3][4];
#pragma unroll
          for (int p = 0; p < 3; ++p)
            ldm4<true>(b[p], sV + (p * M_BN + 16 * kk + (lane & 7) + ((lane >> 3) & 1) * 8) * PITCH + 8 * nd + (lane >> 4) * 8);
          mma_parts(first[nd], rest[nd], pa, b[0][0], b[0][1], b[1][0], b[1][1], b[2][0], b[2][1]);
          mma_parts(first[nd + 1], rest[nd + 1], pa, b[0][2], b[0][3], b[1][2], b[1][3], b[2][2], b[2][3]);
        }
      }
      const unsigned long long down = pack2(V_DOWN, V_DOWN), corr2[2] = {pack2(corr[0], corr[0]), pack2(corr[1], corr[1])};
#pragma unroll
      for (int n = 0; n < ND; ++n)
#pragma unroll
        for (int hi = 0; hi < 2; ++hi) {
          const unsigned long long sum = add2(pack2(first[n][2 * hi], first[n][2 * hi + 1]), pack2(rest[n][2 * hi], rest[n][2 * hi + 1]));
          unpack2(fma2(pack2(o[n][2 * hi], o[n][2 * hi + 1]), corr2[hi], mul2(sum, down)), o[n][2 * hi], o[n][2 * hi + 1]);
        }
    } else {
#pragma unroll
      for (int n = 0; n < ND; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] *= corr[e >> 1];
      // a key that a row does not see has weight 0 there, but 0 times a value that is not finite would be no number
      int lo[2], up[2];
#pragma unroll
      for (int hi = 0; hi < 2; ++hi) {
        const int p = pos0 + wr + g + 8 * hi;
        lo[hi] = max(kbegin, first_seen(p, window)) - j0;
        up[hi] = min(kend, p + 1) - j0;
      }
#pragma unroll
      for (int kn = 0; kn < 8; ++kn)
#pragma unroll 1
        for (int src = 0; src < 4; ++src)      // keys 8 kn + 2 src and + 1, whose weights the lane of the same rows with t4 = src holds
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const float p0 = __shfl_sync(0xffffffffu, s[kn][b], (lane & ~3) + src), p1 = __shfl_sync(0xffffffffu, s[kn][2 + b], (lane & ~3) + src);
            const int j = 8 * kn + 2 * src + b;
            const bool in0 = j >= lo[0] && j < up[0], in1 = j >= lo[1] && j < up[1];
            const float* vr = fV + j * HD + 2 * t4;
#pragma unroll
            for (int n = 0; n < ND; ++n) {
              const float2 v = *reinterpret_cast<const float2*>(vr + 8 * n);
              o[n][0] = fmaf(p0, in0 ? v.x : 0.f, o[n][0]);
              o[n][1] = fmaf(p0, in0 ? v.y : 0.f, o[n][1]);
              o[n][2] = fmaf(p1, in1 ? v.x : 0.f, o[n][2]);
              o[n][3] = fmaf(p1, in1 ? v.y : 0.f, o[n][3]);
            }
          }
      __syncthreads();      // everyone has read the copy
      fetch_next();
    }
  }
#pragma unroll
  for (int hi = 0; hi < 2; ++hi) {
    const int r = wr + g + 8 * hi;
    if (r >= rows_here) continue;
    const size_t row = (size_t)(r_begin + tile * M_BM + r);
    float* dst;
    float f = 1.f;
    if (n_chunks > 1) {
      dst = partial + (((row - row0) * n_head + h) * n_chunks + chunk) * (HD + 4);
      if (t4 == 0) *reinterpret_cast<float2*>(dst + HD) = make_float2(m[hi], l[hi]);
    } else {
      dst = out + row * out_ld + h * HD;
      f = 1.f / l[hi];
    }
#pragma unroll
    for (int n = 0; n < ND; ++n) *reinterpret_cast<float2*>(dst + 8 * n + 2 * t4) = make_float2(o[n][2 * hi] * f, o[n][2 * hi + 1] * f);
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
  // Of the second kernel up to two blocks an SM are spread evenly (a grid that is smaller or fills the SMs anyway gains nothing): packed
  // onto the SMs that the kernel ahead leaves idle, 64 rows behind 4,000 keys, 8 heads of 16, took 17.4 us, the first kernel 16.6;
  // 14.9 so; 16 heads of 32 29.9 -> 24.8, 128 rows behind 4,000, 8 heads of 32, 30.8 -> 25.3.
#define CBIS_PF32(HD_, KERNEL_, BM_, BYTES_)                                                                         \
  if (hd == HD_) {                                                                                                   \
    auto kern = KERNEL_<HD_>;                                                                                        \
    const dim3 grid(((max_seg_rows + BM_ - 1) / BM_) * n_chunks, n_head, n_seg);                                     \
    const long long blocks = (long long)grid.x * grid.y * grid.z;                                                    \
    size_t smem = BYTES_;                                                                                            \
    if (HD_ <= 64 && blocks > 32 && blocks <= 2 * 148) e = spread_evenly(kern, blocks, smem, &smem);                 \
    else e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);                    \
    if (e != cudaSuccess) return (int)e;                                                                             \
    e = launch_pdl(kern, grid, dim3(128), smem, st, q, q_ld, kc, vc, block_table, max_blocks, cu_rows, seg_start, out, \
                   out_ld, seg0, n_head, n_kv_head, ps, scale, window, n_chunks, chunk_keys, partial, row0);         \
  }
#define CBIS_PF32_MMA(HD_) CBIS_PF32(HD_, paged_prefill_f32_mma_kernel, M_BM, F32MmaTile<HD_>::BYTES)
#define CBIS_PF32_FMA(HD_) CBIS_PF32(HD_, paged_prefill_f32_kernel, F32Tile<HD_>::BM, (size_t)F32Tile<HD_>::FLOATS * sizeof(float))
  CBIS_PF32_MMA(16) CBIS_PF32_MMA(32) CBIS_PF32_MMA(48) CBIS_PF32_MMA(64)
  CBIS_PF32_FMA(80) CBIS_PF32_FMA(96) CBIS_PF32_FMA(112) CBIS_PF32_FMA(128)
#undef CBIS_PF32_MMA
#undef CBIS_PF32_FMA
#undef CBIS_PF32
  if (e == cudaSuccess && n_chunks > 1)
    e = launch_pdl(prefill_merge_kernel<float, false>, dim3(n_rows), dim3(128), 0, st, (const float*)partial, positions, (const int*)nullptr, out, out_ld, row0,
                   n_head, hd, window, n_chunks, chunk_keys, (const float*)nullptr, 0);
  return (int)e;
}
