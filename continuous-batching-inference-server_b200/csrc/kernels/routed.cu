// A routed mixture of gated feed-forwards.
//   * route_topk: router logits in 32-bit, a score per expert (sigmoid or softmax), the `top` largest chosen
//     (ties: the lower index), their weights the scores as they are or divided by their sum; a correction per expert may
//     join the scores for the choice alone; one more row of the router may give a number per row whose sigmoid is
//     handed on (the gate of an expert that every row uses);
//   * routed_gate_up / routed_down: the chosen experts of every row, one (row, choice) pair at a time, the experts'
//     matrices streamed by warps (a row's result depends on nothing but the row: no other row of the batch and no
//     position inside it changes a sum's order).  The weight of a choice multiplies the expert's input
//     (`weight_on_input`), which for the two first products is the same as multiplying their 32-bit sums, or its output.
//     The gated product inside an expert takes limit, beta and shift (gated_product in common.cuh).
//   * many rows of bfloat16 go to the tensor cores instead, sorted by expert (routed_tc5.cu).
//   * A chosen index of E or above is an identity expert: its output is the input row itself, times the weight.  It has
//     no matrices; the kernels that sum a row's choices read the row.
#include "common.cuh"

namespace cbis {

constexpr int kScoreSigmoid = 0, kScoreSoftmax = 1;

// grid (rows), blocks of whole warps; shared: 2 (E + 1) floats.  ids [rows, top] int32, weights [rows, top] float.  correction (may
// be null): [E], added to the scores for the choice.  side (may be null): [rows], the sigmoid of router row E's logit.
template <typename TT, int THREADS>
__global__ void __launch_bounds__(THREADS)
route_topk_kernel(const TT* h, int h_ld, const TT* __restrict__ router, int* ids, float* weights, int W, int E, int top,
                  int score, int renormalize, float renorm_eps, float weight_scale, const float* __restrict__ correction,
              float* side) {
  extern __shared__ float z[];
  float* own = z + E + 1;      // with a correction: the scores, while z holds what the choice is made by
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const TT* hr = h + (size_t)r * h_ld;
  constexpr int V = 16 / (int)sizeof(TT);      // elements of a 16-byte load
  const bool vec = W % V == 0 && !(((uintptr_t)hr | (uintptr_t)router) & 15);
  for (int e = warp; e < E + (side ? 1 : 0); e += THREADS == 256 ? 8 : blockDim.x >> 5) {
    const TT* wr = router + (size_t)e * W;
    float acc = 0.f;
    if (vec) {
      float a2 = 0.f;                           // two chains of sums: the loads of a step do not wait for one another
      for (int k = lane * V; k < W; k += 32 * V) {
        TT a[V], b[V];
        *reinterpret_cast<uint4*>(a) = *reinterpret_cast<const uint4*>(hr + k);
        *reinterpret_cast<uint4*>(b) = *reinterpret_cast<const uint4*>(wr + k);
#pragma unroll
        for (int i = 0; i < V; i += 2) {
          acc = fmaf(to_f32(a[i]), to_f32(b[i]), acc);
          a2 = fmaf(to_f32(a[i + 1]), to_f32(b[i + 1]), a2);
        }
      }
      acc += a2;
    } else {
      for (int k = lane; k < W; k += 32) acc = fmaf(to_f32(hr[k]), to_f32(wr[k]), acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) z[e] = acc;
  }
  __syncthreads();
  if (warp != 0) return;
  if (side && lane == 0) side[r] = sigmoid_f32(z[E]);
  float zmax = -INFINITY, denom = 1.f;
  if (score == kScoreSoftmax) {
    for (int e = lane; e < E; e += 32) zmax = fmaxf(zmax, z[e]);
    zmax = warp_max(zmax);
    float d = 0.f;
    for (int e = lane; e < E; e += 32) d += expf(z[e] - zmax);
    denom = warp_sum(d);
  }
  if (correction) {
    for (int e = lane; e < E; e += 32) {
      const float sc = score == kScoreSoftmax ? expf(z[e] - zmax) / denom : sigmoid_f32(z[e]);
      own[e] = sc;
      z[e] = sc + correction[e];
    }
    __syncwarp();
  }
  float total = 0.f;
  for (int k = 0; k < top; ++k) {
    // the largest logit not taken yet; equal logits: the lower index
    float best = -INFINITY;
    int arg = E;
    for (int e = lane; e < E; e += 32) {
      const float v = z[e];
      if (v > best) { best = v; arg = e; }      // within a lane indices rise, so the first of equals stays
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
      if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
    }
    if (arg >= E) arg = k < E ? k : 0;          // rows of not-a-numbers (padding): any valid expert
    const float sc = correction ? own[arg] : (score == kScoreSoftmax ? expf(best - zmax) / denom : sigmoid_f32(best));
    total += sc;
    if (lane == 0) {
      ids[(size_t)r * top + k] = arg;
      weights[(size_t)r * top + k] = sc;
      z[arg] = -INFINITY;
    }
    __syncwarp();
  }
  if (lane == 0 && (renormalize || weight_scale != 1.f)) {
    const float f = renormalize ? weight_scale / (total + renorm_eps) : weight_scale;
    for (int k = 0; k < top; ++k) weights[(size_t)r * top + k] *= f;
  }
}

// grid (pairs, ceil(F / 8)), 256 threads = 8 warps, a warp per hidden column f of pair (row, choice):
//   hid[pair, f] = act(s * (Wg_e[f, :] . h[row])) * (s * (Wu_e[f, :] . h[row])),  s = weight (on input) or 1.
// gate_up: [E, 2F, W] (an expert's gate rows, then its up rows).
template <typename TT>
__global__ void __launch_bounds__(256)
routed_gate_up_kernel(const TT* h, int h_ld, const TT* __restrict__ gate_up, const int* ids, const float* weights,
                      TT* hid, int W, int F, int top, int act, int weight_on_input, int E, float limit, float beta,
                      float shift) {
  extern __shared__ float hs[];
  pdl_trigger();
  pdl_wait();
  const int pair = blockIdx.x, row = pair / top;
  const int e = ids[pair];
  if (e >= E) return;         // an identity expert: nothing to compute
  const TT* hr = h + (size_t)row * h_ld;
  for (int k = threadIdx.x; k < W; k += 256) hs[k] = to_f32(hr[k]);
  __syncthreads();
  const int lane = threadIdx.x & 31, f = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (f >= F) return;
  const TT* wg = gate_up + ((size_t)e * 2 * F + f) * W;
  const TT* wu = wg + (size_t)F * W;
  float g = 0.f, u = 0.f;
  constexpr int V = 16 / (int)sizeof(TT);      // elements of a 16-byte load
  if (W % V == 0 && !(((uintptr_t)wg | (uintptr_t)wu) & 15)) {
    for (int k = lane * V; k < W; k += 32 * V) {
      TT a[V], b[V];
      *reinterpret_cast<uint4*>(a) = *reinterpret_cast<const uint4*>(wg + k);
      *reinterpret_cast<uint4*>(b) = *reinterpret_cast<const uint4*>(wu + k);
#pragma unroll
      for (int i = 0; i < V; ++i) {
        g = fmaf(to_f32(a[i]), hs[k + i], g);
        u = fmaf(to_f32(b[i]), hs[k + i], u);
      }
    }
  } else {
    for (int k = lane; k < W; k += 32) {
      const float x = hs[k];
      g = fmaf(to_f32(wg[k]), x, g);
      u = fmaf(to_f32(wu[k]), x, u);
    }
  }
  g = warp_sum(g);
  u = warp_sum(u);
  if (lane == 0) {
    const float s = weight_on_input ? weights[pair] : 1.f;
    from_f32(hid[(size_t)pair * F + f], gated_product(s * g, s * u, act, limit, beta, shift));
  }
}

// grid (rows, ceil(W / 8)), 256 threads: out[row, n] = sum over the row's choices k of
//   (weight on output ? weight : 1) * (Wd_e[n, :] . hid[row * top + k, :]),   down: [E, W, F].  out is 32-bit and is
// overwritten, or added to with `accumulate`.  A choice of E or above adds weight * h[row, n].
template <typename TT>
__global__ void __launch_bounds__(256)
routed_down_kernel(const TT* hid, const TT* __restrict__ down, const int* ids, const float* weights, float* out,
                   int out_ld, int W, int F, int top, int weight_on_input, int accumulate, int E, const TT* h, int h_ld) {
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x, lane = threadIdx.x & 31, n = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (n >= W) return;
  float total = 0.f;
  for (int k = 0; k < top; ++k) {
    const int pair = row * top + k;
    if (ids[pair] >= E) {      // uniform over the warp
      total += weights[pair] * to_f32(h[(size_t)row * h_ld + n]);
      continue;
    }
    const TT* wd = down + ((size_t)ids[pair] * W + n) * F;
    const TT* hp = hid + (size_t)pair * F;
    float acc = 0.f;
    constexpr int V = 16 / (int)sizeof(TT);
    if (F % V == 0 && !(((uintptr_t)wd | (uintptr_t)hp) & 15)) {
      for (int f = lane * V; f < F; f += 32 * V) {
        TT a[V], b[V];
        *reinterpret_cast<uint4*>(a) = *reinterpret_cast<const uint4*>(wd + f);
        *reinterpret_cast<uint4*>(b) = *reinterpret_cast<const uint4*>(hp + f);
#pragma unroll
        for (int i = 0; i < V; ++i) acc = fmaf(to_f32(a[i]), to_f32(b[i]), acc);
      }
    } else {
      for (int f = lane; f < F; f += 32) acc = fmaf(to_f32(wd[f]), to_f32(hp[f]), acc);
    }
    acc = warp_sum(acc);
    total = weight_on_input ? total + acc : fmaf(acc, weights[pair], total);
  }
  if (lane == 0) {
    float* o = out + (size_t)row * out_ld + n;
    *o = accumulate ? *o + total : total;
  }
}

}  // namespace cbis

using namespace cbis;

CBIS_EXPORT int cbis_route_topk(const void* h, int h_ld, const void* router, int* ids, float* weights, int rows, int W,
                                int E, int top, int score, int renormalize, int dtype, void* stream, float renorm_eps,
                                float weight_scale, const float* correction, float* side) {
  if (rows <= 0) return CBIS_OK;
  if (W <= 0 || E <= 0 || top <= 0 || top > E || (score != kScoreSigmoid && score != kScoreSoftmax)) return CBIS_ERR_BAD_SIZE;
  if (E > 6000) return CBIS_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t smem = (size_t)2 * (E + 1) * sizeof(float);
  // A warp for every router row (up to 32), so that no warp takes two of them one after the other, while the SMs hold the warps
  // of all rows at once, or nearly so; else eight warps a row (of more registers each, hence a kernel of its own).  Eight warps -> more
  // at width 2,048: 148 rows, 64 experts 14.1 -> 9.6 us; 300 rows, 24 experts 9.4 -> 9.8, 64 experts 23.6 -> 18.7; 592 rows, 64
  // experts 20.2 -> 23.2, 256 experts 71 -> 63.
  const int n = E + (side ? 1 : 0), warps = n < 32 ? n : 32, per_sm = (rows + 147) / 148;
  const bool many = n > 8 && ((per_sm <= 3 && (per_sm * warps <= 64 || n >= 48)) || (per_sm == 4 && n >= 128));
#define CBIS_ROUTE(TT, THREADS)                                                                                           \
  return (int)launch_pdl(route_topk_kernel<TT, THREADS>, dim3(rows), dim3(THREADS == 256 ? 256 : 32 * warps), smem, st, \
                         (const TT*)h, h_ld, (const TT*)router, ids, weights, W, E, top, score, renormalize, renorm_eps,  \
                         weight_scale, correction, side)
  if (dtype == CBIS_F32) {
    if (many) CBIS_ROUTE(float, 1024);
    CBIS_ROUTE(float, 256);
  }
  if (dtype == CBIS_BF16) {
    if (many) CBIS_ROUTE(__nv_bfloat16, 1024);
    CBIS_ROUTE(__nv_bfloat16, 256);
  }
#undef CBIS_ROUTE
  return CBIS_ERR_BAD_DTYPE;
}

CBIS_EXPORT int cbis_routed_gate_up(const void* h, int h_ld, const void* gate_up, const int* ids, const float* weights,
                                    void* hid, int rows, int W, int F, int top, int act, int weight_on_input, int dtype,
                                    void* stream, int E, float limit, float beta, float shift) {
  if (rows <= 0) return CBIS_OK;
  if (W <= 0 || F <= 0 || top <= 0) return CBIS_ERR_BAD_SIZE;
  if (W > 12288 || F > 8 * 65535) return CBIS_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  const dim3 grid(rows * top, (F + 7) / 8);
  const size_t smem = (size_t)W * sizeof(float);
  if (dtype == CBIS_F32)
    return (int)launch_pdl(routed_gate_up_kernel<float>, grid, dim3(256), smem, st, (const float*)h, h_ld,
                           (const float*)gate_up, ids, weights, (float*)hid, W, F, top, act, weight_on_input, E, limit,
                           beta, shift);
  if (dtype == CBIS_BF16)
    return (int)launch_pdl(routed_gate_up_kernel<__nv_bfloat16>, grid, dim3(256), smem, st, (const __nv_bfloat16*)h, h_ld,
                           (const __nv_bfloat16*)gate_up, ids, weights, (__nv_bfloat16*)hid, W, F, top, act,
                           weight_on_input, E, limit, beta, shift);
  return CBIS_ERR_BAD_DTYPE;
}

CBIS_EXPORT int cbis_routed_down(const void* hid, const void* down, const int* ids, const float* weights, float* out,
                                 int out_ld, int rows, int W, int F, int top, int weight_on_input, int accumulate,
                                 int dtype, void* stream, int E, const void* h, int h_ld) {
  if (rows <= 0) return CBIS_OK;
  if (W <= 0 || F <= 0 || top <= 0) return CBIS_ERR_BAD_SIZE;
  if (W > 8 * 65535) return CBIS_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  const dim3 grid(rows, (W + 7) / 8);
  if (dtype == CBIS_F32)
    return (int)launch_pdl(routed_down_kernel<float>, grid, dim3(256), 0, st, (const float*)hid, (const float*)down, ids,
                           weights, out, out_ld, W, F, top, weight_on_input, accumulate, E, (const float*)h, h_ld);
  if (dtype == CBIS_BF16)
    return (int)launch_pdl(routed_down_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, (const __nv_bfloat16*)hid,
                           (const __nv_bfloat16*)down, ids, weights, out, out_ld, W, F, top, weight_on_input, accumulate, E,
                           (const __nv_bfloat16*)h, h_ld);
  return CBIS_ERR_BAD_DTYPE;
}
