// Gates and unit norms, all in 32-bit arithmetic whatever the storage type:
//   * rms_norm: rows divided by their root mean square in equal parts, times a weight; an optional gate
//     (act(z), element by element) is applied BEFORE the norm, or (gate_after) to the normalised, weighted values;
//   * gate_mul: out = act(a) * b, the inside of a gated feed-forward (a = gate, b = up) and an output gate
//     (a = the gate's projection, b = the values, act = sigmoid).
#include "common.cuh"

namespace cbis {

// grid (rows, parts); part g of row r covers columns g*pw .. g*pw + pw - 1.
//   v = x[r, c] * (gate ? act(gate[r, c]) : 1);  out[r, c] = v / sqrt(mean_c(v^2) + eps) * (weight ? weight[c] : 1)
// With gate_after the gate stays out of v:  out[r, c] = x / sqrt(mean_c(x^2) + eps) * weight[c] * act(gate[r, c]).
// With `staged` the part's v wait in shared memory (pw floats) between the two passes; else they are read again.
template <typename TI, typename TG, typename TO>
__global__ void rms_norm_kernel(const TI* x, int x_ld, const TG* gate, int gate_ld, int gate_act,
                                const float* __restrict__ weight, float eps, TO* out, int out_ld, int pw, int staged,
                                int gate_after) {
  extern __shared__ float vs[];
  __shared__ float red[33];
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x, c0 = blockIdx.y * pw;
  const TI* xr = x + (size_t)r * x_ld + c0;
  const TG* gr = gate ? gate + (size_t)r * gate_ld + c0 : nullptr;
  float ss = 0.f;
  for (int c = threadIdx.x; c < pw; c += blockDim.x) {
    float v = to_f32(xr[c]);
    if (gr && !gate_after) v *= activate(to_f32(gr[c]), gate_act);
    if (staged) vs[c] = v;
    ss += v * v;
  }
  const float inv = 1.0f / sqrtf(block_sum(ss, red) / (float)pw + eps);
  TO* orow = out + (size_t)r * out_ld + c0;
  for (int c = threadIdx.x; c < pw; c += blockDim.x) {
    float v;
    if (staged) {
      v = vs[c];
    } else {
      v = to_f32(xr[c]);
      if (gr && !gate_after) v *= activate(to_f32(gr[c]), gate_act);
    }
    v *= inv;
    if (weight) v *= weight[c0 + c];
    if (gr && gate_after) v *= activate(to_f32(gr[c]), gate_act);
    from_f32(orow[c], v);
  }
}

// out[r, c] = act(a[r, c]) * b[r, c] (with limit, beta and shift as in gated_product of common.cuh; times row_gate[r], a
// 32-bit number per row, if there is one); with `b_rows` b's row is b_rows[r] instead (rows of a table looked up by token;
// an index outside 0 .. b_n_rows - 1 reads as zeros)
template <typename TT>
__global__ void gate_mul_kernel(const TT* a, int a_ld, const TT* b, int b_ld, TT* out, int out_ld, int act, int rows,
                                int n, const int* b_rows, int b_n_rows, float limit, float beta, float shift, const float* row_gate) {
  pdl_trigger();
  pdl_wait();
  const size_t total = (size_t)rows * n;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t r = i / n;
    const int c = (int)(i % n);
    size_t br = r;
    bool there = true;
    if (b_rows) {
      const int t = b_rows[r];
      there = t >= 0 && t < b_n_rows;
      br = there ? (size_t)t : 0;
    }
    const float bv = there ? to_f32(b[br * b_ld + c]) : 0.f;
    const float v = gated_product(to_f32(a[r * a_ld + c]), bv, act, limit, beta, shift);
    from_f32(out[r * out_ld + c], row_gate ? v * row_gate[r] : v);
  }
}

// rms_norm for parts of a multiple of 8 columns up to 8,192, every row 16-byte aligned: a thread holds 8 neighbouring columns
// (NV times) in registers between the two passes and moves 16 bytes at a time.  1,500 rows of 4,096 with a gate: the kernel
// above took 26 us, four times what its bytes take.
template <typename TI, typename TG, typename TO, int NV>
__global__ void __launch_bounds__(512)
rms_norm_vec_kernel(const TI* x, int x_ld, const TG* gate, int gate_ld, int gate_act, const float* __restrict__ weight, float eps,
                    TO* out, int out_ld, int pw, int gate_after) {
  __shared__ float red[33];
  pdl_trigger();
  const int r = blockIdx.x, c0 = blockIdx.y * pw;
  float w[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 8;
    if (weight && c < pw) load8(w[i], weight + c0 + c);      // the weights do not come from the kernel before
    else
#pragma unroll
      for (int e = 0; e < 8; ++e) w[i][e] = 1.f;
  }
  pdl_wait();
  const TI* xr = x + (size_t)r * x_ld + c0;
  const TG* gr = gate ? gate + (size_t)r * gate_ld + c0 : nullptr;
  float v[NV][8], g[NV][8], ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 8;
    if (c < pw) {
      load8(v[i], xr + c);
      if (gr) load8(g[i], gr + c);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[i][e] = g[i][e] = 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (gr) {
      activate_all(g[i], gate_act);
      if (!gate_after)
#pragma unroll
        for (int e = 0; e < 8; ++e) v[i][e] *= g[i][e];
    }
    if ((threadIdx.x + i * (int)blockDim.x) * 8 < pw)
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += v[i][e] * v[i][e];
  }
  const float inv = 1.0f / sqrtf(block_sum(ss, red) / (float)pw + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (threadIdx.x + i * blockDim.x) * 8;
    if (c >= pw) continue;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      v[i][e] *= inv;
      if (weight) v[i][e] *= w[i][e];
      if (gr && gate_after) v[i][e] *= g[i][e];
    }
    store8(out + (size_t)r * out_ld + c0 + c, v[i]);
  }
}

// gate_mul for rows of a multiple of 8 columns, 16-byte aligned: grid (rows, ceil(n / 2048)), 8 neighbouring columns a thread.
// 1,500 rows of 5,632: the kernel above took 24 us, three times what its bytes take.
template <typename TT>
__global__ void __launch_bounds__(256)
gate_mul_vec_kernel(const TT* a, int a_ld, const TT* b, int b_ld, TT* out, int out_ld, int act, int n, const int* b_rows, int b_n_rows,
                    float limit, float beta, float shift, const float* row_gate) {
  pdl_trigger();
  pdl_wait();
  const size_t r = blockIdx.x;
  const int c = (blockIdx.y * 256 + threadIdx.x) * 8;
  if (c >= n) return;
  size_t br = r;
  bool there = true;
  if (b_rows) {
    const int t = b_rows[r];
    there = t >= 0 && t < b_n_rows;
    br = there ? (size_t)t : 0;
  }
  float g[8], u[8];
  load8(g, a + r * a_ld + c);
  if (there) load8(u, b + br * b_ld + c);
  else
#pragma unroll
    for (int e = 0; e < 8; ++e) u[e] = 0.f;
  const float rg = row_gate ? row_gate[r] : 1.f;
  gated_products(g, u, act, limit, beta, shift);
  if (row_gate)
#pragma unroll
    for (int e = 0; e < 8; ++e) g[e] *= rg;
  store8(out + r * out_ld + c, g);
}

template <typename TI, typename TG, typename TO>
static int launch_rms(const void* x, int x_ld, const void* gate, int gate_ld, int gate_act, const float* weight,
                      float eps, void* out, int out_ld, int rows, int parts, int pw, int gate_after, cudaStream_t st) {
  // (with a gate a thread takes 8 activations one after the other: narrow parts are then faster a value a thread.  Parts of 64, 128 and
  // 256 columns, 64 rows of 8 to 16 of them: 2.3 -> 3.1 us, 2.7 -> 3.2, 2.8 -> 2.3; 1,500 rows of 8 x 160: 14.6 -> 12.8)
  const bool wide = !gate || pw >= 256 || (pw >= 128 && (long long)rows * parts * pw >= 350000);
  const bool vec = wide && pw % 8 == 0 && pw <= 2 * 512 * 8 && x_ld * sizeof(TI) % 16 == 0 && out_ld * sizeof(TO) % 16 == 0 &&
                   (!gate || gate_ld * sizeof(TG) % 16 == 0) &&
                   !(((uintptr_t)x | (uintptr_t)out | (uintptr_t)gate | (uintptr_t)weight) & 15);
  if (vec) {
    const int chunks = pw / 8;
    auto kern = chunks <= 512 ? rms_norm_vec_kernel<TI, TG, TO, 1> : rms_norm_vec_kernel<TI, TG, TO, 2>;
    const int per = chunks <= 512 ? chunks : (chunks + 1) / 2;
    return (int)launch_pdl(kern, dim3(rows, parts), dim3((per + 31) / 32 * 32), 0, st, (const TI*)x, x_ld, (const TG*)gate, gate_ld,
                           gate_act, weight, eps, (TO*)out, out_ld, pw, gate_after);
  }
  const int threads = pw >= 2048 ? 512 : (pw >= 512 ? 256 : (pw >= 128 ? 128 : 64));
  const int staged = pw <= 10240 ? 1 : 0;         // 40 KB of shared memory at most
  return (int)launch_pdl(rms_norm_kernel<TI, TG, TO>, dim3(rows, parts), dim3(threads),
                         staged ? (size_t)pw * sizeof(float) : 0, st, (const TI*)x, x_ld, (const TG*)gate, gate_ld,
                         gate_act, weight, eps, (TO*)out, out_ld, pw, staged, gate_after);
}

}  // namespace cbis

using namespace cbis;

// x: 32-bit or the compute type (x_dtype); gate (may be null) and out: the compute type (dtype).
CBIS_EXPORT int cbis_rms_norm(const void* x, int x_ld, int x_dtype, const void* gate, int gate_ld, int gate_act,
                              const float* weight, float eps, void* out, int out_ld, int dtype, int rows, int parts,
                              int part_width, void* stream, int gate_after) {
  if (rows <= 0) return CBIS_OK;
  if (parts <= 0 || part_width <= 0) return CBIS_ERR_BAD_SIZE;
  if (parts > 65535) return CBIS_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
#define CBIS_RMS(TI, TG) \
  return launch_rms<TI, TG, TG>(x, x_ld, gate, gate_ld, gate_act, weight, eps, out, out_ld, rows, parts, part_width, gate_after, st)
  if (dtype == CBIS_F32 && x_dtype == CBIS_F32) CBIS_RMS(float, float);
  if (dtype == CBIS_BF16 && x_dtype == CBIS_F32) CBIS_RMS(float, __nv_bfloat16);
  if (dtype == CBIS_BF16 && x_dtype == CBIS_BF16) CBIS_RMS(__nv_bfloat16, __nv_bfloat16);
#undef CBIS_RMS
  return CBIS_ERR_BAD_DTYPE;
}

CBIS_EXPORT int cbis_gate_mul(const void* a, int a_ld, const void* b, int b_ld, void* out, int out_ld, int act, int rows,
                              int n, int dtype, void* stream, const int* b_rows, int b_n_rows, float limit, float beta,
                              float shift, const float* row_gate) {
  if (rows <= 0 || n <= 0) return CBIS_OK;
  const size_t total = (size_t)rows * n;
  size_t blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  cudaStream_t st = (cudaStream_t)stream;
  const int per16 = dtype == CBIS_F32 ? 4 : 8;
  // (fewer than 80,000 products are over before eight activations one after the other are: 64 rows of 512 1.5 us -> 1.8, of 1,408 2.1 -> 1.9;
  // a block takes one row, so narrow rows leave its threads idle: 1,500 rows of 128 2.5 -> 2.8, of 256 3.1 -> 2.8)
  if (n >= 256 && total >= 80000 && n % 8 == 0 && a_ld % per16 == 0 && b_ld % per16 == 0 && out_ld % per16 == 0 && n <= 2048 * 65535ll &&
      !(((uintptr_t)a | (uintptr_t)b | (uintptr_t)out) & 15)) {
    const dim3 grid(rows, (n + 2047) / 2048), block(n >= 2048 ? 256 : (n / 8 + 31) / 32 * 32);
    if (dtype == CBIS_F32)
      return (int)launch_pdl(gate_mul_vec_kernel<float>, grid, block, 0, st, (const float*)a, a_ld, (const float*)b, b_ld, (float*)out,
                             out_ld, act, n, b_rows, b_n_rows, limit, beta, shift, row_gate);
    if (dtype == CBIS_BF16)
      return (int)launch_pdl(gate_mul_vec_kernel<__nv_bfloat16>, grid, block, 0, st, (const __nv_bfloat16*)a, a_ld,
                             (const __nv_bfloat16*)b, b_ld, (__nv_bfloat16*)out, out_ld, act, n, b_rows, b_n_rows, limit, beta, shift,
                             row_gate);
  }
  if (dtype == CBIS_F32)
    return (int)launch_pdl(gate_mul_kernel<float>, dim3((int)blocks), dim3(256), 0, st, (const float*)a, a_ld,
                           (const float*)b, b_ld, (float*)out, out_ld, act, rows, n, b_rows, b_n_rows, limit, beta,
                           shift, row_gate);
  if (dtype == CBIS_BF16)
    return (int)launch_pdl(gate_mul_kernel<__nv_bfloat16>, dim3((int)blocks), dim3(256), 0, st, (const __nv_bfloat16*)a,
                           a_ld, (const __nv_bfloat16*)b, b_ld, (__nv_bfloat16*)out, out_ld, act, rows, n, b_rows, b_n_rows, limit, beta,
                           shift, row_gate);
  return CBIS_ERR_BAD_DTYPE;
}
