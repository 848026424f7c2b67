// Reductions, softmax family, NLL loss and the vector/matrix-vector dot family.
//
// Replaces cudnnReduceTensor / cudnnSoftmax* (TensorDslCudnn.scala:1431-1576), the one-thread-per-block nllLoss
// kernels (DslAPI.scala:506-516) and cublasSdot/Sgemv (TensorDslCublas.scala:173-201, 257-264).  Semantics follow
// TensorDslCPU.scala (cited per entry point).  Rows are reduced by one warp each with shuffles; full reductions
// use a block tree in shared memory and, for large inputs, a second pass over per-block partials.
#include <algorithm>
#include <cfloat>

#include "common.cuh"

namespace ltb {

__device__ __forceinline__ float warp_sum(float v) { for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o); return v; }
__device__ __forceinline__ float warp_max(float v) { for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o)); return v; }

__device__ float block_sum(float v) {
  __shared__ float sh[32];
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  int nw = (blockDim.x + 31) >> 5;
  v = threadIdx.x < nw ? sh[threadIdx.x] : 0.0f;
  if (w == 0) v = warp_sum(v);
  return v;   // valid in warp 0
}

// out[0] = scale * sum(x) (single block) or partial[b] = sum of the block's slice.
__global__ void sum_kernel(const float* __restrict__ x, float* out, int64_t n, float scale, bool partial) {
  pdl_enter();
  float s = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) s += x[i];
  s = block_sum(s);
  if (threadIdx.x == 0) out[partial ? blockIdx.x : 0] = partial ? s : s * scale;
}
__global__ void add_scalar_from_kernel(float* dx, const float* __restrict__ dout, float scale, int64_t n) {
  pdl_enter();
  const float v = dout[0];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) dx[i] = fmaf(v, scale, dx[i]);
}
// out[o, l] = sum_s x[o, s, l]
__global__ void sum_dim_kernel(const float* __restrict__ x, float* out, int outer, int d, int inner) {
  pdl_enter();
  int64_t n = (int64_t)outer * inner;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t o = i / inner, l = i % inner;
    const float* p = x + o * d * inner + l;
    float s = 0.0f;
    for (int k = 0; k < d; ++k) s += p[(int64_t)k * inner];
    out[i] = s;
  }
}
// inner == 1: one warp per output
__global__ void sum_lastdim_kernel(const float* __restrict__ x, float* out, int outer, int d) {
  pdl_enter();
  int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; int lane = threadIdx.x & 31;
  if (w >= outer) return;
  float s = 0.0f;
  for (int k = lane; k < d; k += 32) s += x[w * d + k];
  s = warp_sum(s);
  if (lane == 0) out[w] = s;
}
__global__ void sum_dim_grad_kernel(float* dx, const float* __restrict__ dout, int outer, int d, int inner) {
  pdl_enter();
  int64_t n = (int64_t)outer * d * inner;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t l = i % inner, o = i / ((int64_t)d * inner);
    dx[i] += dout[o * inner + l];
  }
}

// One warp per row. MODE 0 softmax, 1 logSoftmax (TensorDslCPU.scala:783-832).  VPT > 0: a row of at most 32 VPT columns stays in registers, all its
// loads in flight at once, and the pieces beyond the row are left out (log-softmax, us, walking the row three times / so: 300 rows of 100 2.8 / 1.6, 9623 of 300 6.2 / 5.0,
// of 1000 16.5 / 11.2, 3000 of 768 4.7 / 5.4, 20000 of 768 23.9 / 19.8); VPT 0: any length.
// Returns log sum exp of the row (MODE 1).
template <int MODE, int VPT>
__device__ __forceinline__ float softmax_row(const float* p, float* q, int cols, int lane) {
  float mx = -FLT_MAX, s = 0.0f;
  if constexpr (VPT > 0) {
    constexpr int G = VPT < 4 ? VPT : 4;                      // pieces of 128 columns, those beyond the row left out
    float v[VPT];
#pragma unroll
    for (int g = 0; g < VPT; g += G) if (g == 0 || 32 * g < cols) {
#pragma unroll
      for (int j = g; j < g + G; ++j) { const int i = lane + 32 * j; v[j] = i < cols ? p[i] : -FLT_MAX; }
    }
#pragma unroll
    for (int g = 0; g < VPT; g += G) if (g == 0 || 32 * g < cols) {
#pragma unroll
      for (int j = g; j < g + G; ++j) mx = fmaxf(mx, v[j]);
    }
    mx = warp_max(mx);
#pragma unroll
    for (int g = 0; g < VPT; g += G) if (g == 0 || 32 * g < cols) {
#pragma unroll
      for (int j = g; j < g + G; ++j) if (lane + 32 * j < cols) s += expf(v[j] - mx);
    }
    s = warp_sum(s);
    const float logsum = mx + logf(s);
#pragma unroll
    for (int g = 0; g < VPT; g += G) if (g == 0 || 32 * g < cols) {
#pragma unroll
      for (int j = g; j < g + G; ++j) { const int i = lane + 32 * j; if (i < cols) q[i] = MODE == 0 ? expf(v[j] - mx) / s : v[j] - logsum; }
    }
    return logsum;
  }
  for (int i = lane; i < cols; i += 32) mx = fmaxf(mx, p[i]);
  mx = warp_max(mx);
  for (int i = lane; i < cols; i += 32) s += expf(p[i] - mx);
  s = warp_sum(s);
  const float logsum = mx + logf(s);
  for (int i = lane; i < cols; i += 32) q[i] = MODE == 0 ? expf(p[i] - mx) / s : p[i] - logsum;
  return logsum;
}
template <int MODE, int VPT>
__global__ void softmax_kernel(const float* __restrict__ x, float* y, int rows, int cols) {
  pdl_enter();
  int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; int lane = threadIdx.x & 31;
  if (r < rows) softmax_row<MODE, VPT>(x + r * cols, y + r * cols, cols, lane);
}
// Log-softmax of a row, the negative log likelihood of its target (nll_kernel) and, with `sum`, scale times the sum of those: three launches of some
// 3 us each on a batch of a few hundred rows, of which there is next to nothing to compute.  The last CTA to finish adds the rows up, in the order in
// which sum_kernel's one CTA of 1024 threads does, so the result is the same to the bit: thirty-two loads of a thread in flight (one after the other the sum of
// 8192 rows took 9 us), rows of at most 32 columns (VPT 1) on as many CTAs as the GPU holds, so that there are fewer tickets to wait for (65536 x 10 24.5 -> 18.2 us).
template <int VPT>
__global__ void __launch_bounds__(256) softmax_nll_kernel(const float* __restrict__ x, float* y, const int32_t* __restrict__ t, float* nll, float* sum, float scale,
                                                          int rows, int cols, unsigned* ticket) {
  pdl_enter();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t first = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  auto row = [&](int64_t r) {
    const int k = t[r];
    const bool in = k >= 0 && k < cols;
    const float xk = in ? x[r * cols + k] : 0.0f;
    const float logsum = softmax_row<1, VPT>(x + r * cols, y + r * cols, cols, lane);
    if (lane == 0) nll[r] = in ? -1.0f * (xk - logsum) : 0.0f;
  };
  if constexpr (VPT == 1) { for (int64_t r = first; r < rows; r += (int64_t)gridDim.x * 8) row(r); }
  else if (first < rows) row(first);
  if (!sum) return;
  __shared__ bool last;
  __shared__ float part[32];
  __syncthreads();
  if (threadIdx.x == 0) { __threadfence(); last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1; __threadfence(); }      // back at zero after the last
  __syncthreads();
  if (!last) return;
  float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  for (int i0 = threadIdx.x; i0 < rows; i0 += 8192) {
    float v[8][4];
#pragma unroll
    for (int e = 0; e < 8; ++e)
#pragma unroll
      for (int q = 0; q < 4; ++q) { const int i = i0 + 1024 * e + 256 * q; v[e][q] = i < rows ? __ldcg(nll + i) : 0.0f; }
#pragma unroll
    for (int e = 0; e < 8; ++e)
#pragma unroll
      for (int q = 0; q < 4; ++q) s[q] += v[e][q];
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) { const float a = warp_sum(s[q]); if (lane == 0) part[w + 8 * q] = a; }
  __syncthreads();
  if (w == 0) { const float a = warp_sum(part[lane]); if (lane == 0) sum[0] = a * scale; }
}
// The gradient's forms.  VPT 1, 8: a row of at most 32 VPT columns in registers, as above.  Longer rows are read twice, VPT 0 in loops that the compiler unrolls by four,
// VPT -1 with four pieces of 32 columns at a time, those of the row's end together too, where the loops' last turns would go one by one.
static int softmax_grad_form(int cols) { return cols <= 32 ? 1 : cols <= 256 ? 8 : cols < 1280 && cols % 128 >= 64 ? -1 : 0; }
// MODE 0: dx += y*(dy - sum dy*y) (cudnnSoftmaxBackward ACCURATE, TensorDslCudnn.scala:1465-1504);
// MODE 1: dx += dy - exp(y)*sum dy (TensorDslCPU.scala:837-846).
// us, VPT 0 / -1 (MODE 1): 1024 columns, 1 row 3.8 / 4.6, 1000 rows 5.6 / 6.8; 4096 columns, 300 rows 15.3 / 20.2; 1000 columns, 1 row 5.4 / 4.6, 1000 rows 7.4 / 6.8,
// 9623 rows 31.4 / 28.7; 600 columns 3.6 / 3.4, 5.0 / 4.8, 11.9 / 10.8.  A row of 1000 in 96 registers: 72 us on 8192 of them, 25 in this form.
template <int MODE, int VPT>
__global__ void softmax_grad_kernel(float* dx, const float* __restrict__ y, const float* __restrict__ dy, int rows, int cols) {
  pdl_enter();
  int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; int lane = threadIdx.x & 31;
  if (r >= rows) return;
  const float* yy = y + r * cols; const float* d = dy + r * cols; float* o = dx + r * cols;
  float s = 0.0f;
  if constexpr (VPT > 0) {
    float v[VPT], w[VPT], old[VPT];
#pragma unroll
    for (int j = 0; j < VPT; ++j) { const int i = lane + 32 * j; v[j] = i < cols ? d[i] : 0.0f; w[j] = i < cols ? yy[i] : 0.0f; old[j] = i < cols ? o[i] : 0.0f; }
#pragma unroll
    for (int j = 0; j < VPT; ++j) if (lane + 32 * j < cols) s += MODE == 0 ? v[j] * w[j] : v[j];
    s = warp_sum(s);
#pragma unroll
    for (int j = 0; j < VPT; ++j) { const int i = lane + 32 * j; if (i < cols) o[i] = old[j] + (MODE == 0 ? w[j] * (v[j] - s) : v[j] - expf(w[j]) * s); }
  } else if constexpr (VPT == 0) {
    for (int i = lane; i < cols; i += 32) s += MODE == 0 ? d[i] * yy[i] : d[i];
    s = warp_sum(s);
    for (int i = lane; i < cols; i += 32) o[i] += MODE == 0 ? yy[i] * (d[i] - s) : d[i] - expf(yy[i]) * s;
  } else {
    for (int i0 = lane; i0 < cols; i0 += 256) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) { const int i = i0 + 32 * j; v[j] = i < cols ? (MODE == 0 ? d[i] * yy[i] : d[i]) : 0.0f; }
#pragma unroll
      for (int j = 0; j < 8; ++j) s += v[j];
    }
    s = warp_sum(s);
    for (int i0 = lane; i0 < cols; i0 += 128) {
      float v[4], w[4], old[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) { const int i = i0 + 32 * j; v[j] = i < cols ? d[i] : 0.0f; w[j] = i < cols ? yy[i] : 0.0f; old[j] = i < cols ? o[i] : 0.0f; }
#pragma unroll
      for (int j = 0; j < 4; ++j) { const int i = i0 + 32 * j; if (i < cols) o[i] = old[j] + (MODE == 0 ? w[j] * (v[j] - s) : v[j] - expf(w[j]) * s); }
    }
  }
}
// What leads from the gradient of a loss to that of the logits, a warp per row: dnll += scale dout (dout set to `value` first when it is seeded here),
// dlogp[target] -= dnll, dx += dlogp - exp(y) sum dlogp; every buffer ends up as the separate launches leave it (four of 2.5 to 4 us each).  Nothing is stored before
// a row's sum, so that its loads go out together (us, 8192 x 1000 apart 25.4, joined 29.4 with the store first, 21.4 so; 8192 x 100 6.8, 4.4).  Rows of 1280 columns and
// more are not joined: the target in the way, the compiler's loops are slow (8192 x 2000 225), and the other form gains nothing (2048 x 2000 apart 15.0, joined 15.0;
// 1024 x 4096 19.1, 23.3).
template <int VPT>
__global__ void __launch_bounds__(256) nll_softmax_grad_kernel(float* __restrict__ dx, const float* __restrict__ y, float* __restrict__ dlogp, float* dnll, float* dout, bool seeded, float value,
                                                               float scale, const int32_t* __restrict__ t, int rows, int cols) {
  pdl_enter();
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; const int lane = threadIdx.x & 31;
  if (r >= rows) return;
  const int target = t[r], k = target < cols ? target : -1;         // (a target may lie beyond the row)
  const float dn = fmaf(seeded ? value : dout[0], scale, dnll[r]);
  if (lane == 0) { dnll[r] = dn; if (seeded && r == 0) dout[0] = value; }
  const float* __restrict__ yy = y + r * cols; float* __restrict__ d = dlogp + r * cols; float* __restrict__ o = dx + r * cols;
  auto with = [&](int i, float v) { return i == k ? v + -1.0f * dn : v; };
  float s = 0.0f;
  if constexpr (VPT > 0) {
    float v[VPT], w[VPT], old[VPT];
#pragma unroll
    for (int j = 0; j < VPT; ++j) { const int i = lane + 32 * j; v[j] = i < cols ? d[i] : 0.0f; w[j] = i < cols ? yy[i] : 0.0f; old[j] = i < cols ? o[i] : 0.0f; }
#pragma unroll
    for (int j = 0; j < VPT; ++j) { const int i = lane + 32 * j; if (i < cols) { if (i == k) { v[j] += -1.0f * dn; d[i] = v[j]; } s += v[j]; } }
    s = warp_sum(s);
#pragma unroll
    for (int j = 0; j < VPT; ++j) { const int i = lane + 32 * j; if (i < cols) o[i] = old[j] + (v[j] - expf(w[j]) * s); }
    return;
  }
  for (int i0 = lane; i0 < cols; i0 += 256) {                       // VPT 0: as softmax_grad_kernel's -1
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) { const int i = i0 + 32 * j; v[j] = i < cols ? d[i] : 0.0f; }
#pragma unroll
    for (int j = 0; j < 8; ++j) s += with(i0 + 32 * j, v[j]);
  }
  s = warp_sum(s);
  for (int i0 = lane; i0 < cols; i0 += 128) {
    float v[4], w[4], old[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) { const int i = i0 + 32 * j; v[j] = i < cols ? d[i] : 0.0f; w[j] = i < cols ? yy[i] : 0.0f; old[j] = i < cols ? o[i] : 0.0f; }
#pragma unroll
    for (int j = 0; j < 4; ++j) { const int i = i0 + 32 * j; if (i < cols) o[i] = old[j] + (with(i, v[j]) - expf(w[j]) * s); }
  }
  if (k >= 0 && lane == (k & 31)) d[k] = with(k, d[k]);             // by the lane that read it
}
__global__ void nll_kernel(const float* __restrict__ x, const int32_t* __restrict__ t, float* out, int rows, int cols) {
  pdl_enter();
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < rows) { int k = t[b]; out[b] = (k >= 0 && k < cols) ? -1.0f * x[(int64_t)b * cols + k] : 0.0f; }
}
__global__ void nll_grad_kernel(float* dx, const float* __restrict__ dout, const int32_t* __restrict__ t, int rows, int cols) {
  pdl_enter();
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < rows) { int k = t[b]; if (k >= 0 && k < cols) dx[(int64_t)b * cols + k] += -1.0f * dout[b]; }
}

// y[m] (+)= A[m,k] x[k]: one warp per row, float4 when k % 4 == 0 (memory-bound: A is read once).
template <bool ACC>
__global__ void gemv_rows_kernel(const float* __restrict__ a, const float* __restrict__ x, float* y, int m, int k) {
  pdl_enter();
  int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; int lane = threadIdx.x & 31;
  if (r >= m) return;
  const float* row = a + r * k;
  float s = 0.0f;
  if ((k & 3) == 0 && ((reinterpret_cast<uintptr_t>(row) | reinterpret_cast<uintptr_t>(x)) & 15) == 0) {
    for (int i = lane * 4; i < k; i += 128) {
      float4 av = *reinterpret_cast<const float4*>(row + i), xv = *reinterpret_cast<const float4*>(x + i);
      s += av.x * xv.x + av.y * xv.y + av.z * xv.z + av.w * xv.w;
    }
  } else for (int i = lane; i < k; i += 32) s += row[i] * x[i];
  s = warp_sum(s);
  if (lane == 0) y[r] = ACC ? y[r] + s : s;
}
// dx[k] += sum_i A[i,k] dout[i]: threads along k (coalesced), loop over rows.
__global__ void gemv_cols_kernel(const float* __restrict__ a, const float* __restrict__ dout, float* dx, int m, int k) {
  pdl_enter();
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= k) return;
  float s = 0.0f;
  for (int i = 0; i < m; ++i) s += a[(int64_t)i * k + j] * dout[i];
  dx[j] += s;
}
__global__ void outer_acc_kernel(float* da, const float* __restrict__ y, const float* __restrict__ dout, int m, int k) {
  pdl_enter();
  int64_t n = (int64_t)m * k;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) da[i] += y[i % k] * dout[i / k];
}
__global__ void dot_kernel(const float* __restrict__ x, const float* __restrict__ y, float* out, int n) {
  pdl_enter();
  float s = 0.0f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += x[i] * y[i];
  s = block_sum(s);
  if (threadIdx.x == 0) out[0] = s;
}
__global__ void axpy_from_scalar_kernel(float* dx, const float* __restrict__ y, const float* __restrict__ a, int n) {
  pdl_enter();
  float av = a[0];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dx[i] += av * y[i];
}

template <int MODE>
static int softmax_issue(const float* x, float* y, int rows, int cols) {
  const unsigned grid = (unsigned)ceil_div((int64_t)rows * 32, 256);
  if (cols <= 32) LTB_LAUNCH((softmax_kernel<MODE, 1>), grid, 256, 0, x, y, rows, cols);
  else if (cols <= 256) LTB_LAUNCH((softmax_kernel<MODE, 8>), grid, 256, 0, x, y, rows, cols);
  else if (cols <= 512) LTB_LAUNCH((softmax_kernel<MODE, 16>), grid, 256, 0, x, y, rows, cols);
  else if (cols <= 1024) LTB_LAUNCH((softmax_kernel<MODE, 32>), grid, 256, 0, x, y, rows, cols);
  else LTB_LAUNCH((softmax_kernel<MODE, 0>), grid, 256, 0, x, y, rows, cols);
  return LTB_OK;
}
template <int MODE>
static int softmax_grad_issue(float* dx, const float* y, const float* dy, int rows, int cols) {
  const unsigned grid = (unsigned)ceil_div((int64_t)rows * 32, 256);
  const int form = softmax_grad_form(cols);
  if (form == 1) LTB_LAUNCH((softmax_grad_kernel<MODE, 1>), grid, 256, 0, dx, y, dy, rows, cols);
  else if (form == 8) LTB_LAUNCH((softmax_grad_kernel<MODE, 8>), grid, 256, 0, dx, y, dy, rows, cols);
  else if (form == 0) LTB_LAUNCH((softmax_grad_kernel<MODE, 0>), grid, 256, 0, dx, y, dy, rows, cols);
  else LTB_LAUNCH((softmax_grad_kernel<MODE, -1>), grid, 256, 0, dx, y, dy, rows, cols);
  return LTB_OK;
}

static int full_sum(const float* x, float* out, int64_t n, float scale) {
  if (n <= (1 << 16)) { LTB_LAUNCH(sum_kernel, 1, 1024, 0, x, out, n, scale, false); return LTB_OK; }
  int blocks = grid_for(n, 1024, 2);
  LTB_LAUNCH(sum_kernel, blocks, 1024, 0, x, g.cur_scratch(), n, 1.0f, true);
  LTB_LAUNCH(sum_kernel, 1, 1024, 0, (const float*)g.cur_scratch(), out, (int64_t)blocks, scale, false);
  return LTB_OK;
}

// ---- the calls around a classifier's loss that look-ahead fusion joins
// The rows up to which the sum joins: not many more than the GPU works on at once, eight CTAs of eight rows an SM, three at 257 to 1024 columns (at most 32
// columns: a CTA takes several rows).  A CTA waits for its ticket before it makes room for another, which costs more than the launch saved: us, the sum apart /
// joined, 4096 x 300 5.8 / 6.6, 5000 x 300 6.3 / 6.9, 4096 x 1000 8.4 / 8.9, 16384 x 100 8.5 / 10.0; 3000 x 1000 8.9 / 7.8, 8192 x 100 6.3 / 5.8, 20000 x 10 8.1 / 7.6,
// but 65536 x 10 17.3 / 18.0.  (One CTA adds them up, as in full_sum: 65536 in all.)
static int head_sum_rows(int cols) { return cols <= 32 ? 1 << 16 : std::min(1 << 16, g.sm_count * 8 * (cols <= 256 || cols > 1024 ? 8 : 3)); }
static int softmax_nll_issue(const Pending& p, float* sum, float scale) {
  const unsigned grid = (unsigned)ceil_div((int64_t)p.N * 32, 256), most = (unsigned)g.sm_count * 8;      // a warp per row
  unsigned* const ticket = g.tickets + (g.in_branch ? 1 : 0);
  if (p.C <= 32) LTB_LAUNCH((softmax_nll_kernel<1>), std::min(grid, most), 256, 0, p.x, p.y, p.target, p.out, sum, scale, p.N, p.C, ticket);
  else if (p.C <= 256) LTB_LAUNCH((softmax_nll_kernel<8>), grid, 256, 0, p.x, p.y, p.target, p.out, sum, scale, p.N, p.C, ticket);
  else if (p.C <= 512) LTB_LAUNCH((softmax_nll_kernel<16>), grid, 256, 0, p.x, p.y, p.target, p.out, sum, scale, p.N, p.C, ticket);
  else if (p.C <= 1024) LTB_LAUNCH((softmax_nll_kernel<32>), grid, 256, 0, p.x, p.y, p.target, p.out, sum, scale, p.N, p.C, ticket);
  else LTB_LAUNCH((softmax_nll_kernel<0>), grid, 256, 0, p.x, p.y, p.target, p.out, sum, scale, p.N, p.C, ticket);
  return LTB_OK;
}
static int nll_softmax_grad_issue(const Pending& p, float* dx, const float* y) {
  const unsigned grid = (unsigned)ceil_div((int64_t)p.N * 32, 256);
  if (p.C <= 32) LTB_LAUNCH((nll_softmax_grad_kernel<1>), grid, 256, 0, dx, y, p.db, p.da, p.d, p.seeded, p.value, p.scale, p.target, p.N, p.C);
  else if (p.C <= 256) LTB_LAUNCH((nll_softmax_grad_kernel<8>), grid, 256, 0, dx, y, p.db, p.da, p.d, p.seeded, p.value, p.scale, p.target, p.N, p.C);
  else LTB_LAUNCH((nll_softmax_grad_kernel<0>), grid, 256, 0, dx, y, p.db, p.da, p.d, p.seeded, p.value, p.scale, p.target, p.N, p.C);
  return LTB_OK;
}
static int sum_grad_issue(float* dx, const float* dout, float scale, int64_t n) {
  if (n) LTB_LAUNCH(add_scalar_from_kernel, grid_for(n, 256), 256, 0, dx, dout, scale, n);
  return LTB_OK;
}
static int nll_grad_issue(float* dx, const float* dout, const int32_t* t, int rows, int cols) {
  LTB_LAUNCH(nll_grad_kernel, (rows + 127) / 128, 128, 0, dx, dout, t, rows, cols);
  return LTB_OK;
}
int head_issue(const Pending& p) {
  if (p.kind == PEND_LSM) return softmax_issue<1>(p.x, p.y, p.N, p.C);
  if (p.kind == PEND_NLL) return softmax_nll_issue(p, nullptr, 0.0f);
  int rc = p.seeded ? fill_issue(p.d, p.value, 1) : LTB_OK;
  if (!rc) rc = sum_grad_issue(p.da, p.d, p.scale, p.n);
  return rc || p.kind == PEND_SUM_GRAD ? rc : nll_grad_issue(p.db, p.da, p.target, p.N, p.C);
}
// Whether [p, p + floats) keeps clear of [q, q + n).
static bool apart(const void* p, int64_t floats, const void* q, int64_t n) { return (const float*)p + floats <= (const float*)q || (const float*)q + n <= (const float*)p; }
static int full_sum_joining(const float* x, float* out, int64_t n, float scale) {
  if (g.pending.kind == PEND_NLL && g.pending.out == x && g.pending.N == n && n <= head_sum_rows(g.pending.C)) {
    const Pending p = g.pending; g.pending.kind = PEND_NONE;
    return softmax_nll_issue(p, out, scale);               // (the last CTA writes out: nothing is read any more)
  }
  if (g.pending.kind) { int rc = flush_pending(); if (rc) return rc; }
  return full_sum(x, out, n, scale);
}
// dx += scale dout.  A held call that cannot be joined is issued before anything else of this one, its zero fills included.
static int sum_grad_joining(float* dx, const float* dout, float scale, int64_t n) {
  const bool clear = apart(dx, n, dout, 1), seeded = g.pending.kind == PEND_SEED && g.pending.d == dout && clear;
  if (g.pending.kind && !seeded) { int rc = flush_pending(); if (rc) return rc; }
  Pending h; h.kind = PEND_SUM_GRAD; h.n = n; h.da = dx; h.d = const_cast<float*>(dout); h.scale = scale; h.seeded = seeded; h.value = g.pending.value;
  LTB_SETTLE(dx); LTB_SETTLE(dout); LTB_WRITES(dx, n);
  g.pending = h;
  if (g.fusion && n > 0 && clear) return LTB_OK;           // the gradient of a negative log likelihood may join it
  return flush_pending();
}

}  // namespace ltb

using namespace ltb;

extern "C" {

// sum / mean and their grads: TensorDslCPU.scala:1115-1124.
int ltb_sum(const float* x, float* out, int64_t n) { LTB_INITED_NOFLUSH(); LTB_REQUIRE(x && out && n >= 0, "ltb_sum: bad argument"); LTB_WRITES(out, 1); return full_sum_joining(x, out, n, 1.0f); }
int ltb_mean(const float* x, float* out, int64_t n) { LTB_INITED_NOFLUSH(); LTB_REQUIRE(x && out && n > 0, "ltb_mean: bad argument"); LTB_WRITES(out, 1); return full_sum_joining(x, out, n, 1.0f / (float)n); }
int ltb_sum_grad(float* dx, const float* dout, int64_t n) {
  LTB_INITED_NOFLUSH(); LTB_REQUIRE(dx && dout && n >= 0, "ltb_sum_grad: bad argument");
  return sum_grad_joining(dx, dout, 1.0f, n);
}
int ltb_mean_grad(float* dx, const float* dout, int64_t n) {
  LTB_INITED_NOFLUSH(); LTB_REQUIRE(dx && dout && n > 0, "ltb_mean_grad: bad argument");
  return sum_grad_joining(dx, dout, 1.0f / (float)n, n);
}
// sum(dim) / sum_grad(dim): TensorDslCPU.scala:1125-1164.
int ltb_sum_dim(const float* x, float* out, int outer, int d, int inner) {
  LTB_INITED(); LTB_REQUIRE(x && out && outer > 0 && d > 0 && inner > 0, "ltb_sum_dim: bad argument"); LTB_WRITES(out, (size_t)outer * inner);
  if (inner == 1) LTB_LAUNCH(sum_lastdim_kernel, (unsigned)ceil_div((int64_t)outer * 32, 256), 256, 0, x, out, outer, d);
  else LTB_LAUNCH(sum_dim_kernel, grid_for((int64_t)outer * inner, 256), 256, 0, x, out, outer, d, inner);
  return LTB_OK;
}
int ltb_sum_dim_grad(float* dx, const float* dout, int outer, int d, int inner) {
  LTB_INITED(); LTB_SETTLE(dx); LTB_SETTLE(dout); LTB_REQUIRE(dx && dout && outer > 0 && d > 0 && inner > 0, "ltb_sum_dim_grad: bad argument"); LTB_WRITES(dx, (size_t)outer * d * inner);
  LTB_LAUNCH(sum_dim_grad_kernel, grid_for((int64_t)outer * d * inner, 256), 256, 0, dx, dout, outer, d, inner);
  return LTB_OK;
}

// ---- the full sum with its partials in a file-scope device array: nothing is allocated, at set-up or per call.
// ltb_sum takes its partials from the workspace that ltb_init obtains with cudaMalloc. This variant is for callers
// for whom an allocation is not acceptable at all: cudaMalloc and cudaFree synchronise the whole device, which
// stalls every other stream of a process that serves requests while it computes, and a process that runs under a
// memory budget fixed at start-up cannot let a library grow its footprint afterwards. No counterpart in the reference.
//   * The first call on a device looks the array's address up (cudaGetSymbolAddress, with that device current); that
//     is set-up work and belongs before any stream capture. Later calls only launch.
//   * Limit: n <= kStaticSumMaxN elements; beyond it the call fails with LTB_E_LIMIT and launches nothing.
//   * Nothing has to start at zero: stage one writes one partial per CTA into slots [0, CTAs), stage two reads exactly
//     those slots, so stale contents of the array are never read.
//   * The array is one per device and process: two calls in flight at once (different streams or threads) race on it.
//     Calls on one stream are ordered and safe.
constexpr int kStaticSumSlots = 2048;
constexpr int64_t kStaticSumMaxN = (int64_t)1 << 30;
constexpr int kStaticSumMaxDevices = 64;
static __device__ __align__(256) float static_sum_scratch[kStaticSumSlots];
static float* static_sum_ptr[kStaticSumMaxDevices] = {};
}  // extern "C"
namespace ltb { void static_sum_forget() { for (auto& p : static_sum_ptr) p = nullptr; } }   // ltb_shutdown: a later context looks the address up again
extern "C" {

int ltb_sum_static_scratch(const float* x, float* out, int64_t n) {
  LTB_INITED(); LTB_REQUIRE(x && out && n >= 0, "ltb_sum_static_scratch: bad argument"); LTB_WRITES(out, 1);
  if (n > kStaticSumMaxN)
    return fail(LTB_E_LIMIT, "ltb_sum_static_scratch: %lld elements exceed the limit of %lld", (long long)n, (long long)kStaticSumMaxN);
  LTB_REQUIRE(g.device >= 0 && g.device < kStaticSumMaxDevices, "ltb_sum_static_scratch: device index out of range");
  if (!static_sum_ptr[g.device]) {                        // set-up, once per device
    // A symbol's address belongs to the device that is current in the calling thread, which need not be the context's
    // (another thread of the host may have selected a different GPU): select ours for the look-up and put the caller's back.
    LTB_REQUIRE(!g.capturing, "ltb_sum_static_scratch: the first call on a device does its set-up and must come before a step is recorded");
    int prev = -1;
    LTB_CUDA(cudaGetDevice(&prev));
    if (prev != g.device) LTB_CUDA(cudaSetDevice(g.device));
    float* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&p, static_sum_scratch);
    if (prev != g.device) cudaSetDevice(prev);
    if (e != cudaSuccess || !p) return fail(LTB_E_CUDA, "ltb_sum_static_scratch: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    static_sum_ptr[g.device] = p;
  }
  float* partial = static_sum_ptr[g.device];
  if (n <= (1 << 16)) { LTB_LAUNCH(sum_kernel, 1, 1024, 0, x, out, n, 1.0f, false); return LTB_OK; }
  int blocks = grid_for(n, 1024, 2);                      // the same grid as ltb_sum: the two agree bit for bit
  if (blocks > kStaticSumSlots) blocks = kStaticSumSlots;
  LTB_LAUNCH(sum_kernel, blocks, 1024, 0, x, partial, n, 1.0f, true);
  LTB_LAUNCH(sum_kernel, 1, 1024, 0, (const float*)partial, out, (int64_t)blocks, 1.0f, false);
  return LTB_OK;
}

// softmax / logSoftmax and grads: TensorDslCPU.scala:783-846.
int ltb_softmax(const float* x, float* y, int rows, int cols) {
  LTB_INITED(); LTB_REQUIRE(x && y && rows > 0 && cols > 0, "ltb_softmax: bad argument"); LTB_WRITES(y, (size_t)rows * cols);
  return softmax_issue<0>(x, y, rows, cols);
}
int ltb_log_softmax(const float* x, float* y, int rows, int cols) {
  LTB_INITED(); LTB_REQUIRE(x && y && rows > 0 && cols > 0, "ltb_log_softmax: bad argument"); LTB_WRITES(y, (size_t)rows * cols);
  if (!g.fusion) return softmax_issue<1>(x, y, rows, cols);
  Pending h; h.kind = PEND_LSM; h.x = x; h.y = y; h.N = rows; h.C = cols;      // the negative log likelihood of y may join it
  g.pending = h;
  return LTB_OK;
}
int ltb_softmax_grad(float* dx, const float* y, const float* dy, int rows, int cols) {
  LTB_INITED(); LTB_SETTLE(dx); LTB_SETTLE(dy); LTB_REQUIRE(dx && y && dy && rows > 0 && cols > 0, "ltb_softmax_grad: bad argument"); LTB_WRITES(dx, (size_t)rows * cols);
  return softmax_grad_issue<0>(dx, y, dy, rows, cols);
}
int ltb_log_softmax_grad(float* dx, const float* y, const float* dy, int rows, int cols) {
  LTB_INITED_NOFLUSH(); LTB_REQUIRE(dx && y && dy && rows > 0 && cols > 0, "ltb_log_softmax_grad: bad argument");
  const Pending p = g.pending;
  const int64_t n = (int64_t)rows * cols;
  const bool joins = p.kind == PEND_NLL_GRAD && p.C < 1280 && p.db == dy && p.N == rows && p.C == cols && apart(dx, n, dy, n) && apart(dx, n, p.da, rows) && apart(dx, n, p.d, 1) &&
                     apart(dx, n, p.target, rows) && apart(y, n, dx, n) && apart(y, n, dy, n) && apart(y, n, p.da, rows) && apart(y, n, p.d, 1);
  if (joins) g.pending.kind = PEND_NONE;
  else if (p.kind) { int rc = flush_pending(); if (rc) return rc; }
  LTB_SETTLE(dx); LTB_SETTLE(dy); LTB_WRITES(dx, (size_t)rows * cols);
  return joins ? nll_softmax_grad_issue(p, dx, y) : softmax_grad_issue<1>(dx, y, dy, rows, cols);
}
// nllLoss / nllLoss_grad: TensorDslCPU.scala:1090-1110.
int ltb_nll(const float* x, const int32_t* t, float* out, int rows, int cols) {
  LTB_INITED_NOFLUSH(); LTB_REQUIRE(x && t && out && rows > 0 && cols > 0, "ltb_nll: bad argument"); LTB_WRITES(out, rows);
  const int64_t n = (int64_t)rows * cols;
  if (g.pending.kind == PEND_LSM && g.pending.y == x && g.pending.N == rows && g.pending.C == cols && apart(out, rows, x, n) && apart(out, rows, g.pending.x, n) &&
      apart(out, rows, t, rows) && apart(t, rows, x, n) && apart(g.pending.x, n, x, n)) {
    g.pending.kind = PEND_NLL; g.pending.target = t; g.pending.out = out;                           // their sum or mean may join it
    return LTB_OK;
  }
  if (g.pending.kind) { int rc = flush_pending(); if (rc) return rc; }
  LTB_LAUNCH(nll_kernel, (rows + 127) / 128, 128, 0, x, t, out, rows, cols); return LTB_OK;
}
int ltb_nll_grad(float* dx, const float* dout, const int32_t* t, int rows, int cols) {
  LTB_INITED_NOFLUSH(); LTB_REQUIRE(dx && dout && t && rows > 0 && cols > 0, "ltb_nll_grad: bad argument");
  const int64_t n = (int64_t)rows * cols;
  const bool joins = g.pending.kind == PEND_SUM_GRAD && g.pending.da == dout && g.pending.n == rows && apart(dx, n, dout, rows) && apart(dx, n, g.pending.d, 1) &&
                     apart(t, rows, dx, n) && apart(t, rows, dout, rows) && apart(t, rows, g.pending.d, 1);
  if (!joins && g.pending.kind) { int rc = flush_pending(); if (rc) return rc; }
  LTB_SETTLE(dx); LTB_SETTLE(dout); LTB_WRITES(dx, (size_t)rows * cols);
  if (!joins) return nll_grad_issue(dx, dout, t, rows, cols);
  g.pending.kind = PEND_NLL_GRAD; g.pending.db = dx; g.pending.target = t; g.pending.N = rows; g.pending.C = cols;      // the log-softmax's gradient may join it
  return LTB_OK;
}

// vectorVectorDot / matrixVectorDot and the (1,1), (2,1) cases of dot_grad: TensorDslCPU.scala:135-206.
int ltb_vv_dot(const float* x, const float* y, float* out, int n) {
  LTB_INITED(); LTB_REQUIRE(x && y && out && n > 0, "ltb_vv_dot: bad argument"); LTB_WRITES(out, 1);
  LTB_LAUNCH(dot_kernel, 1, 1024, 0, x, y, out, n); return LTB_OK;
}
int ltb_vv_dot_grad(float* dx, float* dy, const float* x, const float* y, const float* dout, int n) {
  LTB_INITED(); LTB_SETTLE(dx); LTB_SETTLE(dy); LTB_SETTLE(dout); LTB_REQUIRE(x && y && dout && n > 0, "ltb_vv_dot_grad: bad argument"); LTB_WRITES(dx, n); LTB_WRITES(dy, n);
  if (dx) LTB_LAUNCH(axpy_from_scalar_kernel, grid_for(n, 256), 256, 0, dx, y, dout, n);
  if (dy) LTB_LAUNCH(axpy_from_scalar_kernel, grid_for(n, 256), 256, 0, dy, x, dout, n);
  return LTB_OK;
}
}  // extern "C"
namespace ltb {
// One warp per output row: lanes stride over the columns of W0 (and W1), shuffle reduction, lane 0 adds the bias and
// applies the activation.  150 x 150 gates of a TreeLSTM node: 38 blocks of four warps.
__global__ void affine_act_kernel(const float* __restrict__ W0, const float* __restrict__ a, int cols0, const float* __restrict__ W1,
                                  const float* __restrict__ b, int cols1, const float* __restrict__ bias, int act, float* out, int rows) {
  pdl_enter();
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= rows) return;
  float s0 = 0.0f, s1 = 0.0f;
  const float* w = W0 + (int64_t)r * cols0;
  for (int j = lane; j < cols0; j += 32) s0 += w[j] * a[j];
  if (W1) { w = W1 + (int64_t)r * cols1; for (int j = lane; j < cols1; j += 32) s1 += w[j] * b[j]; }
  for (int o = 16; o > 0; o >>= 1) { s0 += __shfl_xor_sync(0xffffffffu, s0, o); s1 += __shfl_xor_sync(0xffffffffu, s1, o); }
  if (lane == 0) {
    float v = (s0 + s1) + bias[r];
    if (act == LTB_TANH) v = tanhf(v); else if (act == LTB_SIGMOID) v = 1.0f / (expf(-v) + 1.0f);
    out[r] = v;
  }
}
// The gradient of the same row: dpre from the saved output, the row of dW0 (dW1) updated in place, the row's share of
// W0^T dpre added atomically to da (db): rows x cols atomic additions on cols addresses, a few microseconds at these sizes.
__global__ void affine_act_grad_kernel(const float* __restrict__ W0, float* dW0, const float* __restrict__ a, float* da, int cols0,
                                       const float* __restrict__ W1, float* dW1, const float* __restrict__ b, float* db, int cols1,
                                       float* dbias, int act, const float* __restrict__ out, const float* __restrict__ dout, int rows) {
  pdl_enter();
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= rows) return;
  const float y = out[r];
  float dpre = dout[r];
  if (act == LTB_TANH) dpre *= 1.0f - y * y; else if (act == LTB_SIGMOID) dpre *= (1.0f - y) * y;     // TD.scala:789-809
  if (lane == 0) dbias[r] += dpre;
  {
    const float* w = W0 + (int64_t)r * cols0; float* dw = dW0 + (int64_t)r * cols0;
    for (int j = lane; j < cols0; j += 32) { dw[j] += dpre * a[j]; if (da) atomicAdd(da + j, w[j] * dpre); }
  }
  if (W1) {
    const float* w = W1 + (int64_t)r * cols1; float* dw = dW1 + (int64_t)r * cols1;
    for (int j = lane; j < cols1; j += 32) { dw[j] += dpre * b[j]; if (db) atomicAdd(db + j, w[j] * dpre); }
  }
}
}  // namespace ltb
extern "C" {
}  // extern "C"
namespace ltb {
__global__ void lstm_cell_kernel(const float* __restrict__ i, const float* __restrict__ u, const float* __restrict__ fl, const float* __restrict__ cl,
                                 const float* __restrict__ fr, const float* __restrict__ cr, const float* __restrict__ o, float* c, float* tc, float* h, int n) {
  pdl_enter();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  float v = i[k] * u[k];
  if (fl) { v = v + fl[k] * cl[k]; v = v + fr[k] * cr[k]; }
  const float t = tanhf(v);
  c[k] = v; tc[k] = t; h[k] = o[k] * t;
}
__global__ void lstm_cell_grad_kernel(const float* __restrict__ i, float* di, const float* __restrict__ u, float* du, const float* __restrict__ fl, float* dfl,
                                      const float* __restrict__ cl, float* dcl, const float* __restrict__ fr, float* dfr, const float* __restrict__ cr, float* dcr,
                                      const float* __restrict__ o, float* d_o, const float* __restrict__ tc, const float* __restrict__ dc,
                                      const float* __restrict__ dh, int n) {
  pdl_enter();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const float t = tc[k], g = dh[k];
  d_o[k] += g * t;
  const float dct = dc[k] + (g * o[k]) * (1.0f - t * t);
  di[k] += dct * u[k]; du[k] += dct * i[k];
  if (fl) { dfl[k] += dct * cl[k]; dcl[k] += dct * fl[k]; dfr[k] += dct * cr[k]; dcr[k] += dct * fr[k]; }
}
}  // namespace ltb
extern "C" {
int ltb_lstm_cell(const float* i, const float* u, const float* fl, const float* cl, const float* fr, const float* cr,
                  const float* o, float* c, float* tc, float* h, int n) {
  LTB_INITED();
  LTB_REQUIRE(i && u && o && c && tc && h && n > 0, "ltb_lstm_cell: bad argument"); LTB_WRITES(c, n); LTB_WRITES(tc, n); LTB_WRITES(h, n);
  LTB_REQUIRE((fl && cl && fr && cr) || (!fl && !cl && !fr && !cr), "ltb_lstm_cell: the four child operands go together");
  LTB_LAUNCH(lstm_cell_kernel, (unsigned)ceil_div(n, 128), 128, 0, i, u, fl, cl, fr, cr, o, c, tc, h, n);
  return LTB_OK;
}
int ltb_lstm_cell_grad(const float* i, float* di, const float* u, float* du, const float* fl, float* dfl, const float* cl, float* dcl,
                       const float* fr, float* dfr, const float* cr, float* dcr, const float* o, float* d_o,
                       const float* tc, const float* dc, const float* dh, int n) {
  LTB_INITED(); LTB_SETTLE(di); LTB_SETTLE(du); LTB_SETTLE(dfl); LTB_SETTLE(dcl); LTB_SETTLE(dfr); LTB_SETTLE(dcr); LTB_SETTLE(d_o); LTB_SETTLE(dc); LTB_SETTLE(dh);
  LTB_REQUIRE(i && di && u && du && o && d_o && tc && dc && dh && n > 0, "ltb_lstm_cell_grad: bad argument"); LTB_WRITES(di, n); LTB_WRITES(du, n); LTB_WRITES(dfl, n); LTB_WRITES(dcl, n); LTB_WRITES(dfr, n); LTB_WRITES(dcr, n); LTB_WRITES(d_o, n);
  LTB_REQUIRE((fl && dfl && cl && dcl && fr && dfr && cr && dcr) || (!fl && !dfl && !cl && !dcl && !fr && !dfr && !cr && !dcr),
              "ltb_lstm_cell_grad: the child operands and their gradients go together");
  LTB_LAUNCH(lstm_cell_grad_kernel, (unsigned)ceil_div(n, 128), 128, 0, i, di, u, du, fl, dfl, cl, dcl, fr, dfr, cr, dcr, o, d_o, tc, dc, dh, n);
  return LTB_OK;
}
}  // extern "C"
namespace ltb {
__device__ __forceinline__ float act_fwd(int act, float v) { return act == LTB_TANH ? tanhf(v) : act == LTB_SIGMOID ? 1.0f / (expf(-v) + 1.0f) : v; }
__device__ __forceinline__ float act_slope(int act, float y) { return act == LTB_TANH ? 1.0f - y * y : act == LTB_SIGMOID ? (1.0f - y) * y : 1.0f; }
// A thread per output (b, j): the lanes of a warp share b (x is a broadcast) and read consecutive j of a weight row.
__global__ void affine_act_rows_kernel(const float* __restrict__ x0, const float* __restrict__ W0, int cols0, const float* __restrict__ x1,
                                       const float* __restrict__ W1, int cols1, const float* __restrict__ bias, int act, float* out, int batch, int width) {
  pdl_enter();
  const int j = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y;
  if (j >= width) return;
  float s0 = 0.0f, s1 = 0.0f;
  const float* xr = x0 + (int64_t)b * cols0;
#pragma unroll 4
  for (int c = 0; c < cols0; ++c) s0 += xr[c] * W0[(int64_t)c * width + j];
  if (W1) {
    xr = x1 + (int64_t)b * cols1;
#pragma unroll 4
    for (int c = 0; c < cols1; ++c) s1 += xr[c] * W1[(int64_t)c * width + j];
  }
  out[(int64_t)b * width + j] = act_fwd(act, (s0 + s1) + bias[j]);
}
// The whole gradient in one launch, two kinds of blocks.  blockIdx.y < cols0 + cols1 + 1: row c of [dW0; dW1; dbias], a
// thread per column j walks the batch (dpre is recomputed from out and dout: two coalesced loads, nothing stored).
// The blocks after those: input gradients, a thread per (b, c) walks j.
__global__ void affine_act_rows_grad_kernel(const float* __restrict__ x0, float* dx0, const float* __restrict__ W0, float* dW0, int cols0,
                                            const float* __restrict__ x1, float* dx1, const float* __restrict__ W1, float* dW1, int cols1,
                                            float* dbias, int act, const float* __restrict__ out, const float* __restrict__ dout, int batch, int width) {
  pdl_enter();
  const int wrows = cols0 + cols1 + 1;
  if ((int)blockIdx.y < wrows) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (j >= width) return;
    const float* xs; int ld, cc; float* dst;
    if (c < cols0) { xs = x0; ld = cols0; cc = c; dst = dW0 + (int64_t)c * width + j; }
    else if (c < cols0 + cols1) { xs = x1; ld = cols1; cc = c - cols0; dst = dW1 + (int64_t)(c - cols0) * width + j; }
    else { xs = nullptr; ld = 0; cc = 0; dst = dbias + j; }
    float s = 0.0f;
#pragma unroll 4
    for (int b = 0; b < batch; ++b) {
      const float dpre = dout[(int64_t)b * width + j] * act_slope(act, out[(int64_t)b * width + j]);
      s += xs ? xs[(int64_t)b * ld + cc] * dpre : dpre;
    }
    *dst += s;
  } else {
    // input gradients: flat index over dx0 (batch x cols0, when wanted) then dx1 (batch x cols1, when wanted)
    const int64_t n0 = dx0 ? (int64_t)batch * cols0 : 0, n1 = dx1 ? (int64_t)batch * cols1 : 0;
    const int64_t t = ((int64_t)(blockIdx.y - wrows) * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n0 + n1) return;
    const bool first = t < n0;
    const int64_t u = first ? t : t - n0;
    const int ld = first ? cols0 : cols1;
    const int b = (int)(u / ld), c = (int)(u - (int64_t)b * ld);
    const float* w = (first ? W0 : W1) + (int64_t)c * width;
    const float* o = out + (int64_t)b * width; const float* d = dout + (int64_t)b * width;
    float s = 0.0f;
#pragma unroll 4
    for (int j = 0; j < width; ++j) s += d[j] * act_slope(act, o[j]) * w[j];
    (first ? dx0 : dx1)[u] += s;
  }
}
}  // namespace ltb
extern "C" {
int ltb_affine_act_rows(const float* x0, const float* W0, int cols0, const float* x1, const float* W1, int cols1, const float* bias,
                        int act, float* out, int batch, int width) {
  LTB_INITED();
  LTB_REQUIRE(x0 && W0 && bias && out && cols0 > 0 && batch > 0 && batch <= 65535 && width > 0 && (x1 == nullptr) == (W1 == nullptr) && (!W1 || cols1 > 0),
              "ltb_affine_act_rows: bad argument");
  LTB_WRITES(out, (size_t)batch * width);
  LTB_REQUIRE(act == -1 || act == LTB_TANH || act == LTB_SIGMOID, "ltb_affine_act_rows: activation must be tanh, sigmoid or -1");
  LTB_LAUNCH(affine_act_rows_kernel, dim3((unsigned)ceil_div(width, 128), batch), 128, 0, x0, W0, cols0, x1, W1, W1 ? cols1 : 0, bias, act, out, batch, width);
  return LTB_OK;
}
int ltb_affine_act_rows_grad(const float* x0, float* dx0, const float* W0, float* dW0, int cols0, const float* x1, float* dx1,
                             const float* W1, float* dW1, int cols1, float* dbias, int act, const float* out, const float* dout,
                             int batch, int width) {
  LTB_INITED(); LTB_SETTLE(dx0); LTB_SETTLE(dW0); LTB_SETTLE(dx1); LTB_SETTLE(dW1); LTB_SETTLE(dbias); LTB_SETTLE(dout);
  LTB_REQUIRE(x0 && W0 && dW0 && dbias && out && dout && cols0 > 0 && batch > 0 && width > 0, "ltb_affine_act_rows_grad: bad argument");
  LTB_WRITES(dx0, (size_t)batch * cols0); LTB_WRITES(dW0, (size_t)cols0 * width); LTB_WRITES(dx1, (size_t)batch * cols1); LTB_WRITES(dW1, (size_t)cols1 * width); LTB_WRITES(dbias, width);
  LTB_REQUIRE((x1 == nullptr) == (W1 == nullptr) && (W1 == nullptr) == (dW1 == nullptr) && (!W1 || cols1 > 0) && (W1 || !dx1),
              "ltb_affine_act_rows_grad: x1, W1 and dW1 go together");
  LTB_REQUIRE(act == -1 || act == LTB_TANH || act == LTB_SIGMOID, "ltb_affine_act_rows_grad: activation must be tanh, sigmoid or -1");
  const int c1 = W1 ? cols1 : 0;
  const unsigned gx = (unsigned)ceil_div(width, 128);
  const int64_t inputs = (dx0 ? (int64_t)batch * cols0 : 0) + (dx1 ? (int64_t)batch * c1 : 0);
  const int64_t extra = ceil_div(inputs, (int64_t)gx * 128);
  LTB_REQUIRE(cols0 + c1 + 1 + extra <= 65535, "ltb_affine_act_rows_grad: too large for one launch");
  LTB_LAUNCH(affine_act_rows_grad_kernel, dim3(gx, (unsigned)(cols0 + c1 + 1 + extra)), 128, 0, x0, dx0, W0, dW0, cols0, x1, dx1, W1, dW1, c1,
             dbias, act, out, dout, batch, width);
  return LTB_OK;
}
int ltb_affine_act(const float* W0, const float* a, int cols0, const float* W1, const float* b, int cols1, const float* bias,
                   int act, float* out, int rows) {
  LTB_INITED();
  LTB_REQUIRE(W0 && a && bias && out && rows > 0 && cols0 > 0 && (W1 == nullptr) == (b == nullptr) && (!W1 || cols1 > 0), "ltb_affine_act: bad argument"); LTB_WRITES(out, rows);
  LTB_REQUIRE(act == -1 || act == LTB_TANH || act == LTB_SIGMOID, "ltb_affine_act: activation must be tanh, sigmoid or -1");
  LTB_LAUNCH(affine_act_kernel, (unsigned)ceil_div(rows, 4), 128, 0, W0, a, cols0, W1, b, cols1, bias, act, out, rows);
  return LTB_OK;
}
int ltb_affine_act_grad(const float* W0, float* dW0, const float* a, float* da, int cols0, const float* W1, float* dW1,
                        const float* b, float* db, int cols1, float* dbias, int act, const float* out, const float* dout, int rows) {
  LTB_INITED(); LTB_SETTLE(dW0); LTB_SETTLE(da); LTB_SETTLE(dW1); LTB_SETTLE(db); LTB_SETTLE(dbias); LTB_SETTLE(dout);
  LTB_REQUIRE(W0 && dW0 && a && dbias && out && dout && rows > 0 && cols0 > 0, "ltb_affine_act_grad: bad argument"); LTB_WRITES(dW0, (size_t)rows * cols0); LTB_WRITES(da, cols0); LTB_WRITES(dW1, (size_t)rows * cols1); LTB_WRITES(db, cols1); LTB_WRITES(dbias, rows);
  LTB_REQUIRE((W1 == nullptr) == (b == nullptr) && (W1 == nullptr) == (dW1 == nullptr) && (!W1 || cols1 > 0), "ltb_affine_act_grad: W1, dW1 and b go together");
  LTB_REQUIRE(act == -1 || act == LTB_TANH || act == LTB_SIGMOID, "ltb_affine_act_grad: activation must be tanh, sigmoid or -1");
  LTB_LAUNCH(affine_act_grad_kernel, (unsigned)ceil_div(rows, 4), 128, 0, W0, dW0, a, da, cols0, W1, dW1, b, db, cols1, dbias, act, out, dout, rows);
  return LTB_OK;
}
int ltb_mv_dot(const float* a, const float* x, float* out, int m, int k) {
  LTB_INITED(); LTB_REQUIRE(a && x && out && m > 0 && k > 0, "ltb_mv_dot: bad argument"); LTB_WRITES(out, m);
  LTB_LAUNCH(gemv_rows_kernel<false>, (unsigned)ceil_div((int64_t)m * 32, 256), 256, 0, a, x, out, m, k); return LTB_OK;
}
int ltb_add_cartesian(float* da, const float* y, const float* dout, int m, int k) {
  LTB_INITED(); LTB_SETTLE(da); LTB_SETTLE(dout); LTB_REQUIRE(da && y && dout && m > 0 && k > 0, "ltb_add_cartesian: bad argument"); LTB_WRITES(da, (size_t)m * k);
  LTB_LAUNCH(outer_acc_kernel, grid_for((int64_t)m * k, 256), 256, 0, da, y, dout, m, k); return LTB_OK;
}
int ltb_add_composition(float* dx, const float* a, const float* dout, int m, int k) {
  LTB_INITED(); LTB_SETTLE(dx); LTB_SETTLE(dout); LTB_REQUIRE(dx && a && dout && m > 0 && k > 0, "ltb_add_composition: bad argument"); LTB_WRITES(dx, k);
  LTB_LAUNCH(gemv_cols_kernel, (k + 127) / 128, 128, 0, a, dout, dx, m, k); return LTB_OK;
}

}  // extern "C"
