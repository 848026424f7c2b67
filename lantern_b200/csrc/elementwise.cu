// Elementwise, broadcasting, activation, dropout and optimizer kernels: HBM-streaming work.
//
// These replace the reference's fixed <<<28,512>>> grid-stride kernels (src/main/scala/lantern/DslAPI.scala:475-842),
// its staging-time generated broadcast kernels (TensorDslCudnn.scala:153-282), cublasSgeam (TensorDslCublas.scala:318-373)
// and cudnnActivation*/cudnnAddTensor (TensorDslCudnn.scala:476-512, 1349-1429).  Semantics follow the CPU backend
// (TensorDslCPU.scala), cited per entry point.  Design: 128-bit loads/stores whenever every pointer is 16-byte
// aligned, grid sized to the SM count, one pass over memory per op.
#include <cooperative_groups.h>

#include <vector>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace ltb {

// ---- op functors ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float bin_op(int op, float a, float b) {
  switch (op) { case LTB_ADD: return a + b; case LTB_SUB: return a - b; case LTB_MUL: return a * b; default: return a / b; }
}
__device__ __forceinline__ float un_op(int op, float v) {
  switch (op) {
    case LTB_RELU: return v < 0.0f ? 0.0f : v;                    // TensorDslCPU.scala:711-720
    case LTB_TANH: return tanhf(v);
    case LTB_SIGMOID: return 1.0f / (expf(-v) + 1.0f);            // TensorDslCPU.scala:760
    case LTB_EXP: return expf(v);
    case LTB_LOG: return logf(v);
    case LTB_SQRT: return sqrtf(v);
    default: return v * v;
  }
}
// dx += g(x, y, dy): TensorDslCPU.scala:722-781 with the fused helpers of TD.scala:789-809.
__device__ __forceinline__ float un_grad(int op, float x, float y, float dy) {
  switch (op) {
    case LTB_RELU: return x < 0.0f ? 0.0f : dy;
    case LTB_TANH: return (1.0f - y * y) * dy;
    case LTB_SIGMOID: return (1.0f - y) * y * dy;
    case LTB_EXP: return dy * y;
    case LTB_LOG: return dy / x;
    case LTB_SQRT: return dy / y / 2.0f;
    default: return dy * x * 2.0f;
  }
}

// ---- generic vectorised map over up to three inputs -------------------------------------------------------------
// F: float f(float a, float b, float c); a/b/c may be null (then 0 is passed). out may alias any input.
// U items of a thread in flight, bound by memory or, in the L2, by the number of loads under way.  Four of them (1 / 4, us): what lies in the L2 gains from 3.6 million
// elements on (ReLU 3.7 million 4.2 / 3.8, 5.6 million 6.1 / 4.6, 10.3 million 11.3 / 7.6, sum 5.6 million 6.2 / 5.2, ReLU gradient 5.5 / 5.1), fewer leave threads
// without work (sum 2.5 million 3.0 / 3.4, 1.3 million 2.2 / 3.1; with three inputs 2.5 million 3.6 / 3.4, 1.3 million 2.4 / 2.9).  From memory a map of one input gains (25.7 million, ReLU 32.0 / 31.6, tanh 33.3 / 31.7; 100 million
// 121 / 118 and 128 / 117), one of several loses (sum 44.5 / 45.7, 100 million 170 / 173): those go four at a time while their tensors fit the L2 (in place, 10.3
// million, 11.5 / 9.5), which costs them 1 to 2 % if they happen not to be there.
constexpr int64_t kMapL2Bytes = (int64_t)126 << 20;
template <int NIN, int U, class F>
__global__ void __launch_bounds__(256) map_vec4(const float* __restrict__ a, const float* __restrict__ b, const float* __restrict__ c,
                                                float* out, int64_t n4, F f) {
  pdl_enter();
  const int64_t i0 = (int64_t)blockIdx.x * 256 * U + threadIdx.x;
  float4 va[U], vb[U], vc[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t i = i0 + 256 * u;
    if (i >= n4) break;
    va[u] = reinterpret_cast<const float4*>(a)[i];
    vb[u] = NIN > 1 ? reinterpret_cast<const float4*>(b)[i] : make_float4(0, 0, 0, 0);
    vc[u] = NIN > 2 ? reinterpret_cast<const float4*>(c)[i] : make_float4(0, 0, 0, 0);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t i = i0 + 256 * u;
    if (i >= n4) break;
    float4 r;
    r.x = f(va[u].x, vb[u].x, vc[u].x); r.y = f(va[u].y, vb[u].y, vc[u].y); r.z = f(va[u].z, vb[u].z, vc[u].z); r.w = f(va[u].w, vb[u].w, vc[u].w);
    reinterpret_cast<float4*>(out)[i] = r;
  }
}
template <int NIN, class F>
__global__ void map_scalar(const float* a, const float* b, const float* c, float* out, int64_t begin, int64_t n, F f) {
  pdl_enter();
  int64_t i = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) out[i] = f(a[i], NIN > 1 ? b[i] : 0.0f, NIN > 2 ? c[i] : 0.0f);
}
template <int NIN, class F>
int launch_map(const float* a, const float* b, const float* c, float* out, int64_t n, F f) {
  if (n <= 0) return LTB_OK;
  bool vec = aligned16(a) && aligned16(out) && (NIN < 2 || aligned16(b)) && (NIN < 3 || aligned16(c));
  int64_t n4 = vec ? n / 4 : 0;
  LTB_REQUIRE(n4 <= (int64_t)256 * 0x7fffffff, "elementwise operation on too many elements");
  const bool in_place = out == a || (NIN > 1 && out == b) || (NIN > 2 && out == c);
  const bool four = n4 > (int64_t)g.sm_count * (NIN > 2 ? 4096 : 6144) && (NIN == 1 || n4 * 16 * (NIN + (in_place ? 0 : 1)) <= kMapL2Bytes);
  if (four) LTB_LAUNCH((map_vec4<NIN, 4, F>), (unsigned)ceil_div(n4, 1024), 256, 0, a, b, c, out, n4, f);
  else if (n4 > 0) LTB_LAUNCH((map_vec4<NIN, 1, F>), (unsigned)ceil_div(n4, 256), 256, 0, a, b, c, out, n4, f);
  if (n4 * 4 < n) LTB_LAUNCH((map_scalar<NIN, F>), grid_for(n - n4 * 4, 256), 256, 0, a, b, c, out, n4 * 4, n, f);
  return LTB_OK;
}

// ---- fill -----------------------------------------------------------------------------------------------------
__global__ void fill_kernel(float* x, float v, int64_t n) {
  pdl_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) x[i] = v;
}
__global__ void fill_bias_kernel(float* out, const float* __restrict__ bias, int c, int64_t inner, int64_t n) {
  pdl_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) out[i] = bias[(i / inner) % c];
}

// ---- general broadcasting (rank <= 4) --------------------------------------------------------------------------
struct Bcast { int shape[4]; int64_t sa[4]; int64_t sb[4]; };

__device__ __forceinline__ void bcast_index(const Bcast& p, int64_t r, int64_t& ia, int64_t& ib) {
  int64_t i3 = r % p.shape[3]; r /= p.shape[3];
  int64_t i2 = r % p.shape[2]; r /= p.shape[2];
  int64_t i1 = r % p.shape[1]; int64_t i0 = r / p.shape[1];
  ia = i0 * p.sa[0] + i1 * p.sa[1] + i2 * p.sa[2] + i3 * p.sa[3];
  ib = i0 * p.sb[0] + i1 * p.sb[1] + i2 * p.sb[2] + i3 * p.sb[3];
}
__global__ void bcast_binary_kernel(int op, const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, Bcast p, int64_t n) {
  pdl_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) { int64_t ia, ib; bcast_index(p, i, ia, ib); out[i] = bin_op(op, a[ia], b[ib]); }
}
// Gradient of a broadcasting binary op: the operand that was broadcast receives a reduction, done with float atomics;
// the other one is a plain read-modify-write (TensorDslCPU.scala:246-263 and 300-337 for op1/op2).
__global__ void bcast_binary_grad_kernel(int op, const float* __restrict__ a, float* da, bool a_red, const float* __restrict__ b, float* db,
                                         bool b_red, const float* __restrict__ dout, Bcast p, int64_t n) {
  pdl_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    int64_t ia, ib; bcast_index(p, i, ia, ib);
    float x = a[ia], y = b[ib], c = dout[i], g1, g2;
    switch (op) {
      case LTB_ADD: g1 = c; g2 = c; break;
      case LTB_SUB: g1 = c; g2 = 0.0f - c; break;
      case LTB_MUL: g1 = c * y; g2 = c * x; break;
      default: g1 = c / y; g2 = -1.0f * x * c / (y * y); break;
    }
    if (da) { if (a_red) atomicAdd(da + ia, g1); else da[ia] += g1; }
    if (db) { if (b_red) atomicAdd(db + ib, g2); else db[ib] += g2; }
  }
}
// x = x (op) y where y is broadcast over x (no element of x is written twice).
__global__ void bcast_inplace_kernel(int op, float* x, const float* __restrict__ y, Bcast p, int64_t n) {
  pdl_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) { int64_t ix, iy; bcast_index(p, i, ix, iy); x[ix] = bin_op(op, x[ix], y[iy]); }
}
// x = x (op) y where y is REDUCED into x: one warp per element of x walks, in row-major order of the broadcast
// shape, the y elements that map onto it (TensorDslCPU.scala:265-279).  ADD/SUB use a shuffle tree; MUL/DIV fold
// sequentially in lane 0 to keep the reference's order.
struct Reduce { int xshape[4]; int rshape[4]; int64_t sy[4]; };
__global__ void reduce_inplace_kernel(int op, float* x, const float* __restrict__ y, Reduce p, int64_t nx, int64_t per) {
  pdl_enter();
  int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (warp >= nx) return;
  int xi[4]; int64_t r = warp;
  for (int d = 3; d >= 0; --d) { xi[d] = (int)(r % p.xshape[d]); r /= p.xshape[d]; }
  int red[4]; for (int d = 0; d < 4; ++d) red[d] = p.xshape[d] == 1 ? p.rshape[d] : 1;
  auto y_at = [&](int64_t j) {
    int64_t off = 0;
    for (int d = 3; d >= 0; --d) { int k = (int)(j % red[d]); j /= red[d]; off += (int64_t)(p.xshape[d] == 1 ? k : xi[d]) * p.sy[d]; }
    return y[off];
  };
  if (op == LTB_ADD || op == LTB_SUB) {
    float s = 0.0f;
    for (int64_t j = lane; j < per; j += 32) s += y_at(j);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) x[warp] = op == LTB_ADD ? x[warp] + s : x[warp] - s;
  } else if (lane == 0) {
    float v = x[warp];
    for (int64_t j = 0; j < per; ++j) v = bin_op(op, v, y_at(j));
    x[warp] = v;
  }
}

// ---- one operand a vector along one (merged) dimension: biases and their gradients ------------------------------------------------
// Most broadcasts pair a full tensor with a vector: full[outer][mid][inner] and v[mid] (a row of bias: inner 1; a channel: inner =
// pixels).  The general kernels above pay four 64-bit divisions per element and, reducing, let a warp gather one element of x with a
// stride; these pay one 32-bit division per four elements, and the reductions read whole 128-byte rows.  Measured on 8192 x 1000:
// adding the row bias 51 -> 12 us, its gradient 223 -> 11 us (copy bandwidth: 10 and 5 us).
template <int OP, int VEC>
__global__ void bcast_mid_kernel(float* x, const float* __restrict__ v, unsigned n, unsigned inner, unsigned mid) {
  pdl_enter();
  // VEC 1: a thread per element; 4: four elements of one v[m] (inner a multiple of 4; inner in units of 4); 5: four consecutive v (inner 1; mid in units of 4)
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned m = (VEC == 5 ? i : i / inner) % mid;
    if (VEC == 1) x[i] = bin_op(OP, x[i], v[m]);
    else {
      float4 a = reinterpret_cast<float4*>(x)[i];
      const float4 b = VEC == 5 ? reinterpret_cast<const float4*>(v)[m] : make_float4(v[m], v[m], v[m], v[m]);
      a.x = bin_op(OP, a.x, b.x); a.y = bin_op(OP, a.y, b.y); a.z = bin_op(OP, a.z, b.z); a.w = bin_op(OP, a.w, b.w);
      reinterpret_cast<float4*>(x)[i] = a;
    }
  }
}
template <int OP>
static int bcast_mid(float* x, const float* v, int64_t n, int64_t inner, int64_t mid) {
  const bool al = aligned16(x);
  if (al && inner % 4 == 0) LTB_LAUNCH((bcast_mid_kernel<OP, 4>), grid_for(n / 4, 256), 256, 0, x, v, (unsigned)(n / 4), (unsigned)(inner / 4), (unsigned)mid);
  else if (al && inner == 1 && mid % 4 == 0 && aligned16(v)) LTB_LAUNCH((bcast_mid_kernel<OP, 5>), grid_for(n / 4, 256), 256, 0, x, v, (unsigned)(n / 4), 1u, (unsigned)(mid / 4));
  else LTB_LAUNCH((bcast_mid_kernel<OP, 1>), grid_for(n, 256), 256, 0, x, v, (unsigned)n, (unsigned)inner, (unsigned)mid);
  return LTB_OK;
}
// x[m] += sign * sum over outer of y[outer][mid] (inner 1).  A CTA of sixteen warps owns 32 columns, a warp reads whole rows of them; a
// cluster of up to eight CTAs shares the rows, and the sums meet in warp order, then in CTA order: the same bits on every run.
constexpr int kColWarps = 16;
__global__ void __launch_bounds__(kColWarps * 32) reduce_cols_kernel(float* x, const float* __restrict__ y, int64_t rows, int mid, float sign, int cta_per_col) {
  pdl_enter();
  __shared__ float part[kColWarps][32];
  __shared__ float total[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rank = blockIdx.x % cta_per_col;
  const int m = (int)(blockIdx.x / cta_per_col) * 32 + lane;
  float s = 0.0f;
  if (m < mid) {
    const int64_t step = (int64_t)cta_per_col * kColWarps;
    int64_t r = (int64_t)rank * kColWarps + warp;
    const float* p = y + r * mid + m;
    for (; r + 7 * step < rows; r += 8 * step) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = p[u * step * mid];
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
      p += 8 * step * mid;
    }
    for (; r < rows; r += step) { s += *p; p += step * mid; }
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp == 0) {
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < kColWarps; ++w) t += part[w][lane];
    total[lane] = t;
  }
  if (cta_per_col > 1) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (rank == 0 && warp == 0) {
      float t = 0.0f;
      for (int z = 0; z < cta_per_col; ++z) t += *cluster.map_shared_rank(&total[lane], z);
      if (m < mid) x[m] += sign * t;
    }
    cluster.sync();                                      // nobody leaves while its sums may still be read
  } else if (warp == 0 && m < mid) x[m] += sign * total[lane];
}
// x[m] += sign * sum over outer and inner of y[outer][mid][inner]: a CTA per m.
template <int VEC>
__global__ void __launch_bounds__(256) reduce_mid_kernel(float* x, const float* __restrict__ y, int64_t outer, int mid, int inner, float sign) {
  pdl_enter();
  __shared__ float part[8];
  const int m = blockIdx.x;
  const int per = inner / VEC;
  float s = 0.0f;
  const int64_t items = outer * per;
  for (int64_t j = threadIdx.x; j < items; j += 256) {
    const int64_t o = outer == 1 ? 0 : j / per; const int i = (int)(j - o * per);
    const float* p = y + (o * mid + m) * inner;
    if (VEC == 4) { const float4 v = reinterpret_cast<const float4*>(p)[i]; s += (v.x + v.y) + (v.z + v.w); }
    else s += p[i];
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += part[w];
    x[m] += sign * t;
  }
}
static int reduce_mid(float* x, const float* y, int64_t outer, int64_t mid, int64_t inner, float sign) {
  if (inner == 1) {
    const int tiles = (int)ceil_div(mid, 32);
    int cta = 1;                                         // CTAs per 32 columns: about two per SM in all, sixteen rows each at least
    while (cta < 8 && (int64_t)tiles * cta * 2 <= 2 * g.sm_count && outer >= (int64_t)cta * 2 * 2 * kColWarps) cta *= 2;
    LTB_LAUNCH_CLUSTER(reduce_cols_kernel, dim3((unsigned)(tiles * cta)), kColWarps * 32, cta, x, y, outer, (int)mid, sign, cta);
    return LTB_OK;
  }
  if (aligned16(y) && inner % 4 == 0) LTB_LAUNCH(reduce_mid_kernel<4>, (unsigned)mid, 256, 0, x, y, outer, (int)mid, (int)inner, sign);
  else LTB_LAUNCH(reduce_mid_kernel<1>, (unsigned)mid, 256, 0, x, y, outer, (int)mid, (int)inner, sign);
  return LTB_OK;
}

// ---- transpose-aware geam --------------------------------------------------------------------------------------
__global__ void geam_kernel(const float* __restrict__ x, int tx, float alpha, const float* __restrict__ y, int ty, float beta,
                            float* out, int rows, int cols) {
  pdl_enter();
  int64_t n = (int64_t)rows * cols;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    int r = (int)(i / cols), c = (int)(i % cols);
    float xv = tx ? x[(int64_t)c * rows + r] : x[i];
    float yv = ty ? y[(int64_t)c * rows + r] : y[i];
    out[i] = xv * alpha + yv * beta;
  }
}
// 32x32 shared-memory tile transpose; ACC adds into the destination (trans_grad).
template <bool ACC>
__global__ void transpose_kernel(const float* __restrict__ in, float* out, int rows, int cols) {
  pdl_enter();
  __shared__ float tile[32][33];
  int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += 8) {
    int r = by + j, c = bx + threadIdx.x;
    if (r < rows && c < cols) tile[j][threadIdx.x] = in[(int64_t)r * cols + c];
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += 8) {
    int r = bx + j, c = by + threadIdx.x;   // out is [cols, rows]
    if (r < cols && c < rows) { if (ACC) out[(int64_t)r * rows + c] += tile[threadIdx.x][j]; else out[(int64_t)r * rows + c] = tile[threadIdx.x][j]; }
  }
}

// ---- multi-tensor SGD -------------------------------------------------------------------------------------------
struct SgdChunk { float* x; float* d; int64_t n; };
__global__ void sgd_multi_kernel(const SgdChunk* __restrict__ chunks, float lr) {
  pdl_enter();
  SgdChunk c = chunks[blockIdx.y];
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < c.n; i += stride) { c.x[i] = c.x[i] * 1.0f + c.d[i] * (-1.0f * lr); c.d[i] = 0.0f; }
}
// x -= lr*d ; d = 0 in one pass (NNModule.scala:279-285: geam(x,1,d,-lr) then clear_grad): 16 B per parameter.
__global__ void sgd_vec4_kernel(float* x, float* d, float neg_lr, int64_t n4) {
  pdl_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  const float4 z = make_float4(0, 0, 0, 0);
  for (; i < n4; i += stride) {
    float4 xv = reinterpret_cast<float4*>(x)[i], dv = reinterpret_cast<float4*>(d)[i];
    xv.x = xv.x * 1.0f + dv.x * neg_lr; xv.y = xv.y * 1.0f + dv.y * neg_lr; xv.z = xv.z * 1.0f + dv.z * neg_lr; xv.w = xv.w * 1.0f + dv.w * neg_lr;
    reinterpret_cast<float4*>(x)[i] = xv; reinterpret_cast<float4*>(d)[i] = z;
  }
}
__global__ void sgd_scalar_kernel(float* x, float* d, float neg_lr, int64_t begin, int64_t n) {
  pdl_enter();
  int64_t i = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) { x[i] = x[i] * 1.0f + d[i] * neg_lr; d[i] = 0.0f; }
}
__global__ void adagrad_kernel(float* x, float* d, float* h, float lr, float clip, int descent, int64_t n) {
  pdl_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {      // TensorDslCPU.scala:1217-1230
    float t = d[i]; if (t > clip) t = clip; if (t < -clip) t = -clip;
    float hv = h[i] + t * t; h[i] = hv;
    float upd = lr * t / sqrtf(hv + 1e-8f);
    x[i] = descent ? x[i] - upd : x[i] + upd;
    d[i] = 0.0f;
  }
}
__global__ void momentum_kernel(float* x, float* d, float* m, float lr, float mu, float clip, int nesterov, int descent, int64_t n) {
  pdl_enter();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {      // TensorDslCPU.scala:1232-1246
    float t = d[i]; if (t > clip) t = clip; if (t < -clip) t = -clip;
    float mv = m[i] * mu + t; m[i] = mv;
    t = nesterov ? t + mu * mv : mv;
    x[i] = descent ? x[i] - lr * t : x[i] + lr * t;
    d[i] = 0.0f;
  }
}

// Concatenation of up to four pieces [outer][len_k] into [outer][total] (GRAD false) or the gradient back into them: one launch, a thread
// per VEC floats of the whole.  Pieces of the gradient may be missing (null), and those of `fresh` are written instead of added into.
constexpr int kPieces = 4;
struct Pieces { float* p[kPieces]; unsigned len[kPieces], off[kPieces]; int n; unsigned fresh; };
template <bool GRAD, int VEC>
__global__ void concat_kernel(float* whole, const Pieces q, unsigned total, unsigned n) {
  pdl_enter();
  // lengths and offsets in units of VEC floats
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned r = i / total, j = i - r * total;
    int k = 0;
#pragma unroll
    for (int u = 1; u < kPieces; ++u) if (u < q.n && j >= q.off[u]) k = u;
    float* base = q.p[k];
    if (GRAD && !base) continue;
    const size_t at = (size_t)r * q.len[k] + (j - q.off[k]);
    if (VEC == 4) {
      if (!GRAD) reinterpret_cast<float4*>(whole)[i] = reinterpret_cast<const float4*>(base)[at];
      else {
        float4 v = reinterpret_cast<const float4*>(whole)[i];
        if (!(q.fresh >> k & 1)) { const float4 o = reinterpret_cast<const float4*>(base)[at]; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
        reinterpret_cast<float4*>(base)[at] = v;
      }
    } else if (!GRAD) whole[i] = base[at];
    else base[at] = q.fresh >> k & 1 ? whole[i] : base[at] + whole[i];
  }
}
// Issues the pieces [first, first + n) of `total` floats per row; the whole must have fewer than 2^31 elements.
template <bool GRAD>
static int concat_issue(float* whole, float* const* pieces, const int64_t* len, int n, int64_t total, int64_t outer, unsigned fresh) {
  Pieces q; q.n = n; q.fresh = fresh;
  bool vec = aligned16(whole);
  for (int k = 0; k < n; ++k) vec = vec && len[k] % 4 == 0 && (!pieces[k] || aligned16(pieces[k]));
  const int64_t unit = vec ? 4 : 1;
  int64_t off = 0;
  for (int k = 0; k < n; ++k) { q.p[k] = pieces[k]; q.len[k] = (unsigned)(len[k] / unit); q.off[k] = (unsigned)(off / unit); off += len[k]; }
  const int64_t items = outer * total / unit;
  if (vec) LTB_LAUNCH((concat_kernel<GRAD, 4>), grid_for(items, 256), 256, 0, whole, q, (unsigned)(total / unit), (unsigned)items);
  else LTB_LAUNCH((concat_kernel<GRAD, 1>), grid_for(items, 256), 256, 0, whole, q, (unsigned)(total / unit), (unsigned)items);
  return LTB_OK;
}

// One piece of a larger concatenation: a strided row copy, dst[r*dst_stride + j] (op)= src[r*src_stride + j], j < row_len.
template <bool ACC, int VEC>
__global__ void copy_rows_kernel(float* dst, int64_t dst_stride, const float* __restrict__ src, int64_t src_stride, int64_t row_len, int64_t n) {
  pdl_enter();
  // all quantities are in units of VEC floats
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = i / row_len, j = i % row_len;
    if (VEC == 4) {
      float4 v = reinterpret_cast<const float4*>(src)[r * src_stride + j];
      float4* q = reinterpret_cast<float4*>(dst) + r * dst_stride + j;
      if (ACC) { float4 o = *q; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
      *q = v;
    } else {
      float v = src[r * src_stride + j];
      float* q = dst + r * dst_stride + j;
      *q = ACC ? *q + v : v;
    }
  }
}
template <bool ACC>
static int copy_rows(float* dst, int64_t dst_stride, const float* src, int64_t src_stride, int64_t row_len, int64_t rows) {
  if (rows * row_len == 0) return LTB_OK;
  if (aligned16(dst) && aligned16(src) && ((dst_stride | src_stride | row_len) & 3) == 0) {
    int64_t n = rows * (row_len / 4);
    LTB_LAUNCH((copy_rows_kernel<ACC, 4>), grid_for(n, 256), 256, 0, dst, dst_stride / 4, src, src_stride / 4, row_len / 4, n);
  } else {
    int64_t n = rows * row_len;
    LTB_LAUNCH((copy_rows_kernel<ACC, 1>), grid_for(n, 256), 256, 0, dst, dst_stride, src, src_stride, row_len, n);
  }
  return LTB_OK;
}

static bool make_bcast(const int* as, const int* bs, int rank, Bcast& p, int64_t& n, bool& a_b, bool& b_b) {
  if (rank < 1 || rank > 4 || !as || !bs) return false;
  int A[4] = {1, 1, 1, 1}, B[4] = {1, 1, 1, 1};
  for (int i = 0; i < rank; ++i) { A[4 - rank + i] = as[i]; B[4 - rank + i] = bs[i]; }
  n = 1; a_b = b_b = false;
  int64_t sa = 1, sb = 1;
  for (int i = 3; i >= 0; --i) {
    if (A[i] < 1 || B[i] < 1) return false;
    if (A[i] != B[i] && A[i] != 1 && B[i] != 1) return false;
    p.shape[i] = A[i] > B[i] ? A[i] : B[i];
    p.sa[i] = A[i] == 1 ? 0 : sa; p.sb[i] = B[i] == 1 ? 0 : sb;
    if (A[i] == 1 && p.shape[i] != 1) a_b = true;
    if (B[i] == 1 && p.shape[i] != 1) b_b = true;
    sa *= A[i]; sb *= B[i]; n *= p.shape[i];
  }
  return true;
}

// Strides s of an operand over `shape`: when it is a vector along one run of neighbouring dimensions, full = [outer][mid][inner] with the
// operand v[mid]; false otherwise (or when an index does not fit 31 bits).
static bool vector_operand(const int* shape, const int64_t* s, int64_t n, int64_t& outer, int64_t& mid, int64_t& inner) {
  outer = mid = inner = 1;
  int state = 0;                                         // 0 before the run, 1 in it, 2 behind it
  for (int d = 0; d < 4; ++d) {
    if (shape[d] == 1) continue;
    if (s[d] != 0) { if (state == 2) return false; state = 1; mid *= shape[d]; }
    else if (state == 0) outer *= shape[d];
    else { state = 2; inner *= shape[d]; }
  }
  if (state == 0) { inner = outer; outer = 1; }          // a single value
  return n < (1ll << 31);
}

// ---- look-ahead fusion: issue functions and the flush ------------------------------------------------------------
int add_issue(const float* a, const float* b, float* out, int64_t n, bool relu) {
  if (relu) return launch_map<2>(a, b, nullptr, out, n, [] __device__(float x, float y, float) { float v = x + y; return v < 0.0f ? 0.0f : v; });
  return launch_map<2>(a, b, nullptr, out, n, [] __device__(float x, float y, float) { return x + y; });
}
int relu_issue(float* x, int64_t n) { return launch_map<1>(x, nullptr, nullptr, x, n, [] __device__(float v, float, float) { return v < 0.0f ? 0.0f : v; }); }
int relu_grad_issue(const float* y, float* d, int64_t n) {
  return launch_map<2>(y, d, nullptr, d, n, [] __device__(float yv, float g0, float) { return yv > 0.0f ? g0 : 0.0f; });
}
int fill_issue(float* x, float v, int64_t n) {
  if (n) LTB_LAUNCH(fill_kernel, grid_for(n, 256), 256, 0, x, v, n);
  return LTB_OK;
}
int flush_pending() {
  const Pending p = g.pending;
  g.pending.kind = PEND_NONE;
  switch (p.kind) {
    case PEND_BN_FWD: return bn_fwd_issue(p, false);
    case PEND_BN_RELU: { Pending q = p; q.kind = p.inner; return bn_fwd_issue(q, true); }
    case PEND_CONV: return conv_fwd_issue(p, false);
    case PEND_BN_INF: return bn_inference_issue(p, false);
    case PEND_ADD: return add_issue(p.a, p.b, p.out, p.n, false);
    case PEND_RELU_GRAD: return relu_grad_issue(p.relu_y, p.d, p.n);
    case PEND_RELU_ADD_GRAD: return relu_add_grad_issue(p);
    case PEND_SEED: return fill_issue(p.d, p.value, 1);
    case PEND_LSM: case PEND_NLL: case PEND_SUM_GRAD: case PEND_NLL_GRAD: return head_issue(p);
    case PEND_BN_ADD: {                                         // no ReLU came: the two operations on their own, y written
      Pending q = p; q.kind = PEND_BN_FWD;
      int rc = bn_fwd_issue(q, false);
      return rc ? rc : add_issue(p.y, p.a, p.out, p.n, false);
    }
    default: return LTB_OK;
  }
}
// The held in-place ReLU gradient and the gradient of a same-shape add in one pass:
// m = y > 0 ? d : 0;  d = m;  da += m;  db += m   (da, db nullable; fa / fb: that destination holds nothing yet and is written; wb == 0: d itself is not
// rewritten, its owner has declared it dead).
// n4 float4 items, then a scalar tail from `tail`.
__global__ void relu_add_grad_kernel(const float* __restrict__ y, float* d, float* da, float* db, int64_t n4, int64_t tail, int64_t n, int fa, int fb, int wb) {
  pdl_enter();
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = i0; i < n4; i += stride) {
    const float4 yv = reinterpret_cast<const float4*>(y)[i];
    float4 m = reinterpret_cast<const float4*>(d)[i];
    m.x = yv.x > 0.0f ? m.x : 0.0f; m.y = yv.y > 0.0f ? m.y : 0.0f; m.z = yv.z > 0.0f ? m.z : 0.0f; m.w = yv.w > 0.0f ? m.w : 0.0f;
    if (wb) reinterpret_cast<float4*>(d)[i] = m;
    if (da) { float4 v = fa ? make_float4(0.f, 0.f, 0.f, 0.f) : reinterpret_cast<float4*>(da)[i]; v.x += m.x; v.y += m.y; v.z += m.z; v.w += m.w; reinterpret_cast<float4*>(da)[i] = v; }
    if (db) { float4 v = fb ? make_float4(0.f, 0.f, 0.f, 0.f) : reinterpret_cast<float4*>(db)[i]; v.x += m.x; v.y += m.y; v.z += m.z; v.w += m.w; reinterpret_cast<float4*>(db)[i] = v; }
  }
  for (int64_t i = tail + i0; i < n; i += stride) {
    const float m = y[i] > 0.0f ? d[i] : 0.0f;
    if (wb) d[i] = m;
    if (da) da[i] = fa ? m : da[i] + m;
    if (db) db[i] = fb ? m : db[i] + m;
  }
}

int relu_add_grad_issue(const Pending& p) {
  const bool vec = aligned16(p.relu_y) && aligned16(p.d) && (!p.da || aligned16(p.da)) && (!p.db || aligned16(p.db));
  const int64_t n4 = vec ? p.n / 4 : 0;
  LTB_LAUNCH(relu_add_grad_kernel, grid_for(n4 ? n4 : p.n, 256), 256, 0, p.relu_y, p.d, p.da, p.db, n4, n4 * 4, p.n, p.fa, p.fb, g.fusion_no_writeback ? 0 : 1);
  return LTB_OK;
}

// Pinned staging for host-drawn masks: four blocks in turn, each free again when the copy out of it is done.
struct MaskBlock { float* p; size_t bytes; cudaEvent_t done; };
static MaskBlock mask_blocks[4];
static int mask_next = 0;
static int mask_staging(size_t bytes, float** p, cudaEvent_t* done) {
  MaskBlock& b = mask_blocks[mask_next];
  mask_next = (mask_next + 1) % 4;
  if (b.done) LTB_CUDA(cudaEventSynchronize(b.done)); else LTB_CUDA(cudaEventCreateWithFlags(&b.done, cudaEventDisableTiming));
  if (b.bytes < bytes) {
    if (b.p) cudaFreeHost(b.p);
    b.p = nullptr; b.bytes = 0;
    LTB_CUDA(cudaMallocHost((void**)&b.p, bytes));
    b.bytes = bytes;
  }
  *p = b.p; *done = b.done;
  return LTB_OK;
}
void mask_staging_free() {
  for (MaskBlock& b : mask_blocks) { if (b.p) cudaFreeHost(b.p); if (b.done) cudaEventDestroy(b.done); b = MaskBlock{nullptr, 0, nullptr}; }
}

}  // namespace ltb

using namespace ltb;

extern "C" {

static size_t shape_count(const int* shape, int rank) {
  size_t n = 1;
  for (int i = 0; i < rank && i < 8 && shape; ++i) n *= (size_t)(shape[i] > 0 ? shape[i] : 1);
  return n;
}
// fill / fillInPlace: TensorDslCPU.scala:30-35, 65-67.
int ltb_fill(float* x, float v, int64_t n) {
  LTB_INITED(); filter_cache_note_write(x, (size_t)(n > 0 ? n : 0) * 4); LTB_REQUIRE(x && n >= 0, "ltb_fill: bad argument");
  LTB_SETTLE(x);                                            // no longer unset: a later call must not put zeros over the value
  if (n == 1 && g.fusion) { Pending h; h.kind = PEND_SEED; h.n = 1; h.d = x; h.value = v; g.pending = h; return LTB_OK; }   // the gradient of a sum that reads it may join it
  return fill_issue(x, v, n);
}
// fillWithBias: TensorDslCPU.scala:41-61.
int ltb_fill_with_bias(float* out, const float* bias, int outer, int c, int inner) {
  LTB_INITED(); filter_cache_note_write(out, (size_t)outer * c * inner * 4); LTB_REQUIRE(out && bias && outer >= 0 && c > 0 && inner > 0, "ltb_fill_with_bias: bad argument");
  int64_t n = (int64_t)outer * c * inner;
  if (n) LTB_LAUNCH(fill_bias_kernel, grid_for(n, 256), 256, 0, out, bias, c, (int64_t)inner, n);
  return LTB_OK;
}
// clipAt: TensorDslCPU.scala:113-119.
int ltb_clip(float* x, float bound, int64_t n) {
  LTB_INITED(); filter_cache_note_write(x, (size_t)(n > 0 ? n : 0) * 4); LTB_REQUIRE(x && n >= 0, "ltb_clip: bad argument");
  return launch_map<1>(x, nullptr, nullptr, x, n, [bound] __device__(float v, float, float) { return v > bound ? bound : (v < -bound ? -bound : v); });
}

// elementWiseOpWithBroadCast: TensorDslCPU.scala:227-244.
int ltb_ew_binary(int op, const float* a, const int* as, const float* b, const int* bs, float* out, int rank) {
  LTB_INITED_NOFLUSH(); LTB_REQUIRE(a && b && out && op >= LTB_ADD && op <= LTB_DIV, "ltb_ew_binary: bad argument");
  Bcast p; int64_t n; bool ab, bb;
  LTB_REQUIRE(make_bcast(as, bs, rank, p, n, ab, bb), "ltb_ew_binary: shapes do not broadcast");
  LTB_WRITES(out, n);
  if (g.pending.kind == PEND_BN_FWD && g.fusion_single_use && !ab && !bb && op == LTB_ADD && g.pending.n == n && a != b &&
      (a == g.pending.y || b == g.pending.y)) {                 // the held batch norm's result plus a shortcut: held once more, for the ReLU
    const float* other = a == g.pending.y ? b : a;
    if (out != g.pending.y && out != g.pending.x && out != other && aligned16(other) && aligned16(out)) {
      g.pending.kind = PEND_BN_ADD; g.pending.a = other; g.pending.out = out;
      return LTB_OK;
    }
  }
  if (g.pending.kind) { int rc = flush_pending(); if (rc) return rc; }
  if (!ab && !bb && op == LTB_ADD) {
    if (g.fusion && n > 0) { Pending h; h.kind = PEND_ADD; h.n = n; h.a = a; h.b = b; h.out = out; g.pending = h; return LTB_OK; }   // an in-place ReLU of out may join it
    return add_issue(a, b, out, n, false);
  }
  if (!ab && !bb) return launch_map<2>(a, b, nullptr, out, n, [op] __device__(float x, float y, float) { return bin_op(op, x, y); });
  LTB_LAUNCH(bcast_binary_kernel, grid_for(n, 256), 256, 0, op, a, b, out, p, n);
  return LTB_OK;
}
// backpropElementWiseOpWithBroadCast: TensorDslCPU.scala:246-263.
int ltb_ew_binary_grad(int op, const float* a, float* da, const int* as, const float* b, float* db, const int* bs, const float* dout, int rank) {
  LTB_INITED_CHAIN(); LTB_REQUIRE(a && b && dout && op >= LTB_ADD && op <= LTB_DIV, "ltb_ew_binary_grad: bad argument");
  Bcast p; int64_t n; bool ab, bb;
  LTB_REQUIRE(make_bcast(as, bs, rank, p, n, ab, bb), "ltb_ew_binary_grad: shapes do not broadcast");
  // n bounds the size of either operand
  LTB_SIDE_CHECK(da, n, true); LTB_SIDE_CHECK(db, n, true); LTB_SIDE_CHECK(dout, n, true); LTB_SIDE_CHECK(a, n, false); LTB_SIDE_CHECK(b, n, false);
  LTB_WRITES(da, shape_count(as, rank)); LTB_WRITES(db, shape_count(bs, rank));
  if (g.pending.kind == PEND_RELU_GRAD && !ab && !bb && op == LTB_ADD && g.pending.d == dout && g.pending.n == n && n > 0) {
    // the held ReLU gradient of dout and this add's gradient in one pass (dout is rewritten with the masked values)
    const float* y = g.pending.relu_y; float* d = g.pending.d;
    g.pending.kind = PEND_NONE;
    // a destination declared unset (ltb_grad_unset) is written instead of added into; da == db stays an accumulation
    const int fa = da && da != db && grad_take_unset(da, (size_t)n * 4) ? 1 : 0, fb = db && da != db && grad_take_unset(db, (size_t)n * 4) ? 1 : 0;
    LTB_SETTLE(d); if (!fa) LTB_SETTLE(da); if (!fb) LTB_SETTLE(db);
    Pending h; h.kind = PEND_RELU_ADD_GRAD; h.n = n; h.relu_y = y; h.d = d; h.da = da; h.db = db; h.fa = fa; h.fb = fb;
    // level 2: held once more -- a batch-norm backward whose dy is one of the two destinations, written by nobody else before
    // (fresh), reads the masked gradient straight from d and writes the other destination itself (ltb_bn_bwd)
    if (g.fusion_no_writeback && da && db && da != db && (fa || fb)) { g.pending = h; return LTB_OK; }
    return relu_add_grad_issue(h);
  }
  if (g.pending.kind) { int rc = flush_pending(); if (rc) return rc; }
  LTB_SETTLE(dout);
  if (!ab && !bb && op == LTB_ADD) {   // the residual add of ResNet: da += dout, db += dout (a destination declared unset: da = dout)
    const bool fa = da && da != db && grad_take_unset(da, (size_t)n * 4), fb = db && da != db && grad_take_unset(db, (size_t)n * 4);
    if (!fa) LTB_SETTLE(da);
    if (!fb) LTB_SETTLE(db);
    int rc = !da ? 0 : fa ? launch_map<1>(dout, nullptr, nullptr, da, n, [] __device__(float c, float, float) { return c; })
                          : launch_map<2>(da, dout, nullptr, da, n, [] __device__(float g0, float c, float) { return g0 + c; });
    if (rc) return rc;
    return !db ? LTB_OK : fb ? launch_map<1>(dout, nullptr, nullptr, db, n, [] __device__(float c, float, float) { return c; })
                             : launch_map<2>(db, dout, nullptr, db, n, [] __device__(float g0, float c, float) { return g0 + c; });
  }
  LTB_SETTLE(da); LTB_SETTLE(db);
  if (!da && !db) return LTB_OK;
  LTB_LAUNCH(bcast_binary_grad_kernel, grid_for(n, 256), 256, 0, op, a, da, ab, b, db, bb, dout, p, n);
  return LTB_OK;
}
// map(x, s => s op y): TensorDslCPU.scala:298-331.
int ltb_ew_scalar(int op, const float* a, float s, float* out, int64_t n) {
  LTB_INITED(); filter_cache_note_write(out, (size_t)(n > 0 ? n : 0) * 4); LTB_REQUIRE(a && out && n >= 0 && op >= LTB_ADD && op <= LTB_DIV, "ltb_ew_scalar: bad argument");
  return launch_map<1>(a, nullptr, nullptr, out, n, [op, s] __device__(float x, float, float) { return bin_op(op, x, s); });
}
int ltb_ew_inplace_scalar(int op, float* x, float s, int64_t n) { return ltb_ew_scalar(op, x, s, x, n); }

// inplaceElementWiseOpWithBroadCastOrReduce: TensorDslCPU.scala:265-279.
int ltb_ew_inplace(int op, float* x, const int* xs, const float* y, const int* ys, int rank) {
  LTB_INITED(); LTB_SETTLE(x); LTB_SETTLE(y); LTB_WRITES(x, shape_count(xs, rank)); LTB_REQUIRE(x && y && op >= LTB_ADD && op <= LTB_DIV, "ltb_ew_inplace: bad argument");
  Bcast p; int64_t n; bool xb, yb;
  LTB_REQUIRE(make_bcast(xs, ys, rank, p, n, xb, yb), "ltb_ew_inplace: shapes do not broadcast");
  if (!xb && !yb) return launch_map<2>(x, y, nullptr, x, n, [op] __device__(float u, float v, float) { return bin_op(op, u, v); });
  int64_t outer, mid, inner;
  if (!xb && vector_operand(p.shape, p.sb, n, outer, mid, inner)) {
    switch (op) {
      case LTB_ADD: return bcast_mid<LTB_ADD>(x, y, n, inner, mid);
      case LTB_SUB: return bcast_mid<LTB_SUB>(x, y, n, inner, mid);
      case LTB_MUL: return bcast_mid<LTB_MUL>(x, y, n, inner, mid);
      default: return bcast_mid<LTB_DIV>(x, y, n, inner, mid);
    }
  }
  if (xb && !yb && op <= LTB_SUB && vector_operand(p.shape, p.sa, n, outer, mid, inner)) return reduce_mid(x, y, outer, mid, inner, op == LTB_ADD ? 1.0f : -1.0f);
  if (!xb) { LTB_LAUNCH(bcast_inplace_kernel, grid_for(n, 256), 256, 0, op, x, y, p, n); return LTB_OK; }
  // y (possibly itself broadcast on other dims) is reduced into x
  Reduce r; int64_t nx = 1;
  for (int i = 0; i < 4; ++i) { r.xshape[i] = p.sa[i] == 0 && p.shape[i] != 1 ? 1 : p.shape[i]; r.rshape[i] = p.shape[i]; r.sy[i] = p.sb[i]; nx *= r.xshape[i]; }
  int64_t per = n / nx;
  LTB_LAUNCH(reduce_inplace_kernel, (unsigned)ceil_div(nx * 32, 256), 256, 0, op, x, y, r, nx, per);
  return LTB_OK;
}
// plusBias / plusBias_grad: TensorDslCPU.scala:281-288.
int ltb_plus_bias(float* main, const int* ms, const float* bias, const int* bs, int rank) { return ltb_ew_inplace(LTB_ADD, main, ms, bias, bs, rank); }
int ltb_plus_bias_grad(float* dbias, const int* bs, const float* dmain, const int* ms, int rank) { return ltb_ew_inplace(LTB_ADD, dbias, bs, dmain, ms, rank); }

// geam: TensorDslCPU.scala:342-347 / cublasSgeam at TensorDslCublas.scala:318-373.
int ltb_geam(const float* x, int tx, float alpha, const float* y, int ty, float beta, float* out, int rows, int cols) {
  LTB_INITED(); filter_cache_note_write(out, (size_t)rows * cols * 4); LTB_REQUIRE(x && y && out && rows > 0 && cols > 0, "ltb_geam: bad argument");
  LTB_REQUIRE(!((tx || ty) && (out == x || out == y)), "ltb_geam: in-place with transpose");
  int64_t n = (int64_t)rows * cols;
  if (!tx && !ty) return launch_map<2>(x, y, nullptr, out, n, [alpha, beta] __device__(float u, float v, float) { return u * alpha + v * beta; });
  LTB_LAUNCH(geam_kernel, grid_for(n, 256), 256, 0, x, tx, alpha, y, ty, beta, out, rows, cols);
  return LTB_OK;
}
// trans / trans_grad: TensorDslCPU.scala:349-374.
int ltb_trans(const float* x, float* out, int rows, int cols) {
  LTB_INITED(); LTB_REQUIRE(x && out && rows > 0 && cols > 0, "ltb_trans: bad argument");
  LTB_WRITES(out, (size_t)rows * cols);
  LTB_LAUNCH(transpose_kernel<false>, dim3((cols + 31) / 32, (rows + 31) / 32), dim3(32, 8), 0, x, out, rows, cols);
  return LTB_OK;
}
int ltb_trans_grad(float* dx, const float* dy, int rows, int cols) {
  LTB_INITED(); LTB_SETTLE(dx); LTB_SETTLE(dy); LTB_REQUIRE(dx && dy && rows > 0 && cols > 0, "ltb_trans_grad: bad argument");
  LTB_WRITES(dx, (size_t)rows * cols);
  // dy is [cols, rows]; dx[rows, cols] += dy^T
  LTB_LAUNCH(transpose_kernel<true>, dim3((rows + 31) / 32, (cols + 31) / 32), dim3(32, 8), 0, dy, dx, cols, rows);
  return LTB_OK;
}

// relu/tanh/sigmoid/exp/log/sqrt/square: TensorDslCPU.scala:710-781.
int ltb_unary(int op, const float* x, float* out, int64_t n) {
  LTB_INITED_NOFLUSH(); LTB_REQUIRE(x && out && n >= 0 && op >= LTB_RELU && op <= LTB_SQUARE, "ltb_unary: bad argument");
  LTB_WRITES(out, n);
  if (g.pending.kind && op == LTB_RELU && x == out && g.pending.n == n) {      // in-place ReLU of the result that was just held back
    const Pending h = g.pending;
    if ((h.kind == PEND_BN_FWD && h.y == out) || (h.kind == PEND_BN_ADD && h.out == out)) { g.pending.inner = h.kind; g.pending.kind = PEND_BN_RELU; return LTB_OK; }
    if (h.kind == PEND_BN_INF && h.y == out) { g.pending.kind = PEND_NONE; return bn_inference_issue(h, true); }
    if (h.kind == PEND_CONV && h.y == out) { g.pending.kind = PEND_NONE; return conv_fwd_issue(h, true); }
    if (h.kind == PEND_ADD && h.out == out) { g.pending.kind = PEND_NONE; return add_issue(h.a, h.b, h.out, h.n, true); }
  }
  if (g.pending.kind) { int rc = flush_pending(); if (rc) return rc; }
  return launch_map<1>(x, nullptr, nullptr, out, n, [op] __device__(float v, float, float) { return un_op(op, v); });
}
// *_grad.  ReLU in place: the reference's CPU backend tests the clamped value with `< 0` and so never masks
// (TensorDslCPU.scala:726) while its GPU backend masks where y <= 0 (cudnnActivationBackward with beta 0,
// TensorDslCudnn.scala:1392-1429); this library masks where y <= 0, which is the derivative of what was computed.
int ltb_unary_grad(int op, const float* x, float* dx, const float* y, const float* dy, int64_t n, int in_place) {
  LTB_INITED_CHAIN();
  LTB_SIDE_CHECK(dx, n, true); LTB_SIDE_CHECK(x, n, false); LTB_SIDE_CHECK(y, n, false); LTB_SIDE_CHECK(dy, n, false);
  if (g.pending.kind) { int rc_ = flush_pending(); if (rc_) return rc_; }
  LTB_REQUIRE(dx && dy && n >= 0 && op >= LTB_RELU && op <= LTB_SQUARE, "ltb_unary_grad: bad argument");
  LTB_SETTLE(dx); LTB_SETTLE(dy); LTB_WRITES(dx, n);
  if (op == LTB_RELU && in_place) {
    LTB_REQUIRE(y, "ltb_unary_grad: relu in place needs the result");
    if (g.fusion && n > 0) { Pending h; h.kind = PEND_RELU_GRAD; h.n = n; h.relu_y = y; h.d = dx; g.pending = h; return LTB_OK; }   // BN backward or an add's gradient may absorb it
    return relu_grad_issue(y, dx, n);
  }
  const float* xin = x ? x : y; const float* yin = y ? y : x;
  LTB_REQUIRE(xin, "ltb_unary_grad: needs x or y");
  // dx += g(x, y, dy): four streams; fold x/y into the two the op actually needs
  bool needs_x = op == LTB_RELU || op == LTB_LOG || op == LTB_SQUARE;
  const float* s = needs_x ? xin : yin;
  return launch_map<3>(dx, s, dy, dx, n, [op] __device__(float g0, float v, float d) { return g0 + un_grad(op, v, v, d); });
}

// dropout: TensorDslCPU.scala:1066-1088.  The keep mask is drawn on the host from glibc rand() in element order,
// the stream the reference's CPU backend consumes, and uploaded; cudnnDropout in the reference's GPU backend is seeded
// with time(NULL) (TensorDslCudnn.scala:1301) and cannot be reproduced.
int ltb_dropout_masked(const float* x, float* y, const float* mask, int64_t n) {
  LTB_INITED(); LTB_REQUIRE(x && y && mask && n >= 0, "ltb_dropout_masked: bad argument");
  LTB_WRITES(y, n);
  return launch_map<2>(x, mask, nullptr, y, n, [] __device__(float v, float m, float) { return v * m; });
}
int ltb_dropout(const float* x, float* y, float* mask, float p, int64_t n) {
  LTB_INITED(); LTB_REQUIRE(x && y && mask && n >= 0 && p >= 0.0f && p < 1.0f, "ltb_dropout: rate must be in [0,1)");
  LTB_REQUIRE(!g.capturing, "ltb_dropout: host RNG while recording a step");
  LTB_WRITES(mask, n);
  if (n) {
    // drawn into pinned memory that the copy reads later: the stream is not drained (a step of the MNIST program waited here for its
    // whole forward pass, 0.225 -> 0.21 ms).  (float)rand() / RAND_MAX > p compares against p * 2^31: RAND_MAX as a float is 2^31, an exact scale.
    float* h; cudaEvent_t done;
    int rc = mask_staging((size_t)n * 4, &h, &done); if (rc) return rc;
    const float scale = 1.0f / (1.0f - p), bound = p * 2147483648.0f;
    for (int64_t i = 0; i < n; ++i) h[i] = (float)rand() > bound ? scale : 0.0f;
    LTB_CUDA(cudaMemcpyAsync(mask, h, (size_t)n * 4, cudaMemcpyHostToDevice, g.stream));
    LTB_CUDA(cudaEventRecord(done, g.stream));
  }
  return ltb_dropout_masked(x, y, mask, n);
}
int ltb_dropout_grad(float* dx, const float* mask, const float* dy, int64_t n) {
  LTB_INITED(); LTB_SETTLE(dx); LTB_SETTLE(dy); LTB_REQUIRE(dx && mask && dy && n >= 0, "ltb_dropout_grad: bad argument");
  LTB_WRITES(dx, n);
  return launch_map<3>(dx, mask, dy, dx, n, [] __device__(float g0, float m, float d) { return g0 + m * d; });
}

// concat / concat_grad: TensorDslCPU.scala:1166-1212. Input k is [outer, dims[k], inner]; one strided copy per input
// (the reference's GPU kernel handles exactly two 4-D inputs on dim 1, DslAPI.scala:561-623).
int ltb_concat(float* out, const float* const* inputs, const int* dims, int n_inputs, int outer, int inner) {
  LTB_INITED(); LTB_REQUIRE(out && inputs && dims && n_inputs > 0 && outer > 0 && inner > 0, "ltb_concat: bad argument");
  int64_t total = 0;
  for (int k = 0; k < n_inputs; ++k) { LTB_REQUIRE(inputs[k] && dims[k] > 0, "ltb_concat: bad input %d", k); total += dims[k]; }
  LTB_WRITES(out, total * inner * outer);
  int64_t off = 0;
  if (n_inputs <= kPieces && total * inner * outer < (1ll << 31)) {
    float* p[kPieces]; int64_t len[kPieces];
    for (int k = 0; k < n_inputs; ++k) { p[k] = const_cast<float*>(inputs[k]); len[k] = (int64_t)dims[k] * inner; }
    return concat_issue<false>(out, p, len, n_inputs, total * inner, outer, 0);
  }
  for (int k = 0; k < n_inputs; ++k) {
    int64_t len = (int64_t)dims[k] * inner;
    int rc = copy_rows<false>(out + off, total * inner, inputs[k], len, len, outer);
    if (rc) return rc;
    off += len;
  }
  return LTB_OK;
}
int ltb_concat_grad(float* const* dinputs, const float* dout, const int* dims, int n_inputs, int outer, int inner) {
  LTB_INITED_CHAIN();
  if (g.pending.kind) { int rc_ = flush_pending(); if (rc_) return rc_; }
  if (g.side_open && dinputs && dout && dims && n_inputs > 0 && outer > 0 && inner > 0) {
    int64_t all = 0;
    for (int k = 0; k < n_inputs; ++k) { const int64_t len = (int64_t)dims[k] * inner * outer; all += len; LTB_SIDE_CHECK(dinputs[k], len, true); }
    LTB_SIDE_CHECK(dout, all, false);
  }
  LTB_SETTLE(dout); LTB_REQUIRE(dinputs && dout && dims && n_inputs > 0 && outer > 0 && inner > 0, "ltb_concat_grad: bad argument");
  int64_t total = 0;
  for (int k = 0; k < n_inputs; ++k) { LTB_REQUIRE(dims[k] > 0, "ltb_concat_grad: bad input %d", k); total += dims[k]; }
  for (int k = 0; k < n_inputs; ++k) LTB_WRITES(dinputs[k], (size_t)dims[k] * inner * outer);
  int64_t off = 0;
  bool distinct = true;                                       // one buffer named twice is added into piece after piece
  for (int k = 0; k < n_inputs; ++k) for (int j = 0; j < k; ++j) distinct = distinct && (!dinputs[k] || dinputs[k] != dinputs[j]);
  if (n_inputs <= kPieces && distinct && total * inner * outer < (1ll << 31)) {
    float* p[kPieces]; int64_t len[kPieces]; unsigned fresh = 0;
    for (int k = 0; k < n_inputs; ++k) {
      p[k] = dinputs[k]; len[k] = (int64_t)dims[k] * inner;
      if (!p[k]) continue;
      if (grad_take_unset(p[k], (size_t)len[k] * outer * 4)) fresh |= 1u << k; else LTB_SETTLE(p[k]);
    }
    return concat_issue<true>(const_cast<float*>(dout), p, len, n_inputs, total * inner, outer, fresh);
  }
  for (int k = 0; k < n_inputs; ++k) {
    int64_t len = (int64_t)dims[k] * inner;
    if (dinputs[k]) {
      // an input's gradient buffer declared unset (ltb_grad_unset) is written, any other is added into
      const bool fresh = grad_take_unset(dinputs[k], (size_t)len * outer * 4);
      if (!fresh) LTB_SETTLE(dinputs[k]);
      int rc = fresh ? copy_rows<false>(dinputs[k], len, dout + off, total * inner, len, outer) : copy_rows<true>(dinputs[k], len, dout + off, total * inner, len, outer);
      if (rc) return rc;
    }
    off += len;
  }
  return LTB_OK;
}

// SGD.step: NNModule.scala:265-287.
int ltb_sgd_step(float* x, float* d, float lr, int64_t n) {
  LTB_INITED(); filter_cache_note_write(x, (size_t)(n > 0 ? n : 0) * 4); LTB_REQUIRE(x && d && n >= 0, "ltb_sgd_step: bad argument");
  if (!n) return LTB_OK;
  float neg_lr = -1.0f * lr;
  int64_t n4 = (aligned16(x) && aligned16(d)) ? n / 4 : 0;
  if (n4) LTB_LAUNCH(sgd_vec4_kernel, grid_for(n4, 256), 256, 0, x, d, neg_lr, n4);
  if (n4 * 4 < n) LTB_LAUNCH(sgd_scalar_kernel, grid_for(n - n4 * 4, 256), 256, 0, x, d, neg_lr, n4 * 4, n);
  return LTB_OK;
}
// One launch for a whole list of parameter tensors (the reference issues 2 launches per tensor, 267 tensors for ResNet-50).
int ltb_sgd_step_multi(float* const* xs, float* const* ds, const int64_t* sizes, int nt, float lr) {
  LTB_INITED(); filter_cache_note_write(nullptr, 0); LTB_REQUIRE(xs && ds && sizes && nt >= 0, "ltb_sgd_step_multi: bad argument");
  if (!nt) return LTB_OK;
  LTB_REQUIRE((size_t)nt * sizeof(SgdChunk) <= g.cur_scratch_bytes(), "ltb_sgd_step_multi: too many tensors");
  LTB_REQUIRE(!g.capturing, "ltb_sgd_step_multi: uploads its tensor list; use ltb_sgd_step on a slab while recording");
  std::vector<SgdChunk> h(nt);
  int64_t mx = 0;
  for (int i = 0; i < nt; ++i) { h[i] = {xs[i], ds[i], sizes[i]}; if (sizes[i] > mx) mx = sizes[i]; }
  LTB_CUDA(cudaMemcpyAsync(g.cur_scratch(), h.data(), nt * sizeof(SgdChunk), cudaMemcpyHostToDevice, g.stream));
  LTB_CUDA(cudaStreamSynchronize(g.stream));
  int gx = (int)(ceil_div(mx, 256) < 64 ? ceil_div(mx, 256) : 64);
  LTB_LAUNCH(sgd_multi_kernel, dim3(gx < 1 ? 1 : gx, nt), 256, 0, (const SgdChunk*)g.cur_scratch(), lr);
  return LTB_OK;
}
int ltb_adagrad_update(float* x, float* d, float* h, float lr, float clip, int descent, int64_t n) {
  LTB_INITED(); filter_cache_note_write(x, (size_t)(n > 0 ? n : 0) * 4); LTB_REQUIRE(x && d && h && n >= 0, "ltb_adagrad_update: bad argument");
  if (n) LTB_LAUNCH(adagrad_kernel, grid_for(n, 256), 256, 0, x, d, h, lr, clip, descent, n);
  return LTB_OK;
}
int ltb_momentum_update(float* x, float* d, float* m, float lr, float mu, float clip, int nesterov, int descent, int64_t n) {
  LTB_INITED(); filter_cache_note_write(x, (size_t)(n > 0 ? n : 0) * 4); LTB_REQUIRE(x && d && m && n >= 0, "ltb_momentum_update: bad argument");
  if (n) LTB_LAUNCH(momentum_kernel, grid_for(n, 256), 256, 0, x, d, m, lr, mu, clip, nesterov, descent, n);
  return LTB_OK;
}

}  // extern "C"
