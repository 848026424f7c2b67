// A whole unrolled sequence of the vanilla recurrent network in one launch (two for the backward pass).
//
// The reference stages the cell h_t = tanh(x_t Wxh + h_{t-1} Whh + bh) and the output layer o_t = h_t Who + bo operator by
// operator (NNModule.scala:189-200), unrolls T steps (DynamicRNNFix, NNModule.scala:240-253) and adds
// sum(nll(logSoftmax(o_t), y_t)) over the steps: for T = 20 that is some 260 kernels of a few microseconds each, forward and
// backward, and the step runs at the launch rate of the host, not at any limit of the device.
//
// The batch rows of such a sequence never meet: row b of h_t depends on row b of h_{t-1} only.  So the rows are dealt out to
// CTAs (two rows per CTA at batch 256: one CTA per SM); a CTA copies the weight matrices and ALL T steps of its rows into
// shared memory once and never leaves the SM.  Only the recurrence itself is sequential (one matrix-vector product and one
// barrier per step); everything that does not depend on the step before -- x_t Wxh for all t, the output layer, the
// log-softmax, and in the backward pass do_t Who^T and all five gradient sums -- runs as register-tiled matrix products
// over the CTA's T x rows lines at once.  The CTAs' gradient sums are written to slabs and added into the gradient tensors
// in CTA order by a second small launch (no atomics: the same bits on every run).
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace ltb {

constexpr int kSeqThreads = 512;

// CTAs of the running forward launch that have written their part of the loss; back at zero when the launch ends.
__device__ unsigned seq_done_count;

__device__ __forceinline__ float warp_max(float v) { for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o)); return v; }
__device__ __forceinline__ float warp_add(float v) { for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o); return v; }
__host__ __device__ __forceinline__ int up4(int v) { return (v + 3) & ~3; }

// C[m][n] = sum_k A[m][k] W[k][n] (+ bias[n]) on shared memory, a 4 x 4 block of C per thread: the W row is read as one float4
// (consecutive lanes, consecutive columns), the four A values are broadcasts.  Row counts and column pitches are multiples of 4
// (padding rows and columns hold zeros).
__device__ __forceinline__ void mm_tiles(const float* A, int lda, const float* W, int ldw, float* C, int ldc, const float* bias, int M4, int N4, int K) {
  const int nt = N4 >> 2, tiles = (M4 >> 2) * nt;
  for (int tile = threadIdx.x; tile < tiles; tile += kSeqThreads) {
    const int m0 = (tile / nt) << 2, n0 = (tile % nt) << 2;
    float acc[4][4] = {};
    const float* a = A + (size_t)m0 * lda;
    for (int k = 0; k < K; ++k) {
      const float4 w = *reinterpret_cast<const float4*>(W + (size_t)k * ldw + n0);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float av = a[i * lda + k];
        acc[i][0] += av * w.x; acc[i][1] += av * w.y; acc[i][2] += av * w.z; acc[i][3] += av * w.w;
      }
    }
    float4 bv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (bias) bv = *reinterpret_cast<const float4*>(bias + n0);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float4*>(C + (size_t)(m0 + i) * ldc + n0) = make_float4(acc[i][0] + bv.x, acc[i][1] + bv.y, acc[i][2] + bv.z, acc[i][3] + bv.w);
  }
}

// out[a][b] = sum_row A[row][a] B[row][b] for a < Ma, b < Nb (global memory, row pitch Nb), 4 x 4 per thread, both operands read as float4.
__device__ __forceinline__ void outer_tiles(const float* A, int lda, const float* Bm, int ldb, float* out, int Ma, int Nb, int rows) {
  const int nt = up4(Nb) >> 2, tiles = (up4(Ma) >> 2) * nt;
  for (int tile = threadIdx.x; tile < tiles; tile += kSeqThreads) {
    const int a0 = (tile / nt) << 2, b0 = (tile % nt) << 2;
    float acc[4][4] = {};
    for (int r = 0; r < rows; ++r) {
      const float4 av = *reinterpret_cast<const float4*>(A + (size_t)r * lda + a0);
      const float4 bv = *reinterpret_cast<const float4*>(Bm + (size_t)r * ldb + b0);
      const float aa[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) { acc[i][0] += aa[i] * bv.x; acc[i][1] += aa[i] * bv.y; acc[i][2] += aa[i] * bv.z; acc[i][3] += aa[i] * bv.w; }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (a0 + i < Ma && b0 + j < Nb) out[(size_t)(a0 + i) * Nb + b0 + j] = acc[i][j];
  }
}

// Shared memory of the forward kernel (pitches Vq = up4(V), Hq = up4(H); L = up4(T * rows) lines, line (t, r) = t * rows + r):
//   Wxh [V][Hq], Whh [H][Hq], Who [H][Vq], bh [Hq], bo [Vq], x -> o [L][Vq], hx [rows + L][Hq] (h0, then h_0 .. h_{T-1}).
// loss_part[cta] receives the CTA's sum of -logp[y]; the last CTA to finish adds the parts in CTA order into loss[0].
__global__ void __launch_bounds__(kSeqThreads) rnn_seq_fwd_kernel(const float* __restrict__ x, const int32_t* __restrict__ y, const float* __restrict__ h0,
                                                                  const float* __restrict__ Wxh, const float* __restrict__ Whh, const float* __restrict__ bh,
                                                                  const float* __restrict__ Who, const float* __restrict__ bo, float* __restrict__ h_out,
                                                                  float* __restrict__ logp_out, float* loss, float* loss_part,
                                                                  int T, int B, int V, int H, int rows) {
  pdl_enter();
  extern __shared__ float4 sm4[];
  float* sm = reinterpret_cast<float*>(sm4);
  const int Vq = up4(V), Hq = up4(H), L = up4(T * rows);
  float* s_wxh = sm; float* s_whh = s_wxh + V * Hq; float* s_who = s_whh + H * Hq; float* s_bh = s_who + H * Vq; float* s_bo = s_bh + Hq;
  float* s_x = s_bo + Vq; float* s_hx = s_x + L * Vq;
  __shared__ float s_loss[kSeqThreads / 32];
  __shared__ bool s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = blockIdx.x * rows, nr = min(rows, B - b0);
  for (int i = tid; i < V * Hq; i += kSeqThreads) { const int r = i / Hq, c = i - r * Hq; s_wxh[i] = c < H ? Wxh[r * H + c] : 0.0f; }
  for (int i = tid; i < H * Hq; i += kSeqThreads) { const int r = i / Hq, c = i - r * Hq; s_whh[i] = c < H ? Whh[r * H + c] : 0.0f; }
  for (int i = tid; i < H * Vq; i += kSeqThreads) { const int r = i / Vq, c = i - r * Vq; s_who[i] = c < V ? Who[r * V + c] : 0.0f; }
  for (int i = tid; i < Hq; i += kSeqThreads) s_bh[i] = i < H ? bh[i] : 0.0f;
  for (int i = tid; i < Vq; i += kSeqThreads) s_bo[i] = i < V ? bo[i] : 0.0f;
  for (int i = tid; i < L * Vq; i += kSeqThreads) {
    const int line = i / Vq, c = i - line * Vq, t = line / rows, r = line - t * rows;
    s_x[i] = (t < T && r < nr && c < V) ? x[((size_t)t * B + b0 + r) * V + c] : 0.0f;
  }
  for (int i = tid; i < rows * Hq; i += kSeqThreads) { const int r = i / Hq, c = i - r * Hq; s_hx[i] = (h0 && r < nr && c < H) ? h0[(size_t)(b0 + r) * H + c] : 0.0f; }
  __syncthreads();
  // every step's input part at once: hx[line] = x[line] Wxh + bh
  mm_tiles(s_x, Vq, s_wxh, Hq, s_hx + rows * Hq, Hq, s_bh, L, Hq, V);
  __syncthreads();
  // the recurrence: one thread per (row, hidden unit); a warp reads consecutive columns of Whh, h_{t-1} is a broadcast
  for (int t = 0; t < T; ++t) {
    const float* hp = s_hx + (size_t)t * rows * Hq; float* hc = s_hx + (size_t)(t + 1) * rows * Hq;
    for (int i = tid; i < rows * Hq; i += kSeqThreads) {
      const int r = i / Hq, j = i - r * Hq;
      const float* hr = hp + r * Hq;
      float c0 = 0.0f, c1 = 0.0f;
      int k = 0;
      for (; k + 1 < H; k += 2) { c0 += hr[k] * s_whh[k * Hq + j]; c1 += hr[k + 1] * s_whh[(k + 1) * Hq + j]; }
      if (k < H) c0 += hr[k] * s_whh[k * Hq + j];
      hc[i] = j < H ? tanhf(hc[i] + (c0 + c1)) : 0.0f;
    }
    __syncthreads();
  }
  // output layer of every step at once: o[line] = h[line] Who + bo (over the x lines, no longer needed)
  mm_tiles(s_hx + rows * Hq, Hq, s_who, Vq, s_x, Vq, s_bo, L, Vq, H);
  __syncthreads();
  for (int i = tid; i < T * nr * H; i += kSeqThreads) {
    const int c = i % H, rest = i / H, r = rest % nr, t = rest / nr;
    h_out[((size_t)t * B + b0 + r) * H + c] = s_hx[(size_t)((t + 1) * rows + r) * Hq + c];
  }
  // logSoftmax and the loss: one warp per line (max, sum of exponentials, x - (max + log sum): TensorDslCPU.scala:805-835)
  float my_loss = 0.0f;
  for (int line = warp; line < T * rows; line += kSeqThreads / 32) {
    const int t = line / rows, r = line - t * rows;
    if (r >= nr) continue;
    const float* o = s_x + (size_t)line * Vq;
    float m = -3.4028235e38f;
    for (int v = lane; v < V; v += 32) m = fmaxf(m, o[v]);
    m = warp_max(m);
    float s = 0.0f;
    for (int v = lane; v < V; v += 32) s += expf(o[v] - m);
    s = warp_add(s);
    const float lse = m + logf(s);
    float* lp = logp_out + ((size_t)t * B + b0 + r) * V;
    for (int v = lane; v < V; v += 32) lp[v] = o[v] - lse;
    if (lane == 0) { const int target = y[(size_t)t * B + b0 + r]; my_loss += -(o[target] - lse); }
  }
  if (lane == 0) s_loss[warp] = my_loss;
  __syncthreads();
  if (tid == 0) {
    float s = 0.0f;
    for (int w = 0; w < kSeqThreads / 32; ++w) s += s_loss[w];
    loss_part[blockIdx.x] = s;
    __threadfence();
    s_last = atomicAdd(&seq_done_count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (s_last && tid == 0) {                         // the last CTA to finish: the parts are all there; added in CTA order
    __threadfence();
    float s = 0.0f;
    for (unsigned c = 0; c < gridDim.x; ++c) s += ((volatile float*)loss_part)[c];
    loss[0] = s;
    seq_done_count = 0;                             // ready for the next launch
  }
}

// Backward.  Shared memory: Whh^T [H][Hq] and Who^T [V][Hq] (transposed while loading, so that both products below read
// consecutive columns), x [L][Vq], hx [rows + L][Hq] (h0, h_0 .. h_{T-1}), do [L][Vq], dp [L][Hq] (first do Who^T, then the
// gradient at the cell's pre-activation).  The CTA's sums go to slab[cta][...] in the order dWxh, dWhh, dbh, dWho, dbo.
__global__ void __launch_bounds__(kSeqThreads) rnn_seq_bwd_kernel(const float* __restrict__ x, const int32_t* __restrict__ y, const float* __restrict__ h0,
                                                                  const float* __restrict__ Whh, const float* __restrict__ Who, const float* __restrict__ h_all,
                                                                  const float* __restrict__ logp, const float* __restrict__ dloss, float* __restrict__ slab,
                                                                  int T, int B, int V, int H, int rows) {
  pdl_enter();
  extern __shared__ float4 sm4[];
  float* sm = reinterpret_cast<float*>(sm4);
  const int Vq = up4(V), Hq = up4(H), L = up4(T * rows);
  float* s_whhT = sm; float* s_whoT = s_whhT + H * Hq; float* s_x = s_whoT + V * Hq; float* s_hx = s_x + L * Vq;
  float* s_do = s_hx + (rows + L) * Hq; float* s_dp = s_do + L * Vq;
  const int tid = threadIdx.x;
  const int b0 = blockIdx.x * rows, nr = min(rows, B - b0);
  const int n_sums = 2 * V * H + H * H + H + V;
  const float dl = dloss[0];
  for (int i = tid; i < H * Hq; i += kSeqThreads) { const int jp = i / Hq, j = i - jp * Hq; s_whhT[i] = j < H ? Whh[j * H + jp] : 0.0f; }     // [j'][j] = Whh[j][j']
  for (int i = tid; i < V * Hq; i += kSeqThreads) { const int v = i / Hq, j = i - v * Hq; s_whoT[i] = j < H ? Who[j * V + v] : 0.0f; }        // [v][j] = Who[j][v]
  for (int i = tid; i < L * Vq; i += kSeqThreads) {
    const int line = i / Vq, c = i - line * Vq, t = line / rows, r = line - t * rows;
    const bool live = t < T && r < nr && c < V;
    const size_t g = ((size_t)t * B + b0 + r) * V + c;
    s_x[i] = live ? x[g] : 0.0f;
    // nllLoss_grad then logSoftmax_grad (TensorDslCPU.scala:1100-1110, 837-846): do = dl * (exp(logp) - onehot(y))
    s_do[i] = live ? dl * (expf(logp[g]) - (y[(size_t)t * B + b0 + r] == c ? 1.0f : 0.0f)) : 0.0f;
  }
  for (int i = tid; i < (rows + L) * Hq; i += kSeqThreads) {
    const int line = i / Hq, c = i - line * Hq, t = line / rows - 1, r = line % rows;               // line 0 .. rows-1: h0
    float v = 0.0f;
    if (r < nr && c < H && t < T) v = t < 0 ? (h0 ? h0[(size_t)(b0 + r) * H + c] : 0.0f) : h_all[((size_t)t * B + b0 + r) * H + c];
    s_hx[i] = v;
  }
  __syncthreads();
  // what reaches h_t from the output layer, every step at once: dp[line] = do[line] Who^T
  mm_tiles(s_do, Vq, s_whoT, Hq, s_dp, Hq, nullptr, L, Hq, V);
  __syncthreads();
  // the recurrence, backwards in time: dpre_t = (dp_t + dpre_{t+1} Whh^T) (1 - h_t^2)
  for (int t = T - 1; t >= 0; --t) {
    const float* nx = s_dp + (size_t)(t + 1) * rows * Hq; float* cu = s_dp + (size_t)t * rows * Hq;
    const float* hc = s_hx + (size_t)(t + 1) * rows * Hq;
    for (int i = tid; i < rows * Hq; i += kSeqThreads) {
      const int r = i / Hq, j = i - r * Hq;
      float c0 = 0.0f, c1 = 0.0f;
      if (t + 1 < T) {
        const float* dr = nx + r * Hq;
        int k = 0;
        for (; k + 1 < H; k += 2) { c0 += dr[k] * s_whhT[k * Hq + j]; c1 += dr[k + 1] * s_whhT[(k + 1) * Hq + j]; }
        if (k < H) c0 += dr[k] * s_whhT[k * Hq + j];
      }
      const float hv = hc[i];
      cu[i] = j < H ? (cu[i] + (c0 + c1)) * (1.0f - hv * hv) : 0.0f;
    }
    __syncthreads();
  }
  // the five sums over the CTA's lines: dWxh = x^T dpre, dWhh = h_prev^T dpre, dbh, dWho = h^T do, dbo
  float* out = slab + (size_t)blockIdx.x * n_sums;
  const int lines = T * rows;
  outer_tiles(s_x, Vq, s_dp, Hq, out, V, H, lines);
  outer_tiles(s_hx, Hq, s_dp, Hq, out + V * H, H, H, lines);                                       // line (t, r) of hx is h_{t-1}
  outer_tiles(s_hx + rows * Hq, Hq, s_do, Vq, out + V * H + H * H + H, H, V, lines);
  for (int j = tid; j < H; j += kSeqThreads) { float a = 0.0f; for (int l = 0; l < lines; ++l) a += s_dp[(size_t)l * Hq + j]; out[V * H + H * H + j] = a; }
  for (int v = tid; v < V; v += kSeqThreads) { float a = 0.0f; for (int l = 0; l < lines; ++l) a += s_do[(size_t)l * Vq + v]; out[2 * V * H + H * H + H + v] = a; }
}
// ---- hidden sizes up to 128: the recurrent weights in registers -----------------------------------------------------------------
// What bounds a sequence at small batches is its chain of T steps, and around it the copy of the weights by one SM.  Kept in shared
// memory, the recurrent matrix costs a step 2 H dependent loads per thread (about 1000 cycles); here four threads share a hidden unit
// and hold its H weights in registers, so a step is H / 16 vector loads of h, H / 4 FMAs, two shuffles and a barrier.
// Matrices come in by cp.async, all copies in flight at once; Who is never transposed (a product of rows with rows, its pitch
// padded by 4 floats against bank conflicts); with one CTA the gradients are added in place, without the slab and its sum.
// 20 steps, vocabulary 80, hidden 100, batch 1: the step 116 -> 90 us (forward 38 -> 24, backward with its sum 41 -> 27); batch 256: 158 -> 150 (124 with the
// batch uploaded while it is copied).
constexpr int kRegHidden = 128;
__device__ __forceinline__ void copy_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// One row of `cols` floats to shared memory by a warp, zeros up to `pitch`; src null: zeros.
__device__ __forceinline__ void row_to_shared(float* dst, int pitch, const float* src, int cols, int lane) {
  if (!src) { for (int c = lane; c < pitch; c += 32) dst[c] = 0.0f; return; }
  if ((cols & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) { for (int c = lane * 4; c < cols; c += 128) copy_async16(dst + c, src + c); }
  else for (int c = lane; c < cols; c += 32) copy_async4(dst + c, src + c);
  for (int c = cols + lane; c < pitch; c += 32) dst[c] = 0.0f;
}
__device__ __forceinline__ void matrix_to_shared(float* dst, int pitch, const float* src, int rows, int cols) {
  for (int r = threadIdx.x >> 5; r < rows; r += kSeqThreads / 32) row_to_shared(dst + (size_t)r * pitch, pitch, src + (size_t)r * cols, cols, threadIdx.x & 31);
}
// The lines (t, r) of a [T][B][cols] tensor for the batch rows b0 .. b0 + nr - 1; lines beyond them are zeros.
__device__ __forceinline__ void lines_to_shared(float* dst, int pitch, const float* src, int lines, int T, int B, int b0, int rows, int nr, int cols) {
  for (int l = threadIdx.x >> 5; l < lines; l += kSeqThreads / 32) {
    const int t = l / rows, r = l - t * rows;
    row_to_shared(dst + (size_t)l * pitch, pitch, t < T && r < nr ? src + ((size_t)t * B + b0 + r) * cols : nullptr, cols, threadIdx.x & 31);
  }
}
// C[m][n] = sum_k A[m][k] W[k][n] (+ bias[n]), TM x 4 outputs per thread.
template <int TM>
__device__ __forceinline__ void mm_small(const float* A, int lda, const float* W, int ldw, float* C, int ldc, const float* bias, int M, int N4, int K) {
  const int nt = N4 >> 2, tiles = M / TM * nt;
  for (int tile = threadIdx.x; tile < tiles; tile += kSeqThreads) {
    const int m0 = tile / nt * TM, n0 = (tile % nt) << 2;
    float acc[TM][4] = {};
    const float* a = A + (size_t)m0 * lda;
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
      const float4 w = *reinterpret_cast<const float4*>(W + (size_t)k * ldw + n0);
#pragma unroll
      for (int i = 0; i < TM; ++i) { const float av = a[i * lda + k]; acc[i][0] += av * w.x; acc[i][1] += av * w.y; acc[i][2] += av * w.z; acc[i][3] += av * w.w; }
    }
    const float4 bv = *reinterpret_cast<const float4*>(bias + n0);
#pragma unroll
    for (int i = 0; i < TM; ++i) *reinterpret_cast<float4*>(C + (size_t)(m0 + i) * ldc + n0) = make_float4(acc[i][0] + bv.x, acc[i][1] + bv.y, acc[i][2] + bv.z, acc[i][3] + bv.w);
  }
}
__device__ __forceinline__ void mm_lines(const float* A, int lda, const float* W, int ldw, float* C, int ldc, const float* bias, int L, int N4, int K) {
  if ((L >> 2) * (N4 >> 2) >= kSeqThreads) mm_small<4>(A, lda, W, ldw, C, ldc, bias, L, N4, K);      // L is a multiple of 4
  else mm_small<2>(A, lda, W, ldw, C, ldc, bias, L, N4, K);                                          // few lines: more threads with less each
}
// This thread's share of v . w with v in shared memory (`n` floats, n a multiple of 4) and w in registers: float4 number part + 4 i.
__device__ __forceinline__ float part_dot(const float* v, const float* w, int part, int n) {
  float c0 = 0.0f, c1 = 0.0f;
#pragma unroll
  for (int i = 0; i < kRegHidden / 16; ++i) {
    const int q = (part + 4 * i) * 4;
    if (q < n) {
      const float4 h = *reinterpret_cast<const float4*>(v + q);
      c0 += h.x * w[4 * i] + h.y * w[4 * i + 1]; c1 += h.z * w[4 * i + 2] + h.w * w[4 * i + 3];
    }
  }
  float c = c0 + c1;
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c + __shfl_xor_sync(0xffffffffu, c, 2);
}

// Shared memory: Wxh [V][Hq], Who [H][Vq], bh [Hq], bo [Vq], x -> o [L][Vq], hx [rows + L][Hq] (h0, then h_0 .. h_{T-1}).
__global__ void __launch_bounds__(kSeqThreads) rnn_seq_fwd_reg_kernel(const float* __restrict__ x, const int32_t* __restrict__ y, const float* __restrict__ h0,
                                                                      const float* __restrict__ Wxh, const float* __restrict__ Whh, const float* __restrict__ bh,
                                                                      const float* __restrict__ Who, const float* __restrict__ bo, float* __restrict__ h_out,
                                                                      float* __restrict__ logp_out, float* loss, float* loss_part,
                                                                      int T, int B, int V, int H, int rows) {
  pdl_enter();
  extern __shared__ float4 sm4[];
  const int Vq = up4(V), Hq = up4(H), L = up4(T * rows);
  float* s_wxh = reinterpret_cast<float*>(sm4); float* s_who = s_wxh + V * Hq; float* s_bh = s_who + H * Vq; float* s_bo = s_bh + Hq;
  float* s_x = s_bo + Vq; float* s_hx = s_x + L * Vq;
  __shared__ float s_loss[kSeqThreads / 32];
  __shared__ bool s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = blockIdx.x * rows, nr = min(rows, B - b0);
  matrix_to_shared(s_wxh, Hq, Wxh, V, H);
  lines_to_shared(s_x, Vq, x, L, T, B, b0, rows, nr, V);
  matrix_to_shared(s_who, Vq, Who, H, V);
  if (warp == 0) row_to_shared(s_bh, Hq, bh, H, lane);
  if (warp == 1) row_to_shared(s_bo, Vq, bo, V, lane);
  lines_to_shared(s_hx, Hq, h0 ? h0 : nullptr, rows, h0 ? 1 : 0, B, b0, rows, nr, H);
  const int j = tid >> 2, part = tid & 3;
  float w[kRegHidden / 4];
#pragma unroll
  for (int i = 0; i < kRegHidden / 4; ++i) { const int k = (part + 4 * (i >> 2)) * 4 + (i & 3); w[i] = j < H && k < H ? Whh[k * H + j] : 0.0f; }
  copies_done();
  __syncthreads();
  mm_lines(s_x, Vq, s_wxh, Hq, s_hx + rows * Hq, Hq, s_bh, L, Hq, V);              // every step's input part at once
  __syncthreads();
  for (int t = 0; t < T; ++t) {
    for (int r = 0; r < rows; ++r) {
      const float c = part_dot(s_hx + (size_t)(t * rows + r) * Hq, w, part, Hq);
      float* hc = s_hx + (size_t)((t + 1) * rows + r) * Hq;
      if (part == 0 && j < Hq) hc[j] = j < H ? tanhf(hc[j] + c) : 0.0f;
    }
    __syncthreads();
  }
  mm_lines(s_hx + rows * Hq, Hq, s_who, Vq, s_x, Vq, s_bo, L, Vq, H);              // output layer of every step at once
  for (int l = warp; l < T * rows; l += kSeqThreads / 32) {
    const int t = l / rows, r = l - t * rows;
    if (r < nr) for (int c = lane; c < H; c += 32) h_out[((size_t)t * B + b0 + r) * H + c] = s_hx[(size_t)(rows + l) * Hq + c];
  }
  __syncthreads();
  // logSoftmax and the loss: one warp per line (max, sum of exponentials, x - (max + log sum): TensorDslCPU.scala:805-835)
  float my_loss = 0.0f;
  for (int line = warp; line < T * rows; line += kSeqThreads / 32) {
    const int t = line / rows, r = line - t * rows;
    if (r >= nr) continue;
    const float* o = s_x + (size_t)line * Vq;
    const int target = y[(size_t)t * B + b0 + r];
    float m = -3.4028235e38f;
    for (int v = lane; v < V; v += 32) m = fmaxf(m, o[v]);
    m = warp_max(m);
    float s = 0.0f;
    for (int v = lane; v < V; v += 32) s += expf(o[v] - m);
    s = warp_add(s);
    const float lse = m + logf(s);
    float* lp = logp_out + ((size_t)t * B + b0 + r) * V;
    for (int v = lane; v < V; v += 32) lp[v] = o[v] - lse;
    if (lane == 0) my_loss += -(o[target] - lse);
  }
  if (lane == 0) s_loss[warp] = my_loss;
  __syncthreads();
  if (tid == 0) {
    float s = 0.0f;
    for (int u = 0; u < kSeqThreads / 32; ++u) s += s_loss[u];
    if (gridDim.x == 1) { loss[0] = s; s_last = false; }
    else {
      loss_part[blockIdx.x] = s;
      __threadfence();
      s_last = atomicAdd(&seq_done_count, 1u) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (s_last && warp == 0) {                        // the last CTA to finish: the parts are all there; added in a fixed order
    __threadfence();
    float s = 0.0f;
    for (unsigned c = lane; c < gridDim.x; c += 32) s += __ldcg(loss_part + c);
    s = warp_add(s);
    if (lane == 0) { loss[0] = s; seq_done_count = 0; }
  }
}

// out[a][b] (+)= sum_row A[row][a] B[row][b], as outer_tiles.
__device__ __forceinline__ void outer_into(const float* A, int lda, const float* Bm, int ldb, float* out, int Ma, int Nb, int rows, bool add) {
  const int nt = up4(Nb) >> 2, tiles = (up4(Ma) >> 2) * nt;
  for (int tile = threadIdx.x; tile < tiles; tile += kSeqThreads) {
    const int a0 = (tile / nt) << 2, c0 = (tile % nt) << 2;
    float acc[4][4] = {};
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
      const float4 av = *reinterpret_cast<const float4*>(A + (size_t)r * lda + a0);
      const float4 bv = *reinterpret_cast<const float4*>(Bm + (size_t)r * ldb + c0);
      const float aa[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) { acc[i][0] += aa[i] * bv.x; acc[i][1] += aa[i] * bv.y; acc[i][2] += aa[i] * bv.z; acc[i][3] += aa[i] * bv.w; }
    }
    // all old values before the first store: an add per element in turn would wait for memory sixteen times
    if ((Nb & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
      float4* p = reinterpret_cast<float4*>(out + (size_t)a0 * Nb + c0); const int ld = Nb >> 2;
      float4 old[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) old[i] = add && a0 + i < Ma ? p[(size_t)i * ld] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) if (a0 + i < Ma) p[(size_t)i * ld] = make_float4(old[i].x + acc[i][0], old[i].y + acc[i][1], old[i].z + acc[i][2], old[i].w + acc[i][3]);
    } else {
      float old[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int u = 0; u < 4; ++u) old[i][u] = add && a0 + i < Ma && c0 + u < Nb ? out[(size_t)(a0 + i) * Nb + c0 + u] : 0.0f;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int u = 0; u < 4; ++u) if (a0 + i < Ma && c0 + u < Nb) out[(size_t)(a0 + i) * Nb + c0 + u] = old[i][u] + acc[i][u];
    }
  }
}
struct SeqGrads { float *wxh, *whh, *bh, *who, *bo; };
// Shared memory: Who [H][Vq + 4], x [L][Vq], hx [rows + L][Hq], do [L][Vq], dp [L][Hq].  slab null (one CTA): the sums are added into G.
__global__ void __launch_bounds__(kSeqThreads) rnn_seq_bwd_reg_kernel(const float* __restrict__ x, const int32_t* __restrict__ y, const float* __restrict__ h0,
                                                                      const float* __restrict__ Whh, const float* __restrict__ Who, const float* __restrict__ h_all,
                                                                      const float* __restrict__ logp, const float* __restrict__ dloss, float* slab, const SeqGrads G,
                                                                      int T, int B, int V, int H, int rows) {
  pdl_enter();
  extern __shared__ float4 sm4[];
  const int Vq = up4(V), Hq = up4(H), L = up4(T * rows), Vp = Vq + 4;
  float* s_who = reinterpret_cast<float*>(sm4); float* s_x = s_who + H * Vp; float* s_hx = s_x + L * Vq;
  float* s_do = s_hx + (rows + L) * Hq; float* s_dp = s_do + L * Vq;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = blockIdx.x * rows, nr = min(rows, B - b0);
  const float dl = dloss[0];
  matrix_to_shared(s_who, Vp, Who, H, V);
  lines_to_shared(s_x, Vq, x, L, T, B, b0, rows, nr, V);
  lines_to_shared(s_hx, Hq, h0, rows, h0 ? 1 : 0, B, b0, rows, nr, H);
  lines_to_shared(s_hx + rows * Hq, Hq, h_all, L, T, B, b0, rows, nr, H);
  for (int l = warp; l < L; l += kSeqThreads / 32) {
    const int t = l / rows, r = l - t * rows;
    const bool live = t < T && r < nr;
    const size_t at = live ? (size_t)t * B + b0 + r : 0;
    const int target = live ? y[at] : -1;
    // nllLoss_grad then logSoftmax_grad (TensorDslCPU.scala:1100-1110, 837-846): do = dl * (exp(logp) - onehot(y))
    for (int c = lane; c < Vq; c += 32) s_do[(size_t)l * Vq + c] = live && c < V ? dl * (expf(logp[at * V + c]) - (c == target ? 1.0f : 0.0f)) : 0.0f;
  }
  const int j = tid >> 2, part = tid & 3;
  float w[kRegHidden / 4];                          // row j of Whh
#pragma unroll
  for (int i = 0; i < kRegHidden / 4; ++i) { const int k = (part + 4 * (i >> 2)) * 4 + (i & 3); w[i] = j < H && k < H ? Whh[j * H + k] : 0.0f; }
  copies_done();
  __syncthreads();
  // what reaches h_t from the output layer, every step at once: dp[line] = do[line] Who^T, four lines of one hidden unit per thread
  for (int i = tid; i < (L >> 2) * Hq; i += kSeqThreads) {
    const int l0 = i / Hq * 4, u = i % Hq;
    float acc[4] = {};
    if (u < H)
#pragma unroll 4
      for (int v = 0; v < Vq; v += 4) {
        const float4 a = *reinterpret_cast<const float4*>(s_who + (size_t)u * Vp + v);
#pragma unroll
        for (int q = 0; q < 4; ++q) { const float4 d = *reinterpret_cast<const float4*>(s_do + (size_t)(l0 + q) * Vq + v); acc[q] += (a.x * d.x + a.y * d.y) + (a.z * d.z + a.w * d.w); }
      }
#pragma unroll
    for (int q = 0; q < 4; ++q) s_dp[(size_t)(l0 + q) * Hq + u] = acc[q];
  }
  __syncthreads();
  // the recurrence, backwards in time: dpre_t = (dp_t + dpre_{t+1} Whh^T) (1 - h_t^2)
  for (int t = T - 1; t >= 0; --t) {
    for (int r = 0; r < rows; ++r) {
      const float c = t + 1 < T ? part_dot(s_dp + (size_t)((t + 1) * rows + r) * Hq, w, part, Hq) : 0.0f;
      float* cu = s_dp + (size_t)(t * rows + r) * Hq;
      if (part == 0 && j < Hq) { const float hv = s_hx[(size_t)((t + 1) * rows + r) * Hq + j]; cu[j] = j < H ? (cu[j] + c) * (1.0f - hv * hv) : 0.0f; }
    }
    __syncthreads();
  }
  // the five sums over the CTA's lines: dWxh = x^T dpre, dWhh = h_prev^T dpre, dbh, dWho = h^T do, dbo
  const bool add = slab == nullptr;
  float* out = add ? nullptr : slab + (size_t)blockIdx.x * (2 * V * H + H * H + H + V);
  const int lines = T * rows;
  outer_into(s_x, Vq, s_dp, Hq, add ? G.wxh : out, V, H, lines, add);
  outer_into(s_hx, Hq, s_dp, Hq, add ? G.whh : out + V * H, H, H, lines, add);                     // line (t, r) of hx is h_{t-1}
  outer_into(s_hx + rows * Hq, Hq, s_do, Vq, add ? G.who : out + V * H + H * H + H, H, V, lines, add);
  for (int u = tid; u < H + V; u += kSeqThreads) {
    const float* p = u < H ? s_dp + u : s_do + (u - H); const int ld = u < H ? Hq : Vq;
    float a = 0.0f;
#pragma unroll 4
    for (int l = 0; l < lines; ++l) a += p[(size_t)l * ld];
    if (add) { if (u < H) G.bh[u] += a; else G.bo[u - H] += a; }
    else out[u < H ? V * H + H * H + u : 2 * V * H + H * H + H + (u - H)] = a;
  }
}

// d[i] += slab[0][i] + slab[1][i] + ... for the five gradient tensors (segments of the slab row in the order of the kernel above).
// A warp per 32 sums and eighth of the slabs (CTA: 32 sums, eight warps); the eighths meet in order: the same bits on every run.
__global__ void __launch_bounds__(256) rnn_seq_sum_kernel(const float* __restrict__ slab, int ctas, int n_sums, float* dWxh, float* dWhh, float* dbh, float* dWho, float* dbo, int V, int H) {
  pdl_enter();
  __shared__ float part[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
  float a = 0.0f;
  if (i < n_sums) {
    const float* p = slab + i;
#pragma unroll 8
    for (int c = warp; c < ctas; c += 8) a += p[(size_t)c * n_sums];
  }
  part[warp][lane] = a;
  __syncthreads();
  if (warp != 0 || i >= n_sums) return;
#pragma unroll
  for (int w = 1; w < 8; ++w) a += part[w][lane];
  const int o1 = V * H, o2 = o1 + H * H, o3 = o2 + H, o4 = o3 + H * V;
  if (i < o1) dWxh[i] += a; else if (i < o2) dWhh[i - o1] += a; else if (i < o3) dbh[i - o2] += a; else if (i < o4) dWho[i - o3] += a; else dbo[i - o4] += a;
}

static int seq_opted_device = -1;                   // the device whose kernels have been given the large shared-memory limit

// Rows per CTA: one CTA per SM when the batch allows it, fewer rows (more CTAs) when T steps of that many rows do not fit the
// 227 KB of an SM beside the weights.
static bool seq_plan(int T, int B, int V, int H, int* rows, size_t* smem_fwd, size_t* smem_bwd) {
  const size_t Vq = (size_t)up4(V), Hq = (size_t)up4(H);
  int r = (int)ceil_div(B, g.sm_count); if (r < 1) r = 1;
  for (; r >= 1; --r) {
    const size_t L = (size_t)up4(T * r);
    if (H <= kRegHidden) {
      *smem_fwd = ((size_t)V * Hq + (size_t)H * Vq + Hq + Vq + L * Vq + ((size_t)r + L) * Hq) * 4;
      *smem_bwd = ((size_t)H * (Vq + 4) + 2 * L * Vq + ((size_t)r + 2 * L) * Hq) * 4;
      if (*smem_bwd <= (size_t)220 * 1024 && *smem_fwd <= (size_t)220 * 1024 && ceil_div(B, r) <= 65535) { *rows = r; return true; }
      continue;
    }
    *smem_fwd = ((size_t)V * Hq + (size_t)H * Hq + (size_t)H * Vq + Hq + Vq + L * Vq + ((size_t)r + L) * Hq) * 4;
    *smem_bwd = ((size_t)H * Hq + (size_t)V * Hq + L * Vq + ((size_t)r + L) * Hq + L * Vq + (L + (size_t)r) * Hq) * 4;
    if (*smem_bwd <= (size_t)220 * 1024 && *smem_fwd <= (size_t)220 * 1024 && ceil_div(B, r) <= 65535) { *rows = r; return true; }
  }
  return false;
}

}  // namespace ltb

using namespace ltb;

extern "C" {

int ltb_rnn_seq_fwd(const float* x, const int32_t* y, const float* h0, const float* Wxh, const float* Whh, const float* bh, const float* Who,
                    const float* bo, float* h, float* logp, float* loss, int T, int B, int V, int H) {
  LTB_INITED(); LTB_REQUIRE(x && y && Wxh && Whh && bh && Who && bo && h && logp && loss && T > 0 && B > 0 && V > 0 && H > 0, "ltb_rnn_seq_fwd: bad argument");
  LTB_WRITES(h, (size_t)T * B * H); LTB_WRITES(logp, (size_t)T * B * V); LTB_WRITES(loss, 1);
  int rows; size_t sf, sb;
  if (!seq_plan(T, B, V, H, &rows, &sf, &sb))
    return fail(LTB_E_LIMIT, "ltb_rnn_seq_fwd: the weights (vocabulary %d, hidden %d) and %d steps of one batch row do not fit one SM's shared memory", V, H, T);
  if (seq_opted_device != g.device) {
    LTB_REQUIRE(!g.capturing, "ltb_rnn_seq_fwd: the first call sets the kernels up and must come before a step is recorded");
    LTB_CUDA(cudaFuncSetAttribute(rnn_seq_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    LTB_CUDA(cudaFuncSetAttribute(rnn_seq_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    LTB_CUDA(cudaFuncSetAttribute(rnn_seq_fwd_reg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    LTB_CUDA(cudaFuncSetAttribute(rnn_seq_bwd_reg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    seq_opted_device = g.device;
  }
  const int ctas = (int)ceil_div(B, rows);
  LTB_REQUIRE((size_t)ctas * 4 <= g.cur_scratch_bytes(), "ltb_rnn_seq_fwd: batch too large for the library's workspace");
  if (H <= kRegHidden) LTB_LAUNCH(rnn_seq_fwd_reg_kernel, ctas, kSeqThreads, sf, x, y, h0, Wxh, Whh, bh, Who, bo, h, logp, loss, g.cur_scratch(), T, B, V, H, rows);
  else LTB_LAUNCH(rnn_seq_fwd_kernel, ctas, kSeqThreads, sf, x, y, h0, Wxh, Whh, bh, Who, bo, h, logp, loss, g.cur_scratch(), T, B, V, H, rows);
  return LTB_OK;
}

int ltb_rnn_seq_bwd(const float* x, const int32_t* y, const float* h0, const float* Whh, const float* Who, const float* h, const float* logp,
                    const float* dloss, float* dWxh, float* dWhh, float* dbh, float* dWho, float* dbo, int T, int B, int V, int H) {
  LTB_INITED(); LTB_SETTLE(dloss); LTB_SETTLE(dWxh); LTB_SETTLE(dWhh); LTB_SETTLE(dbh); LTB_SETTLE(dWho); LTB_SETTLE(dbo); LTB_REQUIRE(x && y && Whh && Who && h && logp && dloss && dWxh && dWhh && dbh && dWho && dbo && T > 0 && B > 0 && V > 0 && H > 0, "ltb_rnn_seq_bwd: bad argument");
  LTB_WRITES(dWxh, (size_t)V * H); LTB_WRITES(dWhh, (size_t)H * H); LTB_WRITES(dbh, H); LTB_WRITES(dWho, (size_t)H * V); LTB_WRITES(dbo, V);
  int rows; size_t sf, sb;
  if (!seq_plan(T, B, V, H, &rows, &sf, &sb) || seq_opted_device != g.device) return fail(LTB_E_STATE, "ltb_rnn_seq_bwd: no forward call came before");
  const int ctas = (int)ceil_div(B, rows), n_sums = 2 * V * H + H * H + H + V;
  const SeqGrads G{dWxh, dWhh, dbh, dWho, dbo};
  if (H <= kRegHidden && ctas == 1) {
    LTB_LAUNCH(rnn_seq_bwd_reg_kernel, ctas, kSeqThreads, sb, x, y, h0, Whh, Who, h, logp, dloss, (float*)nullptr, G, T, B, V, H, rows);
    return LTB_OK;
  }
  float* slab = (float*)ltb_malloc_uninit((size_t)ctas * n_sums * 4);                 // staging block, given back below (LIFO)
  if (!slab) return g.last;
  if (H <= kRegHidden) LTB_LAUNCH(rnn_seq_bwd_reg_kernel, ctas, kSeqThreads, sb, x, y, h0, Whh, Who, h, logp, dloss, slab, G, T, B, V, H, rows);
  else LTB_LAUNCH(rnn_seq_bwd_kernel, ctas, kSeqThreads, sb, x, y, h0, Whh, Who, h, logp, dloss, slab, T, B, V, H, rows);
  LTB_LAUNCH(rnn_seq_sum_kernel, (unsigned)ceil_div(n_sums, 32), 256, 0, (const float*)slab, ctas, n_sums, dWxh, dWhh, dbh, dWho, dbo, V, H);
  return ltb_free(slab, (size_t)ctas * n_sums * 4);
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------------------------
// One node of the binary tree LSTM per launch.
//
// Operator by operator a node is some 45 kernels forward and backward, gate by gate (ltb_affine_act, ltb_lstm_cell) still 18;
// every one of them works on vectors of 150 floats, so a tree runs at the launch rate of the host.  Here the forward pass of
// a node is one launch: a warp per gate row (750 rows for an inner node: 94 CTAs that read the ten 150x150 matrices out of
// L2 once), and the last CTA to finish combines the gates into the cell, runs the classifier and the loss.  The backward
// pass is one launch too: what precedes the gate gradients in the chain rule (loss, classifier, cell: a few thousand
// operations on vectors of 150) is recomputed by EVERY CTA for itself in shared memory, so no CTA waits for another; CTA 0
// alone writes that part's results.  Then a CTA is one of two kinds: rows of the weight gradients (dW[g][j][:] += dpre in[:]),
// or partial sums of the input gradients (32 inputs x 32 gate rows per warp, added atomically).
namespace ltb {

constexpr int kNodeThreads = 256, kNodeWarps = kNodeThreads / 32;
constexpr int kNodeMaxHidden = 512;                   // the backward prologue keeps 7 vectors of this length in shared memory

__device__ unsigned node_done_count;                  // CTAs of the running forward launch that have stored their gates
constexpr int kNodesPerLaunch = 128;
__device__ unsigned nodes_done_count[kNodesPerLaunch]; // the same, one per node of a batched launch

__device__ __forceinline__ float act_apply(int slot, float v) { return slot == 4 ? tanhf(v) : 1.0f / (1.0f + expf(-v)); }
__device__ __forceinline__ int node_slot(bool inner, int g) { return inner ? g : (g == 0 ? 0 : g + 2); }   // leaf rows: slots 0, 3, 4

// bx: this CTA's index among the n_ctas CTAs that work on node P; done: their completion counter (zero between launches)
__device__ __forceinline__ void node_fwd_body(const ltb_tree_node& P, unsigned* done, unsigned n_ctas, int bx) {
  __shared__ float s_in[kNodeMaxHidden];
  __shared__ float s_pred[32];
  __shared__ bool s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int Hd = P.hidden, L = P.in_len, G = P.inner ? 5 : 3;
  const int row = bx * kNodeWarps + warp;
  if (row < G * Hd) {
    const int slot = node_slot(P.inner, row / Hd), j = row % Hd;
    float a = 0.0f;
    const float* w0 = P.W[slot][0] + (size_t)j * L; const float* x0 = P.in[0];
    for (int k = lane; k < L; k += 32) a += w0[k] * x0[k];
    if (P.inner) {
      float b = 0.0f;
      const float* w1 = P.W[slot][1] + (size_t)j * L; const float* x1 = P.in[1];
      for (int k = lane; k < L; k += 32) b += w1[k] * x1[k];
      a = warp_add(a) + warp_add(b);
    } else {
      a = warp_add(a);
    }
    if (lane == 0) { P.gates[slot * Hd + j] = act_apply(slot, a + P.bias[slot][j]); __threadfence(); }
  }
  __syncthreads();
  if (tid == 0) { __threadfence(); s_last = atomicAdd(done, 1u) == n_ctas - 1; }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // the last CTA: all gates are in memory (read past L1: other SMs wrote them)
  for (int j = tid; j < Hd; j += kNodeThreads) {
    const float ig = __ldcg(P.gates + j), og = __ldcg(P.gates + 3 * Hd + j), uv = __ldcg(P.gates + 4 * Hd + j);
    float c = ig * uv;
    if (P.inner) c = (c + __ldcg(P.gates + Hd + j) * P.cl[j]) + __ldcg(P.gates + 2 * Hd + j) * P.cr[j];
    const float tc = tanhf(c), h = og * tc;
    P.c[j] = c; P.tc[j] = tc; P.h[j] = h;
    s_in[j] = P.classify_cell ? c : h;
  }
  __syncthreads();
  for (int k = warp; k < P.classes; k += kNodeWarps) {
    float a = 0.0f;
    for (int j = lane; j < Hd; j += 32) a += P.Why[(size_t)k * Hd + j] * s_in[j];
    a = warp_add(a);
    if (lane == 0) s_pred[k] = a + P.by[k];
  }
  __syncthreads();
  if (warp == 0) {
    const float o = lane < P.classes ? s_pred[lane] : -3.4028235e38f;
    const float m = warp_max(o);
    const float s = warp_add(lane < P.classes ? expf(o - m) : 0.0f);
    const float lse = m + logf(s);
    if (lane < P.classes) P.logp[lane] = o - lse;
    if (lane == 0) {
      float loss = -(s_pred[P.score[0]] - lse);
      if (P.loss_l) loss += P.loss_l[0];
      if (P.loss_r) loss += P.loss_r[0];
      P.loss[0] = loss;
      *done = 0;                                      // ready for the next launch
    }
  }
}
__global__ void __launch_bounds__(kNodeThreads) tree_node_fwd_kernel(const ltb_tree_node P) { pdl_enter(); node_fwd_body(P, &node_done_count, gridDim.x, (int)blockIdx.x); }
// A level of many CTAs releases the next one only as its CTAs leave (which a kernel without the instruction does): released at the start,
// the next level's waiting CTAs take places that this one's still need (25-leaf tree 229 us against 220).
__device__ __forceinline__ void level_enter() { if (gridDim.x * gridDim.y <= 2u * kSMs) pdl_launch(); pdl_wait(); }
// Several independent nodes (one level of a tree) in one launch: blockIdx.y picks the node out of an array in device memory,
// the CTA copies its node's description into shared memory first.  done[] has one counter per node of the launch.
__device__ __forceinline__ const ltb_tree_node& node_to_shared(const ltb_tree_node* nodes, int i) {
  __shared__ ltb_tree_node sp;
  const int* src = reinterpret_cast<const int*>(nodes + i); int* dst = reinterpret_cast<int*>(&sp);
  for (int k = threadIdx.x; k < (int)(sizeof(ltb_tree_node) / 4); k += blockDim.x) dst[k] = src[k];
  __syncthreads();
  return sp;
}
__global__ void __launch_bounds__(kNodeThreads) tree_nodes_fwd_kernel(const ltb_tree_node* nodes) {
  level_enter();
  unsigned* done = nodes_done_count;
  const ltb_tree_node& P = node_to_shared(nodes, (int)blockIdx.y);
  const unsigned n_ctas = (unsigned)(((P.inner ? 5 : 3) * P.hidden + kNodeWarps - 1) / kNodeWarps);
  if (blockIdx.x >= n_ctas) return;                                    // the grid is sized for an inner node; a leaf needs fewer CTAs
  node_fwd_body(P, done + blockIdx.y, n_ctas, (int)blockIdx.x);
}

// Backward.  Grid: n_w CTAs of weight-gradient rows, then n_x CTAs of input-gradient partial sums (none for a leaf).
// SHARED: several nodes of one launch add into the same parameter gradients (a level of a tree): those additions are atomic.
template <bool SHARED>
__device__ __forceinline__ void node_bwd_body(const ltb_tree_node& P, int n_w, int bx) {
  __shared__ float s_dpre[5 * kNodeMaxHidden];        // gradient at each gate's pre-activation
  __shared__ float s_dpred[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int Hd = P.hidden, L = P.in_len, G = P.inner ? 5 : 3;
  const float dl = P.dloss[0];
  const int score = P.score[0];
  if (tid < 32) s_dpred[tid] = tid < P.classes ? dl * (expf(P.logp[tid]) - (tid == score ? 1.0f : 0.0f)) : 0.0f;   // nllLoss_grad, logSoftmax_grad
  __syncthreads();
  for (int j = tid; j < Hd; j += kNodeThreads) {
    float dcls = 0.0f;                                // classifier's gradient at its input
    for (int k = 0; k < P.classes; ++k) dcls += P.Why[(size_t)k * Hd + j] * s_dpred[k];
    const float dh = P.dh[j] + (P.classify_cell ? 0.0f : dcls), dc = P.dc[j] + (P.classify_cell ? dcls : 0.0f);
    const float ig = P.gates[j], og = P.gates[3 * Hd + j], uv = P.gates[4 * Hd + j], tc = P.tc[j];
    const float dct = dc + dh * og * (1.0f - tc * tc);
    s_dpre[0 * Hd + j] = (dct * uv) * ig * (1.0f - ig);
    s_dpre[3 * Hd + j] = (dh * tc) * og * (1.0f - og);
    s_dpre[4 * Hd + j] = (dct * ig) * (1.0f - uv * uv);
    if (P.inner) {
      const float fl = P.gates[Hd + j], fr = P.gates[2 * Hd + j];
      s_dpre[1 * Hd + j] = (dct * P.cl[j]) * fl * (1.0f - fl);
      s_dpre[2 * Hd + j] = (dct * P.cr[j]) * fr * (1.0f - fr);
      if (bx == 0) {
        if (P.dcl) P.dcl[j] += dct * fl;
        if (P.dcr) P.dcr[j] += dct * fr;
      }
    }
    if (bx == 0) {
      const float v = P.classify_cell ? P.c[j] : P.h[j];
      for (int k = 0; k < P.classes; ++k) { if (SHARED) atomicAdd(P.dWhy + (size_t)k * Hd + j, s_dpred[k] * v); else P.dWhy[(size_t)k * Hd + j] += s_dpred[k] * v; }
    }
  }
  if (bx == 0) {
    if (tid < P.classes) { if (SHARED) atomicAdd(P.dby + tid, s_dpred[tid]); else P.dby[tid] += s_dpred[tid]; }
    if (tid == 0) { if (P.dloss_l) P.dloss_l[0] += dl; if (P.dloss_r) P.dloss_r[0] += dl; }
  }
  __syncthreads();
  if (bx < n_w) {
    const int row = bx * kNodeWarps + warp;
    if (row >= G * Hd) return;
    const int slot = node_slot(P.inner, row / Hd), j = row % Hd;
    const float dp = s_dpre[slot * Hd + j];
    float* d0 = P.dW[slot][0] + (size_t)j * L; const float* x0 = P.in[0];
    for (int k = lane; k < L; k += 32) { if (SHARED) atomicAdd(d0 + k, dp * x0[k]); else d0[k] += dp * x0[k]; }
    if (P.inner) {
      float* d1 = P.dW[slot][1] + (size_t)j * L; const float* x1 = P.in[1];
      for (int k = lane; k < L; k += 32) { if (SHARED) atomicAdd(d1 + k, dp * x1[k]); else d1[k] += dp * x1[k]; }
    }
    if (lane == 0) atomicAdd(P.dbias[slot] + j, dp);   // two slots may share a bias vector
    return;
  }
  // input gradients: warp = (input, block of 32 inputs, gate, block of 32 gate rows); din[k] += sum_j dpre[j] W[j][k]
  const int kb = (L + 31) / 32, jb = (Hd + 31) / 32;
  int w = (bx - n_w) * kNodeWarps + warp;
  const int n_in = P.inner ? 2 : 1;
  if (w >= n_in * kb * G * jb) return;
  const int j0 = (w % jb) * 32; w /= jb;
  const int slot = node_slot(P.inner, w % G); w /= G;
  const int k = (w % kb) * 32 + lane; const int input = w / kb;
  float* din = P.din[input];
  if (!din || k >= L) return;
  const float* wm = P.W[slot][input];
  const int j1 = min(j0 + 32, Hd);
  float a = 0.0f;
  for (int j = j0; j < j1; ++j) a += s_dpre[slot * Hd + j] * wm[(size_t)j * L + k];
  atomicAdd(din + k, a);
}

__global__ void __launch_bounds__(kNodeThreads) tree_node_bwd_kernel(const ltb_tree_node P, int n_w) { pdl_enter(); node_bwd_body<false>(P, n_w, (int)blockIdx.x); }
__global__ void __launch_bounds__(kNodeThreads) tree_nodes_bwd_kernel(const ltb_tree_node* nodes) {
  level_enter();
  const ltb_tree_node& P = node_to_shared(nodes, (int)blockIdx.y);
  const int G = P.inner ? 5 : 3, n_w = (G * P.hidden + kNodeWarps - 1) / kNodeWarps;
  const bool any_din = P.din[0] || (P.inner && P.din[1]);
  const int x_warps = any_din ? (P.inner ? 2 : 1) * ((P.in_len + 31) / 32) * G * ((P.hidden + 31) / 32) : 0;
  if ((int)blockIdx.x >= n_w + (x_warps + kNodeWarps - 1) / kNodeWarps) return;
  node_bwd_body<true>(P, n_w, (int)blockIdx.x);
}

}  // namespace ltb

extern "C" {

// Gradients that were declared unset get their zeros: every one of these is added to.
static int tree_node_settle(const ltb_tree_node& q) {
  for (const float* d : std::initializer_list<const float*>{q.dc, q.dh, q.dloss, q.din[0], q.din[1], q.dcl, q.dcr, q.dloss_l, q.dloss_r, q.dWhy, q.dby}) LTB_SETTLE(d);
  for (int s = 0; s < 5; ++s) for (float* d : {q.dW[s][0], q.dW[s][1], q.dbias[s]}) LTB_SETTLE(d);
  return LTB_OK;
}
static int tree_node_check(const ltb_tree_node* n, const char* who) {
  LTB_REQUIRE(n, "tree_node: null node");
  const int G = n->inner ? 5 : 3;
  LTB_REQUIRE(n->hidden > 0 && n->hidden <= kNodeMaxHidden && n->in_len > 0 && n->classes > 0 && n->classes <= 32, "tree_node: hidden must be 1..512, classes 1..32");
  LTB_REQUIRE(n->in[0] && (!n->inner || (n->in[1] && n->cl && n->cr)) && n->Why && n->by && n->score && n->gates && n->c && n->tc && n->h && n->logp && n->loss,
              "tree_node: missing operand");
  for (int g = 0; g < G; ++g) {
    const int slot = n->inner ? g : (g == 0 ? 0 : g + 2);
    LTB_REQUIRE(n->W[slot][0] && n->bias[slot] && (!n->inner || n->W[slot][1]), "tree_node: missing gate matrix or bias");
  }
  (void)who;
  return LTB_OK;
}

int ltb_tree_node_fwd(const ltb_tree_node* n) {
  LTB_INITED();
  if (int rc = tree_node_check(n, "ltb_tree_node_fwd")) return rc;
  filter_cache_note_write(nullptr, 0);                  // what it writes is a score of vectors: everything is taken as stale
  const int G = n->inner ? 5 : 3;
  LTB_LAUNCH(tree_node_fwd_kernel, (unsigned)ceil_div(G * n->hidden, kNodeWarps), kNodeThreads, 0, *n);
  return LTB_OK;
}

int ltb_tree_node_bwd(const ltb_tree_node* n) {
  LTB_INITED();
  if (int rc = tree_node_check(n, "ltb_tree_node_bwd")) return rc;
  if (int rc = tree_node_settle(*n)) return rc;
  filter_cache_note_write(nullptr, 0);
  const int G = n->inner ? 5 : 3;
  LTB_REQUIRE(n->dc && n->dh && n->dloss && n->dWhy && n->dby, "ltb_tree_node_bwd: missing gradient operand");
  for (int g = 0; g < G; ++g) {
    const int slot = n->inner ? g : (g == 0 ? 0 : g + 2);
    LTB_REQUIRE(n->dW[slot][0] && n->dbias[slot] && (!n->inner || n->dW[slot][1]), "ltb_tree_node_bwd: missing gate gradient");
  }
  const int n_w = (int)ceil_div(G * n->hidden, kNodeWarps);
  const bool any_din = n->din[0] || (n->inner && n->din[1]);
  const int x_warps = any_din ? (n->inner ? 2 : 1) * (int)ceil_div(n->in_len, 32) * G * (int)ceil_div(n->hidden, 32) : 0;
  LTB_LAUNCH(tree_node_bwd_kernel, (unsigned)(n_w + ceil_div(x_warps, kNodeWarps)), kNodeThreads, 0, *n, n_w);
  return LTB_OK;
}

// One level of a tree -- `count` nodes that do not depend on one another -- in one launch each way.  nodes_host and nodes_dev
// are the same array on the host (read here: checks, grid size) and in device memory (read by the kernels); the nodes of the
// call are [first, first + count).
int ltb_tree_nodes_fwd(const ltb_tree_node* nodes_host, const ltb_tree_node* nodes_dev, int first, int count) {
  LTB_INITED(); LTB_REQUIRE(nodes_host && nodes_dev && first >= 0 && count > 0, "ltb_tree_nodes_fwd: bad argument");
  filter_cache_note_write(nullptr, 0);
  for (int at = first; at < first + count; at += kNodesPerLaunch) {
    const int n = first + count - at < kNodesPerLaunch ? first + count - at : kNodesPerLaunch;
    int ctas = 1;
    for (int i = at; i < at + n; ++i) {
      if (int rc = tree_node_check(nodes_host + i, "ltb_tree_nodes_fwd")) return rc;
      const int c = (int)ceil_div((nodes_host[i].inner ? 5 : 3) * nodes_host[i].hidden, kNodeWarps);
      if (c > ctas) ctas = c;
    }
    LTB_LAUNCH(tree_nodes_fwd_kernel, dim3((unsigned)ctas, (unsigned)n), kNodeThreads, 0, nodes_dev + at);
  }
  return LTB_OK;
}
int ltb_tree_nodes_bwd(const ltb_tree_node* nodes_host, const ltb_tree_node* nodes_dev, int first, int count) {
  LTB_INITED(); LTB_REQUIRE(nodes_host && nodes_dev && first >= 0 && count > 0, "ltb_tree_nodes_bwd: bad argument");
  filter_cache_note_write(nullptr, 0);
  for (int at = first; at < first + count; at += kNodesPerLaunch) {
    const int n = first + count - at < kNodesPerLaunch ? first + count - at : kNodesPerLaunch;
    int ctas = 1;
    for (int i = at; i < at + n; ++i) {
      const ltb_tree_node* q = nodes_host + i;
      if (int rc = tree_node_check(q, "ltb_tree_nodes_bwd")) return rc;
      if (int rc = tree_node_settle(*q)) return rc;
      const int G = q->inner ? 5 : 3;
      LTB_REQUIRE(q->dc && q->dh && q->dloss && q->dWhy && q->dby, "ltb_tree_nodes_bwd: missing gradient operand");
      for (int g = 0; g < G; ++g) {
        const int slot = q->inner ? g : (g == 0 ? 0 : g + 2);
        LTB_REQUIRE(q->dW[slot][0] && q->dbias[slot] && (!q->inner || q->dW[slot][1]), "ltb_tree_nodes_bwd: missing gate gradient");
      }
      const bool any_din = q->din[0] || (q->inner && q->din[1]);
      const int x_warps = any_din ? (q->inner ? 2 : 1) * (int)ceil_div(q->in_len, 32) * G * (int)ceil_div(q->hidden, 32) : 0;
      const int c = (int)ceil_div(G * q->hidden, kNodeWarps) + (int)ceil_div(x_warps, kNodeWarps);
      if (c > ctas) ctas = c;
    }
    LTB_LAUNCH(tree_nodes_bwd_kernel, dim3((unsigned)ctas, (unsigned)n), kNodeThreads, 0, nodes_dev + at);
  }
  return LTB_OK;
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------------------------
// A whole tree per call (ltb_tree_fwd / ltb_tree_bwd).
//
// Level by level (above) a level costs 10 us whatever it holds: a launch, the description, the weights out of L2, a counter, the combination by
// the last CTA.  Here the chain of levels runs in ONE thread-block cluster of sixteen CTAs, a warp per hidden unit, and a level is one hardware cluster barrier.
//   tree_leaves_fwd   all leaves, on the whole machine: a warp holds the three gate rows of a unit and takes every `shares`-th leaf.
//   tree_chain_fwd    a warp holds the five gate rows of its unit (50 floats per lane) and computes gates, cell and hidden state of one node after the other; the two
//                     states go into the shared memory of all CTAs, where the next level finds them.  Then a warp per node classifies.
//   tree_chain_bwd    a warp holds the two columns of its unit (50 floats per lane): what reaches the unit in a node's children is the product of those
//                     with the node's 5 Hd gate gradients.  Everything of a unit -- its states, its gradients in every node -- stays in the warp's own part
//                     of shared memory; only the gate gradients are written to all CTAs.
//   tree_weights_bwd  weight gradients on the whole machine: a warp per row, over all nodes in order (a bias that two gates share takes two atomic additions).
// A grid-wide barrier on a counter in memory instead of the cluster's takes 6 us per level (25 leaves, nine levels: 70 us forward, 81 backward).
// Bound: the chain, 0.8 us per level (barrier and exchange) and some 0.5 us per node forward, 0.8 backward; 25 leaves 9 + 33 us forward, 45 + 13 backward
// (event-timed, with some 4 us of the event pair each; level by level 105 and 110 for the two directions), the step 202 -> 123 us.
namespace ltb {

constexpr int kTreeUnits = 160;                        // warps of a chain kernel: CTAS thread blocks of kTreeUnits / CTAS warps
constexpr int kTreeHidden = kTreeUnits, kTreeIn = 320, kTreeNodes = 119, kTreeChunk = 8;      // limits; nodes whose gate gradients are exchanged at once
constexpr int kTreeH = kTreeHidden / 32, kTreeI = kTreeIn / 32, kTreeR = 5 * kTreeHidden / 32;            // floats per lane: half a gate row, a leaf's row, a column

struct TreeView {
  const ltb_tree& t; int n, p;
  const int32_t *left, *right, *score, *word, *first;
  __device__ TreeView(const ltb_tree& t_) : t(t_), n(t_.nodes), p(LTB_TREE_PITCH(t_.hidden)), left(t_.topo), right(left + n), score(right + n), word(score + n), first(word + n) {}
  __device__ float* V(int i) const { return t.values + (size_t)i * (8 * p + 64); }
  __device__ float* G(int i) const { return t.grads + (size_t)i * (2 * p + 64); }
  // a parent's gates read the first state of its children, its cell the second; the classifier reads the first
  __device__ int first_state() const { return (t.classify_cell ? 5 : 7) * p; }
  __device__ int second_state() const { return (t.classify_cell ? 7 : 5) * p; }
};

// Sums of five values over the warp in eight exchanges: a lane ends up with the total of gate five_of(lane) alone.
__device__ __forceinline__ int five_of(int lane) { return lane & 4 ? 4 : (lane & 8 ? 2 : 0) + (lane & 16 ? 1 : 0); }
__device__ __forceinline__ float warp_add_five(const float* a, int lane) {
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
  float v0 = (b4 ? a[1] : a[0]) + __shfl_xor_sync(0xffffffffu, b4 ? a[0] : a[1], 16);
  const float v1 = (b4 ? a[3] : a[2]) + __shfl_xor_sync(0xffffffffu, b4 ? a[2] : a[3], 16);
  float v2 = a[4] + __shfl_xor_sync(0xffffffffu, a[4], 16);
  v0 = (b3 ? v1 : v0) + __shfl_xor_sync(0xffffffffu, b3 ? v0 : v1, 8);
  v2 += __shfl_xor_sync(0xffffffffu, v2, 8);
  v0 = (b2 ? v2 : v0) + __shfl_xor_sync(0xffffffffu, b2 ? v0 : v2, 4);
  v0 += __shfl_xor_sync(0xffffffffu, v0, 2);
  return v0 + __shfl_xor_sync(0xffffffffu, v0, 1);
}

__global__ void __launch_bounds__(kNodeThreads) tree_leaves_fwd_kernel(const ltb_tree tree, int shares) {
  pdl_wait();
  pdl_launch();                   // in this order: the chain kernel reads the weights before it waits for this one
  const TreeView T(tree);
  const int lane = threadIdx.x & 31, Hd = tree.hidden, L = tree.in_len;
  const int at = (int)blockIdx.x * kNodeWarps + ((int)threadIdx.x >> 5), u = at % Hd, share = at / Hd;
  if (share >= shares) return;
  float w[3][kTreeI], bias[3];
#pragma unroll
  for (int g = 0; g < 3; ++g) {
    const int slot = node_slot(false, g);
    bias[g] = tree.leaf_bias[slot][u];
#pragma unroll
    for (int m = 0; m < kTreeI; ++m) { const int k = lane + 32 * m; w[g][m] = k < L ? tree.leaf_W[slot][(size_t)u * L + k] : 0.0f; }
  }
  const int leaves = T.first[1];
  for (int i = share; i < leaves; i += 2 * shares) {           // two leaves' loads in flight; the weights beyond L are zero, so the index may be clamped
    const int i1 = min(i + shares, leaves - 1);
    const float* x0 = tree.table + (size_t)__ldg(T.word + i) * L; const float* x1 = tree.table + (size_t)__ldg(T.word + i1) * L;
    float a[6] = {};
    float v0[kTreeI], v1[kTreeI];
#pragma unroll
    for (int m = 0; m < kTreeI; ++m) { const int k = min(lane + 32 * m, L - 1); v0[m] = __ldg(x0 + k); v1[m] = __ldg(x1 + k); }
#pragma unroll
    for (int m = 0; m < kTreeI; ++m)
#pragma unroll
      for (int g = 0; g < 3; ++g) { a[g] += w[g][m] * v0[m]; a[3 + g] += w[g][m] * v1[m]; }
#pragma unroll
    for (int g = 0; g < 6; ++g) a[g] = warp_add(a[g]) + bias[g % 3];
    if (lane < 2 && (lane == 0 || i + shares < leaves)) {
      const float ig = act_apply(0, lane ? a[3] : a[0]), og = act_apply(3, lane ? a[4] : a[1]), uv = act_apply(4, lane ? a[5] : a[2]), c = ig * uv, tc = tanhf(c);
      float* v = T.V(lane ? i + shares : i);
      v[u] = ig; v[3 * Hd + u] = og; v[4 * Hd + u] = uv;
      v[5 * T.p + u] = c; v[6 * T.p + u] = tc; v[7 * T.p + u] = og * tc;
    }
  }
}

// This CTA's units of `rows` vectors of Hs floats into the same place of the other CTAs, eight bytes at a time (a float at a time from each unit's warp
// the network between the SMs takes 1.5 us per node).
template <int CTAS>
__device__ __forceinline__ void tree_spread(const cg::cluster_group& cluster, float* v, int rows, int Hs, int rank) {
  constexpr int kWarps = kTreeUnits / CTAS, kParts = kWarps / 2;
  for (int i = threadIdx.x; i < rows * CTAS * kParts; i += 32 * kWarps) {
    const int rest = i / kParts, row = rest / CTAS, to = rest - row * CTAS, at = rank * kWarps + (i - rest * kParts) * 2;
    if (to == rank || at >= Hs) continue;
    float* p = v + (size_t)row * Hs + at;
    *reinterpret_cast<float2*>(cluster.map_shared_rank(p, to)) = *reinterpret_cast<const float2*>(p);
  }
}
// Shared memory: state [node][2][Hs] (first, second; Hs = hidden rounded up to 32, zeros beyond hidden), kept [unit of the CTA][inner node][8] (gates, c, tanh c,
// h: they go to memory at the end, because a cluster barrier waits for every store to memory before it), why [classes][hidden], loss [node], left,
// right [node], first [levels + 1].
template <int CTAS>
__global__ void __launch_bounds__(32 * kTreeUnits / CTAS, 1) tree_chain_fwd_kernel(const ltb_tree tree) {
  constexpr int kWarps = kTreeUnits / CTAS, kThreads = 32 * kWarps;
  extern __shared__ float sm[];
  const TreeView T(tree);
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)cluster.block_rank();
  const int Hd = tree.hidden, Hs = (Hd + 31) / 32 * 32, n = T.n, u = rank * kWarps + warp;
  const int inner = n / 2;                                   // room for: of n nodes no more have two children of their own (a tree has as many, nodes that are no one's children make it fewer)
  const int K = tree.classes;
  float* state = sm; float* kept = state + (size_t)n * 2 * Hs; float* why = kept + (size_t)kWarps * inner * 8; float* loss = why + K * Hd;
  int* left = reinterpret_cast<int*>(loss + n); int* right = left + n; int* first = right + n;
  pdl_launch();
  float w0[5][kTreeH], w1[5][kTreeH], bias = 0.0f;
#pragma unroll
  for (int g = 0; g < 5; ++g)
#pragma unroll
    for (int m = 0; m < kTreeH; ++m) {
      const int k = lane + 32 * m; const bool ok = u < Hd && k < Hd && tree.levels > 1;
      w0[g][m] = ok ? tree.W[g][0][(size_t)u * Hd + k] : 0.0f; w1[g][m] = ok ? tree.W[g][1][(size_t)u * Hd + k] : 0.0f;
    }
  const int my_gate = five_of(lane);
  if (u < Hd && tree.levels > 1) bias = tree.bias[my_gate][u];
  pdl_wait();
  for (int i = tid; i < n; i += kThreads) { left[i] = T.left[i]; right[i] = T.right[i]; }
  for (int i = tid; i <= tree.levels; i += kThreads) first[i] = T.first[i];
  const int leaves = T.first[1], quads = leaves * 2 * (Hs / 4);
  for (int i = tid; i < K * Hd; i += kThreads) why[i] = tree.Why[i];
  for (int i = quads + tid; i < n * 2 * (Hs / 4); i += kThreads) reinterpret_cast<float4*>(state)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i0 = tid; i0 < quads; i0 += 4 * kThreads) {   // the leaves' states, four loads of a thread in flight
    float4 v[4]; int k[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 + e * kThreads, row = i / (Hs / 4), q = row >> 1;
      k[e] = (i - row * (Hs / 4)) * 4;
      v[e] = i < quads && k[e] < Hd ? __ldg(reinterpret_cast<const float4*>(T.V(q) + (row & 1 ? T.second_state() : T.first_state()) + k[e])) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 + e * kThreads;
      if (k[e] + 1 >= Hd) v[e].y = 0.0f;
      if (k[e] + 2 >= Hd) v[e].z = 0.0f;
      if (k[e] + 3 >= Hd) v[e].w = 0.0f;
      if (i < quads) reinterpret_cast<float4*>(state)[i] = v[e];
    }
  }
  cluster.sync();                                            // before the first write from another CTA
  for (int level = 1; level < tree.levels; ++level) {
    const int begin = first[level], end = first[level + 1];
    float* const mine = kept + ((size_t)warp * inner + begin - leaves) * 8;      // this unit's values of the level's nodes
    if (u < Hd) {
      // the products, two nodes at a time (one after the other their latencies add up: 1800 cycles a node with the gates below)
      for (int q = begin; q < end; q += 2) {
        const int q1 = min(q + 1, end - 1);
        const float* x[4] = {state + (size_t)left[q] * 2 * Hs, state + (size_t)right[q] * 2 * Hs, state + (size_t)left[q1] * 2 * Hs, state + (size_t)right[q1] * 2 * Hs};
        float a[2][5] = {};
#pragma unroll
        for (int m = 0; m < kTreeH; ++m) {
          if (32 * m >= Hs) break;
          float v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = x[e][lane + 32 * m];
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int g = 0; g < 5; ++g) a[e][g] += w0[g][m] * v[2 * e] + w1[g][m] * v[2 * e + 1];
        }
        const float p0 = warp_add_five(a[0], lane) + bias, p1 = warp_add_five(a[1], lane) + bias;
        if ((lane & 3) == 0 && (lane < 5 || !(lane & 4))) { mine[(q - begin) * 8 + my_gate] = p0; mine[(q1 - begin) * 8 + my_gate] = p1; }
      }
      __syncwarp();
      // the gates and the cell, a lane per node
      for (int i = lane; i < end - begin; i += 32) {
        float* v = mine + i * 8;
        const float ig = act_apply(0, v[0]), fl = act_apply(1, v[1]), fr = act_apply(2, v[2]), og = act_apply(3, v[3]), uv = act_apply(4, v[4]);
        const int q = begin + i;
        const float c = (ig * uv + fl * state[(size_t)(2 * left[q] + 1) * Hs + u]) + fr * state[(size_t)(2 * right[q] + 1) * Hs + u], tc = tanhf(c), h = og * tc;
        *reinterpret_cast<float4*>(v) = make_float4(ig, fl, fr, og); *reinterpret_cast<float4*>(v + 4) = make_float4(uv, c, tc, h);
        state[(size_t)2 * q * Hs + u] = tree.classify_cell ? c : h; state[(size_t)(2 * q + 1) * Hs + u] = tree.classify_cell ? h : c;
      }
    }
    __syncthreads();
    tree_spread<CTAS>(cluster, state + (size_t)begin * 2 * Hs, 2 * (end - begin), Hs, rank);
    cluster.sync();                                          // the level's states are in every CTA
  }
  for (int i = tid; i < (n - leaves) * 8 * kWarps; i += kThreads) {   // neighbouring threads on neighbouring units
    const int ne = i / kWarps, a = i - ne * kWarps, q = ne >> 3, e = ne & 7, unit = rank * kWarps + a;
    if (unit < Hd) T.V(leaves + q)[(e < 5 ? e * Hd : e * T.p) + unit] = kept[((size_t)a * inner + q) * 8 + e];
  }
  // log probabilities and each node's own part of the loss: a warp per node, the parts gathered by CTA 0
  float* const loss0 = cluster.map_shared_rank(loss, 0);
  for (int i = rank * kWarps + warp; i < n; i += CTAS * kWarps) {
    const float* x = state + (size_t)i * 2 * Hs;
    float o = -3.4028235e38f;
    for (int k = 0; k < K; ++k) {
      float a = 0.0f;
      for (int j = lane; j < Hd; j += 32) a += why[k * Hd + j] * x[j];
      a = warp_add(a);
      if (lane == k) o = a + tree.by[k];
    }
    const float m = warp_max(o), lse = m + logf(warp_add(lane < K ? expf(o - m) : 0.0f));
    if (lane < K) T.V(i)[8 * T.p + lane] = o - lse;
    if (lane == T.score[i]) loss0[i] = -(o - lse);
  }
  cluster.sync();
  if (rank != 0 || warp != 0) return;
  for (int level = 0; level < tree.levels; ++level) {
    for (int i = first[level] + lane; i < first[level + 1]; i += 32) {
      const float v = level == 0 ? loss[i] : (loss[i] + loss[left[i]]) + loss[right[i]];
      loss[i] = v; T.V(i)[8 * T.p + 32] = v;
    }
    __syncwarp();
  }
}

// work: per node 5 Hd gate gradients and 32 of the classifier, for tree_weights_bwd.
// Shared memory: dpre [2][kTreeChunk][5][Hs] (Hs as above), per unit of the CTA and node eight values (five gates, tanh c, the children's second states) and
// two gradients (first, second state) and the five gate gradients (to memory at the end, as above), why [classes][unit], dpred [node][classes], dloss [node], left, right [node], first [levels + 1].
template <int CTAS>
__global__ void __launch_bounds__(32 * kTreeUnits / CTAS, 1) tree_chain_bwd_kernel(const ltb_tree tree, float* work) {
  constexpr int kWarps = kTreeUnits / CTAS, kThreads = 32 * kWarps;
  extern __shared__ float sm[];
  const TreeView T(tree);
  cg::cluster_group cluster = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)cluster.block_rank();
  const int Hd = tree.hidden, Hs = (Hd + 31) / 32 * 32, K = tree.classes, n = T.n, R = 5 * Hs, u0 = rank * kWarps, u = u0 + warp, wstride = 5 * Hd + 32;
  float* dpre = sm; float* vals = dpre + 2 * kTreeChunk * R; float* grad = vals + (size_t)kWarps * n * 8; float* kept = grad + (size_t)kWarps * n * 2; float* why = kept + (size_t)kWarps * n * 5;
  float* dpred = why + K * kWarps; float* dloss = dpred + n * K;
  int* left = reinterpret_cast<int*>(dloss + n); int* right = left + n; int* first = right + n;
  pdl_enter();
  float w0[kTreeR], w1[kTreeR];
#pragma unroll
  for (int m = 0; m < kTreeR; ++m) {
    const int g = 32 * m / Hs, j = lane + 32 * m - g * Hs; const bool ok = u < Hd && g < 5 && j < Hd && tree.levels > 1;
    w0[m] = ok ? tree.W[g][0][(size_t)j * Hd + u] : 0.0f; w1[m] = ok ? tree.W[g][1][(size_t)j * Hd + u] : 0.0f;
  }
  const int leaves = T.first[1], second = T.second_state();
  for (int i = tid; i < n; i += kThreads) { left[i] = T.left[i]; right[i] = T.right[i]; dloss[i] = T.G(i)[2 * T.p]; }
  for (int i = tid; i <= tree.levels; i += kThreads) first[i] = T.first[i];
  for (int i = tid; i < 2 * kTreeChunk * R; i += kThreads) dpre[i] = 0.0f;
  for (int i = tid; i < K * kWarps; i += kThreads) { const int k = i / kWarps, a = u0 + i - k * kWarps; why[i] = a < Hd ? tree.Why[(size_t)k * Hd + a] : 0.0f; }
  for (int i0 = tid; i0 < n * 10 * kWarps; i0 += 8 * kThreads) {      // neighbouring threads on neighbouring units, eight loads of a thread in flight
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = i0 + j * kThreads, nu = i / kWarps, a = i - nu * kWarps, q = nu / 10, e = nu - q * 10;
      v[j] = 0.0f;
      if (q < n && u0 + a < Hd) {
        const float* at = nullptr;
        if (e < 5) at = e == 0 || e > 2 || q >= leaves ? T.V(q) + e * Hd : nullptr;
        else if (e == 5) at = T.V(q) + 6 * T.p;
        else if (e < 8) at = q >= leaves ? T.V(e == 6 ? __ldg(T.left + q) : __ldg(T.right + q)) + second : nullptr;
        else at = T.G(q) + ((e == 8) == (tree.classify_cell != 0) ? 0 : T.p);           // first: dc where the cell is classified, else dh
        if (at) v[j] = at[u0 + a];
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int i = i0 + j * kThreads, nu = i / kWarps, a = i - nu * kWarps, q = nu / 10, e = nu - q * 10;
      if (q < n) { if (e < 8) vals[((size_t)a * n + q) * 8 + e] = v[j]; else grad[((size_t)a * n + q) * 2 + e - 8] = v[j]; }
    }
  }
  __syncthreads();
  if (warp == 0) {                                           // the loss gradient goes down the tree unchanged
    for (int level = tree.levels - 1; level > 0; --level) {
      for (int q = first[level] + lane; q < first[level + 1]; q += 32) { dloss[left[q]] += dloss[q]; dloss[right[q]] += dloss[q]; }
      __syncwarp();
    }
  }
  __syncthreads();
  for (int i = tid; i < n * K; i += kThreads) {          // nllLoss_grad, logSoftmax_grad
    const int q = i / K, k = i - q * K;
    const float d = dloss[q] * (expf(T.V(q)[8 * T.p + k]) - (k == T.score[q] ? 1.0f : 0.0f));
    dpred[i] = d;
  }
  if (rank == 0) for (int i = tid; i < n; i += kThreads) T.G(i)[2 * T.p] = dloss[i];
  cluster.sync();                                            // shared memory of every CTA is set up
  float* const my_vals = vals + (size_t)warp * n * 8; float* const my_grad = grad + (size_t)warp * n * 2;
  // gate gradients of node q at this warp's unit; the children's second states get theirs
  auto gates_of = [&](int q, bool inner, float* d) {
    const float* v = my_vals + (size_t)q * 8;
    float dfirst = my_grad[q * 2];
    const float dsecond = my_grad[q * 2 + 1];
    float dcls = 0.0f;
    for (int k = 0; k < K; ++k) dcls += why[k * kWarps + warp] * dpred[q * K + k];
    dfirst += dcls;
    const float dc = tree.classify_cell ? dfirst : dsecond, dh = tree.classify_cell ? dsecond : dfirst;
    const float ig = v[0], fl = v[1], fr = v[2], og = v[3], uv = v[4], tc = v[5];
    const float dct = dc + dh * og * (1.0f - tc * tc);
    d[0] = (dct * uv) * ig * (1.0f - ig); d[3] = (dh * tc) * og * (1.0f - og); d[4] = (dct * ig) * (1.0f - uv * uv);
    d[1] = (dct * v[6]) * fl * (1.0f - fl); d[2] = (dct * v[7]) * fr * (1.0f - fr);       // zero in a leaf
    if (inner) { my_grad[left[q] * 2 + 1] += dct * fl; my_grad[right[q] * 2 + 1] += dct * fr; }
    float* o = kept + ((size_t)warp * n + q) * 5;
#pragma unroll
    for (int e = 0; e < 5; ++e) o[e] = d[e];
  };
  int turn = 0;
  for (int level = tree.levels - 1; level > 0; --level)
    for (int q0 = first[level]; q0 < first[level + 1]; q0 += kTreeChunk, turn ^= 1) {
      const int nq = min(kTreeChunk, first[level + 1] - q0);
      float* const buf = dpre + (size_t)turn * kTreeChunk * R;
      if (u < Hd && lane < nq) {
        float d[5];
        gates_of(q0 + lane, true, d);
#pragma unroll
        for (int e = 0; e < 5; ++e) buf[(size_t)lane * R + e * Hs + u] = d[e];
      }
      __syncthreads();
      tree_spread<CTAS>(cluster, buf, 5 * nq, Hs, rank);
      // everybody has the chunk's gate gradients; the buffer of the chunk before is free again once all have met the next time
      cluster.sync();
      if (u < Hd)
        for (int b = 0; b < nq; b += 2) {                    // two nodes at a time
          const int b1 = min(b + 1, nq - 1);
          float a[4] = {};
#pragma unroll
          for (int m = 0; m < kTreeR; ++m) {
            if (32 * m >= R) break;
            const float x0 = buf[(size_t)b * R + lane + 32 * m], x1 = buf[(size_t)b1 * R + lane + 32 * m];
            a[0] += w0[m] * x0; a[1] += w1[m] * x0; a[2] += w0[m] * x1; a[3] += w1[m] * x1;
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) a[e] = warp_add(a[e]);
          if (lane < (b1 > b ? 4 : 2)) {
            const int q = q0 + (lane < 2 ? b : b1);
            my_grad[(lane & 1 ? right[q] : left[q]) * 2] += lane == 0 ? a[0] : lane == 1 ? a[1] : lane == 2 ? a[2] : a[3];
          }
        }
      __syncwarp();
    }
  if (u < Hd) for (int q = lane; q < leaves; q += 32) { float d[5]; gates_of(q, false, d); }
  __syncthreads();
  for (int i = tid; i < n * 2 * kWarps; i += kThreads) {             // what the nodes' gradients have become
    const int nu = i / kWarps, a = i - nu * kWarps, q = nu >> 1, e = nu & 1;
    if (u0 + a < Hd) T.G(q)[((e == 0) == (tree.classify_cell != 0) ? 0 : T.p) + u0 + a] = grad[((size_t)a * n + q) * 2 + e];
  }
  for (int i = tid; i < n * 5 * kWarps; i += kThreads) {
    const int ne = i / kWarps, a = i - ne * kWarps, q = ne / 5, e = ne - q * 5;
    if (u0 + a < Hd) work[(size_t)q * wstride + e * Hd + u0 + a] = kept[((size_t)a * n + q) * 5 + e];
  }
  if (rank == 0)
    for (int i = tid; i < n * K; i += kThreads) { const int q = i / K, k = i - q * K; work[(size_t)q * wstride + 5 * Hd + k] = dpred[i]; }
  cluster.sync();                                            // nobody leaves while its shared memory may still be written
}

// acc[m] += dp(q) x(q)[m] over the nodes lo <= q < hi, NB nodes' loads in flight; x writes M floats.  Returns the sum of dp.
template <int M, int NB, class DP, class X>
__device__ __forceinline__ float tree_outer(float* acc, int lo, int hi, const DP& dp, const X& x) {
  float total = 0.0f;
  for (int q = lo; q < hi; q += NB) {
    float v[NB][M], d[NB];
#pragma unroll
    for (int e = 0; e < NB; ++e) { const int i = min(q + e, hi - 1); d[e] = q + e < hi ? dp(i) : 0.0f; x(i, v[e]); }
#pragma unroll
    for (int e = 0; e < NB; ++e) {
      total += d[e];
#pragma unroll
      for (int m = 0; m < M; ++m) acc[m] += d[e] * v[e][m];
    }
  }
  return total;
}
// M floats of a vector of `len`, lane + 32 m; the index is clamped, not tested: what comes of the rest is not stored.
template <int M>
__device__ __forceinline__ void tree_lane(float* v, const float* p, int lane, int len) {
#pragma unroll
  for (int m = 0; m < M; ++m) v[m] = __ldg(p + min(lane + 32 * m, len - 1));
}
__global__ void __launch_bounds__(kNodeThreads) tree_weights_bwd_kernel(const ltb_tree tree, const float* __restrict__ work) {
  pdl_enter();
  __shared__ int left[kTreeNodes], right[kTreeNodes], word[kTreeNodes];
  const TreeView T(tree);
  const int lane = threadIdx.x & 31, Hd = tree.hidden, L = tree.in_len, K = tree.classes, wstride = 5 * Hd + 32;
  if ((int)threadIdx.x < T.n) { left[threadIdx.x] = T.left[threadIdx.x]; right[threadIdx.x] = T.right[threadIdx.x]; word[threadIdx.x] = T.word[threadIdx.x]; }
  __syncthreads();
  const int leaves = T.first[1], inner_rows = 5 * Hd, leaf_rows = 3 * Hd, s = T.first_state();
  int item = (int)blockIdx.x * kNodeWarps + ((int)threadIdx.x >> 5);
  float acc[kTreeI], total = 0.0f;
#pragma unroll
  for (int m = 0; m < kTreeI; ++m) acc[m] = 0.0f;
  if (item < inner_rows) {
    if (leaves == T.n) return;                               // a single leaf: the inner gates may not even exist
    const int g = item / Hd, u = item - g * Hd;
    float* d0 = tree.dW[g][0] + (size_t)u * Hd; float* d1 = tree.dW[g][1] + (size_t)u * Hd;
    float old[kTreeI];
#pragma unroll
    for (int m = 0; m < kTreeH; ++m) { const int k = lane + 32 * m; old[m] = k < Hd ? d0[k] : 0.0f; old[kTreeH + m] = k < Hd ? d1[k] : 0.0f; }
    total = tree_outer<kTreeI, 5>(acc, leaves, T.n, [&](int q) { return __ldg(work + (size_t)q * wstride + item); },
                                  [&](int q, float* v) { tree_lane<kTreeH>(v, T.V(left[q]) + s, lane, Hd); tree_lane<kTreeH>(v + kTreeH, T.V(right[q]) + s, lane, Hd); });
#pragma unroll
    for (int m = 0; m < kTreeH; ++m) { const int k = lane + 32 * m; if (k < Hd) { d0[k] = old[m] + acc[m]; d1[k] = old[kTreeH + m] + acc[kTreeH + m]; } }
    if (lane == 0) atomicAdd(tree.dbias[g] + u, total);
    return;
  }
  item -= inner_rows;
  if (item < leaf_rows) {
    const int g = node_slot(false, item / Hd), u = item % Hd;
    float* d0 = tree.leaf_dW[g] + (size_t)u * L;
    float old[kTreeI];
#pragma unroll
    for (int m = 0; m < kTreeI; ++m) { const int k = lane + 32 * m; old[m] = k < L ? d0[k] : 0.0f; }
    total = tree_outer<kTreeI, 5>(acc, 0, leaves, [&](int q) { return __ldg(work + (size_t)q * wstride + g * Hd + u); }, [&](int q, float* v) { tree_lane<kTreeI>(v, tree.table + (size_t)word[q] * L, lane, L); });
#pragma unroll
    for (int m = 0; m < kTreeI; ++m) { const int k = lane + 32 * m; if (k < L) d0[k] = old[m] + acc[m]; }
    if (lane == 0) atomicAdd(tree.leaf_dbias[g] + u, total);
    return;
  }
  item -= leaf_rows;
  if (item >= K) return;
  total = tree_outer<kTreeH, 10>(acc, 0, T.n, [&](int q) { return __ldg(work + (size_t)q * wstride + 5 * Hd + item); }, [&](int q, float* v) { tree_lane<kTreeH>(v, T.V(q) + s, lane, Hd); });
#pragma unroll
  for (int m = 0; m < kTreeH; ++m) { const int u = lane + 32 * m; if (u < Hd) tree.dWhy[(size_t)item * Hd + u] += acc[m]; }
  if (lane == 0) tree.dby[item] += total;
}

static size_t tree_smem_fwd(const ltb_tree& t, int ctas) {
  return ((size_t)t.nodes * (2 * ((t.hidden + 31) / 32 * 32) + 3) + (size_t)(kTreeUnits / ctas) * (t.nodes / 2) * 8 + (size_t)t.classes * t.hidden + t.levels + 1) * 4;
}
static size_t tree_smem_bwd(const ltb_tree& t, int ctas) {
  return ((size_t)2 * kTreeChunk * 5 * ((t.hidden + 31) / 32 * 32) + (size_t)(kTreeUnits / ctas) * ((size_t)t.nodes * 15 + t.classes) + (size_t)t.nodes * (t.classes + 3) + t.levels + 1) * 4;
}
static int tree_check(const ltb_tree* t, bool grads, const char* who) {
  LTB_REQUIRE(t && t->nodes > 0 && t->levels > 0 && t->hidden > 0 && t->in_len > 0 && t->classes > 0 && t->classes <= 32, "%s: bad argument", who);
  if (t->hidden > kTreeHidden || t->in_len > kTreeIn || t->nodes > kTreeNodes) return fail(LTB_E_LIMIT, "%s: hidden at most %d, in_len %d, %d nodes", who, kTreeHidden, kTreeIn, kTreeNodes);
  LTB_REQUIRE(aligned16(t->values), "%s: values must be 16-byte aligned", who);
  LTB_REQUIRE(t->Why && t->by && t->table && t->topo && t->topo_host && t->values && (!grads || (t->grads && t->dWhy && t->dby)), "%s: missing operand", who);
  for (int s = 0; s < 5; ++s) {
    LTB_REQUIRE(s == 1 || s == 2 || (t->leaf_W[s] && t->leaf_bias[s] && (!grads || (t->leaf_dW[s] && t->leaf_dbias[s]))), "%s: missing gate of the leaves", who);
    LTB_REQUIRE(t->levels == 1 || (t->W[s][0] && t->W[s][1] && t->bias[s] && (!grads || (t->dW[s][0] && t->dW[s][1] && t->dbias[s]))), "%s: missing gate", who);
  }
  // the topology the kernels will follow: levels in order, every child in a level below and of one parent
  const int n = t->nodes; const int32_t *left = t->topo_host, *right = left + n, *score = right + n, *word = score + n, *first = word + n;
  LTB_REQUIRE(t->levels <= n && first[0] == 0 && first[t->levels] == n, "%s: levels do not cover the nodes", who);
  bool taken[kTreeNodes] = {};
  for (int l = 0; l < t->levels; ++l) {
    LTB_REQUIRE(first[l] < first[l + 1] && first[l + 1] <= n, "%s: bad level", who);
    for (int i = first[l]; i < first[l + 1]; ++i) {
      LTB_REQUIRE(score[i] >= 0 && score[i] < t->classes, "%s: score out of range", who);
      if (l == 0) LTB_REQUIRE(left[i] < 0 && word[i] >= 0, "%s: bad leaf", who);
      else {
        LTB_REQUIRE(left[i] >= 0 && right[i] >= 0 && left[i] < first[l] && right[i] < first[l], "%s: a child is not below its parent", who);
        LTB_REQUIRE(left[i] != right[i] && !taken[left[i]] && !taken[right[i]], "%s: a node with two parents", who);
        taken[left[i]] = taken[right[i]] = true;
      }
    }
  }
  return LTB_OK;
}
// CTAs of the chain kernels' cluster: sixteen, twice the warps per SM of eight, where the device takes a cluster of that size (25 leaves, before the
// products went two nodes at a time: 43 us forward, 48 with eight), else eight, which every device does.  0: the kernels could not be set up.
template <int CTAS>
static bool tree_set_up() {
  const int smem = 220 * 1024;
  bool ok = cudaFuncSetAttribute(tree_chain_fwd_kernel<CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
            cudaFuncSetAttribute(tree_chain_bwd_kernel<CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess;
  if (ok && CTAS > 8) {
    ok = cudaFuncSetAttribute(tree_chain_fwd_kernel<CTAS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
         cudaFuncSetAttribute(tree_chain_bwd_kernel<CTAS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CTAS); cfg.blockDim = dim3(32 * kTreeUnits / CTAS); cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension; attr[0].val.clusterDim.x = CTAS; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int f = 0, b = 0;
    ok = ok && cudaOccupancyMaxActiveClusters(&f, tree_chain_fwd_kernel<CTAS>, &cfg) == cudaSuccess && f > 0 &&
         cudaOccupancyMaxActiveClusters(&b, tree_chain_bwd_kernel<CTAS>, &cfg) == cudaSuccess && b > 0;
  }
  cudaGetLastError();
  return ok;
}
static int tree_ctas() {
  static int device = -1, ctas = 0;
  if (device != g.device) { ctas = tree_set_up<16>() ? 16 : tree_set_up<8>() ? 8 : 0; device = g.device; }
  return ctas;
}

}  // namespace ltb

extern "C" {

int ltb_tree_fwd(const ltb_tree* t) {
  LTB_INITED();
  if (int rc = tree_check(t, false, "ltb_tree_fwd")) return rc;
  const int ctas = tree_ctas();
  if (!ctas) return fail(LTB_E_CUDA, "the tree kernels could not be set up");
  LTB_WRITES(t->values, (size_t)t->nodes * LTB_TREE_VALUES(t->hidden));
  const int leaves = t->topo_host[4 * t->nodes + 1];
  int shares = g.sm_count * kNodeWarps / t->hidden;           // a warp per unit and share of the leaves, a CTA per SM
  shares = shares < 1 ? 1 : shares > leaves ? leaves : shares;
  LTB_LAUNCH(tree_leaves_fwd_kernel, (unsigned)ceil_div((int64_t)shares * t->hidden, kNodeWarps), kNodeThreads, 0, *t, shares);
  const unsigned threads = 32 * kTreeUnits / ctas;
  if (ctas == 16) LTB_LAUNCH_CLUSTER_XZ(tree_chain_fwd_kernel<16>, dim3(16), dim3(threads), 16, 1, tree_smem_fwd(*t, 16), *t);
  else LTB_LAUNCH_CLUSTER_XZ(tree_chain_fwd_kernel<8>, dim3(8), dim3(threads), 8, 1, tree_smem_fwd(*t, 8), *t);
  return LTB_OK;
}
int ltb_tree_bwd(const ltb_tree* t) {
  LTB_INITED();
  if (int rc = tree_check(t, true, "ltb_tree_bwd")) return rc;
  for (float* d : {t->grads, t->dWhy, t->dby}) LTB_SETTLE(d);
  for (int s = 0; s < 5; ++s) for (float* d : {t->leaf_dW[s], t->leaf_dbias[s], t->dW[s][0], t->dW[s][1], t->dbias[s]}) LTB_SETTLE(d);
  const int ctas = tree_ctas();
  if (!ctas) return fail(LTB_E_CUDA, "the tree kernels could not be set up");
  filter_cache_note_write(nullptr, 0);                  // what it writes is a score of vectors: everything is taken as stale
  const size_t need = (size_t)t->nodes * (5 * t->hidden + 32) * 4;
  if (need > g.cur_scratch_bytes()) return fail(LTB_E_LIMIT, "ltb_tree_bwd: too many nodes for the library's workspace");
  float* work = g.cur_scratch();
  const unsigned threads = 32 * kTreeUnits / ctas;
  if (ctas == 16) LTB_LAUNCH_CLUSTER_XZ(tree_chain_bwd_kernel<16>, dim3(16), dim3(threads), 16, 1, tree_smem_bwd(*t, 16), *t, work);
  else LTB_LAUNCH_CLUSTER_XZ(tree_chain_bwd_kernel<8>, dim3(8), dim3(threads), 8, 1, tree_smem_bwd(*t, 8), *t, work);
  LTB_LAUNCH(tree_weights_bwd_kernel, (unsigned)ceil_div(8 * t->hidden + t->classes, kNodeWarps), kNodeThreads, 0, *t, (const float*)work);
  return LTB_OK;
}

}  // extern "C"
