// FP32 CUDA-core contraction path: GEMM family and implicit-GEMM convolution (forward, data-grad, weight-grad).
//
// This is the 1e-4 path (LTB_MATH_FP32) and the path for shapes the tensor-core engine does not take
// (strides not multiples of 16 bytes, tiny K such as the 1->10 5x5 MNIST convolution or the 3->64 stem).
// Replaces cublasSgemm call sites (TensorDslCublas.scala:204-282, 589-688) and the cuDNN convolution calls
// (TensorDslCudnn.scala:515-831).  Semantics follow TensorDslCPU.scala:379-472 (gemm) and 484-692 (conv).
//
// One kernel template: C[m,n] (op)= sum_k A(m,k) * B(k,n), both operands given by tables, so that the convolution variants never
// materialise the reference's `finput` (im2col) buffer: element (r, k) is p[row(r).off + kk(k).off], or zero where the bits of kk(k) are
// not all among those of row(r) (a tap outside the image).  A table entry costs the divisions once per row or once per k, not per element
// (computed per element they made the data-gradient of SqueezeNet's layers 5 TFLOP/s kernels); the bit test and 32-bit offsets, and 16-byte loads
// where four neighbours lie together, took the contractions of SqueezeNet's step at batch 64 from 1586 to 1448 us, entries made before the
// kernel waits for its predecessors to 1420.
//   tiles      : BM x BN outputs, 16 of k per step, 256 threads with (BM/16) x (BN/16) outputs each; the next step's operands travel to
//                registers while this one is computed, shared memory is double-buffered, one barrier per step.  (Element-wise
//                cp.async with three steps under way was slower: 41 against 48 TFLOP/s.)
//   arithmetic : packed pairs (fma.rn.f32x2): half the issue slots of scalar FMAs, which leaves room for the shared-memory loads.
//   output     : m is the index that is contiguous in memory (the caller swaps the operands for row-major results), so a thread's
//                four consecutive m leave as one 16-byte store or vector reduction.
// Bound: the FP32 pipes (128 FMA per SM and cycle, 74 TFLOP/s at 1.97 GHz) and, for an 8 x 8 tile of a thread as much, the 32 floats per cycle that
// shared memory delivers (four FMAs per float loaded); 55 TFLOP/s on 4096 x 4096 x 2048 with k contiguous, 51 without.  In the 3x3 layers
// that conv3x3_direct_kernel below takes a lane makes 24 PX FMAs of the PX + 2 pixels and 24 weights it loads, 5.6 per float in runs of eight pixels and 3.2 in runs
// of four; but a weight is one for the whole warp, so that six deliveries of 128 bytes hold them all and a warp makes 12 or 8 FMAs per delivery, where the tiles make four.
#include <cooperative_groups.h>

#include <type_traits>

#include "gemm.cuh"

namespace cg = cooperative_groups;

namespace ltb {

constexpr int BKK = 16;
// Narrow entries: element (r, k) is p[row.off + kk.off] where every bit of kk.bits is set in row.bits.  A convolution's row has a bit for
// each kh and each kw that stays inside the image (R + S <= 30 of them), its k the two of its tap; bit 31 says that the entry exists.
// Wide entries are for operands of 2^31 elements or more and for larger filters.
struct Ent { int off; unsigned bits; };
struct WideEnt { long long off; int h, w; };
constexpr unsigned kExists = 1u << 31, kNowhere = 1u << 30;  // no row has kNowhere
constexpr int kOutside = -(1 << 28);                        // an h that no partner brings back into range
__device__ __forceinline__ void outside_row(Ent& e) { e.off = 0; e.bits = 0; }
__device__ __forceinline__ void outside_row(WideEnt& e) { e.off = 0; e.h = kOutside; e.w = 0; }
__device__ __forceinline__ void outside_k(Ent& e) { e.off = 0; e.bits = kNowhere; }
__device__ __forceinline__ void outside_k(WideEnt& e) { e.off = 0; e.h = kOutside; e.w = 0; }
__device__ __forceinline__ bool meets(const Ent& r, const Ent& k) { return (r.bits & k.bits) == k.bits; }
__device__ __forceinline__ bool meets(const WideEnt& r, const WideEnt& k) { return r.h + k.h == 0; }       // entries without a place in an image
template <class E> __device__ __forceinline__ E plain_entry(long long off);
template <> __device__ __forceinline__ Ent plain_entry<Ent>(long long off) { return Ent{(int)off, kExists}; }
template <> __device__ __forceinline__ WideEnt plain_entry<WideEnt>(long long off) { return WideEnt{off, 0, 0}; }

__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

constexpr int kTables = 4;
// How an operand's elements are fetched.  FEED_ROW: single elements, neighbouring threads on neighbouring rows (a thread keeps its row);
// FEED_K: neighbouring threads on neighbouring k (a thread keeps its k).  _4: four neighbours at a time with one 16-byte load, where
// groups of four along the contiguous index are aligned and lie inside together.  That doubles the kernels (and their build), for, us one by one / four at a time:
// products, 32 of eight sizes and both orders of each operand, 0 to 14 % (2048^3 408 / 370 with both along k, 390 / 353 with neither, 397 / 397 and 399 / 393 mixed;
// 512 x 512 x 4096 100 / 92 to 84; 300 x 2000 x 320 23.5 / 21.6); 1x1 layers, fourteen, forward 0 to 7 % (128 -> 256 at 28 x 28 on 8 images 18.4 / 17.3), data-gradient
// 0 to 11 % (48 -> 192 at 8 x 8 on 64 images 12.7 / 11.3), weight gradient 1 to 6 %; larger filters, whose taps leave one operand as it was, 0 to 1 % forward
// (64 -> 64 3x3 at 28 x 28 on 32 images 72.2 / 71.5) and 1 to 3 % of the weight gradient (16 -> 64 at 16 x 16 on 64 images 24.0 / 23.2).  None was slower.
enum { FEED_ROW = 0, FEED_K = 1, FEED_ROW4 = 2, FEED_K4 = 3 };
// One operand's share of a step: T rows x BKK, fetched to registers, then stored k by k.
template <int T, int FEED, class OP>
struct Feed {
  using E = typename OP::Entry;
  static constexpr int P = T + 4;
  static constexpr int N = FEED >= FEED_ROW4 ? (T * BKK / 4 + 255) / 256 : T * BKK / 256;
  static constexpr bool whole = T * BKK / 4 >= 256;             // 16-byte items: fewer than threads for 32-row tiles
  float v[FEED >= FEED_ROW4 ? 4 * N : N];
  __device__ __forceinline__ void fetch(const OP& op, const E& mine, const E* rows, const E* ks, int tid) {
    if constexpr (FEED == FEED_K) {
      const E k = ks[tid & 15];
#pragma unroll
      for (int e = 0; e < N; ++e) v[e] = op.get(rows[(tid >> 4) + 16 * e], k);
    } else if constexpr (FEED == FEED_ROW) {
#pragma unroll
      for (int e = 0; e < N; ++e) v[e] = op.get(mine, ks[tid / T + (256 / T) * e]);
    } else if constexpr (FEED == FEED_ROW4) {
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const int k = tid / (T / 4) + (1024 / T) * e;
        const float4 t = whole || k < BKK ? op.get4(mine, ks[whole ? k : k & 15]) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[4 * e] = t.x; v[4 * e + 1] = t.y; v[4 * e + 2] = t.z; v[4 * e + 3] = t.w;
      }
    } else {
      const E k = ks[(tid & 3) * 4];
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const int r = (tid >> 2) + 64 * e;
        const float4 t = whole || r < T ? op.get4(rows[whole ? r : r & (T - 1)], k) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[4 * e] = t.x; v[4 * e + 1] = t.y; v[4 * e + 2] = t.z; v[4 * e + 3] = t.w;
      }
    }
  }
  // the row that a thread keeps (its first of four)
  static __device__ __forceinline__ int my_row(int tid) { return FEED == FEED_ROW4 ? tid % (T / 4) * 4 : tid % T; }
  static constexpr bool table = FEED == FEED_K || FEED == FEED_K4;
  __device__ __forceinline__ void store(float* s, int tid) const {
    if constexpr (FEED == FEED_ROW4) {
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const int k = tid / (T / 4) + (1024 / T) * e;
        if (whole || k < BKK) *reinterpret_cast<float4*>(s + k * P + tid % (T / 4) * 4) = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
      }
    } else if constexpr (FEED == FEED_K4) {
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const int r = (tid >> 2) + 64 * e;
        if (whole || r < T)
#pragma unroll
          for (int i = 0; i < 4; ++i) s[((tid & 3) * 4 + i) * P + r] = v[4 * e + i];
      }
    } else {
#pragma unroll
      for (int e = 0; e < N; ++e) {
        const int r = FEED == FEED_K ? (tid >> 4) + 16 * e : tid % T, k = FEED == FEED_K ? (tid & 15) : tid / T + (256 / T) * e;
        s[k * P + r] = v[e];
      }
    }
  }
};

template <int BM, int BN> constexpr int igemm_smem() {
  constexpr int operands = 2 * BKK * (BM + BN + 8) * 4, partial = BM * BN * 4;       // a split's partial tile takes the operands' place
  return operands > partial ? operands : partial;
}
template <int BM, int BN, int AF, int BF, class OA, class OB, class ST>
__global__ void __launch_bounds__(256, 2) igemm_kernel(int M, int N, int K, int k_per_split, const OA oa, const OB ob, const ST st) {
  pdl_launch();
  constexpr int PA = BM + 4, PB = BN + 4, TM = BM / 16, TN = BN / 16;
  extern __shared__ __align__(16) float pool[];
  using EA = typename OA::Entry; using EB = typename OB::Entry;
  using FA = Feed<BM, AF, OA>; using FB = Feed<BN, BF, OB>;
  __shared__ EA ka[kTables][BKK]; __shared__ EB kb[kTables][BKK];
  __shared__ EA ra[FA::table ? BM : 1]; __shared__ EB rb[FB::table ? BN : 1];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int k_begin = blockIdx.z * k_per_split, k_end = min(K, k_begin + k_per_split);
  const int steps = k_end > k_begin ? (k_end - k_begin + BKK - 1) / BKK : 0;          // the last splits may have nothing: they contribute zeros
  auto a_row = [&](int r) { EA e; if (m0 + r < M) e = oa.row(m0 + r); else outside_row(e); return e; };
  auto b_row = [&](int r) { EB e; if (n0 + r < N) e = ob.row(n0 + r); else outside_row(e); return e; };
  auto table = [&](int step, int i, bool second) {
    const int k = k_begin + step * BKK + i;
    if (second) { EB e; if (k < k_end) e = ob.kk(k); else outside_k(e); kb[step & (kTables - 1)][i] = e; }
    else { EA e; if (k < k_end) e = oa.kk(k); else outside_k(e); ka[step & (kTables - 1)][i] = e; }
  };
  EA mine_a; EB mine_b;
  if (FA::table) { for (int r = tid; r < BM; r += 256) ra[r] = a_row(r); } else mine_a = a_row(FA::my_row(tid));
  if (FB::table) { for (int r = tid; r < BN; r += 256) rb[r] = b_row(r); } else mine_b = b_row(FB::my_row(tid));
  if (tid < 4 * BKK) table(tid % (2 * BKK) / BKK, tid % BKK, tid >= 2 * BKK);            // steps 0 and 1
  __syncthreads();
  pdl_wait();                                               // the entries touch no memory: they are made while the kernels before run
  FA fa; FB fb;
  auto fetch = [&](int step) {
    fa.fetch(oa, mine_a, ra, ka[step & (kTables - 1)], tid);
    fb.fetch(ob, mine_b, rb, kb[step & (kTables - 1)], tid);
  };
  auto put_down = [&](int step) {
    float* as = pool + (step & 1) * BKK * (PA + PB);
    fa.store(as, tid); fb.store(as + BKK * PA, tid);
  };
  if (steps > 0) { fetch(0); put_down(0); }

  unsigned long long acc[TM / 2][TN];                       // pairs of neighbouring m
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
  const int tm = tid & 15, tn = tid >> 4;                   // rows tm*4 + 64*i.., columns tn*4 + 64*j.. (BN 32: tn*2)
  for (int s = 0; s < steps; ++s) {
    __syncthreads();                                        // step s is in shared memory, and everybody is done with step s - 1
    if (s + 1 < steps) fetch(s + 1);
    if (tid < 2 * BKK && s + 2 < steps) table(s + 2, tid & 15, tid >= BKK);              // read after the next barrier
    const float* as = pool + (s & 1) * BKK * (PA + PB); const float* bs = as + BKK * PA;
#pragma unroll
    for (int k = 0; k < BKK; ++k) {
      unsigned long long a[TM / 2]; float b[TN];
#pragma unroll
      for (int i = 0; i < TM / 4; ++i) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(as + k * PA + tm * 4 + 64 * i);
        a[2 * i] = t.x; a[2 * i + 1] = t.y;
      }
      if (TN >= 4) {
#pragma unroll
        for (int j = 0; j < TN / 4; ++j) *reinterpret_cast<float4*>(b + 4 * j) = *reinterpret_cast<const float4*>(bs + k * PB + tn * 4 + 64 * j);
      } else *reinterpret_cast<float2*>(b) = *reinterpret_cast<const float2*>(bs + k * PB + tn * 2);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const unsigned long long bj = pack2(b[j], b[j]);
#pragma unroll
        for (int i = 0; i < TM / 2; ++i) acc[i][j] = fma2(a[i], bj, acc[i][j]);
      }
    }
    if (s + 1 < steps) put_down(s + 1);
  }
  // Splits of K: up to eight form a thread-block cluster along z.  Every CTA leaves its partial tile in shared memory, then sums one
  // slice of the tile over the cluster in rank order: no zero fill, no atomics, the same bits on every run.
  cg::cluster_group cluster = cg::this_cluster();
  const int cz = (int)cluster.num_blocks();
  if (cz > 1) __syncthreads();                              // the last step's operands have been read
#pragma unroll
  for (int i4 = 0; i4 < TM / 4; ++i4) {
    const int ml = tm * 4 + 64 * i4, m = m0 + ml;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int nl = TN >= 4 ? tn * 4 + 64 * (j / 4) + (j & 3) : tn * 2 + j, n = n0 + nl;
      const float2 lo = unpack2(acc[2 * i4][j]), hi = unpack2(acc[2 * i4 + 1][j]);
      float v[4] = {lo.x, lo.y, hi.x, hi.y};
      if (cz > 1) *reinterpret_cast<float4*>(pool + nl * BM + ml) = make_float4(v[0], v[1], v[2], v[3]);
      else if (m < M && n < N) st(m, n, v, M - m);
    }
  }
  if (cz > 1) {
    cluster.sync();
    const int rank = (int)cluster.block_rank(), items = BM * BN / 4, per = (items + cz - 1) / cz;
    for (int i = rank * per + tid; i < min(items, (rank + 1) * per); i += 256) {
      const int nl = i / (BM / 4), ml = (i - nl * (BM / 4)) * 4, m = m0 + ml, n = n0 + nl;
      if (m >= M || n >= N) continue;
      float4 p[8];
#pragma unroll
      for (int z = 0; z < 8; ++z) if (z < cz) p[z] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(pool, z) + 4 * i);
      float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int z = 0; z < 8; ++z) if (z < cz) { v[0] += p[z].x; v[1] += p[z].y; v[2] += p[z].z; v[3] += p[z].w; }
      st(m, n, v, M - m);
    }
    cluster.sync();                                         // nobody leaves while its tile may still be read
  }
}

// ---- operands ------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float4 load4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
template <class E>
struct MatOpOf {                                            // a strided matrix
  using Entry = E;
  const float* p; long long sr, sk;
  __device__ __forceinline__ E row(int r) const { return plain_entry<E>(r * sr); }
  __device__ __forceinline__ E kk(int k) const { return plain_entry<E>(k * sk); }
  __device__ __forceinline__ float get(const E& r, const E& k) const { return meets(r, k) ? __ldg(p + (r.off + k.off)) : 0.0f; }
  __device__ __forceinline__ float4 get4(const E& r, const E& k) const { return meets(r, k) ? load4(p + (r.off + k.off)) : make_float4(0.f, 0.f, 0.f, 0.f); }
};
using MatOp = MatOpOf<Ent>; using WideMatOp = MatOpOf<WideEnt>;
// Output pixel (n, ho, wo) and tap (ci, kh, kw) of a convolution input.  PIXROW: the pixel is the row index (forward), else k (weight-gradient).
// The entry of whichever is the row carries a bit for each kh and kw (of the pixel: those inside the image; of the tap: its own), the
// other's is matched against it; in the weight gradient the roles of the two bit sets are exchanged: see meets().
template <bool PIXROW>
struct ConvInput {
  using Entry = Ent;
  const float* x; ConvDims d; FastDiv oW, oH, S, R;
  ConvInput(const float* x_, const ConvDims& d_) : x(x_), d(d_), oW(d_.oW), oH(d_.oH), S(d_.S), R(d_.R) {}
  // inside: the kh and kw that lie inside for this pixel
  __device__ __forceinline__ int pixel(int m, unsigned& inside) const {
    int wo, ho; const int n = oH.divmod(oW.divmod(m, wo), ho), h = ho * d.sh - d.ph, w = wo * d.sw - d.pw;
    inside = 0;
    for (int i = 0; i < d.R; ++i) if ((unsigned)(h + i) < (unsigned)d.H) inside |= 1u << i;
    for (int i = 0; i < d.S; ++i) if ((unsigned)(w + i) < (unsigned)d.W) inside |= 1u << (d.R + i);
    return (n * d.C * d.H + h) * d.W + w;
  }
  __device__ __forceinline__ int tap(int k, unsigned& own) const {
    int kw, kh; const int ci = R.divmod(S.divmod(k, kw), kh);
    own = (1u << kh) | (1u << (d.R + kw));
    return (ci * d.H + kh) * d.W + kw;
  }
  // own bits of the tap must be among the pixel's inside bits: with the tap as the row, the complements change sides
  __device__ __forceinline__ unsigned all() const { return (1u << (d.R + d.S)) - 1u; }
  __device__ __forceinline__ Ent row(int r) const {
    unsigned b; int off;
    if (PIXROW) off = pixel(r, b); else { off = tap(r, b); b = all() & ~b; }
    return Ent{off, b | kExists};
  }
  __device__ __forceinline__ Ent kk(int k) const {
    unsigned b; int off;
    if (PIXROW) off = tap(k, b); else { off = pixel(k, b); b = all() & ~b; }
    return Ent{off, b | kExists};
  }
  __device__ __forceinline__ float get(const Ent& r, const Ent& k) const { return meets(r, k) ? __ldg(x + (r.off + k.off)) : 0.0f; }
  __device__ __forceinline__ float4 get4(const Ent& r, const Ent& k) const { return meets(r, k) ? load4(x + (r.off + k.off)) : make_float4(0.f, 0.f, 0.f, 0.f); }
};
template <bool PIXROW>
struct WideConvInput {
  using Entry = WideEnt;
  const float* x; ConvDims d; FastDiv oW, oH, S, R;
  WideConvInput(const float* x_, const ConvDims& d_) : x(x_), d(d_), oW(d_.oW), oH(d_.oH), S(d_.S), R(d_.R) {}
  __device__ __forceinline__ WideEnt pixel(int m) const {
    int wo, ho; const int n = oH.divmod(oW.divmod(m, wo), ho), h = ho * d.sh - d.ph, w = wo * d.sw - d.pw;
    return WideEnt{(long long)n * d.C * d.H * d.W + (long long)h * d.W + w, h, w};
  }
  __device__ __forceinline__ WideEnt tap(int k) const {
    int kw, kh; const int ci = R.divmod(S.divmod(k, kw), kh);
    return WideEnt{((long long)ci * d.H + kh) * d.W + kw, kh, kw};
  }
  __device__ __forceinline__ WideEnt row(int r) const { return PIXROW ? pixel(r) : tap(r); }
  __device__ __forceinline__ WideEnt kk(int k) const { return PIXROW ? tap(k) : pixel(k); }
  __device__ __forceinline__ float get(const WideEnt& r, const WideEnt& k) const {
    return (unsigned)(r.h + k.h) < (unsigned)d.H && (unsigned)(r.w + k.w) < (unsigned)d.W ? x[r.off + k.off] : 0.0f;
  }
  __device__ __forceinline__ float4 get4(const WideEnt&, const WideEnt&) const { return make_float4(0.f, 0.f, 0.f, 0.f); }
};
// Input pixel (n, h, w) against (co, kh, kw) of dy: the element at ((h + ph - kh) / sh, (w + pw - kw) / sw) where that exists.  Where it does,
// h + ph and kh leave the same remainder, so the quotient is the difference of the two quotients and the offset still a sum.
struct ConvDy {
  using Entry = Ent;
  const float* dy; ConvDims d; FastDiv W, H, S, R, sh, sw;
  ConvDy(const float* dy_, const ConvDims& d_) : dy(dy_), d(d_), W(d_.W), H(d_.H), S(d_.S), R(d_.R), sh(d_.sh), sw(d_.sw) {}
  __device__ __forceinline__ Ent row(int m) const {
    int w, h, rh, rw; const int n = H.divmod(W.divmod(m, w), h);
    const int qh = sh.divmod(h + d.ph, rh), qw = sw.divmod(w + d.pw, rw);
    unsigned b = kExists;
    for (int i = rh, q = qh; i < d.R; i += d.sh, --q) if ((unsigned)q < (unsigned)d.oH) b |= 1u << i;
    for (int i = rw, q = qw; i < d.S; i += d.sw, --q) if ((unsigned)q < (unsigned)d.oW) b |= 1u << (d.R + i);
    return Ent{(n * d.K * d.oH + qh) * d.oW + qw, b};
  }
  __device__ __forceinline__ Ent kk(int k) const {
    int kw, kh; const int co = R.divmod(S.divmod(k, kw), kh);
    return Ent{(co * d.oH - sh.div(kh)) * d.oW - sw.div(kw), kExists | (1u << kh) | (1u << (d.R + kw))};
  }
  __device__ __forceinline__ float get(const Ent& r, const Ent& k) const { return meets(r, k) ? __ldg(dy + (r.off + k.off)) : 0.0f; }
  __device__ __forceinline__ float4 get4(const Ent& r, const Ent& k) const { return meets(r, k) ? load4(dy + (r.off + k.off)) : make_float4(0.f, 0.f, 0.f, 0.f); }
};
struct WideConvDy {
  using Entry = WideEnt;
  const float* dy; ConvDims d; FastDiv W, H, S, R;
  WideConvDy(const float* dy_, const ConvDims& d_) : dy(dy_), d(d_), W(d_.W), H(d_.H), S(d_.S), R(d_.R) {}
  __device__ __forceinline__ WideEnt row(int m) const {
    int w, h; const int n = H.divmod(W.divmod(m, w), h);
    return WideEnt{(long long)n * d.K * d.oH * d.oW, h + d.ph, w + d.pw};
  }
  __device__ __forceinline__ WideEnt kk(int k) const {
    int kw, kh; const int co = R.divmod(S.divmod(k, kw), kh);
    return WideEnt{(long long)co * d.oH * d.oW, -kh, -kw};
  }
  __device__ __forceinline__ float get(const WideEnt& r, const WideEnt& k) const {
    const int h = r.h + k.h, w = r.w + k.w;
    if (h < 0 || w < 0) return 0.0f;
    const int ho = h / d.sh, wo = w / d.sw;
    return ho * d.sh == h && wo * d.sw == w && ho < d.oH && wo < d.oW ? dy[r.off + k.off + (long long)ho * d.oW + wo] : 0.0f;
  }
  __device__ __forceinline__ float4 get4(const WideEnt&, const WideEnt&) const { return make_float4(0.f, 0.f, 0.f, 0.f); }
};
// Filter w[co][ci][tap] with row ci and k = (co, tap).
template <class E>
struct FilterByInput {
  using Entry = E;
  const float* w; int C, rs; FastDiv by;
  FilterByInput(const float* w_, int C_, int rs_) : w(w_), C(C_), rs(rs_), by(rs_) {}
  __device__ __forceinline__ E row(int ci) const { return plain_entry<E>((long long)ci * rs); }
  __device__ __forceinline__ E kk(int k) const { const int co = by.div(k); return plain_entry<E>((long long)co * C * rs + (k - co * rs)); }
  __device__ __forceinline__ float get(const E& r, const E& k) const { return meets(r, k) ? __ldg(w + (r.off + k.off)) : 0.0f; }
  __device__ __forceinline__ float4 get4(const E& r, const E& k) const { return meets(r, k) ? load4(w + (r.off + k.off)) : make_float4(0.f, 0.f, 0.f, 0.f); }
};
// dy[n][co][pixel] with row co and k = (n, pixel).
template <class E>
struct DyByPixel {
  using Entry = E;
  const float* dy; int K, hw; FastDiv by;
  DyByPixel(const float* dy_, int K_, int hw_) : dy(dy_), K(K_), hw(hw_), by(hw_) {}
  __device__ __forceinline__ E row(int co) const { return plain_entry<E>((long long)co * hw); }
  __device__ __forceinline__ E kk(int k) const { const int n = by.div(k); return plain_entry<E>((long long)n * K * hw + (k - n * hw)); }
  __device__ __forceinline__ float get(const E& r, const E& k) const { return meets(r, k) ? __ldg(dy + (r.off + k.off)) : 0.0f; }
  __device__ __forceinline__ float4 get4(const E& r, const E& k) const { return meets(r, k) ? load4(dy + (r.off + k.off)) : make_float4(0.f, 0.f, 0.f, 0.f); }
};

// ---- results: four consecutive m of column n, of which `left` exist -------------------------------------------------------------
// mode 0: = v (+ bias), 1: += v, 2: += v atomically (more splits of K than one cluster holds)
__device__ __forceinline__ void put(float* q, float v, int mode) { if (mode == 2) atomicAdd(q, v); else *q = mode == 1 ? *q + v : v; }
__device__ __forceinline__ void put4(float* q, const float* v, int mode) {
  float4 t = make_float4(v[0], v[1], v[2], v[3]);
  float4* q4 = reinterpret_cast<float4*>(q);
  if (mode == 2) { atomicAdd(q4, t); return; }
  if (mode == 1) { const float4 o = *q4; t.x += o.x; t.y += o.y; t.z += o.z; t.w += o.w; }
  *q4 = t;
}
struct MatPut {                                             // p[m * sm + n * sn]; vec: sm 1 and every group of four aligned
  float* p; long long sm, sn; float alpha; int mode, vec;
  __device__ __forceinline__ void operator()(int m, int n, float* v, int left) const {
    float* q = p + m * sm + n * sn;
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] *= alpha;
    if (vec && left >= 4) { put4(q, v, mode); return; }
#pragma unroll
    for (int u = 0; u < 4; ++u) if (u < left) put(q + u * sm, v[u], mode);
  }
};
struct PixelPut {                                           // p[img][n][pixel] of `chan` channels; vec: hw a multiple of 4, p aligned
  float* p; const float* bias; int chan, hw, mode, vec, relu; FastDiv by;
  PixelPut(float* p_, const float* bias_, int chan_, int hw_, int mode_, bool relu_) : p(p_), bias(bias_), chan(chan_), hw(hw_), mode(mode_), vec(hw_ % 4 == 0 && aligned16(p_)), relu(relu_), by(hw_) {}
  __device__ __forceinline__ void operator()(int m, int n, float* v, int left) const {
    const float b = bias ? bias[n] : 0.0f;
#pragma unroll
    for (int u = 0; u < 4; ++u) { v[u] += b; if (relu && v[u] < 0.0f) v[u] = 0.0f; }
    if (vec && left >= 4) { const int img = by.div(m); put4(p + ((long long)img * chan + n) * hw + (m - img * hw), v, mode); return; }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (u < left) { const int img = by.div(m + u); put(p + ((long long)img * chan + n) * hw + (m + u - img * hw), v[u], mode); }
  }
};

// ---- tile and split choice ---------------------------------------------------------------------------------------------------------
// The widest tile that N fills, 64 columns at most when 128-wide tiles do not cover the SMs; when the tiles are still too few K is split
// until three CTAs per SM have work: up to eight splits per cluster of 128 of k at least (with 64 the cluster's sum costs what the
// shorter chains save), and where the caller's sums may meet atomically several clusters per tile, 64 of k each at least.  (The weight
// gradients of SqueezeNet's layers at batch 64: three CTAs per SM 0.71 ms, two 0.77.)
struct Tiling { int bm, bn, cz, groups, kps; };
static Tiling choose_tiling(int M, int N, int K, bool may_add_atomically) {
  Tiling t;
  t.bn = N > 64 ? 128 : N > 32 ? 64 : 32;
  t.bm = 128;
  auto tiles = [&] { return ceil_div(M, t.bm) * ceil_div(N, t.bn); };
  if (t.bn == 128 && tiles() < g.sm_count) t.bn = 64;
  if (t.bn <= 64 && ceil_div(M, 64) * 64 * 5 <= ceil_div(M, 128) * 128 * 4) t.bm = 64;      // a fifth less padding
  int splits = 1;
  if (tiles() < g.sm_count) {
    const int chain = may_add_atomically ? 64 : 128, most = K / chain < 1 ? 1 : K / chain;
    if (tiles() * (may_add_atomically ? most : most < 8 ? most : 8) < 2 * g.sm_count) t.bm = 64;
    splits = (int)ceil_div(3 * g.sm_count, tiles());
    if (splits > most) splits = most;
  }
  t.cz = splits < 8 ? splits : 8;
  t.groups = may_add_atomically ? (int)ceil_div(splits, t.cz) : 1;
  t.kps = (int)(ceil_div(ceil_div(K, t.cz * t.groups), BKK) * BKK);
  t.groups = (int)ceil_div(K, (int64_t)t.kps * t.cz);                     // only clusters that have work
  return t;
}
template <int AF, int BF, class OA, class OB, class ST>
static int launch_igemm(const char* label, const Tiling& t, int M, int N, int K, const OA& oa, const OB& ob, const ST& st) {
  const dim3 grid((unsigned)ceil_div(M, t.bm), (unsigned)ceil_div(N, t.bn), (unsigned)(t.cz * t.groups));
  auto go = [&](auto igemm, int smem, int& ready) -> int {
    if (ready != g.device) { LTB_CUDA(cudaFuncSetAttribute(igemm, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); ready = g.device; }
    g.label = label;
    LTB_LAUNCH_CLUSTER_Z(igemm, grid, 256, t.cz, smem, M, N, K, t.kps, oa, ob, st);
    g.label = nullptr;
    return LTB_OK;
  };
  static int ready[5] = {-1, -1, -1, -1, -1};              // the device whose kernels have been given the larger shared memory
#define LTB_TILE(BM, BN, I) go(igemm_kernel<BM, BN, AF, BF, OA, OB, ST>, igemm_smem<BM, BN>(), ready[I])
  if (t.bm == 128) return t.bn == 128 ? LTB_TILE(128, 128, 0) : t.bn == 64 ? LTB_TILE(128, 64, 1) : LTB_TILE(128, 32, 2);
  return t.bn == 64 ? LTB_TILE(64, 64, 3) : LTB_TILE(64, 32, 4);
#undef LTB_TILE
}

// ---- skinny products: one extent of 16 or less (a 10-way classifier and its gradients) -----------------------------------
// The 64 x 64 tiles above leave such products to one or two CTAs walking a long K; these three kernels give every output
// (or every output column) its own thread or warp instead.
// N <= 16, A and B both contiguous along k: a block of sixteen warps per row m, each warp a sixteenth of K, lanes stride over
// k (at K = 2048 a lane makes four independent iterations: the loads of a row are all in flight at once).  The warps' sums are
// added in warp order by one thread per column: the same bits on every run.
constexpr int kSkinnyNWarps = 16;
template <bool ACC>
__global__ void __launch_bounds__(kSkinnyNWarps * 32) skinny_n_kernel(const float* __restrict__ a, int64_t sam, const float* __restrict__ b, int64_t sbn, float* c,
                                                                      int64_t scm, int64_t scn, int N, int K, float alpha) {
  pdl_enter();
  __shared__ float part[kSkinnyNWarps][16];
  const int m = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k0 = (int)((int64_t)K * warp / kSkinnyNWarps), k1 = (int)((int64_t)K * (warp + 1) / kSkinnyNWarps);
  float acc[16];
#pragma unroll
  for (int n = 0; n < 16; ++n) acc[n] = 0.0f;
  const float* ar = a + (int64_t)m * sam;
#pragma unroll 4
  for (int k = k0 + lane; k < k1; k += 32) {
    const float av = ar[k];
#pragma unroll
    for (int n = 0; n < 16; ++n) if (n < N) acc[n] += av * b[(int64_t)n * sbn + k];
  }
#pragma unroll
  for (int n = 0; n < 16; ++n) {
    float v = acc[n];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) part[warp][n] = v;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    const int n = threadIdx.x;
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < kSkinnyNWarps; ++w) v += part[w][n];
    v *= alpha;
    float* q = c + (int64_t)m * scm + (int64_t)n * scn;
    *q = ACC ? *q + v : v;
  }
}
// K <= 16: a thread per output element.
template <bool ACC>
__global__ void skinny_k_kernel(const float* __restrict__ a, int64_t sam, int64_t sak, const float* __restrict__ b, int64_t sbk, int64_t sbn,
                                float* c, int64_t scm, int64_t scn, int M, int N, int K, float alpha) {
  pdl_enter();
  const int64_t total = (int64_t)M * N;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int n = (int)(i % N); const int64_t m = i / N;
    float v = 0.0f;
    for (int k = 0; k < K; ++k) v += a[m * sam + k * sak] * b[k * sbk + n * sbn];
    float* q = c + m * scm + n * scn;
    *q = ACC ? *q + alpha * v : alpha * v;
  }
}
// M <= 16: a block is 32 output columns x 8 slices of K (blockIdx.y splits K further when it is long); a thread keeps all
// rows of its column in registers over its slice, B is read once, coalesced when contiguous along n.  The slices of a block
// are added in slice order through shared memory (a lane's loop over k is a chain of dependent steps: the classifier's weight
// gradient, 10 x 2048 over a batch of 128, took 89 us as sixteen blocks walking all of K, 19 us as sixteen slabs and a second
// launch).  With blockIdx.y > 1 a block's sum goes to its own slab and skinny_sum_kernel adds the slabs in order.
constexpr int kSkinnyMSlices = 8, kSkinnyMChunk = 32 * kSkinnyMSlices;
template <bool ACC>
__global__ void __launch_bounds__(32 * kSkinnyMSlices) skinny_m_kernel(const float* __restrict__ a, int64_t sam, int64_t sak, const float* __restrict__ b, int64_t sbk,
                                                                       int64_t sbn, float* c, int64_t scm, int64_t scn, int M, int N, int K, float alpha, float* part) {
  pdl_enter();
  __shared__ float sums[kSkinnyMSlices][16][33];
  __shared__ float rows[16][kSkinnyMChunk + 1];                                     // a's share: every lane of a column's loop reads the same ones
  const int n = blockIdx.x * 32 + threadIdx.x, slice = threadIdx.y, tid = slice * 32 + threadIdx.x;
  const int q0 = (int)((int64_t)K * blockIdx.y / gridDim.y), q1 = (int)((int64_t)K * (blockIdx.y + 1) / gridDim.y);
  float acc[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) acc[m] = 0.0f;
  for (int c0 = q0; c0 < q1; c0 += kSkinnyMChunk) {
    const int len = min(kSkinnyMChunk, q1 - c0), k0 = len * slice / kSkinnyMSlices, k1 = len * (slice + 1) / kSkinnyMSlices;
    __syncthreads();
    if (sak == 1) { for (int m = slice; m < M; m += kSkinnyMSlices) for (int k = threadIdx.x; k < len; k += 32) rows[m][k] = a[(int64_t)m * sam + c0 + k]; }
    else for (int i = tid; i < M * len; i += 32 * kSkinnyMSlices) { const int k = i / M, m = i - k * M; rows[m][k] = a[(int64_t)m * sam + (int64_t)(c0 + k) * sak]; }
    __syncthreads();
    if (n >= N) continue;
    const float* p = b + (int64_t)(c0 + k0) * sbk + (int64_t)n * sbn;
    for (int k = k0; k < k1; k += 8, p += 8 * sbk) {                             // eight loads in flight
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = k + e < k1 ? p[e * sbk] : 0.0f;
#pragma unroll
      for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int m = 0; m < 16; ++m) if (m < M && k + e < k1) acc[m] += rows[m][k + e] * v[e];
    }
  }
#pragma unroll
  for (int m = 0; m < 16; ++m) sums[slice][m][threadIdx.x] = acc[m];
  __syncthreads();
  if (n >= N) return;
  for (int m = slice; m < M; m += kSkinnyMSlices) {                              // the rows are dealt out to the slices' threads
    float v = 0.0f;
#pragma unroll
    for (int z = 0; z < kSkinnyMSlices; ++z) v += sums[z][m][threadIdx.x];
    float* q = c + (int64_t)m * scm + (int64_t)n * scn;
    if (part) part[((int64_t)blockIdx.y * M + m) * N + n] = v;                   // K was split over blocks too: this block's share goes to its own slab
    else *q = ACC ? *q + alpha * v : alpha * v;
  }
}
// c[m][n] (+)= alpha * (part[0][m][n] + part[1][m][n] + ...), in that order: the second half of skinny_m_kernel when K is split.
template <bool ACC>
__global__ void skinny_sum_kernel(const float* __restrict__ part, int slabs, float* c, int64_t scm, int64_t scn, int M, int N, float alpha) {
  pdl_enter();
  const int64_t total = (int64_t)M * N;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    float v = 0.0f;
    for (int z = 0; z < slabs; ++z) v += part[(int64_t)z * total + i];
    float* q = c + (i / N) * scm + (i % N) * scn;
    *q = ACC ? *q + alpha * v : alpha * v;
  }
}
static int skinny_gemm(const float* a, int64_t sam, int64_t sak, const float* b, int64_t sbk, int64_t sbn, float* c, int64_t scm, int64_t scn,
                       int M, int N, int K, float alpha, bool accumulate, bool* taken) {
  *taken = true;
  if (N <= 16 && sak == 1 && sbk == 1 && K >= 128 && M <= 65535) {
    // one block per row, its warps share K and are added in a fixed order: the same bits on every run (splitting K over
    // more blocks would need atomics, whose order changes from run to run)
    if (accumulate) LTB_LAUNCH(skinny_n_kernel<true>, dim3(M), kSkinnyNWarps * 32, 0, a, sam, b, sbn, c, scm, scn, N, K, alpha);
    else LTB_LAUNCH(skinny_n_kernel<false>, dim3(M), kSkinnyNWarps * 32, 0, a, sam, b, sbn, c, scm, scn, N, K, alpha);
  } else if (K <= 16) {
    const unsigned grid = (unsigned)grid_for((int64_t)M * N, 256);
    if (accumulate) LTB_LAUNCH(skinny_k_kernel<true>, grid, 256, 0, a, sam, sak, b, sbk, sbn, c, scm, scn, M, N, K, alpha);
    else LTB_LAUNCH(skinny_k_kernel<false>, grid, 256, 0, a, sam, sak, b, sbk, sbn, c, scm, scn, M, N, K, alpha);
  } else if (M <= 16 && N >= 256 && K <= 4096) {
    const unsigned gx = (unsigned)ceil_div(N, 32);
    // a thread's loop over k is a chain of dependent steps: beyond 64 steps per in-block slice K is also split over blockIdx.y,
    // every such split writes its share into a slab of the library's workspace and a second small launch adds the slabs in
    // order (no atomics: same bits every run)
    int ks = (int)ceil_div(K, 64 * kSkinnyMSlices);
    const size_t room = g.cur_scratch_bytes() / ((size_t)M * N * sizeof(float));
    if ((size_t)ks > room) ks = (int)room;
    if (ks < 1) ks = 1;
    float* part = ks > 1 ? g.cur_scratch() : nullptr;
    if (accumulate) LTB_LAUNCH(skinny_m_kernel<true>, dim3(gx, ks), dim3(32, kSkinnyMSlices), 0, a, sam, sak, b, sbk, sbn, c, scm, scn, M, N, K, alpha, part);
    else LTB_LAUNCH(skinny_m_kernel<false>, dim3(gx, ks), dim3(32, kSkinnyMSlices), 0, a, sam, sak, b, sbk, sbn, c, scm, scn, M, N, K, alpha, part);
    if (part) {
      const unsigned gr = (unsigned)grid_for((int64_t)M * N, 256);
      if (accumulate) LTB_LAUNCH(skinny_sum_kernel<true>, gr, 256, 0, (const float*)part, ks, c, scm, scn, M, N, alpha);
      else LTB_LAUNCH(skinny_sum_kernel<false>, gr, 256, 0, (const float*)part, ks, c, scm, scn, M, N, alpha);
    }
  } else *taken = false;
  return LTB_OK;
}

// ---- small products: so few outputs that one round of 32 x 32 tiles covers them ------------------------------------------------
// The time of such a product is latency: the tiles above walk K in steps of 16, each a round trip to memory and a barrier.  Here a CTA of sixteen warps
// fetches all of k of both operands at once (up to sixteen loads of a thread in flight; 4-byte cp.async leave an SM at one warp's worth per 18 cycles:
// 100 x 50 x 320 8.4 us), each warp takes a sixteenth of k and the whole T x T tile, and their sums meet in shared memory in warp order: the same bits on
// every run, and shorter chains than the tiles above have.  T is 16 where that is the faster tile: a quarter of the arithmetic per SM.
constexpr int kSmallWarps = 16, kSmallPart = 33;
template <int T> constexpr int kSmallK = 16384 / T;       // what shared memory holds of both operands: 1024 of k, or 512
template <int T>
__device__ __forceinline__ void small_fetch(float* dst, const float* p, int64_t row, int64_t kst, int rows, int len, int units, int warp, int lane) {
  const bool along_k = kst == 1 && row != 1;                                          // a warp reads 8 of k by 4 rows (whole sectors), or T rows
  auto at = [&](int u, int& k, int& m) {
    if (along_k) { k = u / (T / 4) * 8 + (lane & 7); m = u % (T / 4) * 4 + (lane >> 3); }
    else { k = u * (32 / T) + lane / T; m = lane % T; }
  };
  for (int u0 = warp; u0 < units; u0 += 16 * kSmallWarps) {
    float v[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) { int k, m; at(u0 + e * kSmallWarps, k, m); v[e] = k < len && m < rows ? p[m * row + k * kst] : 0.0f; }
#pragma unroll
    for (int e = 0; e < 16; ++e) { int k, m; at(u0 + e * kSmallWarps, k, m); if (u0 + e * kSmallWarps < units) dst[k * (T + 4) + m] = v[e]; }     // pitch T + 4: 8 of k by 4 rows hit 32 banks
  }
}
template <bool ACC, int T>
__global__ void __launch_bounds__(kSmallWarps * 32) small_gemm_kernel(const float* __restrict__ a, int64_t sam, int64_t sak, const float* __restrict__ b, int64_t sbk, int64_t sbn,
                                                                      float* c, int64_t scm, int64_t scn, int M, int N, int K, float alpha) {
  extern __shared__ __align__(16) float small_smem[];
  constexpr int TM = T / 8, TN = T / 4, P = T + 4;                                    // a lane's rows and columns
  pdl_enter();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m0 = blockIdx.x * T, n0 = blockIdx.y * T;
  const int lenp = (K + 15) / 16 * 16, per = lenp / kSmallWarps;
  float* const as = small_smem; float* const bs = small_smem + lenp * P;
  small_fetch<T>(as, a + m0 * sam, sam, sak, M - m0, K, lenp * T / 32, warp, lane);
  small_fetch<T>(bs, b + n0 * sbn, sbn, sbk, N - n0, K, lenp * T / 32, warp, lane);
  __syncthreads();
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
  const int lm = lane & 7, ln = lane >> 3;                                            // rows TM lm .., columns TN ln ..
#pragma unroll 4
  for (int k = warp * per; k < (warp + 1) * per; ++k) {
    float u[TM], v[TN];
#pragma unroll
    for (int i = 0; i < TM; i += 2) { const float2 x = *reinterpret_cast<const float2*>(as + k * P + TM * lm + i); u[i] = x.x; u[i + 1] = x.y; }
#pragma unroll
    for (int j = 0; j < TN; j += 4) { const float4 y = *reinterpret_cast<const float4*>(bs + k * P + TN * ln + j); v[j] = y.x; v[j + 1] = y.y; v[j + 2] = y.z; v[j + 3] = y.w; }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] += u[i] * v[j];
  }
  __syncthreads();
  constexpr int kWarpSums = TM * TN * kSmallPart;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) small_smem[warp * kWarpSums + (i * TN + j) * kSmallPart + lane] = acc[i][j];
  __syncthreads();
  const bool by_rows = scm == 1 && scn != 1;                                          // neighbouring lanes: neighbouring addresses of c
#pragma unroll
  for (int e = threadIdx.x; e < T * T; e += kSmallWarps * 32) {
    const int m = by_rows ? e % T : e / T, n = by_rows ? e / T : e % T;
    const float* q = small_smem + (m % TM * TN + n % TN) * kSmallPart + n / TN * 8 + m / TM;
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < kSmallWarps; ++w) v += q[w * kWarpSums];
    if (m0 + m < M && n0 + n < N) {
      float* d = c + (m0 + m) * scm + (n0 + n) * scn;
      *d = ACC ? *d + alpha * v : alpha * v;
    }
  }
}
// The tile of a small product, or 0: the tiles above.  One round of CTAs, one fetch of all of k (walking a longer K in several fetches lost: 200 x 300 x 1500 20.9 / 24.8 us,
// 128 x 128 x 2048 16 / 33), and where that was the faster one of the three; sums that may be added atomically are split over CTAs by the tiles above, from K = 128 on.
// Measured in recordings of twenty, us, tiles above / 16 / 32:
//                    stored                                                               added
//   64 x 64          K 48 3.2/3.2/3.7, 64 3.9/3.2/3.8, 512 7.8/4.8/8.4, 1024 8.0/8.0        K 32 3.1/3.1/3.7, 64 4.3/3.2/3.8, 400 5.9/4.4, 512 5.3/4.9, 640 4.5/6.5
//   8 x 8            K 48 2.6/3.0/3.3, 64 3.2/3.1/3.4, 512 6.2/4.4/7.7, 640 6.3/6.4         K 48 2.9/2.9/3.3, 320 4.2/3.7/6.1, 512 4.2/4.5, 640 3.6/6.1
//   192 x 192        K 64 4.1/5.0/3.9, 128 6.6/5.4/4.4, 400 8.7/6.6/7.6, 640 8.2/10.9, 768 8.1/7.1   K 64 4.9/4.7/4.1, 192 5.8/5.2/5.4, 256 5.5/5.5/5.8
//   384 x 384 (32)   K 48 3.4/3.9, 64 4.0/4.0, 512 12.0/8.7                                 K 48 4.6/4.2, 400 9.0/7.9
// (More than one CTA of 16 x 16 for two SMs is slow where two of them fit one SM, up to K = 640: they are not spread evenly.)
static int small_tile(int M, int N, int K, bool adds) {
  const int64_t t16 = ceil_div(M, 16) * ceil_div(N, 16), t32 = ceil_div(M, 32) * ceil_div(N, 32), sms = g.sm_count;
  const bool few = 2 * t16 <= sms;
  if (K < (adds ? 48 : 64)) return 0;
  if (adds) {
    if (few) return K <= (t16 >= 8 && t16 <= 32 ? 512 : 400) ? 16 : 0;
    return t32 <= sms && K <= (5 * t32 >= 2 * sms ? 400 : 192) ? 32 : 0;
  }
  if (K > 512) return t16 >= 16 && t16 <= sms && K <= kSmallK<16> && (K >= 704 || t16 <= 32) ? 16 : 0;
  if (t16 <= sms && (few || K > 256)) return 16;
  return t32 <= sms ? 32 : 0;
}
template <int T>
static int small_gemm(const float* a, int64_t sam, int64_t sak, const float* b, int64_t sbk, int64_t sbn, float* c, int64_t scm, int64_t scn,
                      int M, int N, int K, float alpha, bool accumulate) {
  constexpr int kMost = 2 * kSmallK<T> * (T + 4) * 4, kSums = kSmallWarps * T * T / 32 * kSmallPart * 4;
  static int ready = -1;
  if (ready != g.device) {
    LTB_CUDA(cudaFuncSetAttribute((small_gemm_kernel<false, T>), cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
    LTB_CUDA(cudaFuncSetAttribute((small_gemm_kernel<true, T>), cudaFuncAttributeMaxDynamicSharedMemorySize, kMost));
    ready = g.device;
  }
  const int panels = 2 * ((K + 15) / 16 * 16) * (T + 4) * 4, smem = panels > kSums ? panels : kSums;
  const dim3 grid((unsigned)ceil_div(M, T), (unsigned)ceil_div(N, T));
  if (accumulate) LTB_LAUNCH((small_gemm_kernel<true, T>), grid, kSmallWarps * 32, smem, a, sam, sak, b, sbk, sbn, c, scm, scn, M, N, K, alpha);
  else LTB_LAUNCH((small_gemm_kernel<false, T>), grid, kSmallWarps * 32, smem, a, sam, sak, b, sbk, sbn, c, scm, scn, M, N, K, alpha);
  return LTB_OK;
}

// C[M,N] (op)= alpha * A B with arbitrary strides; accumulate selects += (gradients) over = (forward).
static int strided_gemm(const float* a, int64_t sam, int64_t sak, const float* b, int64_t sbk, int64_t sbn, float* c, int64_t scm,
                        int64_t scn, int M, int N, int K, float alpha, bool accumulate) {
  { bool taken = false; int rc = skinny_gemm(a, sam, sak, b, sbk, sbn, c, scm, scn, M, N, K, alpha, accumulate, &taken); if (rc || taken) return rc; }
  const bool adds = accumulate && !g.deterministic;
  if (const int tile = small_tile(M, N, K, adds))
    return tile == 16 ? small_gemm<16>(a, sam, sak, b, sbk, sbn, c, scm, scn, M, N, K, alpha, accumulate) : small_gemm<32>(a, sam, sak, b, sbk, sbn, c, scm, scn, M, N, K, alpha, accumulate);
  // m of the kernel is the contiguous index of C
  const bool swap = scn == 1 && scm != 1;
  const int m = swap ? N : M, n = swap ? M : N;
  const long long sm = swap ? scn : scm, sn = swap ? scm : scn;
  const float* pa = swap ? b : a; const float* pb = swap ? a : b;
  const int64_t ar = swap ? sbn : sam, ak = swap ? sbk : sak, br = swap ? sam : sbn, bk = swap ? sak : sbk;
  const Tiling t = choose_tiling(m, n, K, adds);
  const MatPut st{c, sm, sn, alpha, t.groups > 1 ? 2 : accumulate ? 1 : 0, sm == 1 && sn % 4 == 0 && aligned16(c)};
  const int64_t most = ((int64_t)1 << 31) - 1;
  if (m * ar + K * ak > most || n * br + K * bk > most) {
    const WideMatOp oa{pa, ar, ak}, ob{pb, br, bk};
    if (ak == 1 && ar != 1) return bk == 1 && br != 1 ? launch_igemm<FEED_K, FEED_K>("igemm[gemm]", t, m, n, K, oa, ob, st) : launch_igemm<FEED_K, FEED_ROW>("igemm[gemm]", t, m, n, K, oa, ob, st);
    return bk == 1 && br != 1 ? launch_igemm<FEED_ROW, FEED_K>("igemm[gemm]", t, m, n, K, oa, ob, st) : launch_igemm<FEED_ROW, FEED_ROW>("igemm[gemm]", t, m, n, K, oa, ob, st);
  }
  const MatOp oa{pa, ar, ak}, ob{pb, br, bk};
  // four at a time along the contiguous index, which must then end on a multiple of four (k also where a split begins, a multiple of 16)
  auto feed = [&](const float* p, int64_t sr, int64_t sk, int rows) {
    if (sk == 1 && sr != 1) return sr % 4 == 0 && K % 4 == 0 && aligned16(p) ? FEED_K4 : FEED_K;
    return sr == 1 && sk % 4 == 0 && rows % 4 == 0 && aligned16(p) ? FEED_ROW4 : FEED_ROW;
  };
  int fa = feed(pa, ar, ak, m), fb = feed(pb, br, bk, n);
  if (fa < FEED_ROW4 || fb < FEED_ROW4) { fa &= FEED_K; fb &= FEED_K; }          // both or neither: half as many kernels
#define LTB_FEEDS(A, B) if (fa == A && fb == B) return launch_igemm<A, B>("igemm[gemm]", t, m, n, K, oa, ob, st)
  LTB_FEEDS(FEED_K4, FEED_K4); LTB_FEEDS(FEED_K4, FEED_ROW4); LTB_FEEDS(FEED_ROW4, FEED_K4); LTB_FEEDS(FEED_ROW4, FEED_ROW4);
  LTB_FEEDS(FEED_K, FEED_K); LTB_FEEDS(FEED_K, FEED_ROW); LTB_FEEDS(FEED_ROW, FEED_K); LTB_FEEDS(FEED_ROW, FEED_ROW);
#undef LTB_FEEDS
  return fail(LTB_E_STATE, "igemm: no such feed");
}

// dbias[co] += sum over n, ho, wo of dy (TensorDslCPU.scala:607-617); MASK: dy is the gradient of a ReLU that ran in place and is
// masked on the way (dy = y > 0 ? dy : 0, the held ltb_unary_grad), which saves that kernel and one of the two reads of dy.
// A cluster of CTAs owns a channel and shares its images; their sums meet in rank order: the same bits on every run.
// VEC: hw is a multiple of 4 and the tensors are 16-byte aligned.  Bound by latency on small maps; 96 x 32 x 32 at batch 64 (75 MB) 14.4 -> 11.8 us with four
// items of a thread in flight, 512 threads and half the CTAs.
constexpr int kBiasThreads = 512;
template <bool VEC, bool MASK>
__global__ void __launch_bounds__(kBiasThreads) conv_bias_grad_kernel(float* dy, const float* __restrict__ y, float* dbias, int N, int K, int hw, FastDiv by_per, int ctas) {
  pdl_enter();
  __shared__ float sh[kBiasThreads / 32];
  __shared__ float total;
  const int co = blockIdx.x / ctas, rank = blockIdx.x - co * ctas;
  const int n0 = (int)((long long)N * rank / ctas), n1 = (int)((long long)N * (rank + 1) / ctas);
  float s = 0.0f;
  const int per = VEC ? hw / 4 : hw, items = (n1 - n0) * per;          // the threads run over (image, element) pairs: small maps keep every lane busy
  using T = typename std::conditional<VEC, float4, float>::type;
  for (int j0 = threadIdx.x; j0 < items; j0 += 4 * kBiasThreads) {      // four items of a thread in flight
    T v[4], a[4]; long long at[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = j0 + u * kBiasThreads;
      int i; const int n = by_per.divmod(j < items ? j : 0, i);
      at[u] = ((long long)(n0 + n) * K + co) * hw + (VEC ? 4 * i : i);
      if (j < items) { v[u] = *reinterpret_cast<const T*>(dy + at[u]); if (MASK) a[u] = *reinterpret_cast<const T*>(y + at[u]); }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (j0 + u * kBiasThreads >= items) break;
      if constexpr (VEC) {
        if (MASK) {
          v[u].x = a[u].x > 0.0f ? v[u].x : 0.0f; v[u].y = a[u].y > 0.0f ? v[u].y : 0.0f; v[u].z = a[u].z > 0.0f ? v[u].z : 0.0f; v[u].w = a[u].w > 0.0f ? v[u].w : 0.0f;
          *reinterpret_cast<T*>(dy + at[u]) = v[u];
        }
        s += (v[u].x + v[u].y) + (v[u].z + v[u].w);
      } else {
        if (MASK) { v[u] = a[u] > 0.0f ? v[u] : 0.0f; dy[at[u]] = v[u]; }
        s += v[u];
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < kBiasThreads / 32; ++w) t += sh[w];
    if (ctas == 1) dbias[co] += t; else total = t;
  }
  if (ctas > 1) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (rank == 0 && threadIdx.x == 0) {
      float t = 0.0f;
      for (int z = 0; z < ctas; ++z) t += *cluster.map_shared_rank(&total, z);
      dbias[co] += t;
    }
    cluster.sync();
  }
}

// ---- 3x3, stride 1, padding 1 on maps of 4, 8, 16 or 32 columns: direct -----------------------------------------------------------
// Forward (FLIP false): out[n][o][p] = sum over (i, r, s) of w[o][i][r][s] in[n][i][p + (r-1, s-1)].  Data gradient (FLIP true): in = dy, out = dx and
// w[i][o][2-r][2-s], added to what out holds.  A warp owns 32 runs of PX neighbouring pixels (a lane each) times 8 output channels; the CTA's NW warps
// share the input tile and have 8 channels each.  For one input channel and filter row a lane loads PX + 2 pixels and three times eight
// weights (the same for the whole warp) and makes 24 PX products of them, so that the FP32 pipes and not the loads are the limit; the
// matrix form above loads every element of the unfolded operand on its own.  Packed pairs run along the output channel.
//   shared memory : rows of in with four zeros in front (the left edge of a row and the right edge of the one before), W + 4 floats an odd
//                   multiple of four so that lanes on neighbouring rows meet no bank twice; weights [channel][tap][output channel].  Double-buffered,
//                   the next 8 channels arrive by cp.async.
//   splits        : input channels are dealt to a cluster of up to 8 CTAs, whose tiles are summed in rank order, as in igemm_kernel.
struct DirectGeo { int N, Ci, Co, H, W; int rows, imgs, rs, ci_per; const float* bias; int relu; FastDiv by_q, by_line, by_ch, by_seg, by_rows, by_group; };
// Asynchronous copies into shared memory; zeros (and nothing read) where ok is false.
__device__ __forceinline__ void copy16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
constexpr int kDirectCh = 8;                                // input channels per step
template <int PX, int NW> int direct_smem(int tile) {      // tile: floats of one input channel
  const int steps = 2 * kDirectCh * (tile + 9 * (NW * 8 + 4)), partial = 32 * PX * NW * 8;
  return (steps > partial ? steps : partial) * 4;
}
template <int PX, int NW, bool FLIP>
__global__ void __launch_bounds__(NW * 32) conv3x3_direct_kernel(const float* __restrict__ in, const float* __restrict__ w, float* out, const DirectGeo G) {
  pdl_launch();
  constexpr int T = NW * 32, KT = NW * 8, KP = KT + 4;       // pitch of the weights: the copies below meet a bank four times at most
  extern __shared__ __align__(16) float pool[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int hw = G.H * G.W, img_tile = (G.rows + 2) * G.rs, tile = G.imgs * img_tile + 4;    // four more: the right edge of the last row
  // the group's first image and row, and the lane's own place in it; lanes of neighbouring rows first (see above)
  int h0, row, r_all;
  const int n0 = G.by_group.divmod(blockIdx.x, h0) * G.imgs, seg = G.by_seg.divmod(lane, r_all), img = G.by_rows.divmod(r_all, row);
  h0 *= G.rows;
  const int o0 = blockIdx.y * KT, c_begin = blockIdx.z * G.ci_per, c_end = min(G.Ci, c_begin + G.ci_per);
  const int steps = c_end > c_begin ? (c_end - c_begin + kDirectCh - 1) / kDirectCh : 0;
  float* const buf[2] = {pool, pool + kDirectCh * (tile + 9 * KP)};

  // input rows as 16-byte items: (channel, image, row, quarter), W / 4 quarters; the zeros around them are written once
  const int q = G.W / 4, per_ch = G.imgs * (G.rows + 2) * q, items = kDirectCh * per_ch;
  constexpr int kItems = ((PX == 8 ? 640 : 384) + T - 1) / T;      // items of a thread: 4 to 32 columns make 576 or 640 with runs of eight, 320 or 384 with four
  constexpr int kWeights = kDirectCh * 9 * KT / T;          // 18
  int src[kItems], dst[kItems];                             // within a channel block; src -1: outside the image, dst -1: no item
#pragma unroll
  for (int e = 0; e < kItems; ++e) {
    const int i = tid + e * T;
    src[e] = -1; dst[e] = -1;
    if (i < items) {
      int j, c4, y;
      const int c = G.by_ch.divmod(i, j), line = G.by_q.divmod(j, c4), im = G.by_line.divmod(line, y), h = h0 + y - 1;
      c4 *= 4;
      dst[e] = c * tile + im * img_tile + y * G.rs + 4 + c4;
      if ((unsigned)h < (unsigned)G.H && n0 + im < G.N) src[e] = ((im * G.Ci + c) * G.H + h) * G.W + c4;
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u)
    for (int i = tid; i < kDirectCh * tile / 4; i += T) reinterpret_cast<float4*>(buf[u])[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();                                          // the zeros are down
  pdl_wait();
  auto fetch = [&](int step) {
    float* b = buf[step & 1];
    const int c0 = c_begin + step * kDirectCh, live = c_end - c0;
    const float* base = in + ((long long)n0 * G.Ci + c0) * hw;
#pragma unroll
    for (int e = 0; e < kItems; ++e)
      if (dst[e] >= 0) { const bool ok = src[e] >= 0 && tid + e * T < live * per_ch; copy16(b + dst[e], base + (ok ? src[e] : 0), ok); }
    // weights in the order of memory: (channel, tap) of one output channel after the other, FLIP: (output channel, tap) of one channel after the other
    float* wb = b + kDirectCh * tile;
#pragma unroll
    for (int e = 0; e < kWeights; ++e) {
      const int i = tid + e * T, a = i / (FLIP ? KT * 9 : kDirectCh * 9), j = i - a * (FLIP ? KT * 9 : kDirectCh * 9), u = j / 9, t = j - u * 9;
      const int c = FLIP ? a : u, o = FLIP ? u : a;
      const bool ok = c < live && o0 + o < G.Co;
      const float* from = FLIP ? w + ((long long)(c0 + c) * G.Co + o0) * 9 + j : w + ((long long)(o0 + o) * G.Ci + c0) * 9 + j;
      copy4(wb + (c * 9 + (FLIP ? 8 - t : t)) * KP + o, ok ? from : w, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  unsigned long long acc[PX][4];
#pragma unroll
  for (int p = 0; p < PX; ++p)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[p][j] = 0ull;
  if (steps > 0) fetch(0);
  const int at = img * img_tile + row * G.rs + seg * PX + 3;      // the pixel left of the lane's first, one row up
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                        // step s is down for everybody, and everybody is done with step s - 1
    if (s + 1 < steps) fetch(s + 1);
    const float* xb = buf[s & 1] + at; const float* wb = buf[s & 1] + kDirectCh * tile + warp * 8;
#pragma unroll 1
    for (int c = 0; c < kDirectCh; ++c) {
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        float x[PX + 2];
        const float* xr = xb + c * tile + r * G.rs;
        x[0] = xr[0]; x[PX + 1] = xr[PX + 1];
#pragma unroll
        for (int p = 0; p < PX; p += 4) *reinterpret_cast<float4*>(x + 1 + p) = *reinterpret_cast<const float4*>(xr + 1 + p);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
          const ulonglong2 wa = *reinterpret_cast<const ulonglong2*>(wb + (c * 9 + r * 3 + t) * KP), wc = *reinterpret_cast<const ulonglong2*>(wb + (c * 9 + r * 3 + t) * KP + 4);
#pragma unroll
          for (int p = 0; p < PX; ++p) {
            const unsigned long long xx = pack2(x[p + t], x[p + t]);
            acc[p][0] = fma2(wa.x, xx, acc[p][0]); acc[p][1] = fma2(wa.y, xx, acc[p][1]);
            acc[p][2] = fma2(wc.x, xx, acc[p][2]); acc[p][3] = fma2(wc.y, xx, acc[p][3]);
          }
        }
      }
    }
  }
  cg::cluster_group cluster = cg::this_cluster();
  const int cz = (int)cluster.num_blocks();
  // eight channels of PX neighbouring pixels leave as 16-byte stores
  auto emit = [&](int o, int lane_img, int lane_row, int lane_seg, float4 v, int part) {
    if (n0 + lane_img >= G.N || o >= G.Co) return;
    float4* dst4 = reinterpret_cast<float4*>(out + ((long long)(n0 + lane_img) * G.Co + o) * hw + (h0 + lane_row) * G.W + lane_seg * PX) + part;
    if (FLIP) { const float4 old = *dst4; v.x += old.x; v.y += old.y; v.z += old.z; v.w += old.w; }
    else {
      const float b = G.bias ? G.bias[o] : 0.0f;
      v.x += b; v.y += b; v.z += b; v.w += b;
      if (G.relu) { v.x = v.x < 0.0f ? 0.0f : v.x; v.y = v.y < 0.0f ? 0.0f : v.y; v.z = v.z < 0.0f ? 0.0f : v.z; v.w = v.w < 0.0f ? 0.0f : v.w; }
    }
    *dst4 = v;
  };
  if (cz > 1) __syncthreads();
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int p = 0; p < PX; p += 4) {
      const float2 a = unpack2(acc[p][j]), b = unpack2(acc[p + 1][j]), c = unpack2(acc[p + 2][j]), d = unpack2(acc[p + 3][j]);
      const float4 lo = make_float4(a.x, b.x, c.x, d.x), hi = make_float4(a.y, b.y, c.y, d.y);
      const int o = warp * 8 + 2 * j;
      if (cz > 1) {                                         // [output channel][part][lane]: the sum below runs along the lanes
        float4* t = reinterpret_cast<float4*>(pool) + (o * (PX / 4) + p / 4) * 32 + lane;
        t[0] = lo; t[(PX / 4) * 32] = hi;
      } else { emit(o0 + o, img, row, seg, lo, p / 4); emit(o0 + o + 1, img, row, seg, hi, p / 4); }
    }
  if (cz > 1) {
    cluster.sync();
    const int rank = (int)cluster.block_rank(), all = KT * (PX / 4) * 32, per = all / cz / 32 * 32 + (all / cz % 32 ? 32 : 0);
    for (int i = rank * per + tid; i < min(all, (rank + 1) * per); i += T) {
      float4 p[8];
#pragma unroll
      for (int z = 0; z < 8; ++z) if (z < cz) p[z] = reinterpret_cast<const float4*>(cluster.map_shared_rank(pool, z))[i];
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int z = 0; z < 8; ++z) if (z < cz) { v.x += p[z].x; v.y += p[z].y; v.z += p[z].z; v.w += p[z].w; }
      const int part = (i >> 5) % (PX / 4), o = (i >> 5) / (PX / 4);
      emit(o0 + o, img, row, seg, v, part);                 // T is a multiple of 32: item i belongs to this thread's lane
    }
    cluster.sync();
  }
}
template <int PX, int NW, bool FLIP>
static int launch_direct(const float* in, const float* w, float* out, DirectGeo& G, int warps, const char* label) {
  const int segs = G.W / PX, lines = 32 / segs;             // rows of a group
  G.rows = lines < G.H ? lines : G.H; G.imgs = lines / G.rows;
  G.rs = G.W + 4; if (G.rs % 8 == 0) G.rs += 4;
  G.by_q = FastDiv(G.W / 4); G.by_line = FastDiv(G.rows + 2); G.by_ch = FastDiv(G.imgs * (G.rows + 2) * (G.W / 4));
  G.by_seg = FastDiv(32 / segs); G.by_rows = FastDiv(G.rows); G.by_group = FastDiv(G.H / G.rows);
  const int groups = (int)ceil_div(G.N, G.imgs) * (G.H / G.rows);
  const int tiles = groups * (int)ceil_div(G.Co, NW * 8);
  // CTAs share the input channels until every SM has `warps` warps; small problems of more than 32 channels also until a chain is 144 products
  // long (the matrix form's in such cases: 64 -> 256 on 8 x 8 at batch 64 is 1.9e-7 off in both, 2.6e-7 with chains of 288)
  int cz = 1;
  while (cz < 8 && G.Ci >= kDirectCh * (cz + 1) && (tiles * cz * NW < warps * g.sm_count || (G.Ci > 32 && G.Ci > 16 * cz && tiles * NW < 12 * g.sm_count))) ++cz;
  G.ci_per = (int)ceil_div(ceil_div(G.Ci, cz), kDirectCh) * kDirectCh;
  cz = (int)ceil_div(G.Ci, G.ci_per);
  const int smem = direct_smem<PX, NW>(G.imgs * (G.rows + 2) * G.rs + 4);
  static int most = 0, device = -1;
  if (device != g.device || smem > most) { LTB_CUDA(cudaFuncSetAttribute((conv3x3_direct_kernel<PX, NW, FLIP>), cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); most = smem; device = g.device; }
  g.label = label;
  LTB_LAUNCH_CLUSTER_Z((conv3x3_direct_kernel<PX, NW, FLIP>), dim3((unsigned)groups, (unsigned)ceil_div(G.Co, NW * 8), (unsigned)cz), NW * 32, cz, smem, in, w, out, G);
  g.label = nullptr;
  return LTB_OK;
}
// Few channels into many: runs of eight pixels and 32 output channels per CTA, split until an SM has six warps (a split's sum costs what it
// saves beyond that).  Many into few: the sums are long and the outputs few, so runs of four and 16 output channels, split until an SM has
// sixteen warps.  Swept on SqueezeNet's layers at batch 64 (us, 16 -> 64 and 32 -> 128 on 16 x 16, 48 -> 192 and 64 -> 256 on 8 x 8): the first rule
// 14, 31, 29, 34 forward and 25, 45, 36, 55 in the data gradient, the second 17, 39, 29, 43 and 14, 38, 30, 38.
template <bool FLIP>
static int conv_direct(const float* in, const float* w, float* out, DirectGeo& G, const char* label) {
  if (G.Ci <= G.Co && G.W >= 8 && G.H >= 8) return launch_direct<8, 4, FLIP>(in, w, out, G, 6, label);
  return launch_direct<4, 2, FLIP>(in, w, out, G, G.Ci <= G.Co ? 6 : 16, label);
}
// 3x3, stride 1, padding 1 on maps of 4 to 32 rows and columns (powers of two: whole groups of 32 runs), 16-byte aligned tensors, at least a step of
// channels on both sides; and where it is the faster one.  Measured against the matrix form on 1328 sizes each way (4 to 32 rows, 1 to 128 images, 8 to 512 channels): from 24
// channels summed over it takes 0.4 to 1.0 of the time but where less than half of a group's pixels exist and there are splits all the same (128 -> 512, one
// image of 8 x 8, 10.1 us in matrix form, 18.2 here; 96 -> 256, two images, 9.5 / 12.5); with fewer a chain is too short for what it costs, so that only large outputs
// gain (16 channels: 24 outputs on 16 images of 8 x 8 6.9 / 9.0, 96 outputs on 32 of 32 x 32 32.2 / 26.1; 12, a step and a half, at 32 x 32 on 16 images, 256 outputs
// 26.7 / 33.7), and maps of 4 rows, whose tiles are half as wide (16 -> 64, 8.2 / 5.6; back from 8 channels to fewer than 32, 4.9 / 5.8).
static bool direct_takes(const ConvDims& d, const float* a, const float* b, bool back) {
  if (d.R != 3 || d.S != 3 || d.sh != 1 || d.sw != 1 || d.ph != 1 || d.pw != 1 || !aligned16(a) || !aligned16(b)) return false;
  if (d.W != 4 && d.W != 8 && d.W != 16 && d.W != 32) return false;
  if (d.C < 8 || d.K < 8) return false;
  const int from = back ? d.K : d.C, to = back ? d.C : d.K;
  const int64_t pixels = (int64_t)d.N * d.H * d.W;
  const bool wide = d.W >= 8 && d.H >= 8;
  if (from < 24 && (from % 8 || (wide ? pixels * ceil_div(to, 32) * 32 < 1200000 : back && from == 8 && to < 32))) return false;
  if (wide && from > 64 && from <= to && pixels <= 128) return false;
  return d.H <= 32 && (d.H & (d.H - 1)) == 0 && d.H >= 4 && (int64_t)d.C * d.H * d.W * 32 < (1ll << 31) && (int64_t)d.K * d.H * d.W * 32 < (1ll << 31);
}

// ---- convolution as implicit GEMM -----------------------------------------------------------------------------
// Whether narrow entries hold this convolution, and whether its pixels are plain runs (1x1, stride 1, no padding, whole groups of four).
static bool narrow(const ConvDims& d) {
  const int64_t most = ((int64_t)1 << 31) - 1 - (int64_t)(d.R + d.ph) * (d.W + d.oW) - d.S - d.pw;      // an entry's own offset may lie a filter or the padding outside
  return d.R + d.S <= 30 && (int64_t)d.N * d.C * d.H * d.W <= most && (int64_t)d.N * d.K * d.oH * d.oW <= most && (int64_t)d.K * d.C * d.R * d.S <= most;
}
static bool plain_pixels(const ConvDims& d) { return d.R == 1 && d.S == 1 && d.sh == 1 && d.sw == 1 && d.ph == 0 && d.pw == 0 && d.H * d.W % 4 == 0; }
int conv_fwd_fp32(const float* x, const float* w, const float* bias, float* y, const ConvDims& d, bool relu) {
  const int hw = d.oH * d.oW, M = d.N * hw, Kd = d.C * d.R * d.S;
  if (direct_takes(d, x, y, false)) {
    DirectGeo G{d.N, d.C, d.K, d.H, d.W, 0, 0, 0, 0, bias, relu ? 1 : 0};
    return conv_direct<false>(x, w, y, G, "direct[conv_fwd]");
  }
  const Tiling t = choose_tiling(M, d.K, Kd, false);
  const PixelPut st(y, bias, d.K, hw, 0, relu);
  if (!narrow(d)) return launch_igemm<FEED_ROW, FEED_K>("igemm[conv_fwd]", t, M, d.K, Kd, WideConvInput<true>(x, d), WideMatOp{w, Kd, 1}, st);
  const ConvInput<true> in(x, d); const MatOp fw{w, Kd, 1};
  const bool w4 = Kd % 4 == 0 && aligned16(w);
  if (w4 && plain_pixels(d) && aligned16(x)) return launch_igemm<FEED_ROW4, FEED_K4>("igemm[conv_fwd]", t, M, d.K, Kd, in, fw, st);
  if (w4) return launch_igemm<FEED_ROW, FEED_K4>("igemm[conv_fwd]", t, M, d.K, Kd, in, fw, st);
  return launch_igemm<FEED_ROW, FEED_K>("igemm[conv_fwd]", t, M, d.K, Kd, in, fw, st);
}
int conv_dgrad_fp32(const float* dy, const float* w, float* dx, const ConvDims& d) {
  const int hw = d.H * d.W, M = d.N * hw, rs = d.R * d.S, Kd = d.K * rs;
  if (direct_takes(d, dy, dx, true)) {
    DirectGeo G{d.N, d.K, d.C, d.H, d.W, 0, 0, 0, 0, nullptr, 0};
    return conv_direct<true>(dy, w, dx, G, "direct[conv_dgrad]");
  }
  const Tiling t = choose_tiling(M, d.C, Kd, false);
  const PixelPut st(dx, nullptr, d.C, hw, 1, false);
  if (!narrow(d)) return launch_igemm<FEED_ROW, FEED_K>("igemm[conv_dgrad]", t, M, d.C, Kd, WideConvDy(dy, d), FilterByInput<WideEnt>(w, d.C, rs), st);
  const FilterByInput<Ent> fw(w, d.C, rs);
  const ConvDy in(dy, d);
  if (rs > 1) return launch_igemm<FEED_ROW, FEED_K>("igemm[conv_dgrad]", t, M, d.C, Kd, in, fw, st);
  const bool w4 = d.C % 4 == 0 && aligned16(w);
  if (w4 && plain_pixels(d) && aligned16(dy)) return launch_igemm<FEED_ROW4, FEED_ROW4>("igemm[conv_dgrad]", t, M, d.C, Kd, in, fw, st);
  return launch_igemm<FEED_ROW, FEED_ROW>("igemm[conv_dgrad]", t, M, d.C, Kd, in, fw, st);
}
int conv_wgrad_fp32(const float* x, const float* dy, float* dw, const ConvDims& d) {
  const int M = d.C * d.R * d.S, hw = d.oH * d.oW, Kd = d.N * hw;       // dw[co][(ci, kh, kw)]: the filter element is the contiguous index
  const Tiling t = choose_tiling(M, d.K, Kd, !g.deterministic);
  const MatPut st{dw, 1, M, 1.0f, t.groups > 1 ? 2 : 1, M % 4 == 0 && aligned16(dw)};
  if (!narrow(d)) return launch_igemm<FEED_K, FEED_K>("igemm[conv_wgrad]", t, M, d.K, Kd, WideConvInput<false>(x, d), DyByPixel<WideEnt>(dy, d.K, hw), st);
  const ConvInput<false> in(x, d); const DyByPixel<Ent> g4(dy, d.K, hw);
  const bool d4 = hw % 4 == 0 && aligned16(dy);
  if (d4 && plain_pixels(d) && aligned16(x)) return launch_igemm<FEED_K4, FEED_K4>("igemm[conv_wgrad]", t, M, d.K, Kd, in, g4, st);
  if (d4) return launch_igemm<FEED_K, FEED_K4>("igemm[conv_wgrad]", t, M, d.K, Kd, in, g4, st);
  return launch_igemm<FEED_K, FEED_K>("igemm[conv_wgrad]", t, M, d.K, Kd, in, g4, st);
}
int conv_bias_grad(float* dy, const float* relu_y, float* dbias, const ConvDims& d) {
  const int hw = d.oH * d.oW;
  int ctas = 1;                                             // per channel: two per SM in all at most, 16 KB of dy each at least
  while (ctas < 8 && (int64_t)d.K * ctas <= g.sm_count && (int64_t)d.N * hw >= (int64_t)ctas * 2 * 4096 && d.N >= ctas * 2) ctas *= 2;
  const bool vec = hw % 4 == 0 && aligned16(dy) && (!relu_y || aligned16(relu_y));
  const FastDiv per(vec ? hw / 4 : hw);
  const dim3 grid((unsigned)(d.K * ctas));
  if (relu_y) {
    if (vec) LTB_LAUNCH_CLUSTER((conv_bias_grad_kernel<true, true>), grid, kBiasThreads, ctas, dy, relu_y, dbias, d.N, d.K, hw, per, ctas);
    else LTB_LAUNCH_CLUSTER((conv_bias_grad_kernel<false, true>), grid, kBiasThreads, ctas, dy, relu_y, dbias, d.N, d.K, hw, per, ctas);
  } else if (vec) LTB_LAUNCH_CLUSTER((conv_bias_grad_kernel<true, false>), grid, kBiasThreads, ctas, dy, relu_y, dbias, d.N, d.K, hw, per, ctas);
  else LTB_LAUNCH_CLUSTER((conv_bias_grad_kernel<false, false>), grid, kBiasThreads, ctas, dy, relu_y, dbias, d.N, d.K, hw, per, ctas);
  return LTB_OK;
}

// Entry used by the other translation units (declared in gemm.cuh).
int gemm_fp32(const float* a, int64_t sam, int64_t sak, const float* b, int64_t sbk, int64_t sbn, float* c, int64_t scm, int64_t scn,
              int M, int N, int K, float alpha, bool accumulate) {
  return strided_gemm(a, sam, sak, b, sbk, sbn, c, scm, scn, M, N, K, alpha, accumulate);
}

}  // namespace ltb
