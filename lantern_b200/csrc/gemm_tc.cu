// TF32 tensor-core engine for sm_100a: one warp-specialised kernel for every dense contraction of the training step
// (convolution forward / data-grad / weight-grad and gemm), driven by the plans of tc_plan.cpp.
//
//   warp 0      : TMA producer: cp.async.bulk.tensor loads of the A and B boxes of each k-iteration into a shared-memory ring of
//                 four stages (three for 128-wide tiles, so that two CTAs share an SM); completion is signalled on the stage's
//                 "full" mbarrier by byte count.  With one box per operand the elected lane issues both, with several
//                 boxes or the im2col mode every lane its own (BoxLane::issue).
//   warp 1      : owns the tensor memory (tcgen05.alloc / dealloc) and issues tcgen05.mma.kind::tf32 (M = 128, N = tile
//                 width, K = 8) from the elected lane, four per stage, accumulating in TMEM; tcgen05.commit releases the stage
//                 ("empty" mbarrier) and finally signals the epilogue.
//   warps 2..9  : epilogue.  Each warp reads its 32-lane quarter of the accumulator with tcgen05.ld (32 columns at a time)
//                 and writes the result: pixel-major for convolutions (a warp store covers 32 consecutive pixels of one
//                 channel: 128 contiguous bytes), row-major for gemm / weight-grad; optional bias, alpha, accumulation,
//                 and atomic accumulation under split-K.
// Activations are NCHW at the boundary.  For 1x1 convolutions on images of 32 pixels or more the pixel index is the
// contiguous one and the activation operand is fed M/N-major (tcgen05 allows it for tf32) straight from the tensor with a
// 4-D tiled tensor map.  R x S convolutions with stride 1 run in tap-loop form from a channels-last copy (one transposing
// pass, see channels_last_kernel): a TMA box is then a window of whole image rows whose coordinates the tap shifts, and
// zero fill outside the image is the padding.  Images that fill no tiles, and strides, go through the TMA unit's im2col mode on the
// same copies (conv_fwd_any and its neighbours), 1x1 convolutions on such images through several clipped boxes per tile.  1x1
// convolutions on maps of 4 and 16 pixels are gathered by the epilogue warps.  Filters over a few channels, and strided ones where
// the unfolded matrix is no larger than two copies, are unfolded by the helper kernels below (wants_im2col).
// Every mbarrier wait is bounded: after about a second it records a code in the library's device status word and the CTA
// runs to its normal teardown (TMEM is released on every path).  The single issuing lanes of warps 0 and 1 are rejoined by
// their warps (__syncwarp) before the block-wide barrier, which needs converged warps.
#include <cooperative_groups.h>
#include <cuda.h>

#include <vector>

#include "gemm.cuh"
#include "tc_plan.h"

void* arena_alloc(size_t bytes, bool zero);
namespace ltb { void* step_alloc(size_t bytes); }
extern "C" int ltb_free(void* p, size_t bytes);

namespace cg = cooperative_groups;

namespace ltb {

constexpr int kMaxStages = 6;
constexpr int kPartPitch = 129;                    // floats per column of a CTA's partial tile in shared memory (odd: reads along either axis are conflict-free)
constexpr int kTapChunk = 40, kTapPitch = 161;     // TC_EPI_TAPS staging: floats from chunk to chunk of 32 columns (lanes = 8 channels x 4 chunks hit 32 banks) and from row to row
constexpr int kTcThreads = 320;                    // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue

// One moving part of a box coordinate: coordinate `dim` += ((i / div) % mod) * mul, i the tile or the k-iteration.
struct TcTerm { FastDiv div, mod; int dim, mul; };
struct TcOperandDev {
  TcTerm tile[3], k[3];
  FastDiv n0, n1;                             // of the walk
  int n_tile, n_k, c_off[5];
  TcWalk walk;                                // the k part as a mixed-radix counter (tc_plan.h)
  int rank, nk;
  uint32_t stage_bytes, desc_lo, desc_hi;     // descriptor without the start address
  uint32_t kstep_off[8];
  int load, nbox, dim0;                       // TcLoad; boxes per stage; extent of dimension 0 (TC_LOAD_BOXES skips boxes beyond it)
  TcIm2col im;
};
struct TcParams {
  TcOperandDev a, b;
  int M, N, bn, k_iters, k_per_split, epilogue, accumulate, atomic, stages;
  uint32_t idesc;
  float* out; const float* bias; float alpha;
  long long split_stride;      // floats between the result slabs of consecutive clusters of splits (see launch_plan)
  int cluster_z;               // splits whose partial results are summed inside the kernel: a thread-block cluster of this many CTAs along z
  long long pix_per_img, img_stride, chan_stride, ld;
  FastDiv by_pix;              // by the tile rows of an image (pix_pad)
  int col_mod, col_mul;        // TC_EPI_TAPS: col_mod channels in blocks of 32, col_mul taps
  // Gather mode (gather_src != null): the A operand is not loaded by TMA but collected by the epilogue warps, which are idle
  // during the main loop, straight from an activation tensor src[img][chan][pix] with pix = 4 or 16 (images too small for a
  // 128-byte run of pixels), transposing it on the way into the K-major rows the tensor core reads.
  const float* gather_src; int g_pix, g_chan, g_imgs;
  int relu;                    // clamp the result at zero (store epilogues, mode 0)
  int* status;
  long long wait_cycles;       // bound of every spin wait, in clock64 ticks (the context's limit, ~1 s by default)
};

// ---- PTX wrappers ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait: false when it gave up (the code is recorded, the shared abort flag raised).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int code, long long limit) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > limit) { *abort_flag = 1; atomicExch(status, code); return false; }
  }
  return true;
}
__device__ __forceinline__ void tma_load(const CUtensorMap* map, uint64_t* bar, void* dst, int rank, const int* c) {
  const uint32_t d = smem_u32(dst), b = smem_u32(bar);
  const uint64_t m = reinterpret_cast<uint64_t>(map);
  if (rank == 2)
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(d), "l"(m), "r"(b), "r"(c[0]), "r"(c[1]) : "memory");
  else if (rank == 3)
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(d), "l"(m), "r"(b), "r"(c[0]), "r"(c[1]), "r"(c[2]) : "memory");
  else if (rank == 4)
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                 ::"r"(d), "l"(m), "r"(b), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]) : "memory");
  else
    asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
                 ::"r"(d), "l"(m), "r"(b), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(c[4]) : "memory");
}
// The same for a CTA of a pair: `bar` is a barrier of the pair's first CTA, as an address of the cluster's shared memory.
__device__ __forceinline__ void tma_load_pair(const CUtensorMap* map, uint32_t b, void* dst, int rank, const int* c) {
  const uint32_t d = smem_u32(dst);
  const uint64_t m = reinterpret_cast<uint64_t>(map);
  if (rank == 2)
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(d), "l"(m), "r"(b), "r"(c[0]), "r"(c[1]) : "memory");
  else if (rank == 3)
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(d), "l"(m), "r"(b), "r"(c[0]), "r"(c[1]), "r"(c[2]) : "memory");
  else if (rank == 4)
    asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
                 ::"r"(d), "l"(m), "r"(b), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]) : "memory");
  else
    asm volatile("cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
                 ::"r"(d), "l"(m), "r"(b), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]), "r"(c[4]) : "memory");
}
__device__ __forceinline__ void tma_im2col_pair(const CUtensorMap* map, uint32_t b, void* dst, int c, int w, int h, int n, int s, int r) {
  asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(b), "r"(c), "r"(w), "r"(h), "r"(n), "h"((uint16_t)s), "h"((uint16_t)r) : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t first_of_pair(const void* p) {      // where p's namesake lies in the pair's first CTA
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(cluster_rank() & ~1u));
  return a;
}
__device__ __forceinline__ void pair_sync() { asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// One im2col-mode load: the map's walk starts at base pixel (w, h) of image n, tap (s, r) is added as an offset.
__device__ __forceinline__ void tma_im2col(const CUtensorMap* map, uint64_t* bar, void* dst, int c, int w, int h, int n, int s, int r) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c), "r"(w), "r"(h), "r"(n), "h"((uint16_t)s), "h"((uint16_t)r) : "memory");
}
// True in one lane of the (converged) warp, the same one every time.  The tensor-core and TMA instructions take their operands from
// the warp's uniform registers; behind this the compiler knows that one lane runs them, behind `lane == 0` it makes a loop over the
// lanes of every such instruction (four MMAs and a commit then took 670 cycles to issue, two and a half times the MMAs themselves).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {        // arrives at this barrier of both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)(3u << (cluster_rank() & ~1u))) : "memory");
}
__device__ __forceinline__ void tc_mma_tf32_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_mma_tf32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
      "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The producer warp.  Lanes 0..7 are the A operand's loads of a stage, lanes 8..15 the B operand's: a lane owns one box (or im2col
// load) for the CTA's whole life, so the coordinates cost the warp what one lane costs.  Box coordinates: c[d] = c_off[d] + tile part (fixed for the CTA)
// + ((kiter / k_div[d]) % k_mod[d]) * k_mul[d]; the k part is advanced with additions only, the plan's TcWalk says what each level
// of the counter adds, and the common case (level 0) uses increments kept in registers.
struct BoxLane {
  int c[5], inc0[5], i0, i1, n0, n1;
  int load, rank;
  int pi, pj, pn;                     // im2col modes: output pixel (pi, pj) of image pn; tap of TC_LOAD_IM2COL_MN in c[1], c[2]
  uint32_t offset;                    // of this lane's box within a stage
  bool active;

  // Start coordinates of the lane's operand.  Every lane computes its own, from multiplications only: the start of a CTA is exposed
  // in launches as short as these (five coordinates by integer division, one lane each, took 1500 cycles).  Returns the bytes
  // a stage receives.
  template <bool GEN>
  __device__ __forceinline__ uint32_t init(const TcParams& P, int m_tile, int n_tile, int k0, int lane, bool gather) {
    const bool second = (lane & 8) != 0;
    const TcOperandDev& o = second ? P.b : P.a;
    const int tile = second ? n_tile : m_tile, d = lane & 7;
#pragma unroll
    for (int j = 0; j < 5; ++j) { c[j] = o.c_off[j]; inc0[j] = o.walk.inc[0][j]; }
    auto add = [&](const TcTerm& t, int i) {
      int r; t.mod.divmod(t.div.div(i), r);
      r *= t.mul;
#pragma unroll
      for (int j = 0; j < 5; ++j) if (t.dim == j) c[j] += r;
    };
    if (tile) for (int j = 0; j < o.n_tile; ++j) add(o.tile[j], tile);
    i0 = i1 = 0;
    if (k0) {
      for (int j = 0; j < o.n_k; ++j) add(o.k[j], k0);
      const int q = o.n0.divmod(k0, i0);
      o.n1.divmod(q, i1);
    }
    n0 = o.walk.n0; n1 = o.walk.n1; rank = o.rank; load = GEN ? o.load : (int)TC_LOAD_BOX;
    active = lane < 16 && !(gather && !second) && d < (GEN ? o.nbox : 1);
    offset = second ? P.a.stage_bytes : 0u;
    uint32_t bytes = o.stage_bytes;
    if (GEN && load == TC_LOAD_BOXES) {
      c[0] += 32 * d; offset += 4096u * d; bytes = 4096u;
      if (c[0] >= o.dim0) active = false;
    } else if (GEN && load == TC_LOAD_TAPS) {
      const int q = n_tile * o.nbox + d, blk = q / o.im.taps, tap = q - blk * o.im.taps, r = tap / o.im.tap_s;
      c[1] += tap - r * o.im.tap_s; c[2] += r; c[4] = blk;
      offset += 4096u * d; bytes = 4096u;
      if (blk >= o.im.ch_blocks) active = false;
    } else if (GEN && load == TC_LOAD_IM2COL) start(o.im, (long long)m_tile * 128);
    else if (GEN && load == TC_LOAD_IM2COL_MN) {
      const int q = n_tile * o.nbox + d, blk = q / o.im.taps, tap = q - blk * o.im.taps;
      c[0] = blk * 32; c[2] = tap / o.im.tap_s; c[1] = tap - c[2] * o.im.tap_s;
      offset += 4096u * d; bytes = 4096u;
      if (blk >= o.im.ch_blocks) active = false;
      start(o.im, (long long)k0 * 32);
    }
    return __reduce_add_sync(0xffffffffu, active ? bytes : 0u);
  }
  __device__ __forceinline__ void start(const TcIm2col& m, long long pixel) {
    const int per = m.grid_w * m.grid_h;
    pn = (int)(pixel / per); const int q = (int)(pixel - (long long)pn * per);
    pj = q / m.grid_w; pi = q - pj * m.grid_w;
  }
  // Issues a stage's loads and moves on to the next k-iteration.  GEN false: one box per operand, issued by the elected lane, which gets the
  // coordinates by shuffles.  GEN true: up to eight boxes per operand; every lane issues its own (the shuffles would cost more than the
  // compiler's loop over the lanes: 56 x 56, 3x3 layer 323 us instead of 282).
  // PAIR: `pair_bar` instead of bar.
  template <bool GEN, bool PAIR>
  __device__ __forceinline__ void issue(const TcParams& P, bool both, const CUtensorMap* map_a, const CUtensorMap* map_b, const TcOperandDev& o, int lane, uint64_t* bar, uint32_t pair_bar, uint8_t* stage) {
    if (!GEN) {
      int va[5], vb[5];
#pragma unroll
      for (int j = 0; j < 5; ++j) { va[j] = __shfl_sync(0xffffffffu, c[j], 0); vb[j] = __shfl_sync(0xffffffffu, c[j], 8); }
      if (elect_one()) {
        if (PAIR) { tma_load_pair(map_a, pair_bar, stage, P.a.rank, va); tma_load_pair(map_b, pair_bar, stage + P.a.stage_bytes, P.b.rank, vb); }
        else {
          if (both) tma_load(map_a, bar, stage, P.a.rank, va);
          tma_load(map_b, bar, stage + P.a.stage_bytes, P.b.rank, vb);
        }
      }
    } else {
      const CUtensorMap* const map = lane & 8 ? map_b : map_a;
      if (load != TC_LOAD_IM2COL && load != TC_LOAD_IM2COL_MN) { if (active) { if (PAIR) tma_load_pair(map, pair_bar, stage + offset, rank, c); else tma_load(map, bar, stage + offset, rank, c); } }
      else if (active) {
        const int w = o.im.low_w + pi * o.im.step_w, h = o.im.low_h + pj * o.im.step_h;
        if (PAIR) tma_im2col_pair(map, pair_bar, stage + offset, c[0], w, h, pn, c[1], c[2]); else tma_im2col(map, bar, stage + offset, c[0], w, h, pn, c[1], c[2]);
      }
    }
    if (GEN && load == TC_LOAD_IM2COL_MN) {
      pi += o.im.adv_i; pj += o.im.adv_j; pn += o.im.adv_n;
      if (pi >= o.im.grid_w) { pi -= o.im.grid_w; ++pj; }
      if (pj >= o.im.grid_h) { pj -= o.im.grid_h; ++pn; }
      return;
    }
    if (++i0 != n0) {
#pragma unroll
      for (int d = 0; d < 5; ++d) c[d] += inc0[d];
    } else {
      i0 = 0;
      int lvl = 1;
      if (++i1 == n1) { i1 = 0; lvl = 2; }
#pragma unroll
      for (int d = 0; d < 5; ++d) c[d] += o.walk.inc[lvl][d];
    }
  }
};

// ---- the engine -------------------------------------------------------------------------------------------------------
// Epilogue store helpers: pointers advance by the column stride instead of being recomputed, and the mode (plain, bias,
// accumulate, atomic) is decided outside the 32-element loops, so that a column costs two or three instructions.  With one
// epilogue warp per scheduler every extra dependent instruction is exposed latency.
__device__ __forceinline__ float clamp_if(float v, int relu) { return relu && v < 0.0f ? 0.0f : v; }
template <bool FULL>
__device__ __forceinline__ void store_columns(float* p, long long stride, const uint32_t* r, float alpha, const float* bias, int lim, int mode, int relu) {
  if (mode == 2) {                               // split-K, default mode: atomic accumulation (the bias pointer is set for split 0 only)
#pragma unroll
    for (int j = 0; j < 32; ++j) { if (FULL || j < lim) atomicAdd(p, alpha * __uint_as_float(r[j]) + (bias ? bias[j] : 0.0f)); p += stride; }
  } else if (mode == 1) {                        // accumulate: all loads first, a load-add-store chain per element would serialise on latency
    // sixteen at a time: thirty-two loads in flight next to the thirty-two accumulator registers spill
#pragma unroll
    for (int h = 0; h < 32; h += 16) {
      float old[16]; const float* q = p;
#pragma unroll
      for (int j = 0; j < 16; ++j) { old[j] = (FULL || h + j < lim) ? *q : 0.0f; q += stride; }
#pragma unroll
      for (int j = 0; j < 16; ++j) { if (FULL || h + j < lim) *p = old[j] + alpha * __uint_as_float(r[h + j]); p += stride; }
    }
  } else if (bias) {
#pragma unroll
    for (int j = 0; j < 32; ++j) { if (FULL || j < lim) *p = clamp_if(alpha * __uint_as_float(r[j]) + bias[j], relu); p += stride; }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) { if (FULL || j < lim) *p = clamp_if(alpha * __uint_as_float(r[j]), relu); p += stride; }
  }
}

// Where D column n of a row-major result goes; negative: nowhere.
template <int EPI>
__device__ __forceinline__ long long out_column(const TcParams& P, int n) {
  if (EPI == TC_EPI_TAPS) {
    const int q = n >> 5, blk = q / P.col_mul, c = blk * 32 + (n & 31);
    return c < P.col_mod ? (long long)c * P.col_mul + (q - blk * P.col_mul) : -1;
  }
  return n;
}

// EPI (TcEpilogue) and MODE (0 store, 1 accumulate, 2 atomic accumulate) are compile-time: each launch then carries one
// epilogue instead of six, a third of the instructions -- these CTAs live for a few microseconds and the instruction cache
// starts cold (measured hit rate 66 % with all variants in one kernel).
// PAIR: a cluster of two CTAs along x works on 256 rows.  Each loads its own 128 rows of A and half of B's columns, signalling the first one's barriers; the
// first one issues the MMAs over both CTAs' shared memory (cta_group::2), whose commits arrive in both; each has its rows' accumulator and stores them.
// The arrivals at the other CTA's barriers are relaxed (the copies are what the barrier orders): released at cluster scope, each waited about a
// microsecond and a product took twice as long.
template <int EPI, int MODE, bool GEN, bool PAIR>
__global__ void __launch_bounds__(kTcThreads, PAIR ? 1 : 2)
tc_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ TcParams P) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kMaxStages];
  __shared__ __align__(8) uint64_t empty_bar[kMaxStages];
  __shared__ __align__(8) uint64_t accum_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // the shuffle tells the compiler that warp is uniform
  const int m_tile = blockIdx.x, n_tile = blockIdx.y;
  const bool second_cta = PAIR && (blockIdx.x & 1);
  const int k_begin = blockIdx.z * P.k_per_split;
  const int k_end = min(P.k_iters, k_begin + P.k_per_split);
  const int n_iter = k_end - k_begin;
  const int stages = P.stages;
  const bool gather = P.gather_src != nullptr;

  // stage buffers, aligned to the 1024-byte swizzle atom
  uint8_t* stage_base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t stage_bytes = P.a.stage_bytes + P.b.stage_bytes;

  // Set-up.  Warp 1 initialises the barriers while the producer warp works out its coordinates; those two meet, and the producer
  // starts to fill the ring while warp 1 allocates tensor memory.
  BoxLane box;
  uint32_t tx = 0;             // bytes a stage receives through TMA
  if (warp == 0) {
    if (lane < 2) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(lane ? &map_b : &map_a)) : "memory");
    tx = box.init<GEN>(P, m_tile, PAIR ? 2 * n_tile + (second_cta ? 1 : 0) : n_tile, k_begin, lane, gather);
    asm volatile("bar.sync 5, 64;" ::: "memory");
    pdl_wait();
  }
  if (warp == 1) {
    if (lane == 0) {
      // a stage is full when the TMA bytes have landed (one arrival with the byte count) and, in gather mode, the eight
      // gathering warps have stored their rows (one arrival each)
      for (int s = 0; s < stages; ++s) { mbar_init(&full_bar[s], PAIR ? 2 : gather ? 9 : 1); mbar_init(&empty_bar[s], 1); }      // (of a pair: an arrival with the byte count from each CTA)
      mbar_init(&accum_bar, 1);
      abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    asm volatile("bar.sync 5, 64;" ::: "memory");
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)P.bn) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)P.bn) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  // gather mode: the first two k-iterations' loads leave before the warps meet
  float4 cur[4], nxt[4], nx2[4];                                               // the loads of two k-iterations are in flight while one is stored
  const int gw = warp - 2, pix = P.g_pix, chan = P.g_chan;
  const int runs = pix == 16 ? 1 : 4;                                         // 1 run of 16 floats or 4 runs of 4
  const long long img0 = ((long long)m_tile * 128 + gw * 16) >> (runs == 1 ? 4 : 2);     // image of the warp's first tile row (pix 16), or the first of four (pix 4)
  const uint32_t col = (uint32_t)(lane >> 2), sub = (uint32_t)(lane & 3) << 2;
  auto fetch = [&](int it, float4* v) {
    const int c = (k_begin + it) * 32 + lane;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long img = runs == 1 ? img0 : img0 + j;
      const bool ok = c < chan && img < P.g_imgs;
      const float4* src = reinterpret_cast<const float4*>(P.gather_src + (img * chan + c) * pix) + (runs == 1 ? j : 0);
      v[j] = ok ? __ldg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  if (warp == 0) pdl_launch();
  if (warp >= 2) pdl_wait();
  if (gather && warp >= 2 && n_iter > 0) { fetch(0, cur); if (n_iter > 1) fetch(1, nxt); }
  // The producer goes on issuing; the others meet here (the tensor memory's address, the barriers), so that the first MMA waits for
  // its own stage only.
  tc_fence_before();
  if (PAIR) { __syncwarp(); pair_sync(); }                     // both CTAs' barriers and tensor memory are there
  else if (warp != 0) asm volatile("bar.sync 6, 288;" ::: "memory");
  tc_fence_after();
  const uint32_t tmem_base = warp != 0 ? tmem_slot : 0u;

  if (warp == 0) {
    int s = 0; uint32_t ph = 0;
    const TcOperandDev& o = lane & 8 ? P.b : P.a;
    for (int it = 0; it < n_iter; ++it) {
      if (it >= stages) {                                      // the first fills find the ring empty and wait for nobody
        const bool ok = mbar_wait(&empty_bar[s], ph ^ 1u, &abort_flag, P.status, 1, P.wait_cycles);
        if (!__all_sync(0xffffffffu, ok)) break;
      }
      uint32_t pair_bar = 0;
      if (PAIR) {
        pair_bar = first_of_pair(&full_bar[s]);
        if (elect_one()) asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(pair_bar), "r"(tx) : "memory");
      } else if (elect_one()) mbar_expect_tx(&full_bar[s], tx);
      __syncwarp();
      box.issue<GEN, PAIR>(P, !gather, &map_a, &map_b, o, lane, &full_bar[s], pair_bar, stage_base + (size_t)s * stage_bytes);
      if (++s == stages) { s = 0; ph ^= 1u; }
    }
    __syncwarp();          // the block-wide barrier below needs converged warps
  } else if (warp == 1) {
    if (n_iter > 0 && !second_cta) {
      int s = 0; uint32_t ph = 0;
      // descriptor pieces that do not change: kept in registers so that an MMA costs two additions and the instruction
      uint32_t koa[4], kob[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) { koa[k] = P.a.kstep_off[k] >> 4; kob[k] = P.b.kstep_off[k] >> 4; }
      const uint64_t a_hi = (uint64_t)P.a.desc_hi << 32, b_hi = (uint64_t)P.b.desc_hi << 32;
      const uint32_t a_lo = P.a.desc_lo, b_lo = P.b.desc_lo, idesc = P.idesc, a_bytes = P.a.stage_bytes;
      const uint32_t ring = smem_u32(stage_base);
      for (int it = 0; it < n_iter; ++it) {
        const bool ok = mbar_wait(&full_bar[s], ph, &abort_flag, P.status, 2, P.wait_cycles);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_fence_after();
        if (elect_one()) {
        const uint32_t sa = (ring + (uint32_t)s * stage_bytes) >> 4, sb = sa + (a_bytes >> 4);   // in 16-byte units (ring < 256 KB: 14 bits)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t adesc = a_hi | (uint64_t)(a_lo | ((sa + koa[k]) & 0x3FFFu));
          const uint64_t bdesc = b_hi | (uint64_t)(b_lo | ((sb + kob[k]) & 0x3FFFu));
          if (PAIR) tc_mma_tf32_pair(tmem_base, adesc, bdesc, idesc, (it > 0 || k > 0) ? 1u : 0u);
          else tc_mma_tf32(tmem_base, adesc, bdesc, idesc, (it > 0 || k > 0) ? 1u : 0u);
        }
        if (PAIR) { tc_commit_pair(&empty_bar[s]); if (it + 1 == n_iter) tc_commit_pair(&accum_bar); }
        else {
        tc_commit(&empty_bar[s]);       // the stage may be refilled once these MMAs have read it
        if (it + 1 == n_iter) tc_commit(&accum_bar);    // accumulator complete
        }
        }
        __syncwarp();
        if (++s == stages) { s = 0; ph ^= 1u; }
      }
    }
    __syncwarp();
  } else if (n_iter > 0) {
    // ---- warps 2..9.  In gather mode they first feed the A operand: warp g owns rows 16 g .. 16 g + 15 of the tile (one image
    // of 16 pixels, or four images of 4), lane = channel within the 32-channel block of the k-iteration.  A lane reads its
    // channel's 16 pixels (64 contiguous bytes, or four runs of 16) and stores them down its column of the tile: for a fixed
    // pixel the 32 lanes write one whole 128-byte row (128-byte swizzle: 16-byte chunk j of row r sits at chunk j ^ (r & 7)),
    // so the stores are free of bank conflicts.  The loads of the next two k-iterations are issued before this one is stored.
    if (gather) {
      int s = 0; uint32_t ph = 0;
      for (int it = 0; it < n_iter; ++it) {
        if (it + 2 < n_iter) fetch(it + 2, nx2);
        bool ok = true;
        if (it >= stages) { if (lane == 0) ok = mbar_wait(&empty_bar[s], ph ^ 1u, &abort_flag, P.status, 4, P.wait_cycles); ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0; }
        if (!ok) break;
        uint8_t* sa = stage_base + (size_t)s * stage_bytes + (size_t)gw * 16 * 128;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float e[4] = {cur[j].x, cur[j].y, cur[j].z, cur[j].w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t r = (uint32_t)(j * 4 + i);                            // row within this warp's sixteen (gw * 16 is a multiple of 8: r & 7 is the swizzle phase)
            *reinterpret_cast<float*>(sa + r * 128 + (((col ^ (r & 7u)) << 4) | sub)) = e[i];
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");             // the tensor core reads shared memory through the async proxy
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full_bar[s])) : "memory");
#pragma unroll
        for (int j = 0; j < 4; ++j) { cur[j] = nxt[j]; nxt[j] = nx2[j]; }
        if (++s == stages) { s = 0; ph ^= 1u; }
      }
    }
    // ---- epilogue: TMEM lane quarter = warp index mod 4; the two warps of a quarter take alternate 32-column chunks
    const int q = warp & 3, half = (warp - 2) >> 2;
    // where this lane's pixel goes, worked out while the contraction runs
    float* dst = nullptr;
    if (EPI == TC_EPI_PIXEL) {
      const int m = m_tile * 128 + q * 32 + lane;
      int pix; const int img = P.by_pix.divmod(m, pix);
      if (m < P.M && pix < P.pix_per_img) dst = P.out + (long long)(blockIdx.z / P.cluster_z) * P.split_stride + (long long)img * P.img_stride + pix;
    }
    const bool ok = mbar_wait(&accum_bar, 0, &abort_flag, P.status, 3, P.wait_cycles);
    tc_fence_after();
    if (ok) {
      const int n0 = n_tile * P.bn;
      const float alpha = P.alpha;
      constexpr int mode = MODE;
      const uint32_t tmem_row = tmem_base + ((uint32_t)(q * 32) << 16);
      float* const out_base = P.out + (long long)(blockIdx.z / P.cluster_z) * P.split_stride;   // a cluster of splits writes its own slab of partial results
      if (P.cluster_z > 1) {
        // Split-K inside a cluster: the accumulator goes to this CTA's shared memory (the pipeline stages are idle by now);
        // the cluster then adds the tiles up (below, after the block has met).  The tile is laid out so that the reads of
        // that sum run along contiguous addresses (reads from another SM's shared memory are slow when scattered):
        // part[column][row] for the pixel-major epilogue, part[row][column] for the row-major one, odd pitches.
        float* part = reinterpret_cast<float*>(stage_base);
        const int row = q * 32 + lane, rp = P.bn + 1;
        for (int c0 = half * 32; c0 < P.bn; c0 += 64) {
          uint32_t r[32];
          tc_ld32(tmem_row + (uint32_t)c0, r);
#pragma unroll
          for (int j = 0; j < 32; ++j) part[EPI == TC_EPI_PIXEL ? (c0 + j) * kPartPitch + row : row * rp + c0 + j] = __uint_as_float(r[j]);
        }
      } else if (EPI == TC_EPI_PIXEL) {
        // lane = pixel, register j = channel: for a fixed j a warp covers 32 consecutive pixels (128 contiguous bytes)
        const long long cs = P.chan_stride;
        for (int c0 = half * 32; c0 < P.bn; c0 += 64) {
          if (n0 + c0 >= P.N) break;                         // uniform across the warp
          uint32_t r[32];
          tc_ld32(tmem_row + (uint32_t)c0, r);
          if (dst) {
            const int lim = P.N - n0 - c0;
            const float* bias = (P.bias && (!P.atomic || blockIdx.z == 0)) ? P.bias + n0 + c0 : nullptr;
            if (lim >= 32) store_columns<true>(dst + (long long)(n0 + c0) * cs, cs, r, alpha, bias, 32, mode, P.relu);
            else store_columns<false>(dst + (long long)(n0 + c0) * cs, cs, r, alpha, bias, lim, mode, P.relu);
          }
        }
      } else if (EPI == TC_EPI_TAPS) {
        // stage this warp's chunks of 32 columns; they are written out below, when the other warp of the quarter has staged its own
        float* tile = reinterpret_cast<float*>(stage_base) + (size_t)q * 32 * kTapPitch;
        for (int c0 = half * 32; c0 < P.bn; c0 += 64) {
          if (n0 + c0 >= P.N) break;
          uint32_t r[32];
          tc_ld32(tmem_row + (uint32_t)c0, r);
#pragma unroll
          for (int j = 0; j < 32; ++j) tile[lane * kTapPitch + (c0 >> 5) * kTapChunk + j] = __uint_as_float(r[j]);
        }
      } else {
        // row-major output: transpose each 32x32 block through shared memory so that a warp writes 32 consecutive columns
        // of one row (128 contiguous bytes) per instruction.  The staging tile lives in the pipeline stages, which are idle
        // once the accumulator is complete (every load has landed and every MMA has read its operands).
        float (*tile)[33] = reinterpret_cast<float (*)[33]>(stage_base + (size_t)(warp - 2) * 32 * 33 * 4);
        const long long m0 = (long long)m_tile * 128 + q * 32;
        const int rows = (int)min(32ll, (long long)P.M - m0);
        const long long ld = P.ld;
        for (int c0 = half * 32; c0 < P.bn; c0 += 64) {
          if (n0 + c0 >= P.N) break;
          uint32_t r[32];
          tc_ld32(tmem_row + (uint32_t)c0, r);
#pragma unroll
          for (int j = 0; j < 32; ++j) tile[lane][j] = __uint_as_float(r[j]);
          __syncwarp();
          const int n = n0 + c0 + lane;
          const long long col = out_column<EPI>(P, n);
          if (n < P.N && col >= 0 && rows > 0) {
            uint32_t t[32];
#pragma unroll
            for (int rr = 0; rr < 32; ++rr) t[rr] = __float_as_uint(tile[rr][lane]);
            // after the transpose the "columns" of store_columns are the 32 rows of this block, `ld` apart
            const float* bias = nullptr;
            float* p = out_base + m0 * ld + col;
            if (P.bias && mode == 0) {
              const float bv = P.bias[n];
#pragma unroll
              for (int rr = 0; rr < 32; ++rr) { if (rr < rows) *p = alpha * __uint_as_float(t[rr]) + bv; p += ld; }
            } else if (rows == 32) store_columns<true>(p, ld, t, alpha, bias, 32, mode, 0);
            else store_columns<false>(p, ld, t, alpha, bias, rows, mode, 0);
          }
          __syncwarp();
        }
      }
    }
    if (EPI == TC_EPI_TAPS && P.cluster_z == 1) {
      // Weight gradient of a multi-tap filter, dw[row][channel][tap].  The tile's chunks are taps of one channel block (mostly), so
      // the elements of a row are taken channel by channel, chunk by chunk: 32 lanes then touch about ten 32-byte sectors instead of
      // 36 (a chunk at a time, stride `taps`), and L2 handles the atomics of split-K sector by sector (256 -> 256, 3x3, 4 x 4, batch
      // 128: 35 -> 29 us).
      // Both warps of a quarter meet here on every path, also after a wait that gave up.
      asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
      if (ok) {
        const float* tile = reinterpret_cast<const float*>(stage_base) + (size_t)q * 32 * kTapPitch;
        const long long m0 = (long long)m_tile * 128 + q * 32;
        const int r_end = min(half * 16 + 16, (int)min(32ll, (long long)P.M - m0)), nch = P.bn >> 5, shift = nch == 4 ? 2 : 1;
        for (int i = 0; i < nch; ++i) {
          const int e = i * 32 + lane, ch = e & (nch - 1), c = e >> shift, n = n_tile * P.bn + ch * 32 + c;
          const long long col = n < P.N ? out_column<EPI>(P, n) : -1;
          if (col < 0) continue;
          const float* src = tile + ch * kTapChunk + c + half * 16 * kTapPitch;
          float* p = P.out + (m0 + half * 16) * P.ld + col;
          const int rows = r_end - half * 16;
          float old[16];
          if (MODE == 1)                          // all loads first: added one after the other these take 25 us where everything else takes 11
#pragma unroll
            for (int r = 0; r < 16; ++r) old[r] = r < rows ? p[r * P.ld] : 0.0f;
#pragma unroll
          for (int r = 0; r < 16; ++r) {
            if (r >= rows) break;
            const float v = P.alpha * src[r * kTapPitch];
            if (MODE == 2) atomicAdd(p + r * P.ld, v); else p[r * P.ld] = MODE == 1 ? old[r] + v : v;
          }
        }
      }
    }
  }
  if (P.cluster_z > 1 && n_iter <= 0 && warp >= 2) {
    // a split without k-iterations (the split count was rounded up to the cluster size) contributes zeros
    float* part = reinterpret_cast<float*>(stage_base);
    const int part_floats = EPI == TC_EPI_PIXEL ? P.bn * kPartPitch : 128 * (P.bn + 1);
    for (int i = threadIdx.x - 64; i < part_floats; i += kTcThreads - 64) part[i] = 0.0f;
  }
  tc_fence_before();
  __syncthreads();
  if (P.cluster_z > 1) {
    // ---- the cluster sums its partial tiles in a fixed order.  The hardware cluster barrier is safe to wait at: the CTAs
    // of a cluster are scheduled together.  CTA (of a pair's halves each) number zr of the cluster owns a slice of the tile -- columns for the
    // pixel-major epilogue, rows for the row-major one, so that its global stores coalesce -- reads that slice from the
    // shared memory of every CTA of the cluster, rank 0 first, and writes the result the way the epilogue would.
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (warp >= 2 && !abort_flag) {
      const int cz = P.cluster_z, zr = (int)cluster.block_rank() >> (PAIR ? 1 : 0);
      float* part = reinterpret_cast<float*>(stage_base);
      const float* remote[8];
#pragma unroll
      for (int z = 0; z < 8; ++z) remote[z] = z < cz ? cluster.map_shared_rank(part, PAIR ? 2 * z + (second_cta ? 1 : 0) : z) : part;
      const int t = threadIdx.x - 64;                                  // 0 .. 255
      const int n0 = n_tile * P.bn;
      float* const out_base = P.out + (long long)(blockIdx.z / cz) * P.split_stride;
      const float alpha = P.alpha;
      // Eight outputs at a time per thread: their partial tiles are read and, when the destination is accumulated into, its
      // old values loaded, all before the first store (a load-add-store chain per element would pay the memory latency
      // once per element).
      const bool acc = MODE == 1;
      if (EPI == TC_EPI_PIXEL) {
        const TcSlice slice(P.bn, cz, zr, P.N - n0);
        const int c_lo = slice.lo + (t >> 7), c_hi = slice.hi;
        const int row = t & 127;
        const int m = m_tile * 128 + row;
        int pix; const int img = P.by_pix.divmod(m, pix);
        if (m < P.M && pix < P.pix_per_img) {
          float* dst = out_base + (long long)img * P.img_stride + pix + (long long)n0 * P.chan_stride;
          for (int cb = c_lo; cb < c_hi; cb += 16) {                   // this thread's columns cb, cb + 2, ..., cb + 14
            float v[8], old[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int c = cb + 2 * u; v[u] = 0.0f; old[u] = 0.0f;
              if (c < c_hi) {
#pragma unroll
                for (int z = 0; z < 8; ++z) if (z < cz) v[u] += remote[z][c * kPartPitch + row];
                if (acc) old[u] = dst[(long long)c * P.chan_stride];
              }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int c = cb + 2 * u;
              if (c < c_hi) dst[(long long)c * P.chan_stride] = clamp_if(old[u] + alpha * v[u] + (P.bias ? P.bias[n0 + c] : 0.0f), P.relu);
            }
          }
        }
      } else {
        // rows of the slice go round the eight warps, a lane takes every 32nd column: a warp's stores cover 128 contiguous bytes
        const TcSliceRows rows(TcSlice(128, cz, zr, (int)min(128ll, (long long)P.M - (long long)m_tile * 128)), P.bn, t >> 5);
        for (int ib = 0; ib < rows.items; ib += 8) {
          float v[8], old[8]; float* o[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int i = ib + u; v[u] = 0.0f; old[u] = 0.0f; o[u] = nullptr;
            const int row = rows.row(i), c = (rows.run(i) << 5) + lane, n = n0 + c;
            if (i < rows.items && n < P.N) {
#pragma unroll
              for (int z = 0; z < 8; ++z) if (z < cz) v[u] += remote[z][row * (P.bn + 1) + c];
              const long long col = out_column<EPI>(P, n);
              o[u] = col >= 0 ? out_base + ((long long)m_tile * 128 + row) * P.ld + col : nullptr;
              if (acc && o[u]) old[u] = *o[u];
            }
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) if (o[u]) *o[u] = old[u] + alpha * v[u];
        }
      }
    }
    cluster.sync();                // no CTA leaves while its shared memory may still be read
  }
  if (PAIR) { __syncwarp(); pair_sync(); }           // neither CTA's barriers, stages or tensor memory are used by the other any more
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)P.bn) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)P.bn) : "memory");
  }
}

// ---- unfold / fold helpers for convolutions that are not 1x1 stride 1 ---------------------------------------------------
// col[n][(c*R+r)*S+s][p] = x[n][c][ho*sh-ph+r][wo*sw-pw+s] (0 outside): the reference's `finput` (TensorDslCPU.scala:484-530).
// A thread owns one output pixel of one input plane (n, c) and writes all R*S taps of it: the plane and pixel
// decomposition (the only integer divisions) is paid once per R*S elements, the writes of a warp stay contiguous.
__global__ void unfold_rows_kernel(const float* __restrict__ x, float* __restrict__ col, ConvDims d, int planes_per_block, int threads_per_plane, const ZeroFill zero) {
  pdl_enter();
  zero_fill(zero);
  const int pix = d.oH * d.oW, rs = d.R * d.S;
  const int64_t planes = (int64_t)d.N * d.C;
  const int lane_p = threadIdx.x % threads_per_plane;
  for (int64_t plane = (int64_t)blockIdx.x * planes_per_block + threadIdx.x / threads_per_plane; plane < planes;
       plane += (int64_t)gridDim.x * planes_per_block) {
  const float* src = x + plane * (int64_t)d.H * d.W;
  float* dst = col + plane * rs * pix;                         // rows (c*R + r)*S + s of image n are consecutive
  for (int p = lane_p; p < pix; p += threads_per_plane) {
    const int ho = p / d.oW, wo = p - ho * d.oW;
    const int ih0 = ho * d.sh - d.ph, iw0 = wo * d.sw - d.pw;
    float* q = dst + p;
    for (int r = 0; r < d.R; ++r) {
      const int ih = ih0 + r;
      const bool row_ok = ih >= 0 && ih < d.H;
      for (int s = 0; s < d.S; ++s) {
        const int iw = iw0 + s;
        *q = (row_ok && iw >= 0 && iw < d.W) ? src[ih * d.W + iw] : 0.0f;
        q += pix;
      }
    }
  }
  }
}
// Channels-last copy dst[n][p][ld] of src[n][chan][p] for any channel and pixel count; channels chan .. ld - 1 are written as zeros.
// A CTA moves 32 channels x 64 pixels through shared memory, coalesced on both sides, eight loads in flight per thread (tiles of 32 x 32
// with four took 19 us instead of 15 on 32 x 64 x 56 x 56).  grid (ceil(pix/64), ceil(ld/32), N), block 256.
__global__ void __launch_bounds__(256) channels_last_kernel(const float* __restrict__ src, float* __restrict__ dst, int chan, int pix, int ld, const ZeroFill zero) {
  pdl_enter();
  zero_fill(zero);
  __shared__ float tile[32][65];
  const int p0 = blockIdx.x * 64, c0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
  const float* s = src + ((int64_t)blockIdx.z * chan + c0) * pix + p0;
#pragma unroll
  for (int c = ty; c < 32; c += 4) tile[c][tx] = (c0 + c < chan && p0 + tx < pix) ? s[(int64_t)c * pix + tx] : 0.0f;
  __syncthreads();
  const int c = threadIdx.x & 31;
  float* d = dst + ((int64_t)blockIdx.z * pix + p0) * ld + c0 + c;
  if (c0 + c < ld) {
#pragma unroll
    for (int p = threadIdx.x >> 5; p < 64; p += 8) if (p0 + p < pix) d[(int64_t)p * ld] = tile[c][p];
  }
}
// The same copy of small images (fewer than 32 pixels: 64-pixel rows of the tile above would be mostly idle), 32 channels of one image
// per CTA; chan a multiple of 32.  grid (1, chan/32, N).
__global__ void to_rows_tiled_kernel(const float* __restrict__ src, float* __restrict__ dst, int chan, int pix, const ZeroFill zero) {
  pdl_enter();
  zero_fill(zero);
  __shared__ float tile[32][33];
  const int n = blockIdx.z, c0 = blockIdx.y * 32;
  const float* s = src + ((int64_t)n * chan + c0) * pix;
  for (int i = threadIdx.x; i < 32 * pix; i += blockDim.x) { const int c = i / pix; tile[c][i - c * pix] = s[i]; }
  __syncthreads();
  float* d = dst + (int64_t)n * pix * chan + c0;
  for (int i = threadIdx.x; i < 32 * pix; i += blockDim.x) { const int p = i >> 5, c = i & 31; d[(int64_t)p * chan + c] = tile[c][p]; }
}
// Channels-last copy of dy with sh - 1 / sw - 1 zeros between neighbouring pixels: up[n][sh a][sw b][k] = dy[n][k][a][b], 0 elsewhere
// (up is uH x uW pixels of ld channels).  The data-gradient of a strided convolution is the stride-1 data-gradient of this tensor,
// so no fold-back pass is needed.  A CTA writes the sh rows that one row of dy owns, 32 channels, through shared memory; wide rows
// go 32 pixels at a time.  grid (ceil(uH/sh), ceil(ld/32), N), block 256.
__global__ void __launch_bounds__(256) channels_last_up_kernel(const float* __restrict__ dy, float* __restrict__ up, int K, int ld, int oH, int oW, int uH, int uW, int sh, int sw, const ZeroFill zero) {
  pdl_enter();
  zero_fill(zero);
  __shared__ float tile[32][33];
  const int a = blockIdx.x, k0 = blockIdx.y * 32, n = blockIdx.z;
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  for (int b0 = 0; b0 * sw < uW; b0 += 32) {
    if (a < oH)
      for (int k = row; k < 32; k += 8) tile[k][lane] = (k0 + k < K && b0 + lane < oW) ? dy[(((int64_t)n * K + k0 + k) * oH + a) * oW + b0 + lane] : 0.0f;
    __syncthreads();
    if (k0 + lane < ld) {
      const int w_end = min(uW, (b0 + 32) * sw);
      for (int hu = sh * a; hu < sh * a + sh && hu < uH; ++hu)
        for (int wu = b0 * sw + row; wu < w_end; wu += 8) {
          const int b = wu / sw;
          up[(((int64_t)n * uH + hu) * uW + wu) * ld + k0 + lane] = (hu == sh * a && a < oH && b * sw == wu && b < oW) ? tile[lane][b - b0] : 0.0f;
        }
    }
    __syncthreads();
  }
}
// Filters w[k][c][tap] (OIHW) as one matrix per tap: out[tap][k][c] (by_c == 0, forward) or out[tap][c][k] (data-grad).
// Rows of the inner index are ld floats long, zeros beyond it.
__global__ void permute_taps_kernel(const float* __restrict__ w, float* __restrict__ out, int K, int C, int taps, int by_c, int ld, int64_t total) {
  pdl_enter();
  const int inner = by_c ? K : C, outer = by_c ? C : K;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int a = (int)(i % ld); const int64_t t2 = i / ld; const int b = (int)(t2 % outer); const int t = (int)(t2 / outer);
    const int k = by_c ? a : b, c = by_c ? b : a;
    out[i] = a < inner ? w[((int64_t)k * C + c) * taps + t] : 0.0f;
  }
}
// The per-tap matrices of several filters w[k][c][tap] in one launch (every filter the optimizer has just written: one launch per step
// instead of one per layer): form[tap][k][c], and form_c[tap][c][k] where the data-gradient wants that too (C no multiple of 32).  A CTA takes a tile
// of 32 output channels x 32 input channels x all taps of one filter through shared memory, runs of 32 consecutive floats on both sides.
// 3x3 filters of whole channel blocks move 16 bytes at a time with nine loads of a thread in flight.  Bound by memory (ResNet-50: 45 MB each way);
// 65 us with one load in flight and both forms.  Jobs are laid end to end over the tile index.
struct FormJob { const float* w; float *form, *form_c; int K, C, taps; int begin; };    // begin: first tile of this job
constexpr int kFormJobs = 24;
struct FormJobs { FormJob j[kFormJobs]; int n; int total; };
constexpr int kFormTaps = 9, kFormRow = 32 * kFormTaps;        // filters with more taps go element by element inside their tile
__global__ void __launch_bounds__(256) filter_forms_multi_kernel(const FormJobs J) {
  pdl_enter();
  __shared__ float tile[32][kFormRow + 1];
  int q = 0;
  while (q + 1 < J.n && (int)blockIdx.x >= J.j[q + 1].begin) ++q;
  const FormJob& f = J.j[q];
  const int K = f.K, C = f.C, taps = f.taps;
  const int ctiles = (C + 31) / 32, id = (int)blockIdx.x - f.begin;
  const int k0 = (id / ctiles) * 32, c0 = (id % ctiles) * 32;
  const int kn = min(32, K - k0), cn = min(32, C - c0);
  if (taps == kFormTaps && !f.form_c) {
    float4 v[kFormTaps];
#pragma unroll
    for (int e = 0; e < kFormTaps; ++e) {                      // 32 rows of 72 items over 256 threads
      const int i = threadIdx.x + e * 256, kk = i / (kFormRow / 4), r = i - kk * (kFormRow / 4);
      v[e] = kk < kn ? __ldg(reinterpret_cast<const float4*>(f.w + ((long long)(k0 + kk) * C + c0) * kFormTaps) + r) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int e = 0; e < kFormTaps; ++e) {
      const int i = threadIdx.x + e * 256, kk = i / (kFormRow / 4), r = (i - kk * (kFormRow / 4)) * 4;
      tile[kk][r] = v[e].x; tile[kk][r + 1] = v[e].y; tile[kk][r + 2] = v[e].z; tile[kk][r + 3] = v[e].w;
    }
    __syncthreads();
    const int kk = threadIdx.x >> 3, c = (threadIdx.x & 7) * 4;
    if (kk < kn)
#pragma unroll
      for (int e = 0; e < kFormTaps; ++e) {                    // tap e: 32 rows of 8 items
        const float* t = tile[kk] + c * kFormTaps + e;
        *reinterpret_cast<float4*>(f.form + ((long long)e * K + k0 + kk) * C + c0 + c) = make_float4(t[0], t[kFormTaps], t[2 * kFormTaps], t[3 * kFormTaps]);
      }
    return;
  }
  if (taps > kFormTaps) {
    for (int i = threadIdx.x; i < kn * cn * taps; i += 256) {
      const int t = i % taps, cc = (i / taps) % cn, kk = i / (taps * cn);
      const float v = f.w[((long long)(k0 + kk) * C + c0 + cc) * taps + t];
      f.form[((long long)t * K + k0 + kk) * C + c0 + cc] = v;
      if (f.form_c) f.form_c[((long long)t * C + c0 + cc) * K + k0 + kk] = v;
    }
    return;
  }
  const int run = cn * taps;                                   // floats of one output channel's row inside the tile
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int kk = warp; kk < kn; kk += 8) {                      // a warp per row of the tile: no index arithmetic per element
    const float* src = f.w + ((long long)(k0 + kk) * C + c0) * taps;
    for (int r = lane; r < run; r += 32) tile[kk][r] = src[r];
  }
  __syncthreads();
  // both forms leave as rows of up to 32 consecutive floats, a warp per row: form[t][k][c0 ..] and form_c[t][c][k0 ..]
  for (int row = warp; row < taps * kn; row += 8) {
    const int t = row / kn, kk = row - t * kn;
    if (lane < cn) f.form[((long long)t * K + k0 + kk) * C + c0 + lane] = tile[kk][lane * taps + t];
  }
  if (!f.form_c) return;
  for (int row = warp; row < taps * cn; row += 8) {
    const int t = row / cn, cc = row - t * cn;
    if (lane < kn) f.form_c[((long long)t * C + c0 + cc) * K + k0 + lane] = tile[lane][cc * taps + t];
  }
}
// Filter matrix w[rows][cols] copied with its rows padded by zeros to ld floats (the engine's tensor maps want a row length
// of 4 floats for K-major and 32 floats for N-major operands; 3x3 filters over 3 or 16 channels have 27 or 144).
// A warp per 128 floats of a row: the row number is the only division, and both sides run along the row.
__global__ void __launch_bounds__(256) pad_rows_kernel(const float* __restrict__ w, float* __restrict__ out, int rows, int cols, int ld) {
  pdl_enter();
  const int lane = threadIdx.x & 31, per = (ld + 127) / 128;
  const int64_t items = (int64_t)rows * per;
  for (int64_t i = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); i < items; i += (int64_t)gridDim.x * 8) {
    const int64_t r = i / per; const int c0 = (int)(i - r * per) * 128 + lane;
    const float* src = w + r * cols; float* dst = out + r * ld;
    float v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = c0 + 32 * u < cols ? src[c0 + 32 * u] : 0.0f;
#pragma unroll
    for (int u = 0; u < 4; ++u) if (c0 + 32 * u < ld) dst[c0 + 32 * u] = v[u];
  }
}
// dx[n][c][h][w] += sum over the (r,s) taps that reach (h,w): gather form of unfoldedAcc (TensorDslCPU.scala:647-692).
// One block row per (n, c) plane; the tap loops run over at most R*S entries of the unfolded gradient.
// STRIDE 1 and 2 avoid the per-tap division and remainder (0 = any stride).
template <int STRIDE>
__global__ void fold_acc_kernel(const float* __restrict__ col, float* dx, ConvDims d, int planes_per_block, int threads_per_plane) {
  pdl_enter();
  const int pix = d.oH * d.oW, hw = d.H * d.W;
  const int64_t planes = (int64_t)d.N * d.C;
  const int lane_p = threadIdx.x % threads_per_plane;
  for (int64_t plane = (int64_t)blockIdx.x * planes_per_block + threadIdx.x / threads_per_plane; plane < planes;
       plane += (int64_t)gridDim.x * planes_per_block) {
  const float* src = col + plane * d.R * d.S * pix;          // rows (c*R + r)*S + s of image n start here
  float* dst = dx + plane * hw;
  for (int i = lane_p; i < hw; i += threads_per_plane) {
    const int h = i / d.W, w = i - h * d.W;
    float acc = 0.0f;
    for (int r = 0; r < d.R; ++r) {
      const int hs = h + d.ph - r;
      if (hs < 0) continue;
      int ho;
      if (STRIDE == 1) ho = hs;
      else if (STRIDE == 2) { if (hs & 1) continue; ho = hs >> 1; }
      else { if (hs % d.sh) continue; ho = hs / d.sh; }
      if (ho >= d.oH) continue;
      for (int s = 0; s < d.S; ++s) {
        const int ws = w + d.pw - s;
        if (ws < 0) continue;
        int wo;
        if (STRIDE == 1) wo = ws;
        else if (STRIDE == 2) { if (ws & 1) continue; wo = ws >> 1; }
        else { if (ws % d.sw) continue; wo = ws / d.sw; }
        if (wo >= d.oW) continue;
        acc += src[(r * d.S + s) * pix + ho * d.oW + wo];
      }
    }
    if (acc != 0.0f || STRIDE == 1) dst[i] += acc;
  }
  }
}

// ---- split-K beyond one cluster: the slabs of partial results are summed in a fixed order -----------------------------------
// out[i] (+)= alpha * sum over the slabs of ws[slab][i] (+ bias of i's channel).  A CTA owns 128 consecutive outputs (32
// float4 per warp row); its eight warps each add every eighth slab, in order, and warp 0 adds the eight partial sums, in
// order: the association is fixed, so the result has the same bits on every run (sums combined by atomics do not).  The
// slabs have the layout of the output itself.  chan_div / chan_mod locate the bias entry: channel = (i / chan_div) % chan_mod.
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* __restrict__ ws, int slabs, long long slab, float* out, long long n, float alpha, int accumulate,
                                                            const float* __restrict__ bias, long long chan_div, int chan_mod, int vec) {
  pdl_enter();
  __shared__ float4 partial[8][32];
  const int lane = threadIdx.x & 31, zl = threadIdx.x >> 5;
  const long long base = ((long long)blockIdx.x * 32 + lane) * 4;                  // this lane's four outputs
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  if (base < n) {
    for (int z = zl; z < slabs; z += 8) {
      const float* p = ws + (long long)z * slab + base;
      float4 b;
      if (vec) b = *reinterpret_cast<const float4*>(p);
      else { b.x = p[0]; b.y = base + 1 < n ? p[1] : 0.f; b.z = base + 2 < n ? p[2] : 0.f; b.w = base + 3 < n ? p[3] : 0.f; }
      a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
  }
  partial[zl][lane] = a;
  __syncthreads();
  if (zl != 0 || base >= n) return;
#pragma unroll
  for (int z = 1; z < 8; ++z) { const float4 b = partial[z][lane]; a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
  const float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const long long i = base + e;
    if (i >= n) break;
    const float bv = bias ? bias[(i / chan_div) % chan_mod] : 0.0f;
    out[i] = (accumulate ? out[i] : 0.0f) + alpha * v[e] + bv;
  }
}

// ---- host side ----------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled = nullptr;
typedef CUresult (*EncodeIm2colFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const int*, const int*,
                                   cuuint32_t, cuuint32_t, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeIm2colFn encode_im2col = nullptr;
static int smem_opted_device = -1;                 // the device whose kernels have been given the larger shared memory

static void* driver_entry(const char* name) {
  void* fn = nullptr; cudaDriverEntryPointQueryResult qres;
  cudaError_t e = cudaGetDriverEntryPoint(name, &fn, cudaEnableDefault, &qres);
  return e == cudaSuccess && qres == cudaDriverEntryPointSuccess ? fn : nullptr;
}
static int encode_map(const TcOperand& o, CUtensorMap* out) {
  const TcTensorMap& m = o.map;
  if (!encode_tiled) {
    encode_tiled = (EncodeTiledFn)driver_entry("cuTensorMapEncodeTiled"); encode_im2col = (EncodeIm2colFn)driver_entry("cuTensorMapEncodeIm2col");
    if (!encode_tiled || !encode_im2col) { encode_tiled = nullptr; return fail(LTB_E_CUDA, "the tensor-map encoders are not available from the driver"); }
  }
  cuuint64_t dims[5], strides[4]; cuuint32_t box[5], estr[5];
  for (int d = 0; d < m.rank; ++d) { dims[d] = m.dims[d]; box[d] = m.box[d]; estr[d] = 1; if (d > 0) strides[d - 1] = m.strides[d]; }
  const CUtensorMapSwizzle sw = m.swizzle == TC_SW_128_32B ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B
                                : m.swizzle == TC_SW_128 ? CU_TENSOR_MAP_SWIZZLE_128B : m.swizzle == TC_SW_64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                : m.swizzle == TC_SW_32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE;
  if (o.load == TC_LOAD_IM2COL || o.load == TC_LOAD_IM2COL_MN) {
    const int lower[2] = {o.im.low_w, o.im.low_h}, upper[2] = {o.im.upper_w, o.im.upper_h};
    estr[1] = (cuuint32_t)o.im.step_w; estr[2] = (cuuint32_t)o.im.step_h;
    CUresult r = encode_im2col(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(m.base), dims, strides, lower, upper, 32, (cuuint32_t)o.im.pixels, estr,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(LTB_E_CUDA, "cuTensorMapEncodeIm2col failed with code %d (walk of %d x %d pixels)", (int)r, o.im.grid_w, o.im.grid_h);
    return LTB_OK;
  }
  CUresult r = encode_tiled(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)m.rank, const_cast<void*>(m.base), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(LTB_E_CUDA, "cuTensorMapEncodeTiled failed with code %d (rank %d, inner box %u)", (int)r, m.rank, m.box[0]);
  return LTB_OK;
}

static bool to_dev(const TcOperand& o, TcOperandDev& v) {
  v.n_tile = v.n_k = 0;
  for (int d = 0; d < 5; ++d) {
    v.c_off[d] = o.c_off[d];
    if (o.t_mul[d] != 0) { if (v.n_tile == 3) return false; v.tile[v.n_tile++] = TcTerm{FastDiv(o.t_div[d]), FastDiv(o.t_mod[d]), d, o.t_mul[d]}; }
    if (o.k_mul[d] != 0 && o.k_mod[d] > 1) { if (v.n_k == 3) return false; v.k[v.n_k++] = TcTerm{FastDiv(o.k_div[d]), FastDiv(o.k_mod[d]), d, o.k_mul[d]}; }
  }
  if (!tc_walk_of(o, v.walk)) return false;
  v.n0 = FastDiv(v.walk.n0); v.n1 = FastDiv(v.walk.n1);
  v.rank = o.map.rank; v.nk = o.nk; v.stage_bytes = o.stage_bytes;
  // UMMA layout type: 0 none, 1 128-byte swizzle with 32-byte atoms (M/N-major 32-bit operands), 2 128 B, 4 64 B, 6 32 B
  const uint32_t layout = o.map.swizzle == TC_SW_128_32B ? 1u : o.map.swizzle == TC_SW_128 ? 2u : o.map.swizzle == TC_SW_64 ? 4u : o.map.swizzle == TC_SW_32 ? 6u : 0u;
  v.desc_lo = ((o.lbo >> 4) & 0x3FFFu) << 16;                                     // leading byte offset, bits [16,30)
  v.desc_hi = ((o.sbo >> 4) & 0x3FFFu) | (1u << 14) | (layout << 29);             // stride byte offset [32,46), version 1 at [46,48), layout [61,64)
  for (int i = 0; i < 8; ++i) v.kstep_off[i] = o.kstep_off[i];
  v.load = o.load; v.nbox = o.nbox; v.dim0 = (int)o.map.dims[0]; v.im = o.im;
  return true;
}

static void temp_free(float* p, size_t floats);
static float* temp_alloc(size_t floats);

typedef void (*EngineFn)(const CUtensorMap, const CUtensorMap, const TcParams);
#define LTB_MODES(EPI, GEN, PAIR) tc_gemm_kernel<EPI, 0, GEN, PAIR>, tc_gemm_kernel<EPI, 1, GEN, PAIR>, tc_gemm_kernel<EPI, 2, GEN, PAIR>
static const EngineFn kEngine[2][9] = {                                          // by load modes, epilogue and store mode
    {LTB_MODES(TC_EPI_PIXEL, false, false), LTB_MODES(TC_EPI_ROWMAJOR, false, false), LTB_MODES(TC_EPI_TAPS, false, false)},
    {LTB_MODES(TC_EPI_PIXEL, true, false), LTB_MODES(TC_EPI_ROWMAJOR, true, false), LTB_MODES(TC_EPI_TAPS, true, false)}};
static const EngineFn kEnginePair[2][6] = {{LTB_MODES(TC_EPI_PIXEL, false, true), LTB_MODES(TC_EPI_ROWMAJOR, false, true)},
                                           {LTB_MODES(TC_EPI_PIXEL, true, true), LTB_MODES(TC_EPI_ROWMAJOR, true, true)}};
#undef LTB_MODES
static size_t plan_out_floats(const TcPlan& p) {
  return p.epilogue == TC_EPI_PIXEL ? (size_t)ceil_div(p.M, p.pix_pad ? p.pix_pad : p.pix_per_img ? p.pix_per_img : 1) * (size_t)p.img_stride : (size_t)p.M * (size_t)p.ld;
}
// What a plan's launch wants cleared first: a result that its splits add into.  As a node of its own a clearing costs 2.5 to 3 us of a chain of
// launches and the early start of the launch behind it, 50 times in a step of ResNet-50 at batch 8; beside a kernel that runs anyway
// nothing measurable.
static Clear plan_clear(const TcPlan& p) {
  Clear c;
  if (p.splits > 1 && !g.deterministic && !p.accumulate) { c.p = p.out; c.floats = plan_out_floats(p); }
  return c;
}
ZeroFill take_clear(Clear* c) {
  ZeroFill z;
  if (!c || !c->p || c->done || c->floats % 4 || !aligned16(c->p)) return z;
  c->done = true; z.p = reinterpret_cast<float4*>(c->p); z.n4 = (int64_t)(c->floats / 4);
  return z;
}
static bool overlaps(const void* a, size_t an, const void* b, size_t bn) {      // floats
  return a && b && (const char*)a < (const char*)b + bn * 4 && (const char*)b < (const char*)a + an * 4;
}
int issue_ahead(Clear* clear, float* cl) {
  if (!g.ahead.kind) return LTB_OK;
  Pending p = g.ahead;
  g.ahead.kind = PEND_NONE;
  p.kind = p.inner;
  BnExtra extra;
  extra.cl = cl;
  if (clear && clear->p && clear->floats <= 8 * (size_t)p.n) {       // not what the batch norm itself reads or writes, and in proportion to its grid
    bool apart = true;
    for (const float* q : {p.x, p.a, (const float*)p.y, (const float*)p.out}) apart = apart && !overlaps(q, (size_t)p.n, clear->p, clear->floats);
    for (const float* q : {p.gamma, p.beta, (const float*)p.run_mean, (const float*)p.run_var, (const float*)p.save_mean, (const float*)p.save_istd})
      apart = apart && !overlaps(q, (size_t)p.C, clear->p, clear->floats);
    if (apart) extra.zero = take_clear(clear);
  }
  return bn_fwd_issue(p, true, extra);
}
// *relu: the caller wants max(0, result); false on return when the kernel has done it, still true when splits meet outside it.
// clear: plan_clear of this plan, if a kernel before this one was to do it.
static int launch_plan(const TcPlan& p, const char* label, bool* relu = nullptr, Clear clear = Clear()) {
  if (!clear.p) clear = plan_clear(p);
  { int rc = issue_ahead(&clear); if (rc) return rc; }
  CUtensorMap ma, mb;
  int rc = encode_map(p.a, &ma); if (rc) return rc;
  rc = encode_map(p.b, &mb); if (rc) return rc;
  TcParams P;
  if (!to_dev(p.a, P.a) || !to_dev(p.b, P.b)) return fail(LTB_E_STATE, "tensor-core plan whose k-iteration order has no incremental walk");
  P.M = p.M; P.N = p.N; P.bn = p.bn; P.k_iters = p.k_iters;
  // Split-K: up to eight splits of a tile form a thread-block cluster and add their partial tiles up inside the kernel
  // (through distributed shared memory, in a fixed order).  More than eight splits (four, of pairs): every cluster writes a slab of
  // partial results (a staging block with the layout of the output) and one more launch adds the slabs up, again in a fixed
  // order, and applies alpha, bias and accumulation.  No atomics, no zero fill, the same bits on every run.
  // That is the deterministic mode (ltb_set_deterministic): measured, it costs the contraction kernels about a third more
  // time (cluster barriers, partial tiles through shared memory).  By default the splits add their tiles into the output
  // atomically, as cuDNN's default algorithms do: faster, and the last bits of a sum depend on the order of arrival.
  int splits = p.splits < 1 ? 1 : p.splits, cz = 1, nslabs = 1;
  const bool atomic = splits > 1 && !g.deterministic;
  if (splits > 1 && !atomic) {
    cz = splits <= 2 ? 2 : splits <= 4 || p.pair ? 4 : 8;                           // (four pairs)
    nslabs = (int)ceil_div(splits, cz);
  }
  const size_t out_floats = plan_out_floats(p);
  float* ws = nullptr;
  if (nslabs > 1) {
    ws = temp_alloc((size_t)nslabs * out_floats);
    if (!ws) nslabs = 1;                                                           // no room for the slabs: one cluster per tile
  }
  if (!atomic) splits = nslabs * cz;
  P.k_per_split = (int)ceil_div(p.k_iters, splits);                                // a split may end up without iterations: it contributes zeros
  if (atomic) splits = (int)ceil_div(p.k_iters, P.k_per_split);                    // atomic mode: only splits that have work
  P.cluster_z = cz;
  P.epilogue = p.epilogue; P.accumulate = ws ? 0 : p.accumulate; P.atomic = atomic ? 1 : 0;
  if (atomic && !p.accumulate && !clear.done) LTB_CUDA(cudaMemsetAsync(p.out, 0, out_floats * 4, g.stream));     // overwrite semantics: start from zero, then add
  // tf32 x tf32 -> f32: D format 1 at [4,6), A/B format 2 at [7,10)/[10,13), major bits 15/16, N>>3 at [17,23), M>>4 at [24,29)
  P.idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)p.a.mn_major << 15) | ((uint32_t)p.b.mn_major << 16) | ((uint32_t)(p.bn >> 3) << 17) | ((uint32_t)(p.pair ? 256 : 128) >> 4 << 24);
  P.out = ws ? ws : p.out; P.bias = ws ? nullptr : p.bias; P.alpha = ws ? 1.0f : p.alpha; P.split_stride = ws ? (long long)out_floats : 0;
  P.pix_per_img = p.pix_per_img ? p.pix_per_img : 1; P.by_pix = FastDiv((int)(p.pix_pad ? p.pix_pad : P.pix_per_img));
  P.img_stride = p.img_stride; P.chan_stride = p.chan_stride; P.ld = p.ld; P.col_mod = p.col_mod; P.col_mul = p.col_mul;
  P.gather_src = p.gather_src; P.g_pix = p.g_pix; P.g_chan = p.g_chan; P.g_imgs = p.g_imgs;
  P.relu = relu && *relu && !atomic && !ws ? 1 : 0;
  if (P.relu) *relu = false;
  P.status = g.dev_status; P.wait_cycles = g.wait_limit_cycles;
  // 4 stages, except 3 for 128-wide tiles so that two CTAs (2 x 97 KB) share an SM and one's epilogue overlaps the other's main loop
  // (256-wide tiles: four stages of 48 KB, one CTA per SM; six of 32 KB in a pair).
  P.stages = p.pair ? kMaxStages : p.bn == 128 ? 3 : 4;
  const size_t smem = (size_t)P.stages * (p.a.stage_bytes + p.b.stage_bytes) + 1024;
  if (cz > 1 && (size_t)128 * (p.bn + 1) * 4 > smem - 1024) return fail(LTB_E_STATE, "tensor-core plan whose partial tile does not fit the pipeline stages");
  if (smem_opted_device != g.device) {
    const int max_smem = 4 * (16384 + 32768) + 1024;                              // as much as six of 32 KB
    for (auto& set : kEngine) for (auto k : set) LTB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    for (auto& set : kEnginePair) for (auto k : set) LTB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    smem_opted_device = g.device;
  }
  const int mode = atomic ? 2 : (P.accumulate ? 1 : 0);
  const bool gen = p.a.load != TC_LOAD_BOX || p.b.load != TC_LOAD_BOX;
  const EngineFn kernel = p.pair ? kEnginePair[gen][p.epilogue * 3 + mode] : kEngine[gen][p.epilogue * 3 + mode];
  {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.pair ? (p.m_tiles + 1) / 2 * 2 : p.m_tiles, p.n_tiles, splits); cfg.blockDim = dim3(kTcThreads); cfg.dynamicSmemBytes = smem; cfg.stream = g.stream;
    cudaLaunchAttribute attr[2];
    pdl_attribute(attr[1]);
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.pair ? 2 : 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = (unsigned)cz;
    cfg.attrs = attr; cfg.numAttrs = g.profiling ? 1 : 2;
    if (g.profiling) profile_before(label);
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, ma, mb, P);
    if (g.profiling) profile_after();
    ++g.launches;
    if (e != cudaSuccess) return fail(LTB_E_CUDA, "launch of the tensor-core engine failed: %s (grid %d x %d x %d, cluster %d)", cudaGetErrorString(e), p.m_tiles, p.n_tiles, splits, cz);
  }
  if (ws) {
    const bool pixel = p.epilogue == TC_EPI_PIXEL;
    const long long chan_div = pixel ? (long long)(p.pix_per_img ? p.pix_per_img : 1) : 1;
    const int chan_mod = pixel ? p.N : (int)(p.ld > 0 ? p.ld : 1);
    const int vec = aligned16(ws) && out_floats % 4 == 0 ? 1 : 0;
    const unsigned grid_r = (unsigned)ceil_div((int64_t)out_floats, 128);
    LTB_LAUNCH(splitk_reduce_kernel, grid_r, 256, 0, (const float*)ws, nslabs, (long long)out_floats, p.out, (long long)out_floats, p.alpha, p.accumulate, p.bias, chan_div, chan_mod, vec);
    temp_free(ws, (size_t)nslabs * out_floats);
  }
  return LTB_OK;
}

// Self-test of the bounded wait: one warp waits, through the engine's own mbar_wait, on a barrier at which nothing ever
// arrives.  No copy is in flight and no tensor memory is held, so when the limit runs out the kernel simply records code 9
// in the status word and returns; the context stays usable.
__global__ void wait_selftest_kernel(int* status, long long limit) {
  pdl_enter();
  __shared__ __align__(8) uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) { mbar_init(&bar, 1); abort_flag = 0; asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
  __syncthreads();
  if (threadIdx.x == 0) mbar_wait(&bar, 0, &abort_flag, status, 9, limit);
  __syncthreads();
}

}  // namespace ltb
extern "C" {
int ltb_set_wait_limit(int64_t cycles) {
  LTB_INITED(); LTB_REQUIRE(cycles > 0, "ltb_set_wait_limit: the limit must be positive");
  ltb::g.wait_limit_cycles = cycles; return LTB_OK;
}
int ltb_selftest_bounded_wait(int64_t cycles) {
  LTB_INITED(); LTB_REQUIRE(cycles > 0 && cycles <= 4000000000ll, "ltb_selftest_bounded_wait: limit out of range (1 .. 4e9 cycles)");
  LTB_LAUNCH(ltb::wait_selftest_kernel, 1, 32, 0, ltb::g.dev_status, (long long)cycles);
  return LTB_OK;
}
}
namespace ltb {

// ---- channels-last copies of activations ---------------------------------------------------------------------------------------
// The tap-loop convolutions read act[n][h][w][c].  Without the operand cache (ltb_set_filter_cache) every call makes its own
// copy in a staging block and gives it back.  With it, a copy made by a forward convolution, or of dy at the start of a
// convolution's backward call, is kept in a block taken from the far end of the arena (those blocks live until ltb_reset)
// and found again by address and shape: the weight-gradient of that convolution reads the forward copy of x, and data-grad
// and weight-grad share one copy of dy.  Only backward looks a copy up, dy's within its own call: a forward call makes its copy in any
// case, and so does a backward call for dy, because the caller may have written the buffer by its own means.  A copy is dropped when
// any entry point writes its source (LTB_WRITES), when ltb_free releases the source, where a recording begins or ends, and at ltb_reset.
struct ClCopy { const float* src; size_t src_floats; int n_img, chan, pix; float* cl; int geom; };   // geom 0: channels-last copy; else the key of an unfolded matrix (unfold_key)
static std::vector<ClCopy> cl_cache;
void cl_cache_clear() { cl_cache.clear(); }
void cl_cache_drop_from(const void* p) {                   // ltb_free: everything at or above p is gone
  for (size_t i = 0; i < cl_cache.size();) { if (in_arena_from(cl_cache[i].src, p)) { cl_cache[i] = cl_cache.back(); cl_cache.pop_back(); } else ++i; }
}
static void cl_cache_drop(const void* p, size_t bytes) {       // every copy whose source overlaps [p, p + bytes); p null: all
  for (size_t i = 0; i < cl_cache.size();) {
    const char* sl = (const char*)cl_cache[i].src; const char* sh = sl + cl_cache[i].src_floats * 4;
    if (!p || ((const char*)p < sh && sl < (const char*)p + bytes)) { cl_cache[i] = cl_cache.back(); cl_cache.pop_back(); } else ++i;
  }
}
// A block for a new copy of src that is to be kept (null: no room): the block of the copy it replaces where that has the same shape, so
// that calls on the same buffers without an ltb_reset between do not use the arena up.  Every reader of the old copy runs before on
// the same stream or has been waited for; not so in a branch region, whose two streams may read one source.
static float* kept_block(const float* src, size_t src_floats, int n_img, int chan, int pix, int geom, size_t floats) {
  for (size_t i = 0; i < cl_cache.size(); ++i) {
    ClCopy& e = cl_cache[i];
    if (e.src != src || e.geom != geom) continue;
    if (e.n_img == n_img && e.chan == chan && e.pix == pix && !g.branch_marked) return e.cl;
    e = cl_cache.back(); cl_cache.pop_back();
    break;
  }
  float* p = (float*)step_alloc(floats * 4);
  if (p) cl_cache.push_back(ClCopy{src, src_floats, n_img, chan, pix, p, geom});
  return p;
}
static float* cl_lookup(const float* src, int n_img, int chan, int pix) {
  for (auto& e : cl_cache) if (e.src == src && e.n_img == n_img && e.chan == chan && e.pix == pix && e.geom == 0) return e.cl;
  return nullptr;
}
// The unfolded matrix col[n][(c, r, s)][p] of a convolution input (the forward pass of a strided or 3-channel convolution
// makes it, the weight gradient of the same convolution reads it again): kept and found like the channels-last copies.
static int unfold_key(const ConvDims& d) { return 1 + ((((((d.R * 8 + d.S) * 4 + d.sh) * 4 + d.sw) * 8 + d.ph) * 8 + d.pw) * 64 + d.W % 64); }
static float* unfold_lookup(const float* src, const ConvDims& d) {
  const int ck = d.C * d.R * d.S, pix = d.oH * d.oW, key = unfold_key(d);
  for (auto& e : cl_cache) if (e.src == src && e.n_img == d.N && e.chan == ck && e.pix == pix && e.geom == key) return e.cl;
  return nullptr;
}
static int launch_unfold(const float* x, float* col, const ConvDims& d, Clear* clear = nullptr) {
  { int rc = issue_ahead(clear); if (rc) return rc; }
  const ZeroFill zero = clear && !overlaps(clear->p, clear->floats, x, (size_t)d.N * d.C * d.H * d.W) ? take_clear(clear) : ZeroFill();
  const int pix = d.oH * d.oW;
  int tpp = 4; while (tpp < pix && tpp < 256) tpp <<= 1;       // threads per input plane: a power of two in [4, 256] (4 x 4 and 2 x 2 outputs leave no lane idle)
  const int ppb = 256 / tpp;
  const int64_t planes = (int64_t)d.N * d.C;
  LTB_LAUNCH(unfold_rows_kernel, grid_for(ceil_div(planes, ppb) * 256, 256, 16), 256, 0, x, col, d, ppb, tpp, zero);
  return LTB_OK;
}
// 1x1 convolution with stride 2 and no padding (ResNet's downsampling branch): every gradient element goes to exactly
// one input pixel, dx[n][c][2a][2b] += col[n][c][a][b]; a thread per element of col.
__global__ void fold_1x1_s2_kernel(const float* __restrict__ col, float* dx, int oH, int oW, int H, int W, int64_t total) {
  pdl_enter();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int b = (int)(i % oW); const int64_t t = i / oW; const int a = (int)(t % oH); const int64_t plane = t / oH;
    dx[(plane * H + 2 * a) * W + 2 * b] += col[i];
  }
}
static int launch_fold(const float* col, float* dx, const ConvDims& d) {
  const int hw = d.H * d.W;
  int tpp = 32; while (tpp < hw && tpp < 256) tpp <<= 1;
  const int ppb = 256 / tpp;
  const int64_t planes = (int64_t)d.N * d.C;
  const unsigned grid = (unsigned)grid_for(ceil_div(planes, ppb) * 256, 256, 16);
  if (d.R == 1 && d.S == 1 && d.sh == 2 && d.sw == 2 && d.ph == 0 && d.pw == 0) {
    const int64_t total = planes * d.oH * d.oW;
    LTB_LAUNCH(fold_1x1_s2_kernel, grid_for(total, 256), 256, 0, col, dx, d.oH, d.oW, d.H, d.W, total);
    return LTB_OK;
  }
  if (d.sh == 1 && d.sw == 1) LTB_LAUNCH(fold_acc_kernel<1>, grid, 256, 0, col, dx, d, ppb, tpp);
  else if (d.sh == 2 && d.sw == 2) LTB_LAUNCH(fold_acc_kernel<2>, grid, 256, 0, col, dx, d, ppb, tpp);
  else LTB_LAUNCH(fold_acc_kernel<0>, grid, 256, 0, col, dx, d, ppb, tpp);
  return LTB_OK;
}
static bool is_pointwise(const ConvDims& d) { return d.R == 1 && d.S == 1 && d.sh == 1 && d.sw == 1 && d.ph == 0 && d.pw == 0; }
// Staging blocks go back to the arena (a LIFO pop, host arithmetic only) unless the caller holds them: conv backward runs
// its two halves on two streams and pops both halves' blocks together once both are issued.
// Nor inside a branch region (ltb_branch_mark .. ltb_branch_join): the other stream's next call would reuse the block.
static void temp_free(float* p, size_t floats) { if (!g.hold_workspace && !g.branch_marked && !g.side_open) ltb_free(p, floats * 4); }
static float* temp_alloc(size_t floats) {
  size_t bytes = (floats * 4 + kGranule - 1) / kGranule * kGranule;
  if (g.used + bytes + g.top_used > g.heap_bytes) return nullptr;   // no room for the staging buffer: let the FP32 path run
  return (float*)arena_alloc(floats * 4, false);
}
// The unfolded form col[n][(c, r, s)][p] of a convolution input for the forward pass: kept for the weight gradient of the same
// convolution when the operand cache is on, else a staging block of *floats floats to give back (*floats == 0: kept).  *col stays
// null when there is no room.
static int unfolded(const float* x, const ConvDims& d, const float** col, float** temp, size_t* floats, Clear* clear) {
  const int ck = d.C * d.R * d.S, pix = d.oH * d.oW;
  const size_t n = (size_t)d.N * ck * pix;
  *temp = nullptr; *floats = 0; *col = nullptr;
  if (g.filter_cache && !(g.tune & 4)) {
    if (float* kept = kept_block(x, (size_t)d.N * d.C * d.H * d.W, d.N, ck, pix, unfold_key(d), n)) {
      *col = kept;
      int rc = launch_unfold(x, kept, d, clear); if (rc) cl_cache_drop(x, 1);
      return rc;
    }
  }
  float* buf = temp_alloc(n);
  if (!buf) return LTB_OK;
  *temp = buf; *floats = n; *col = buf;
  return launch_unfold(x, buf, d, clear);
}

// ---- tap-loop (implicit) path for R x S convolutions with stride 1 ---------------------------------------------------------
static bool taps_geometry(const ConvDims& d, TcConvGeom& gm) {
  if (d.R * d.S == 1 || d.sh != 1 || d.sw != 1) return false;
  gm.n_img = d.N; gm.C = d.C; gm.H = d.H; gm.W = d.W; gm.K = d.K; gm.R = d.R; gm.S = d.S; gm.ph = d.ph; gm.pw = d.pw; gm.oH = d.oH; gm.oW = d.oW;
  return true;
}
static int up4(int v) { return (v + 3) / 4 * 4; }
static int channels_last_into(const float* src, int n_img, int chan, int pix, float* out, Clear* clear) {
  const int ld = up4(chan);
  if (g.ahead.kind && g.ahead.N == n_img && g.ahead.C == chan && g.ahead.HW == pix && bn_fwd_writes_copy(g.ahead)) return issue_ahead(clear, out);      // (g.ahead makes src)
  { int rc = issue_ahead(clear); if (rc) return rc; }
  ZeroFill zero = clear && !overlaps(clear->p, clear->floats, src, (size_t)n_img * chan * pix) ? take_clear(clear) : ZeroFill();
  if (chan % 32 == 0 && pix < 32 && n_img <= 65535) {
    LTB_LAUNCH(to_rows_tiled_kernel, dim3(1, chan / 32, n_img), 32 * pix < 256 ? 128 : 256, 0, src, out, chan, pix, zero);
    return LTB_OK;
  }
  for (int n0 = 0; n0 < n_img; n0 += 65535) {                       // gridDim.z holds at most 65535 images
    const int nn = n_img - n0 < 65535 ? n_img - n0 : 65535;
    LTB_LAUNCH(channels_last_kernel, dim3((unsigned)ceil_div(pix, 64), (unsigned)ceil_div(ld, 32), (unsigned)nn), 256, 0, src + (size_t)n0 * chan * pix, out + (size_t)n0 * pix * ld, chan, pix, ld, zero);
    zero = ZeroFill();
  }
  return LTB_OK;
}
// Channels-last copy [N][pix][ld] of a tensor [N][chan][pix], ld = chan rounded up to 4 (zeros beyond chan: the tensor maps want
// rows of a multiple of 16 bytes).  keep: put it where it outlives the call and remember it (when the cache is on and the arena has
// room); otherwise a staging block of *floats floats to give back (*floats == 0: kept).  *out stays null when there is no room at all.
static int channels_last(const float* src, int n_img, int chan, int pix, float** out, size_t* floats, bool keep = false, Clear* clear = nullptr) {
  const size_t n = (size_t)n_img * up4(chan) * pix;
  *floats = 0; *out = nullptr;
  if (keep && g.filter_cache && !(g.tune & 4)) {
    if (float* kept = kept_block(src, (size_t)n_img * chan * pix, n_img, chan, pix, 0, n)) {
      *out = kept;
      int rc = channels_last_into(src, n_img, chan, pix, kept, clear); if (rc) cl_cache_drop(src, 1);
      return rc;
    }
  }
  *out = temp_alloc(n); *floats = n;
  if (!*out) return LTB_OK;
  return channels_last_into(src, n_img, chan, pix, *out, clear);
}
// ---- filter cache (ltb_set_filter_cache) ------------------------------------------------------------------------------------
// The per-tap forms of a filter are needed twice per step (forward and data-grad) and change once per step (the optimizer).
// With the cache on they live in private device memory, keyed by the filter's address and shape, and are refreshed -- all
// stale filters together, in ONE launch -- at the first use after a write that overlaps a filter (LTB_WRITES in every entry point that
// writes; a replayed step and ltb_params_changed mark every filter).  A filter first seen while a step is being recorded takes
// the uncached path (no allocation inside a capture).
struct FilterForms { const float* w; int K, C, taps; float *form, *form_c; bool stale, gone; };
static std::vector<FilterForms> filter_cache;
static size_t filter_cache_bytes = 0;
void filter_cache_clear() {
  for (auto& e : filter_cache) { cudaFree(e.form); cudaFree(e.form_c); }
  filter_cache.clear(); filter_cache_bytes = 0;
}
// ltb_reset / ltb_free: filters at or above p exist no more and are not refreshed with the next program's.  Their blocks stay (a
// recorded step may name them) until a filter of that address and shape comes again or the cache is cleared.
void filter_cache_drop_from(const void* p) { for (auto& e : filter_cache) if (in_arena_from(e.w, p)) { e.gone = true; e.stale = true; } }
void filter_cache_note_write(const void* p, size_t bytes) {
  cl_cache_drop(p, bytes);
  if (filter_cache.empty()) return;
  const char* lo = (const char*)p; const char* hi = lo + bytes;
  for (auto& e : filter_cache) {
    const char* wl = (const char*)e.w; const char* wh = wl + (size_t)e.K * e.C * e.taps * 4;
    if (!p || (lo < wh && wl < hi)) e.stale = true;
  }
}
static FilterForms* filter_cache_entry(const float* w, const ConvDims& d) {
  const int taps = d.R * d.S;
  for (auto& e : filter_cache) if (e.w == w && e.K == d.K && e.C == d.C && e.taps == taps) { e.gone = false; return &e; }
  if (g.capturing) return nullptr;
  const size_t bytes = (size_t)d.K * d.C * taps * 4;
  if (filter_cache_bytes + 2 * bytes > ((size_t)2 << 30)) { cudaStreamSynchronize(g.stream); cudaStreamSynchronize(g.side); cudaStreamSynchronize(g.branch); filter_cache_clear(); }
  FilterForms e{w, d.K, d.C, taps, nullptr, nullptr, true, false};
  if (cudaMalloc((void**)&e.form, bytes) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  if (d.C % 32 && cudaMalloc((void**)&e.form_c, bytes) != cudaSuccess) { cudaGetLastError(); cudaFree(e.form); return nullptr; }
  filter_cache_bytes += d.C % 32 ? 2 * bytes : bytes;
  filter_cache.push_back(e);
  return &filter_cache.back();
}
// The per-tap matrices of w: out[tap][k][c], rows padded to 4 floats, for forward and, of a filter whose C is a multiple of 32, data-gradient;
// or out[tap][c][k] for the data-gradient of any other.  *floats is the size of the staging block to give back afterwards, 0 when the matrices live in the cache.
static int tap_matrices(const float* w, const ConvDims& d, bool dgrad, float** out, size_t* floats) {
  const int by_c = dgrad && d.C % 32 != 0;
  const int ld = up4(by_c ? d.K : d.C);
  const size_t n = (size_t)(by_c ? d.C : d.K) * ld * d.R * d.S;
  if (!by_c && d.R * d.S == 1 && ld == d.C && aligned16(w)) { *out = const_cast<float*>(w); *floats = 0; return LTB_OK; }   // one tap: the filter is that matrix
  // Only filters in the arena are kept: a refresh reads every filter it knows, and memory of the caller's own may be gone by then,
  // or be another filter written by other means.
  const bool in_arena = (const char*)w >= g.heap && (const char*)w < g.heap + g.heap_bytes;
  if (g.filter_cache && in_arena && d.R * d.S > 1 && d.C % 4 == 0 && d.K % 4 == 0 && aligned16(w)) {
    if (FilterForms* e = filter_cache_entry(w, d)) {
      if (e->stale) {
        // every stale filter at once: after an optimizer step all of them are, and their values are final until the next write
        // (which marks them again), so the forms of the layers still to come are made here too
        FormJobs jobs; jobs.n = 0; jobs.total = 0;
        auto flush = [&]() -> int {
          if (jobs.n == 0) return LTB_OK;
          LTB_LAUNCH(filter_forms_multi_kernel, (unsigned)jobs.total, 256, 0, jobs);
          jobs.n = 0; jobs.total = 0;
          return LTB_OK;
        };
        for (auto& o : filter_cache) {
          if (!o.stale || o.gone) continue;
          if (jobs.n == kFormJobs) { int rc = flush(); if (rc) return rc; }
          jobs.j[jobs.n++] = FormJob{o.w, o.form, o.form_c, o.K, o.C, o.taps, jobs.total};
          jobs.total += (int)(ceil_div(o.K, 32) * ceil_div(o.C, 32));
          o.stale = false;
        }
        int rc = flush(); if (rc) return rc;
      }
      *out = by_c ? e->form_c : e->form; *floats = 0;
      return LTB_OK;
    }
  }
  *out = temp_alloc(n); *floats = n;
  if (!*out) return LTB_OK;
  LTB_LAUNCH(permute_taps_kernel, grid_for((int64_t)n, 256), 256, 0, w, *out, d.K, d.C, d.R * d.S, by_c, ld, (int64_t)n);
  return LTB_OK;
}
// w[rows][cols] with rows of ld floats, 16-byte aligned: the tensor itself when it is that already, else a zero-padded copy in a staging block
// (*out stays null when the arena has no room for it).
static int padded_filter(const float* w, int rows, int cols, int ld, const float** out, float** temp, size_t* floats) {
  *temp = nullptr; *floats = 0; *out = w;
  if (ld == cols && aligned16(w)) return LTB_OK;
  const size_t n = (size_t)rows * ld;
  float* buf = temp_alloc(n);
  *out = buf;
  if (!buf) return LTB_OK;
  *temp = buf; *floats = n;
  LTB_LAUNCH(pad_rows_kernel, grid_for((int64_t)rows * ceil_div(ld, 128) * 32, 256), 256, 0, w, buf, rows, cols, ld);
  return LTB_OK;
}
int gemm_tc(const float* a, bool a_kmajor, const float* b, bool b_kmajor, float* c, bool, int M, int N, int K, float alpha, bool accumulate) {
  TcPlan p;
  if (tc_plan_gemm(p, a, a_kmajor, b, b_kmajor, c, M, N, K, alpha, accumulate, g.sm_count)) {
    int rc = launch_plan(p, "tc_gemm_kernel[gemm]");
    return rc ? rc : 1;
  }
  // A large product whose rows the tensor maps cannot address (a length or a start that is no multiple of 16 bytes), or with one
  // extent below half a tile: worth a padded copy of the operands that need one.  Below about 0.2 GFLOP the CUDA-core kernels take as
  // long as the copy and the engine's launch together.
  if (2.0 * M * N * K < 2e8 || M < 16 || N < 16 || K < 32) return 0;
  const int ca = a_kmajor ? K : M, cb = b_kmajor ? K : N;                        // row lengths of the operands as they are stored
  const int lda = up4(ca), ldb = up4(cb);
  const float *ap, *bp; float *at, *bt; size_t an, bn;
  int rc = padded_filter(a, a_kmajor ? M : K, ca, lda, &ap, &at, &an); if (rc) return rc;
  if (!ap) return 0;
  rc = padded_filter(b, b_kmajor ? N : K, cb, ldb, &bp, &bt, &bn);
  const bool ok = !rc && bp && tc_plan_gemm_ld(p, ap, a_kmajor, lda, bp, b_kmajor, ldb, c, M, N, K, alpha, accumulate, g.sm_count);
  if (ok) rc = launch_plan(p, "tc_gemm_kernel[gemm padded]");
  if (bt) temp_free(bt, bn);
  if (at) temp_free(at, an);
  return rc ? rc : (ok ? 1 : 0);
}

// Each returns 1 when it took the problem, 0 when not eligible (the unfolding path then runs), negative on error.
static int conv_fwd_taps(const float* x, const float* w, const float* bias, float* y, const ConvDims& d, bool* relu) {
  TcConvGeom gm; TcPlan p;
  if (!taps_geometry(d, gm) || !tc_plan_conv_taps_fwd(p, y, y, bias, y, gm, g.sm_count)) return 0;     // eligibility with any aligned pointers
  float *xr = nullptr, *wt = nullptr; size_t nx = 0, nw = 0;
  Clear clear = plan_clear(p);
  int rc = channels_last(x, d.N, d.C, d.H * d.W, &xr, &nx, /*keep=*/true, &clear); if (rc) return rc;     // the weight-gradient of this convolution reads it again
  if (!xr) return 0;
  rc = tap_matrices(w, d, false, &wt, &nw);
  bool ok = !rc && wt && tc_plan_conv_taps_fwd(p, xr, wt, bias, y, gm, g.sm_count);
  if (ok) rc = launch_plan(p, "tc_gemm_kernel[conv_fwd taps]", relu, clear);
  if (wt && nw) temp_free(wt, nw);
  if (nx) temp_free(xr, nx);
  return rc ? rc : (ok ? 1 : 0);
}
static int conv_dgrad_taps(const float* dy, const float* w, float* dx, const ConvDims& d, bool accumulate) {
  TcConvGeom gm; TcPlan p;
  if (!taps_geometry(d, gm) || !tc_plan_conv_taps_dgrad(p, dx, dx, dx, gm, true, g.sm_count)) return 0;
  float *dyr = cl_lookup(dy, d.N, d.K, d.oH * d.oW), *wd = nullptr; size_t ny = 0, nw = 0;
  int rc = dyr ? LTB_OK : channels_last(dy, d.N, d.K, d.oH * d.oW, &dyr, &ny); if (rc) return rc;
  if (!dyr) return 0;
  rc = tap_matrices(w, d, true, &wd, &nw);
  bool ok = !rc && wd && tc_plan_conv_taps_dgrad(p, dyr, wd, dx, gm, accumulate, g.sm_count);
  if (ok) rc = launch_plan(p, "tc_gemm_kernel[conv_dgrad taps]");
  if (wd && nw) temp_free(wd, nw);
  if (ny) temp_free(dyr, ny);
  return rc ? rc : (ok ? 1 : 0);
}

// ---- any image size, stride and channel count: the TMA unit's im2col mode ----------------------------------------------------
// The tap loop above needs output rows that fill a tile of 128 pixels exactly (widths that divide 128) and channels in whole blocks
// of 32.  In im2col mode the TMA unit walks the output pixels itself, image after image, at any stride, so a tile is any 128
// consecutive output pixels and nothing is unfolded or folded back: per call one channels-last copy of the activation (shared with
// the other passes when the operand cache is on) and the contraction.  Before, such a convolution was unfolded into a matrix R x S
// times the size of its input element by element (56 x 56, 64 -> 64, 3x3, batch 32: forward 476 us, with this path 67 us; the layer's
// whole training pass 920 -> 310 us, 215 with what followed).
// A filter of fewer than 32 elements per output channel fills less than one k-iteration and stays with the other paths, and so do
// forward and data-gradient of such images when their rows would need padding (below): those have always been computed in FP32.
static bool any_geometry(const ConvDims& d, TcConvAny& a) {
  if (d.C * d.R * d.S < 32) return false;
  a.n_img = d.N; a.C = d.C; a.H = d.H; a.W = d.W; a.K = d.K; a.R = d.R; a.S = d.S; a.sh = d.sh; a.sw = d.sw; a.ph = d.ph; a.pw = d.pw;
  a.oH = d.oH; a.oW = d.oW; a.ldc = up4(d.C); a.ldk = up4(d.K);
  return true;
}
static int conv_fwd_any(const float* x, const float* w, const float* bias, float* y, const ConvDims& d, bool* relu) {
  TcConvAny a; TcPlan p;
  if (tc_conv_needs_rows(d.oH * d.oW) && d.C * d.R * d.S % 4) return 0;
  if (!any_geometry(d, a) || !tc_plan_conv_any_fwd(p, (const float*)g.heap, (const float*)g.heap, bias, y, a, g.sm_count)) return 0;     // eligibility with any aligned pointers
  float *xr = nullptr, *wt = nullptr; size_t nx = 0, nw = 0;
  Clear clear = plan_clear(p);
  int rc = channels_last(x, d.N, d.C, d.H * d.W, &xr, &nx, /*keep=*/true, &clear); if (rc) return rc;
  if (!xr) return 0;
  rc = tap_matrices(w, d, false, &wt, &nw);
  bool ok = !rc && wt && tc_plan_conv_any_fwd(p, xr, wt, bias, y, a, g.sm_count);
  if (ok) rc = launch_plan(p, "tc_gemm_kernel[conv_fwd im2col]", relu, clear);
  if (wt && nw) temp_free(wt, nw);
  if (nx) temp_free(xr, nx);
  return rc ? rc : (ok ? 1 : 0);
}
// A stride is taken out by zeros between the pixels of dy (channels_last_up_kernel): dx is then a stride-1 data-gradient.
static int conv_dgrad_any(const float* dy, const float* w, float* dx, const ConvDims& d, bool accumulate) {
  TcConvAny a; TcPlan p; TcConvGeom gm;
  if (!any_geometry(d, a) || d.N > 65535 || (tc_conv_needs_rows(d.oH * d.oW) && d.K % 4)) return 0;
  const bool strided = d.sh != 1 || d.sw != 1;
  if (strided) {
    a.sh = a.sw = 1; a.oH = d.H + 2 * d.ph - d.R + 1; a.oW = d.W + 2 * d.pw - d.S + 1;              // the stride-1 output grid
    if (a.oH < 1 || a.oW < 1) return 0;
  }
  gm.n_img = d.N; gm.C = d.C; gm.H = d.H; gm.W = d.W; gm.K = d.K; gm.R = d.R; gm.S = d.S; gm.ph = d.ph; gm.pw = d.pw; gm.oH = a.oH; gm.oW = a.oW;
  const float* any = (const float*)g.heap;
  const bool window = tc_plan_conv_taps_dgrad(p, any, any, dx, gm, accumulate, g.sm_count);
  if (!window && !tc_plan_conv_any_dgrad(p, any, any, dx, a, accumulate, g.sm_count)) return 0;
  Clear clear = plan_clear(p);
  float *dyr = strided ? nullptr : cl_lookup(dy, d.N, d.K, d.oH * d.oW), *wd = nullptr; size_t ny = 0, nw = 0;
  int rc = LTB_OK;
  if (strided) {
    ny = (size_t)d.N * a.oH * a.oW * a.ldk;
    if (!(dyr = temp_alloc(ny))) return 0;
    const ZeroFill zero = overlaps(clear.p, clear.floats, dy, (size_t)d.N * d.K * d.oH * d.oW) ? ZeroFill() : take_clear(&clear);
    LTB_LAUNCH(channels_last_up_kernel, dim3((unsigned)ceil_div(a.oH, d.sh), (unsigned)ceil_div(a.ldk, 32), (unsigned)d.N), 256, 0, dy, dyr, d.K, a.ldk, d.oH, d.oW, a.oH, a.oW, d.sh, d.sw, zero);
  } else if (!dyr) rc = channels_last(dy, d.N, d.K, d.oH * d.oW, &dyr, &ny, false, &clear);
  if (rc) return rc;
  if (!dyr) return 0;
  rc = tap_matrices(w, d, true, &wd, &nw);
  bool ok = !rc && wd && (window ? tc_plan_conv_taps_dgrad(p, dyr, wd, dx, gm, accumulate, g.sm_count) : tc_plan_conv_any_dgrad(p, dyr, wd, dx, a, accumulate, g.sm_count));
  if (ok) rc = launch_plan(p, window ? "tc_gemm_kernel[conv_dgrad taps up]" : "tc_gemm_kernel[conv_dgrad im2col]", nullptr, clear);
  if (wd && nw) temp_free(wd, nw);
  if (ny) temp_free(dyr, ny);
  return rc ? rc : (ok ? 1 : 0);
}
static int conv_wgrad_any(const float* x, const float* dy, float* dw, const ConvDims& d) {
  TcConvAny a; TcPlan p;
  const float* any = (const float*)g.heap;
  if (!any_geometry(d, a) || !tc_plan_conv_any_wgrad(p, any, any, dw, a, g.sm_count)) return 0;
  float *dyr = cl_lookup(dy, d.N, d.K, d.oH * d.oW), *xr = cl_lookup(x, d.N, d.C, d.H * d.W); size_t ny = 0, nx = 0;
  int rc = dyr ? LTB_OK : channels_last(dy, d.N, d.K, d.oH * d.oW, &dyr, &ny); if (rc) return rc;
  if (!dyr) return 0;
  if (!xr) rc = channels_last(x, d.N, d.C, d.H * d.W, &xr, &nx);
  bool ok = !rc && xr && tc_plan_conv_any_wgrad(p, dyr, xr, dw, a, g.sm_count);
  if (ok) rc = launch_plan(p, "tc_gemm_kernel[conv_wgrad im2col]");
  if (xr && nx) temp_free(xr, nx);
  if (ny) temp_free(dyr, ny);
  return rc ? rc : (ok ? 1 : 0);
}

static int conv_wgrad_taps(const float* x, const float* dy, float* dw, const ConvDims& d) {
  TcConvGeom gm; TcPlan p;
  if (!taps_geometry(d, gm) || !tc_plan_conv_taps_wgrad(p, dw, dw, dw, gm, g.sm_count)) return 0;
  float *dyr = cl_lookup(dy, d.N, d.K, d.oH * d.oW), *xr = cl_lookup(x, d.N, d.C, d.H * d.W); size_t ny = 0, nx = 0;
  // Both operands are read channels-last.  With the copies already there (x from this convolution's forward call, dy shared
  // with the data-grad) the tap loop reads each of them once; having to make both first only pays once the unfolded
  // matrix, nine times the size of x, would be large.
  if ((!dyr || !xr || (g.tune & 2)) && (size_t)d.N * d.C * d.R * d.S * d.oH * d.oW * 4 < ((size_t)64 << 20)) return 0;
  int rc = dyr ? LTB_OK : channels_last(dy, d.N, d.K, d.oH * d.oW, &dyr, &ny); if (rc) return rc;
  if (!dyr) return 0;
  if (!xr) rc = channels_last(x, d.N, d.C, d.H * d.W, &xr, &nx);
  bool ok = !rc && xr && tc_plan_conv_taps_wgrad(p, dyr, xr, dw, gm, g.sm_count);
  if (ok) rc = launch_plan(p, "tc_gemm_kernel[conv_wgrad taps]");
  if (xr && nx) temp_free(xr, nx);
  if (ny) temp_free(dyr, ny);
  return rc ? rc : (ok ? 1 : 0);
}
// Which form a convolution whose filter is more than one tap or whose stride is not 1 takes when the tap loop declines it.  A filter
// over a few channels (an image's three) fills whole k-iterations only when unfolded, and a strided 1x1 reads a quarter of its input,
// which the unfolding copies alone: both stay unfolded where the image size allows it, and so does a strided filter, whose unfolded
// matrix (R S / stride^2 times its input, shared by forward and weight gradient) is no larger than two channels-last copies
// (ResNet-50 at batch 128: 2 % of the step).
static bool flat_pixels(int pix) { return !tc_conv_needs_rows(pix) || (pix % 4 == 0 && pix >= 64); }
static bool wants_im2col(const ConvDims& d) {
  const int pix = d.oH * d.oW;
  if (is_pointwise(d)) return tc_conv_needs_rows(pix) && !(pix % 4 == 0 && pix >= 64) && pix != 1 && !((pix == 4 || pix == 16) && d.C % 4 == 0 && d.K % 4 == 0);
  const bool reread = d.R * d.S > 3 * d.sh * d.sw;
  if (d.C < 16 || !reread) return !flat_pixels(pix) && pix != 4 && pix != 16;     // (fewer channels leave a 32-channel block more than half empty)
  return true;
}

// Start of a convolution's backward call, before its two halves part onto two streams: one channels-last copy of dy for both.
int conv_bwd_prestage(const float* dy, const ConvDims& d, bool both_halves) {
  TcConvGeom gm; TcConvAny a;
  const bool window = taps_geometry(d, gm) && d.C % 64 == 0 && d.K % 32 == 0;
  if (!g.filter_cache || !both_halves || (!window && !(wants_im2col(d) && d.sh == 1 && d.sw == 1 && any_geometry(d, a)))) {
    cl_cache_drop(dy, (size_t)d.N * d.K * d.oH * d.oW * 4);              // a copy from an earlier call is not this gradient's
    return LTB_OK;
  }
  float* dyr; size_t ny;
  int rc = channels_last(dy, d.N, d.K, d.oH * d.oW, &dyr, &ny, /*keep=*/true);
  if (!rc && dyr && ny) temp_free(dyr, ny);                 // no room to keep it: each half makes its own, as before
  return rc;
}

int conv_fwd_tc(const float* x, const float* w, const float* bias, float* y, const ConvDims& d, bool* relu) {
  const int ck = d.C * d.R * d.S, pix = d.oH * d.oW;
  TcPlan p;
  { int t = conv_fwd_taps(x, w, bias, y, d, relu); if (t != 0) return t; }      // the tap-loop form when the shape allows it
  if (wants_im2col(d)) { int t = conv_fwd_any(x, w, bias, y, d, relu); if (t != 0) return t; }
  const bool rows = tc_conv_needs_rows(pix);
  // an image size that does not fill tiles goes image by image, as long as a filter fills a k-iteration (see wants_im2col)
  const bool ragged = rows && pix % 4 == 0 && pix >= 64 && ck >= 32 && ck % 4 == 0;
  const int ldw = up4(ck);                                                 // K-major filter rows must be a multiple of 16 bytes
  if (ragged ? !tc_plan_conv_ragged_fwd(p, (const float*)g.heap, (const float*)g.heap, ldw, bias, y, d.N, ck, d.K, pix, g.sm_count)
             : !tc_plan_conv_fwd(p, y /* any aligned pointer: eligibility only */, rows, y, ldw, bias, y, d.N, ck, d.K, pix, g.sm_count)) return 0;
  // Small images (4 or 16 pixels): the kernel collects the activation itself, from x or from its unfolded form.
  const bool gathered = rows && !ragged && pix > 1 && !(g.tune & 1) && tc_gather_possible(y, ck, pix);
  if (rows && !ragged && !gathered && pix > 1) return 0;
  const float* op = x; float* temp = nullptr; size_t tn = 0;
  Clear clear = plan_clear(p);
  int rc = is_pointwise(d) ? LTB_OK : unfolded(x, d, &op, &temp, &tn, &clear);
  if (rc || !op) return rc;
  float* wtemp; size_t wn; const float* wp;
  rc = padded_filter(w, d.K, ck, ldw, &wp, &wtemp, &wn);
  bool ok = !rc && wp && (ragged ? tc_plan_conv_ragged_fwd(p, op, wp, ldw, bias, y, d.N, ck, d.K, pix, g.sm_count)
                                 : tc_plan_conv_fwd(p, op, rows, wp, ldw, bias, y, d.N, ck, d.K, pix, g.sm_count));
  if (ok && gathered) tc_plan_gather(p, op, d.N, ck, pix);
  if (ok) rc = launch_plan(p, gathered ? "tc_gemm_kernel[conv_fwd gather]" : "tc_gemm_kernel[conv_fwd]", relu, clear);
  if (wtemp) temp_free(wtemp, wn);
  if (temp) temp_free(temp, tn);
  return rc ? rc : (ok ? 1 : 0);
}

// *fresh: dx was declared unset (ltb_grad_unset) and holds nothing: a path that can writes its result instead of adding, the
// unfold-and-fold path fills dx with zeros first; either way *fresh is false once dx holds data.
int conv_dgrad_tc(const float* dy, const float* w, float* dx, const ConvDims& d, bool* fresh) {
  const int ck = d.C * d.R * d.S, pix = d.oH * d.oW;
  TcPlan p;
  const bool rows = tc_conv_needs_rows(pix), direct = is_pointwise(d);
  { int t = conv_dgrad_taps(dy, w, dx, d, !*fresh); if (t != 0) { if (t > 0) *fresh = false; return t; } }
  // a strided 1x1 keeps the unfolded form where the image size allows it: its one-to-one fold is cheaper than the zeros
  if (d.R * d.S > 1 || wants_im2col(d)) { int t = conv_dgrad_any(dy, w, dx, d, !*fresh); if (t != 0) { if (t > 0) *fresh = false; return t; } }
  const bool ragged = rows && pix % 4 == 0 && pix >= 64 && ck >= 32 && d.K % 4 == 0;
  const int ldw = up4(ck);                                                 // N-major filter rows must be a multiple of 16 bytes
  if (ragged ? !tc_plan_conv_ragged_dgrad(p, (const float*)g.heap, (const float*)g.heap, ldw, dx, d.N, ck, d.K, pix, direct, g.sm_count)
             : !tc_plan_conv_dgrad(p, dx, rows, dx, ldw, dx, d.N, ck, d.K, pix, direct, g.sm_count)) return 0;
  const bool gathered = rows && !ragged && pix > 1 && !(g.tune & 1) && tc_gather_possible(dy, d.K, pix);    // dy of a small map: collected by the kernel itself
  if (rows && !ragged && !gathered && pix > 1) return 0;
  int rc = LTB_OK;
  float* col = nullptr; const size_t ncol = (size_t)d.N * ck * pix;
  if (!direct) { col = temp_alloc(ncol); if (!col) return 0; }
  float* wtemp; size_t wn; const float* wp;
  rc = padded_filter(w, d.K, ck, ldw, &wp, &wtemp, &wn);
  float* out = direct ? dx : col; const bool acc = direct && !*fresh;
  bool ok = !rc && wp && (ragged ? tc_plan_conv_ragged_dgrad(p, dy, wp, ldw, out, d.N, ck, d.K, pix, acc, g.sm_count)
                                 : tc_plan_conv_dgrad(p, dy, rows, wp, ldw, out, d.N, ck, d.K, pix, acc, g.sm_count));
  if (ok && !direct && *fresh) {                                  // the fold-back adds into dx: start from zeros
    if (cudaMemsetAsync(dx, 0, (size_t)d.N * d.C * d.H * d.W * 4, g.stream) != cudaSuccess) { ok = false; rc = fail(LTB_E_CUDA, "conv data-grad: zero fill failed"); }
  }
  if (ok && gathered) tc_plan_gather(p, dy, d.N, d.K, pix);
  if (ok) rc = launch_plan(p, gathered ? "tc_gemm_kernel[conv_dgrad gather]" : "tc_gemm_kernel[conv_dgrad]");
  if (ok && !rc && !direct) rc = launch_fold(col, dx, d);
  if (ok && !rc) *fresh = false;
  if (wtemp) temp_free(wtemp, wn);
  if (col) temp_free(col, ncol);
  return rc ? rc : (ok ? 1 : 0);
}

int conv_wgrad_tc(const float* x, const float* dy, float* dw, const ConvDims& d) {
  const int ck = d.C * d.R * d.S, pix = d.oH * d.oW;
  TcPlan p;
  { int t = conv_wgrad_taps(x, dy, dw, d); if (t != 0) return t; }
  // forward left its unfolded matrix behind (the small-channel stems), or the layer is one that is unfolded anyway
  float* kept = is_pointwise(d) ? nullptr : unfold_lookup(x, d);
  if (!kept && wants_im2col(d)) { int t = conv_wgrad_any(x, dy, dw, d); if (t != 0) return t; }
  const bool ragged = tc_conv_needs_rows(pix) && pix % 4 == 0 && pix >= 64 && ck >= 32;
  auto plan = [&](const float* xin) {
    return ragged ? tc_plan_conv_ragged_wgrad(p, xin, dy, dw, d.N, ck, d.K, pix, g.sm_count) : tc_plan_conv_wgrad(p, xin, dy, dw, d.N, ck, d.K, pix, g.sm_count);
  };
  if (!plan(dy)) return 0;
  const float* xin = x; float* col = nullptr; const size_t n = (size_t)d.N * ck * pix;
  if (!is_pointwise(d)) {
    if (kept) xin = kept;
    else {
      col = temp_alloc(n); if (!col) return 0;
      int rc0 = launch_unfold(x, col, d); if (rc0) return rc0;
      xin = col;
    }
  }
  // the probe above used dy in place of x: the caller's x may still be declined (a view that is not 16-byte aligned)
  if (!plan(xin)) { if (col) temp_free(col, n); return 0; }
  int rc = launch_plan(p, "tc_gemm_kernel[conv_wgrad]");
  if (col) temp_free(col, n);
  return rc ? rc : 1;
}

}  // namespace ltb
