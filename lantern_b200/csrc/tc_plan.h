// Host-side plans for the TF32 tensor-core engine (pure C++, no CUDA: also compiled into the CPU layout test).
//
// The engine kernel (gemm_tc.cu) is generic: for every operand it is told how to turn (output tile, k-iteration) into
// TMA box coordinates, how many bytes a stage holds, and the UMMA shared-memory descriptors of the MMA steps of a stage.
// Everything that depends on the tensor layout (NCHW activations with pixels contiguous, OIHW filters, row-major
// matrices, tiny images) is decided here and expressed in those numbers.
//
// Shared-memory layouts are the canonical UMMA layouts for 32-bit operands:
//   K-major,  swizzle span X bytes : rows of X bytes (X/4 floats of K), 8-row groups SBO apart; an MMA step covers 32 B of K
//   MN-major (32-bit operands)     : the only layout the tensor core accepts is the 128-byte swizzle with 32-byte atoms:
//                                    chunks of 32 elements of M (or N) contiguous (128 B), one row per k, 4 k-rows per group
//                                    (512 B), groups SBO apart, chunks LBO apart; an MMA step (K = 8) spans two groups.
//   no swizzle (K-major only)      : 16-byte rows, 8-row groups SBO apart, the second 16-byte k-chunk LBO apart.
// A TMA box whose inner extent is X bytes, loaded with the matching swizzle mode, lands in exactly that layout.
// Operands whose contiguous axis is shorter than 128 bytes cannot be fed MN-major; the callers hand those in as K-major
// row matrices instead (`a_rows`), produced by a small transposing copy.
#pragma once
#include <cstdint>

namespace ltb {

enum TcSwizzle { TC_SW_NONE = 0, TC_SW_32 = 1, TC_SW_64 = 2, TC_SW_128 = 3, TC_SW_128_32B = 4 };

struct TcTensorMap {          // arguments of cuTensorMapEncodeTiled for one FP32 operand
  const void* base;
  int rank;
  uint64_t dims[5];           // innermost first
  uint64_t strides[5];        // bytes; strides[0] is implied (4) and unused
  uint32_t box[5];
  int swizzle;                // TcSwizzle
};

// TC_LOAD_BOX        one tiled box
// TC_LOAD_BOXES      `nbox` tiled boxes of 32 x 32 floats; box j is 32 further along dimension 0 (rows whose length is no multiple
//                    of 32: the part of a box beyond the row is zero-filled, a box wholly beyond it is not loaded)
// TC_LOAD_IM2COL     one im2col-mode load: 128 consecutive pixels of the walk, 32 channels, at the tap given by coordinates 1 and 2
// TC_LOAD_IM2COL_MN  `nbox` im2col-mode loads of 32 pixels x 32 channels; box j is chunk tile * nbox + j of (tap, channel block)
// TC_LOAD_TAPS       `nbox` tiled boxes of 32 pixels x 32 channels of a channels-last image; box j is chunk tile * nbox + j of (tap, channel
//                    block), its tap (s, r) added to coordinates 1 and 2, its channel block to coordinate 4
enum TcLoad { TC_LOAD_BOX = 0, TC_LOAD_BOXES = 1, TC_LOAD_IM2COL = 2, TC_LOAD_IM2COL_MN = 3, TC_LOAD_TAPS = 4 };

// The walk of an im2col-mode tensor map over channels-last images: base pixels (low_w + i * step_w, low_h + j * step_h), i < grid_w,
// j < grid_h, image after image; upper_* is the bounding box's upper corner as cuTensorMapEncodeIm2col wants it.
struct TcIm2col { int grid_w, grid_h, step_w, step_h, low_w, low_h, upper_w, upper_h, pixels; int adv_i, adv_j, adv_n; int taps, tap_s, ch_blocks; };   // adv_*: what `pixels` base pixels further on adds to (i, j, image)

struct TcOperand {
  TcTensorMap map;
  // box coordinate d = c_off[d] + ((tile / t_div[d]) % t_mod[d]) * t_mul[d] + ((kiter / k_div[d]) % k_mod[d]) * k_mul[d]
  // (c_off and k_mul may be negative: the taps of a convolution window start left of / above the image, where TMA fills zeros)
  int t_div[5], t_mod[5], t_mul[5];
  int k_div[5], k_mod[5], k_mul[5];
  int c_off[5];
  uint32_t stage_bytes;       // bytes one stage of this operand occupies (== bytes the TMA box delivers)
  int mn_major;               // 0: K-major, 1: M/N-major (instruction descriptor transpose bit)
  uint32_t lbo, sbo;          // bytes
  int nk;                     // MMA steps (K = 8 each) per stage
  uint32_t kstep_off[8];      // start-address offset of each step within the stage
  // How a stage is filled (TcLoad).  The last three modes are described at their operands in tc_plan.cpp.
  int load;
  int nbox;                   // boxes per stage, 4096 bytes each (TC_LOAD_BOXES, TC_LOAD_IM2COL_MN, TC_LOAD_TAPS); 1 otherwise
  TcIm2col im;
};

// The k part of the coordinates as a mixed-radix counter, so that the single producer thread advances them with additions
// only: level 0 steps n0 times, then level 1 steps once (and level 0 returns to its start), after n1 of those level 2
// steps.  inc[j][d] is what reaching level j adds to coordinate d (returns of the lower levels included).
struct TcWalk { int n0, n1; int inc[3][5]; };
bool tc_walk_of(const TcOperand& o, TcWalk& w);

// A cluster of `cz` splits adds its partial tiles up: CTA `rank` owns rows (row-major epilogues) or columns (pixel-major) lo .. hi - 1 of
// the tile, `extent` of them in the tile and `limit` inside the result.  Used by the kernel and by the CPU check of the plans.
#ifdef __CUDACC__
#define LTB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define LTB_HOST_DEVICE inline
#endif
struct TcSlice {
  int lo, hi;
  LTB_HOST_DEVICE TcSlice(int extent, int cz, int rank, int limit) {
    const int per = (extent + cz - 1) / cz;
    lo = rank * per; hi = lo + per < extent ? lo + per : extent;
    if (limit < hi) hi = limit;
  }
};
// The rows of a slice as eight warps share them: warp w takes the rows lo + w, lo + w + 8, .., each as bn / 32 runs of 32 columns.
struct TcSliceRows {
  int first, items, shift;
  LTB_HOST_DEVICE TcSliceRows(const TcSlice& s, int bn, int w) : first(s.lo + w), shift(0) {
    while ((64 << shift) <= bn) ++shift;                       // runs of a row: 1 << shift
    items = s.hi > first ? ((s.hi - first + 7) / 8) << shift : 0;
  }
  LTB_HOST_DEVICE int row(int i) const { return first + 8 * (i >> shift); }
  LTB_HOST_DEVICE int run(int i) const { return i & ((1 << shift) - 1); }
};

enum TcEpilogue {
  TC_EPI_PIXEL = 0,   // D row = pixel, D column = channel: out[img][chan][pix]   (conv forward / data-grad)
  TC_EPI_ROWMAJOR = 1,// D row = row, D column contiguous:   out[row*ld + col]      (gemm, weight-grad)
  TC_EPI_TAPS = 2     // D row = row, D column (tap, channel block of 32, channel): out[row*ld + channel*taps + tap], channels beyond col_mod not stored
};

struct TcPlan {
  TcOperand a, b;             // a: the M-side operand (128 rows per tile), b: the N-side operand (bn columns per tile)
  int M, N;                   // logical extents of D
  int bn;                     // tile width: 64, 128 or 256
  int pair;                   // two neighbouring row tiles share a CTA pair: one MMA over 256 rows, each CTA loads its own rows of A and half of B's columns (b is planned with tiles of bn / 2)
  int m_tiles, n_tiles, k_iters, splits;
  int epilogue;
  float* out;
  const float* bias;          // per D column, or null
  float alpha;
  int accumulate;             // 1: out += ..., 0: out = ...   (split-K > 1 forces atomic accumulation)
  int64_t pix_per_img, img_stride, chan_stride;   // TC_EPI_PIXEL
  int64_t pix_pad;            // TC_EPI_PIXEL: tile rows per image, at least pix_per_img (0: pix_per_img); rows beyond the image are not stored
  int64_t ld;                                     // TC_EPI_ROWMAJOR
  int col_mod, col_mul;                           // TC_EPI_TAPS: channels, taps
  // Gather mode (tc_plan_gather): operand a keeps its K-major row descriptors but is not loaded by TMA; the kernel's
  // epilogue warps collect it from gather_src[img][chan][pix] (pix = 4 or 16), warp g filling rows 16 g .. 16 g + 15 of
  // the tile, lane = channel within the 32-channel block, 128-byte swizzle.
  const float* gather_src;
  int g_pix, g_chan, g_imgs;
};

// "Flat" convolution view: activations X[n][k][p] with p contiguous (k = channels, or channels*kh*kw after unfolding),
// weights W[co][k] row-major with ldw >= k floats per row (zeros beyond k: the caller pads a copy when the engine needs a
// wider row, ldw a multiple of 4), outputs Y[n][co][p].  P is the number of pixels per image.
//   forward : Y[n][co][p]  = sum_k  W[co][k] X[n][k][p] (+ bias[co])         D = pixels x co
//   dgrad   : dX[n][k][p] (+)= sum_co W[co][k] dY[n][co][p]                   D = pixels x k
//   wgrad   : dW[co][k]  += sum_{n,p} dY[n][co][p] X[n][k][p]                 D = co x k
// Each returns false when the shape is not eligible (the caller then uses the FP32 path).
// a_rows: the activation operand (x for forward, dy for dgrad) is given as a K-major row matrix [n_img*pix][channels]
// instead of [n_img][channels][pix]; tc_conv_needs_rows says when that form is required.
bool tc_conv_needs_rows(int pix);
// Whether an activation [n_img][chan][pix] that needs the row form can be gathered by the kernel itself instead of being
// copied into a row matrix first; tc_plan_gather switches a plan made with a_rows = true (x = src as base) to that mode.
bool tc_gather_possible(const float* src, int chan, int pix);
void tc_plan_gather(TcPlan& p, const float* src, int n_img, int chan, int pix);
bool tc_plan_conv_fwd(TcPlan& p, const float* x, bool a_rows, const float* w, int ldw, const float* bias, float* y, int n_img, int ck, int co, int pix, int sm_count);
bool tc_plan_conv_dgrad(TcPlan& p, const float* dy, bool a_rows, const float* w, int ldw, float* dx, int n_img, int ck, int co, int pix, bool accumulate, int sm_count);
bool tc_plan_conv_wgrad(TcPlan& p, const float* x, const float* dy, float* dw, int n_img, int ck, int co, int pix, int sm_count);
// Implicit ("tap loop") forms for R x S convolutions with stride 1.  The activations are channels-last copies
// xr[n][h][w][c] and dyr[n][oh][ow][k] (made by a transposing copy); a TMA box then is a window of whole image rows
// with 32 channels, and the tap (r, s) only shifts the box coordinates -- the nine-fold unfolded matrix never exists.
//   forward : rows = output pixels, K loop = (r, s, channel block); weights permuted to wt[r*S+s][k][c]
//   dgrad   : rows = input pixels,  K loop = (r, s, k block);       the same weights wt[r*S+s][k][c], read N-major
//   wgrad   : D = k x (channel block, tap, c), K loop = blocks of 32 pixels, both operands M/N-major; stored to OIHW by TC_EPI_TAPS
struct TcConvGeom { int n_img, C, H, W, K, R, S, ph, pw, oH, oW; };
bool tc_plan_conv_taps_fwd(TcPlan& p, const float* xr, const float* wt, const float* bias, float* y, const TcConvGeom& g, int sm_count);
bool tc_plan_conv_taps_dgrad(TcPlan& p, const float* dyr, const float* wt, float* dx, const TcConvGeom& g, bool accumulate, int sm_count);
bool tc_plan_conv_taps_wgrad(TcPlan& p, const float* dyr, const float* xr, float* dw, const TcConvGeom& g, int sm_count);
// The same three contractions for any image size, stride and channel count, from channels-last copies whose channel counts
// are padded to a multiple of 4 (ldc, ldk): the TMA unit's im2col mode walks the output pixels itself, so that a tile is
// any 128 consecutive ones (a tiled window needs rows of the image that fill a tile exactly).
//   fwd   : wt[r*S+s][k][ldc];  dgrad (stride 1): the same for C a multiple of 32, else wd[r*S+s][c][ldk];  wgrad: D = k x (tap, channel block, channel)
struct TcConvAny { int n_img, C, H, W, K, R, S, sh, sw, ph, pw, oH, oW, ldc, ldk; };
bool tc_plan_conv_any_fwd(TcPlan& p, const float* xr, const float* wt, const float* bias, float* y, const TcConvAny& g, int sm_count);
bool tc_plan_conv_any_dgrad(TcPlan& p, const float* dyr, const float* wp, float* dx, const TcConvAny& g, bool accumulate, int sm_count);
bool tc_plan_conv_any_wgrad(TcPlan& p, const float* dyr, const float* xr, float* dw, const TcConvAny& g, int sm_count);
// The flat convolution view straight from x[n][k][p] for image sizes that do not fill tiles (pix a multiple of 4, at least 64):
// every image is cut into tiles of 128 pixels, the last one partly beyond the image.
bool tc_plan_conv_ragged_fwd(TcPlan& p, const float* x, const float* w, int ldw, const float* bias, float* y, int n_img, int ck, int co, int pix, int sm_count);
bool tc_plan_conv_ragged_dgrad(TcPlan& p, const float* dy, const float* w, int ldw, float* dx, int n_img, int ck, int co, int pix, bool accumulate, int sm_count);
bool tc_plan_conv_ragged_wgrad(TcPlan& p, const float* x, const float* dy, float* dw, int n_img, int ck, int co, int pix, int sm_count);
// C[M,N] (op)= alpha * A B; a_kmajor: A stored [M,K] (else [K,M]); b_kmajor: B stored [N,K] (else [K,N]).
bool tc_plan_gemm(TcPlan& p, const float* a, bool a_kmajor, const float* b, bool b_kmajor, float* c, int M, int N, int K, float alpha,
                  bool accumulate, int sm_count);
// The same for any extents and for operands whose rows are lda / ldb floats long (zeros between the row's own length and that: a
// padded copy, where the matrix itself has rows of no whole number of 16-byte units).
bool tc_plan_gemm_ld(TcPlan& p, const float* a, bool a_kmajor, int lda, const float* b, bool b_kmajor, int ldb, float* c, int M, int N, int K, float alpha,
                     bool accumulate, int sm_count);

}  // namespace ltb
