// CPU check of the tensor-core engine's bookkeeping (test infrastructure).
//
// Emulates, for every kind of plan the planner produces, (1) what the TMA loads of a stage write to shared memory (one box, several
// boxes clipped at the row's end, the im2col mode's walk over output pixels; box order, out-of-bounds zero fill, 32/64/128-byte
// swizzle as an XOR of address bits [4,7) with bits [7,10)), (2) which element the tensor core reads for (row, k) of an MMA step
// from the canonical UMMA layout described by the step's descriptor (start offset, LBO, SBO, swizzle, major-ness), and (3) the
// epilogue's output indexing.  The result of the emulated engine is compared with a direct evaluation of the convolution / GEMM.
// The splits are added up in any order here; how a cluster deals a tile out to its CTAs in deterministic mode is checked by itself.
// This pins coordinates, strides, descriptors and tile/split arithmetic without a GPU; it does not prove that the hardware follows
// the emulated conventions.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "../lantern_b200/csrc/tc_plan.h"

using namespace ltb;

static uint32_t swz(uint32_t off, int mode) {
  if (mode == TC_SW_128_32B) return off ^ (((off >> 7) & 3u) << 5);       // 32-byte atoms: bits [5,7) ^= bits [7,9)
  int bits = mode == TC_SW_128 ? 3 : mode == TC_SW_64 ? 2 : mode == TC_SW_32 ? 1 : 0;
  return off ^ (((off >> 7) & ((1u << bits) - 1)) << 4);
}
static int span(int mode) { return (mode == TC_SW_128 || mode == TC_SW_128_32B) ? 128 : mode == TC_SW_64 ? 64 : mode == TC_SW_32 ? 32 : 16; }

static void coords_of(const TcOperand& o, int tile, int kiter, int64_t* c) {
  for (int d = 0; d < 5; ++d) c[d] = (int64_t)o.c_off[d] + (int64_t)((tile / o.t_div[d]) % o.t_mod[d]) * o.t_mul[d] + (int64_t)((kiter / o.k_div[d]) % o.k_mod[d]) * o.k_mul[d];
}
// The im2col mode: `pixels` consecutive output pixels of the walk from `first` on, 32 channels from `chan` on at tap (s, r), written to
// shared memory from `at` on, a row of 128 bytes per pixel.
static void im2col_box(const TcOperand& o, int64_t first, int64_t chan, int64_t s, int64_t r, uint32_t at, std::vector<float>& smem) {
  const TcTensorMap& m = o.map; const TcIm2col& g = o.im;
  for (int64_t q = 0; q < g.pixels; ++q) {
    const int64_t per = (int64_t)g.grid_w * g.grid_h, img = (first + q) / per, j = (first + q) % per / g.grid_w, i = (first + q) % g.grid_w;
    const int64_t w = g.low_w + i * g.step_w + s, h = g.low_h + j * g.step_h + r;
    for (int64_t c = 0; c < 32; ++c) {
      const bool inb = chan + c < (int64_t)m.dims[0] && w >= 0 && w < (int64_t)m.dims[1] && h >= 0 && h < (int64_t)m.dims[2] && img < (int64_t)m.dims[3];
      const float v = inb ? *(const float*)((const char*)m.base + (chan + c) * 4 + w * m.strides[1] + h * m.strides[2] + img * m.strides[3]) : 0.0f;
      smem[swz(at + (uint32_t)(q * 128 + c * 4), m.swizzle) / 4] = v;
    }
  }
}
static bool im2col_load(const TcOperand& o, int tile, int kiter, std::vector<float>& smem) {
  const TcIm2col& g = o.im;
  for (int d = 1; d < 4; ++d) if (o.map.strides[d] % 16) { printf("stride %d not a multiple of 16 bytes\n", d); return false; }
  // the box corners of the map: the walk's first and last base pixel relative to the image's first and last pixel
  if (g.upper_w != g.low_w + (g.grid_w - 1) * g.step_w - ((int)o.map.dims[1] - 1) || g.upper_h != g.low_h + (g.grid_h - 1) * g.step_h - ((int)o.map.dims[2] - 1)) { printf("im2col corners\n"); return false; }
  smem.assign(o.stage_bytes / 4, 1e30f);                       // a box that is not loaded leaves what was there before
  if (o.load == TC_LOAD_IM2COL) {
    int64_t c[5]; coords_of(o, 0, kiter, c);
    if (g.pixels * 128 != (int)o.stage_bytes || c[0] % 4) { printf("im2col stage\n"); return false; }
    im2col_box(o, (int64_t)tile * g.pixels, c[0], c[1], c[2], 0, smem);
    return true;
  }
  if (o.nbox * 4096 != (int)o.stage_bytes) { printf("im2col boxes\n"); return false; }
  for (int b = 0; b < o.nbox; ++b) {
    const int q = tile * o.nbox + b, blk = q / g.taps, tap = q - blk * g.taps;
    if (blk < g.ch_blocks) im2col_box(o, (int64_t)kiter * g.pixels, (int64_t)blk * 32, tap % g.tap_s, tap / g.tap_s, (uint32_t)b * 4096, smem);
  }
  return true;
}
// The producer advances the walk's pixel by additions: from any starting iteration it must be where the division says.
static bool pixel_walk_matches(const TcOperand& o, int k_iters) {
  const TcIm2col& g = o.im;
  for (int k0 = 0; k0 < k_iters; k0 += (k_iters > 5 ? k_iters / 5 : 1)) {
    const int per = g.grid_w * g.grid_h;
    int pn = k0 * 32 / per, pj = k0 * 32 % per / g.grid_w, pi = k0 * 32 % g.grid_w;
    for (int it = k0; it < k_iters; ++it) {
      if (pn != it * 32 / per || pj != it * 32 % per / g.grid_w || pi != it * 32 % g.grid_w) { printf("pixel walk at iteration %d from %d\n", it, k0); return false; }
      pi += g.adv_i; pj += g.adv_j; pn += g.adv_n;
      if (pi >= g.grid_w) { pi -= g.grid_w; ++pj; }
      if (pj >= g.grid_h) { pj -= g.grid_h; ++pn; }
    }
  }
  return true;
}
static bool tma_load(const TcOperand& o, int tile, int kiter, std::vector<float>& smem) {
  const TcTensorMap& m = o.map;
  if (o.load == TC_LOAD_IM2COL || o.load == TC_LOAD_IM2COL_MN) return im2col_load(o, tile, kiter, smem);
  int64_t c[5]; coords_of(o, tile, kiter, c);
  if ((c[0] * 4) % 16) { printf("unaligned innermost TMA coordinate %lld\n", (long long)c[0]); return false; }
  for (int d = 1; d < m.rank; ++d) if (m.strides[d] % 16) { printf("stride %d not a multiple of 16 bytes\n", d); return false; }
  if ((m.box[0] * 4) % 16 || (int)m.box[0] * 4 > span(m.swizzle) && m.swizzle != TC_SW_NONE) { printf("bad inner box\n"); return false; }
  int64_t total = 1; for (int d = 0; d < m.rank; ++d) { if (m.box[d] > 256) { printf("box > 256\n"); return false; } total *= m.box[d]; }
  const bool taps = o.load == TC_LOAD_TAPS;
  const int boxes = o.load == TC_LOAD_BOXES || taps ? o.nbox : 1;
  if (boxes > 1 && total * 4 != 4096) { printf("box of several not 4096 bytes\n"); return false; }
  if (total * 4 * boxes != o.stage_bytes) { printf("stage_bytes %u != box bytes %lld\n", o.stage_bytes, (long long)total * 4); return false; }
  smem.assign(o.stage_bytes / 4, 1e30f);
  const int64_t w0 = c[1], h0 = c[2];
  for (int b = 0; b < boxes; ++b, c[0] += taps ? 0 : 32) {
    if (o.load == TC_LOAD_BOXES && c[0] >= (int64_t)m.dims[0]) break;       // wholly beyond the row: not loaded
    if (taps) {
      const int q = tile * o.nbox + b, blk = q / o.im.taps, tap = q - blk * o.im.taps;
      if (blk >= o.im.ch_blocks) break;
      c[1] = w0 + tap % o.im.tap_s; c[2] = h0 + tap / o.im.tap_s; c[4] = blk;
    }
    for (int64_t lin = 0; lin < total; ++lin) {
      int64_t r = lin, goff = 0; bool inb = true;
      for (int d = 0; d < m.rank; ++d) {
        int64_t i = r % m.box[d]; r /= m.box[d];
        int64_t g = c[d] + i;
        if (g < 0 || g >= (int64_t)m.dims[d]) inb = false;
        goff += g * (d == 0 ? 4 : (int64_t)m.strides[d]);
      }
      float v = inb ? *(const float*)((const char*)m.base + goff) : 0.0f;
      smem[swz((uint32_t)(b * 4096 + lin * 4), m.swizzle) / 4] = v;
    }
  }
  return true;
}
// What the kernel's gathering warps store for operand a of a plan in gather mode (gemm_tc.cu): warp g, lane l, run j, element
// i write row 16 g + 4 j + i, channel l of the 32-channel block, at 16-byte chunk (l >> 2) ^ (row & 7) of the 128-byte row.
static bool gather_load(const TcPlan& p, int tile, int kiter, std::vector<float>& smem) {
  if (p.a.stage_bytes != 128 * 128 || p.a.mn_major || p.a.map.swizzle != TC_SW_128) { printf("gather mode needs a K-major 128-byte-swizzled operand\n"); return false; }
  smem.assign(p.a.stage_bytes / 4, 0.0f);
  const int pix = p.g_pix, chan = p.g_chan, runs = 16 / pix;
  for (int gw = 0; gw < 8; ++gw) for (int lane = 0; lane < 32; ++lane) {
    const int64_t row0 = (int64_t)tile * 128 + gw * 16, img0 = row0 / pix;
    const int c = kiter * 32 + lane;
    for (int j = 0; j < 4; ++j) for (int i = 0; i < 4; ++i) {
      const int64_t img = runs == 1 ? img0 : img0 + j;
      const int q = runs == 1 ? j * 4 + i : i;
      const float v = (c < chan && img < p.g_imgs) ? p.gather_src[(img * chan + c) * pix + q] : 0.0f;
      const uint32_t r = (uint32_t)(j * 4 + i);
      const uint32_t off = (uint32_t)gw * 16 * 128 + r * 128 + (((((uint32_t)lane >> 2) ^ (r & 7u)) << 4) | (((uint32_t)lane & 3u) << 2));
      smem[off / 4] = v;
    }
  }
  return true;
}
// Element (r, kk) of MMA step `ks`: r = row (M or N index within the tile), kk in [0,8).
static float umma_fetch(const TcOperand& o, const std::vector<float>& smem, int ks, int r, int kk) {
  const int X = span(o.map.swizzle); uint32_t off = o.kstep_off[ks];
  if (!o.mn_major) {
    if (o.map.swizzle != TC_SW_NONE) off += (uint32_t)(r / 8) * o.sbo + (uint32_t)(r % 8) * X + (uint32_t)kk * 4;
    else off += (uint32_t)(r / 8) * o.sbo + (uint32_t)(r % 8) * 16 + (uint32_t)(kk / 4) * o.lbo + (uint32_t)(kk % 4) * 4;
  } else {
    // 32-bit operands: only the 128-byte swizzle with 32-byte atoms exists (chunks of 32 elements, 4 k-rows per group)
    if (o.map.swizzle != TC_SW_128_32B) { printf("MN-major operand with an unsupported swizzle mode\n"); exit(1); }
    off += (uint32_t)(r / 32) * o.lbo + (uint32_t)(kk / 4) * o.sbo + (uint32_t)(kk % 4) * 128 + (uint32_t)(r % 32) * 4;
  }
  off = swz(off, o.map.swizzle);
  if (off / 4 >= smem.size()) { printf("MMA read beyond the stage (%u >= %zu)\n", off, smem.size() * 4); exit(1); }
  return smem[off / 4];
}

// The producer's incremental walk (TcWalk) must visit the coordinates the closed formula gives, from any starting iteration.
static bool walk_matches(const TcOperand& o, int tile, int k_iters) {
  TcWalk w;
  if (!tc_walk_of(o, w)) { printf("operand has no walk\n"); return false; }
  for (int k0 = 0; k0 < k_iters; k0 += (k_iters > 7 ? k_iters / 7 : 1)) {
    int64_t c[5]; coords_of(o, tile, k0, c);
    int i0 = k0 % w.n0, i1 = (k0 / w.n0) % w.n1;
    for (int it = k0; it < k_iters; ++it) {
      int64_t want[5]; coords_of(o, tile, it, want);
      for (int d = 0; d < 5; ++d) if (c[d] != want[d]) { printf("walk: coordinate %d at iteration %d (start %d): %lld, formula %lld\n", d, it, k0, (long long)c[d], (long long)want[d]); return false; }
      int lvl = 0;
      if (++i0 == w.n0) { i0 = 0; lvl = 1; if (++i1 == w.n1) { i1 = 0; lvl = 2; } }
      for (int d = 0; d < 5; ++d) c[d] += w.inc[lvl][d];
    }
  }
  return true;
}

static bool run_plan(const TcPlan& p, size_t out_count) {
  if (p.a.nk != p.b.nk) { printf("nk mismatch\n"); return false; }
  if (!walk_matches(p.a, p.m_tiles - 1, p.k_iters) || !walk_matches(p.b, (p.pair + 1) * p.n_tiles - 1, p.k_iters)) return false;
  if (p.pair && (p.bn != 256 || p.gather_src || p.epilogue == TC_EPI_TAPS)) { printf("a pair where the kernel has none\n"); return false; }
  for (const TcOperand* o : {&p.a, &p.b}) if (o->load == TC_LOAD_IM2COL_MN && !pixel_walk_matches(*o, p.k_iters)) return false;
  // overwrite semantics under split-K: the partial results of the splits are summed and then stored; emulated by zeroing first
  if (p.splits > 1 && !p.accumulate) for (size_t i = 0; i < out_count; ++i) p.out[i] = 0.0f;
  std::vector<float> sa, sb, sc, fa(128 * 8), fb((size_t)p.bn * 8);
  // a pair's second CTA loads what stands where a row tile beyond the last one would be; nothing of it is stored
  if (p.pair && p.m_tiles % 2) {
    if (p.a.load != TC_LOAD_BOX && p.a.load != TC_LOAD_BOXES) { printf("a pair whose second row tile has no place to be read from\n"); return false; }
    for (int it = 0; it < p.k_iters; it += 7) if (!tma_load(p.a, p.m_tiles, it, sa)) return false;
  }
  for (int mt = 0; mt < p.m_tiles; ++mt) for (int nt = 0; nt < p.n_tiles; ++nt) for (int z = 0; z < p.splits; ++z) {
    int per = (p.k_iters + p.splits - 1) / p.splits, k0 = z * per, k1 = k0 + per < p.k_iters ? k0 + per : p.k_iters;
    if (k0 >= k1) continue;
    std::vector<double> D((size_t)128 * p.bn, 0.0);
    for (int it = k0; it < k1; ++it) {
      if (!(p.gather_src ? gather_load(p, mt, it, sa) : tma_load(p.a, mt, it, sa)) || !tma_load(p.b, p.pair ? 2 * nt : nt, it, sb)) return false;
      if (p.pair && !tma_load(p.b, 2 * nt + 1, it, sc)) return false;             // the other CTA's half of the columns
      for (int ks = 0; ks < p.a.nk; ++ks) {
        for (int r = 0; r < 128; ++r) for (int kk = 0; kk < 8; ++kk) fa[r * 8 + kk] = umma_fetch(p.a, sa, ks, r, kk);
        for (int c = 0; c < p.bn; ++c) for (int kk = 0; kk < 8; ++kk) fb[c * 8 + kk] = p.pair && c >= 128 ? umma_fetch(p.b, sc, ks, c - 128, kk) : umma_fetch(p.b, sb, ks, c, kk);
        for (int r = 0; r < 128; ++r) for (int c = 0; c < p.bn; ++c) {
          double s = 0; for (int kk = 0; kk < 8; ++kk) s += (double)fa[r * 8 + kk] * fb[c * 8 + kk];
          D[(size_t)r * p.bn + c] += s;
        }
      }
    }
    bool atomic = p.splits > 1;
    for (int r = 0; r < 128; ++r) for (int c = 0; c < p.bn; ++c) {
      int64_t m = (int64_t)mt * 128 + r, n = (int64_t)nt * p.bn + c;
      if (m >= p.M || n >= p.N) continue;
      int64_t idx;
      if (p.epilogue == TC_EPI_PIXEL) {
        const int64_t per = p.pix_pad ? p.pix_pad : p.pix_per_img;
        if (m % per >= p.pix_per_img) continue;                       // a row of the image's last tile beyond the image
        idx = m / per * p.img_stride + n * p.chan_stride + m % per;
      } else if (p.epilogue == TC_EPI_TAPS) {
        const int64_t q = n / 32, blk = q / p.col_mul, ch = blk * 32 + n % 32;
        if (ch >= p.col_mod) continue;                                // a channel that only fills up the last block
        idx = m * p.ld + ch * p.col_mul + q % p.col_mul;
      } else idx = m * p.ld + n;
      if ((size_t)idx >= out_count) { printf("epilogue index out of range\n"); return false; }
      float v = p.alpha * (float)D[(size_t)r * p.bn + c] + ((p.bias && z == 0) ? p.bias[n] : 0.0f);
      if (p.accumulate || atomic) p.out[idx] += v; else p.out[idx] = v;
    }
  }
  return true;
}

// The deterministic mode's sum over a cluster of splits: whatever the tile's width, the cluster's size and the part of the tile inside
// the result, its CTAs together write every output of the tile once.
static bool slices_cover() {
  for (int bn : {64, 128, 256}) for (int cz : {2, 4, 8}) for (int limit = 1; limit <= 256; ++limit) {
    std::vector<int> rows((size_t)128 * bn, 0), cols(bn, 0);
    for (int rank = 0; rank < cz; ++rank) {
      if (limit <= 128) for (int w = 0; w < 8; ++w) {
        const TcSliceRows s(TcSlice(128, cz, rank, limit), bn, w);
        for (int i = 0; i < s.items; ++i) {
          if (s.row(i) >= limit || s.run(i) >= bn / 32) { printf("slice of %d columns, %d CTAs: row %d, run %d\n", bn, cz, s.row(i), s.run(i)); return false; }
          for (int lane = 0; lane < 32; ++lane) ++rows[(size_t)s.row(i) * bn + s.run(i) * 32 + lane];
        }
      }
      const TcSlice c(bn, cz, rank, limit);
      for (int half = 0; half < 2; ++half) for (int j = c.lo + half; j < c.hi; j += 2) ++cols[j];
    }
    for (int r = 0; r < 128 && limit <= 128; ++r) for (int c = 0; c < bn; ++c)
      if (rows[(size_t)r * bn + c] != (r < limit)) { printf("tile of %d columns, %d CTAs, %d rows: (%d, %d) written %d times\n", bn, cz, limit, r, c, rows[(size_t)r * bn + c]); return false; }
    for (int c = 0; c < bn; ++c) if (cols[c] != (c < limit)) { printf("tile of %d columns, %d CTAs, %d inside: column %d written %d times\n", bn, cz, limit, c, cols[c]); return false; }
  }
  return true;
}

static std::vector<float> rnd(size_t n, unsigned seed) { std::vector<float> v(n); srand(seed); for (auto& x : v) x = (float)(rand() % 17 - 8) / 4.0f; return v; }
static bool close(const std::vector<float>& a, const std::vector<float>& b, const char* what) {
  for (size_t i = 0; i < a.size(); ++i) if (std::fabs(a[i] - b[i]) > 1e-3f * (1.0f + std::fabs(a[i]))) { printf("%s: mismatch at %zu: %f vs %f\n", what, i, a[i], b[i]); return false; }
  return true;
}

static std::map<std::string, int> pairs, split_pairs, odd_pairs;      // by planner: plans for pairs of CTAs emulated, those with splits, those of an odd number of row tiles
static bool holds(const TcPlan& p, const std::vector<float>& want, const std::vector<float>& got, const char* what) {
  if (p.pair) { ++pairs[what]; split_pairs[what] += p.splits > 1; odd_pairs[what] += p.m_tiles % 2; }
  return run_plan(p, got.size()) && close(want, got, what);
}

static int conv_case(int n_img, int ck, int co, int pix, int sms = 148) {
  auto x = rnd((size_t)n_img * ck * pix, 1), w = rnd((size_t)co * ck, 2), dy = rnd((size_t)n_img * co * pix, 3), bias = rnd(co, 4);
  // TMA bases must be 16-byte aligned: std::vector<float> storage from operator new is.
  std::vector<float> y((size_t)n_img * co * pix, 7.0f), yr(y.size()), dx((size_t)n_img * ck * pix, 0.5f), dxr(dx), dw((size_t)co * ck, -1.0f), dwr(dw);
  for (int n = 0; n < n_img; ++n) for (int c = 0; c < co; ++c) for (int q = 0; q < pix; ++q) {
    double s = bias[c]; for (int k = 0; k < ck; ++k) s += (double)w[(size_t)c * ck + k] * x[((size_t)n * ck + k) * pix + q];
    yr[((size_t)n * co + c) * pix + q] = (float)s;
  }
  for (int n = 0; n < n_img; ++n) for (int k = 0; k < ck; ++k) for (int q = 0; q < pix; ++q) {
    double s = 0; for (int c = 0; c < co; ++c) s += (double)w[(size_t)c * ck + k] * dy[((size_t)n * co + c) * pix + q];
    dxr[((size_t)n * ck + k) * pix + q] += (float)s;
  }
  for (int c = 0; c < co; ++c) for (int k = 0; k < ck; ++k) {
    double s = 0; for (int n = 0; n < n_img; ++n) for (int q = 0; q < pix; ++q) s += (double)dy[((size_t)n * co + c) * pix + q] * x[((size_t)n * ck + k) * pix + q];
    dwr[(size_t)c * ck + k] += (float)s;
  }
  int taken = 0; TcPlan p;
  const bool rows = tc_conv_needs_rows(pix);
  std::vector<float> xt, dyt;           // K-major row copies [n*pix + q][channel], what the library's transposing copy produces
  if (rows) {
    xt.resize(x.size()); dyt.resize(dy.size());
    for (int n = 0; n < n_img; ++n) for (int q = 0; q < pix; ++q) {
      for (int k = 0; k < ck; ++k) xt[((size_t)n * pix + q) * ck + k] = x[((size_t)n * ck + k) * pix + q];
      for (int c = 0; c < co; ++c) dyt[((size_t)n * pix + q) * co + c] = dy[((size_t)n * co + c) * pix + q];
    }
  }
  // filter rows padded with zeros to 4 floats, the way the library stages them
  auto padded = [&](int ld) { std::vector<float> o((size_t)co * ld, 0.0f); for (int c = 0; c < co; ++c) for (int k = 0; k < ck; ++k) o[(size_t)c * ld + k] = w[(size_t)c * ck + k]; return o; };
  const int ld4 = (ck + 3) / 4 * 4;
  const std::vector<float> w4 = padded(ld4);
  if (tc_plan_conv_fwd(p, rows ? xt.data() : x.data(), rows, w4.data(), ld4, bias.data(), y.data(), n_img, ck, co, pix, sms)) { ++taken; if (!holds(p, yr, y, "fwd")) return -1; }
  if (tc_plan_conv_dgrad(p, rows ? dyt.data() : dy.data(), rows, w4.data(), ld4, dx.data(), n_img, ck, co, pix, true, sms)) { ++taken; if (!holds(p, dxr, dx, "dgrad")) return -1; }
  // the same two contractions with the kernel gathering the activation itself (small images: 4 or 16 pixels)
  if (rows && tc_gather_possible(x.data(), ck, pix) && tc_gather_possible(dy.data(), co, pix)) {
    std::fill(y.begin(), y.end(), 7.0f); std::fill(dx.begin(), dx.end(), 0.5f);
    if (tc_plan_conv_fwd(p, x.data(), true, w4.data(), ld4, bias.data(), y.data(), n_img, ck, co, pix, sms)) {
      tc_plan_gather(p, x.data(), n_img, ck, pix); ++taken; if (!holds(p, yr, y, "fwd (gather)")) return -1; }
    if (tc_plan_conv_dgrad(p, dy.data(), true, w4.data(), ld4, dx.data(), n_img, ck, co, pix, true, sms)) {
      tc_plan_gather(p, dy.data(), n_img, co, pix); ++taken; if (!holds(p, dxr, dx, "dgrad (gather)")) return -1; }
  }
  if (tc_plan_conv_wgrad(p, x.data(), dy.data(), dw.data(), n_img, ck, co, pix, sms)) { ++taken; if (!holds(p, dwr, dw, "wgrad")) return -1; }
  printf("conv n=%d ck=%d co=%d pix=%d: %d of 3 plans (5 with the gathered ones) taken, all match\n", n_img, ck, co, pix, taken);
  return taken;
}

// Images of a size that fills no tiles, straight from x[n][k][p].
static int ragged_case(int n_img, int ck, int co, int pix, int sms = 148) {
  auto x = rnd((size_t)n_img * ck * pix, 1), w = rnd((size_t)co * ck, 2), dy = rnd((size_t)n_img * co * pix, 3), bias = rnd(co, 4);
  std::vector<float> y(dy.size(), 7.0f), yr(y.size()), dx(x.size(), 0.5f), dxr(dx), dw(w.size(), -1.0f), dwr(dw);
  for (int n = 0; n < n_img; ++n) for (int q = 0; q < pix; ++q) {
    for (int c = 0; c < co; ++c) {
      double s = bias[c]; for (int k = 0; k < ck; ++k) s += (double)w[(size_t)c * ck + k] * x[((size_t)n * ck + k) * pix + q];
      yr[((size_t)n * co + c) * pix + q] = (float)s;
    }
    for (int k = 0; k < ck; ++k) {
      double s = 0; for (int c = 0; c < co; ++c) s += (double)w[(size_t)c * ck + k] * dy[((size_t)n * co + c) * pix + q];
      dxr[((size_t)n * ck + k) * pix + q] += (float)s;
    }
  }
  for (int c = 0; c < co; ++c) for (int k = 0; k < ck; ++k) {
    double s = 0; for (int n = 0; n < n_img; ++n) for (int q = 0; q < pix; ++q) s += (double)dy[((size_t)n * co + c) * pix + q] * x[((size_t)n * ck + k) * pix + q];
    dwr[(size_t)c * ck + k] += (float)s;
  }
  const int ld = (ck + 3) / 4 * 4; std::vector<float> wp((size_t)co * ld, 0.0f);
  for (int c = 0; c < co; ++c) for (int k = 0; k < ck; ++k) wp[(size_t)c * ld + k] = w[(size_t)c * ck + k];
  int taken = 0; TcPlan p;
  if (tc_plan_conv_ragged_fwd(p, x.data(), wp.data(), ld, bias.data(), y.data(), n_img, ck, co, pix, sms)) { ++taken; if (!holds(p, yr, y, "ragged fwd")) return -1; }
  if (tc_plan_conv_ragged_dgrad(p, dy.data(), wp.data(), ld, dx.data(), n_img, ck, co, pix, true, sms)) { ++taken; if (!holds(p, dxr, dx, "ragged dgrad")) return -1; }
  if (tc_plan_conv_ragged_wgrad(p, x.data(), dy.data(), dw.data(), n_img, ck, co, pix, sms)) { ++taken; if (!holds(p, dwr, dw, "ragged wgrad")) return -1; }
  printf("ragged conv n=%d ck=%d co=%d pix=%d: %d of 3 plans taken, all match\n", n_img, ck, co, pix, taken);
  return taken;
}

// R x S convolution against a direct evaluation: through the tap-loop plans (stride 1), and through the im2col-mode plans from
// channels-last copies whose channels are padded to a multiple of 4.
static int taps_case(int n_img, int C, int K, int H, int W, int R, int S, int ph, int pw, int sh = 1, int sw = 1, int sms = 148) {
  const int oH = (H + 2 * ph - R) / sh + 1, oW = (W + 2 * pw - S) / sw + 1, taps = R * S;
  TcConvGeom g{n_img, C, H, W, K, R, S, ph, pw, oH, oW};
  auto x = rnd((size_t)n_img * C * H * W, 11), w = rnd((size_t)K * C * taps, 12), dy = rnd((size_t)n_img * K * oH * oW, 13), bias = rnd(K, 14);
  std::vector<float> y((size_t)n_img * K * oH * oW, 7.0f), yr(y.size()), dx(x.size(), 0.5f), dxr(dx), dw(w.size(), -1.0f), dwr(dw);
  auto X = [&](int n, int c, int h, int ww) -> double { return (h < 0 || h >= H || ww < 0 || ww >= W) ? 0.0 : x[(((size_t)n * C + c) * H + h) * W + ww]; };
  for (int n = 0; n < n_img; ++n) for (int k = 0; k < K; ++k) for (int oh = 0; oh < oH; ++oh) for (int ow = 0; ow < oW; ++ow) {
    double s = bias[k];
    for (int c = 0; c < C; ++c) for (int r = 0; r < R; ++r) for (int q = 0; q < S; ++q) s += X(n, c, oh * sh - ph + r, ow * sw - pw + q) * w[(((size_t)k * C + c) * R + r) * S + q];
    yr[(((size_t)n * K + k) * oH + oh) * oW + ow] = (float)s;
    const double d = dy[(((size_t)n * K + k) * oH + oh) * oW + ow];
    for (int c = 0; c < C; ++c) for (int r = 0; r < R; ++r) for (int q = 0; q < S; ++q) {
      const int h = oh * sh - ph + r, ww = ow * sw - pw + q;
      if (h < 0 || h >= H || ww < 0 || ww >= W) continue;
      dxr[(((size_t)n * C + c) * H + h) * W + ww] += (float)(d * w[(((size_t)k * C + c) * R + r) * S + q]);
      dwr[(((size_t)k * C + c) * R + r) * S + q] += (float)(d * x[(((size_t)n * C + c) * H + h) * W + ww]);
    }
  }
  // what the library's staging kernels produce: channels-last copies and per-tap weight matrices
  std::vector<float> xr(x.size()), dyr(dy.size()), wt(w.size()), wd(w.size());
  for (int n = 0; n < n_img; ++n) for (int c = 0; c < C; ++c) for (int i = 0; i < H * W; ++i) xr[((size_t)n * H * W + i) * C + c] = x[((size_t)n * C + c) * H * W + i];
  for (int n = 0; n < n_img; ++n) for (int k = 0; k < K; ++k) for (int i = 0; i < oH * oW; ++i) dyr[((size_t)n * oH * oW + i) * K + k] = dy[((size_t)n * K + k) * oH * oW + i];
  for (int k = 0; k < K; ++k) for (int c = 0; c < C; ++c) for (int t = 0; t < taps; ++t) {
    wt[((size_t)t * K + k) * C + c] = w[((size_t)k * C + c) * taps + t];
    wd[((size_t)t * C + c) * K + k] = w[((size_t)k * C + c) * taps + t];
  }
  int taken = 0; TcPlan p;
  if (sh == 1 && sw == 1) {
    if (tc_plan_conv_taps_fwd(p, xr.data(), wt.data(), bias.data(), y.data(), g, sms)) { ++taken; if (!holds(p, yr, y, "taps fwd")) return -1; }
    if (tc_plan_conv_taps_dgrad(p, dyr.data(), wt.data(), dx.data(), g, true, sms)) { ++taken; if (!holds(p, dxr, dx, "taps dgrad")) return -1; }
    if (tc_plan_conv_taps_wgrad(p, dyr.data(), xr.data(), dw.data(), g, sms)) { ++taken; if (!holds(p, dwr, dw, "taps wgrad")) return -1; }
  }
  // im2col mode; the data gradient of a strided convolution is a stride-1 one of dy with zeros between its pixels
  const int ldc = (C + 3) / 4 * 4, ldk = (K + 3) / 4 * 4, uH = H + 2 * ph - R + 1, uW = W + 2 * pw - S + 1;
  std::vector<float> xp((size_t)n_img * H * W * ldc, 0.0f), dyp((size_t)n_img * oH * oW * ldk, 0.0f), up((size_t)n_img * uH * uW * ldk, 0.0f), wtp((size_t)taps * K * ldc, 0.0f), wdp((size_t)taps * C * ldk, 0.0f);
  for (size_t i = 0; i < (size_t)n_img * H * W; ++i) for (int c = 0; c < C; ++c) xp[i * ldc + c] = xr[i * C + c];
  for (int n = 0; n < n_img; ++n) for (int a = 0; a < oH; ++a) for (int b = 0; b < oW; ++b) for (int k = 0; k < K; ++k) {
    const float v = dyr[(((size_t)n * oH + a) * oW + b) * K + k];
    dyp[(((size_t)n * oH + a) * oW + b) * ldk + k] = v; up[(((size_t)n * uH + a * sh) * uW + b * sw) * ldk + k] = v;
  }
  for (int t = 0; t < taps; ++t) for (int k = 0; k < K; ++k) for (int c = 0; c < C; ++c) {
    wtp[((size_t)t * K + k) * ldc + c] = wt[((size_t)t * K + k) * C + c]; wdp[((size_t)t * C + c) * ldk + k] = wd[((size_t)t * C + c) * K + k];
  }
  std::fill(y.begin(), y.end(), 7.0f); std::fill(dx.begin(), dx.end(), 0.5f); std::fill(dw.begin(), dw.end(), -1.0f);
  TcConvAny a{n_img, C, H, W, K, R, S, sh, sw, ph, pw, oH, oW, ldc, ldk}, u{n_img, C, H, W, K, R, S, 1, 1, ph, pw, uH, uW, ldc, ldk};
  int any = 0;
  if (tc_plan_conv_any_fwd(p, xp.data(), wtp.data(), bias.data(), y.data(), a, sms)) { ++any; if (!holds(p, yr, y, "im2col fwd")) return -1; }
  if (tc_plan_conv_any_dgrad(p, up.data(), C % 32 == 0 ? wtp.data() : wdp.data(), dx.data(), u, true, sms)) { ++any; if (!holds(p, dxr, dx, "im2col dgrad")) return -1; }
  if (tc_plan_conv_any_wgrad(p, dyp.data(), xp.data(), dw.data(), a, sms)) { ++any; if (!holds(p, dwr, dw, "im2col wgrad")) return -1; }
  if (any != 3) { printf("only %d of 3 im2col plans taken\n", any); return -1; }
  printf("taps conv n=%d C=%d K=%d %dx%d k%dx%d pad %d,%d stride %d,%d: %d of 3 window plans and 3 im2col plans taken, all match\n", n_img, C, K, H, W, R, S, ph, pw, sh, sw, taken);
  return taken;
}

static int gemm_case(int M, int N, int K, bool ak, bool bk, bool acc, int sms = 148) {
  auto a = rnd((size_t)M * K, 5), b = rnd((size_t)N * K, 6);
  std::vector<float> c((size_t)M * N, 2.0f), cr(c);
  for (int m = 0; m < M; ++m) for (int n = 0; n < N; ++n) {
    double s = 0; for (int k = 0; k < K; ++k) s += (double)(ak ? a[(size_t)m * K + k] : a[(size_t)k * M + m]) * (bk ? b[(size_t)n * K + k] : b[(size_t)k * N + n]);
    cr[(size_t)m * N + n] = (acc ? cr[(size_t)m * N + n] : 0.0f) + 0.5f * (float)s;
  }
  TcPlan p;
  const int wa = ak ? K : M, ha = ak ? M : K, wb = bk ? K : N, hb = bk ? N : K;
  if (wa % 4 == 0 && wb % 4 == 0) {
    if (!tc_plan_gemm(p, a.data(), ak, b.data(), bk, c.data(), M, N, K, 0.5f, acc, sms)) { printf("gemm %dx%dx%d ak=%d bk=%d: not eligible\n", M, N, K, ak, bk); return 0; }
    if (!holds(p, cr, c, "gemm")) return -1;
  } else {                     // rows of no whole 16-byte unit: copies padded with zeros, as the library makes them
    const int lda = (wa + 3) / 4 * 4, ldb = (wb + 3) / 4 * 4;
    std::vector<float> ap((size_t)ha * lda, 0.0f), bp((size_t)hb * ldb, 0.0f);
    for (int i = 0; i < ha; ++i) for (int j = 0; j < wa; ++j) ap[(size_t)i * lda + j] = a[(size_t)i * wa + j];
    for (int i = 0; i < hb; ++i) for (int j = 0; j < wb; ++j) bp[(size_t)i * ldb + j] = b[(size_t)i * wb + j];
    if (!tc_plan_gemm_ld(p, ap.data(), ak, lda, bp.data(), bk, ldb, c.data(), M, N, K, 0.5f, acc, sms)) { printf("gemm %dx%dx%d ak=%d bk=%d: padded copies not eligible\n", M, N, K, ak, bk); return -1; }
    if (!holds(p, cr, c, "padded gemm")) return -1;
  }
  printf("gemm %dx%dx%d ak=%d bk=%d acc=%d: bn=%d splits=%d match\n", M, N, K, ak, bk, acc, p.bn, p.splits);
  return 1;
}

// "forward splits, data-gradient splits" of a layer on 148 SMs, 0 where its plan is not for pairs of CTAs, in the order in which the library asks the planners.
static int print_pairs(char** v) {
  int n[8]; for (int i = 0; i < 8; ++i) n[i] = atoi(v[i]);
  const int N = n[0], C = n[1], H = n[2], W = n[3], K = n[4], R = n[5], st = n[6], pad = n[7], oH = (H + 2 * pad - R) / st + 1, oW = (W + 2 * pad - R) / st + 1;
  alignas(16) static float some[4];
  TcPlan f{}, d{};
  bool ok = true;
  if (R == 1 && st == 1 && tc_conv_needs_rows(H * W)) {
    ok = tc_plan_conv_ragged_fwd(f, some, some, (C + 3) / 4 * 4, nullptr, some, N, C, K, H * W, 148) && tc_plan_conv_ragged_dgrad(d, some, some, (C + 3) / 4 * 4, some, N, C, K, H * W, true, 148);
  } else if (R == 1 && st == 1) {
    ok = tc_plan_conv_fwd(f, some, false, some, (C + 3) / 4 * 4, nullptr, some, N, C, K, H * W, 148) && tc_plan_conv_dgrad(d, some, false, some, (C + 3) / 4 * 4, some, N, C, K, H * W, true, 148);
  } else {
    const TcConvGeom g{N, C, H, W, K, R, R, pad, pad, oH, oW};
    const TcConvAny a{N, C, H, W, K, R, R, st, st, pad, pad, oH, oW, (C + 3) / 4 * 4, (K + 3) / 4 * 4};
    ok = ((st == 1 && tc_plan_conv_taps_fwd(f, some, some, nullptr, some, g, 148)) || tc_plan_conv_any_fwd(f, some, some, nullptr, some, a, 148)) &&
         ((st == 1 && tc_plan_conv_taps_dgrad(d, some, some, some, g, true, 148)) || tc_plan_conv_any_dgrad(d, some, some, some, a, true, 148));
  }
  printf("%d %d\n", f.pair ? f.splits : 0, d.pair ? d.splits : 0);
  return ok ? 0 : 1;
}

int main(int argc, char** argv) {
  if (argc == 9) return print_pairs(argv + 1);
  int bad = slices_cover() ? 0 : 1, taken = 0;
  const int convs[][4] = {{2, 64, 64, 256}, {3, 64, 256, 256}, {4, 128, 96, 64}, {5, 256, 128, 64}, {11, 256, 128, 16}, {35, 512, 64, 4}, {1, 32, 48, 1024},
                          {8, 576, 64, 256}, {2, 40, 64, 32}, {3, 64, 64, 36}, {2, 2048, 512, 4}, {9, 1024, 256, 16}, {70, 512, 32, 1},
                          // filter rows that need padding (3x3 over 3, 16 and 48 channels; 1x1 over 16 and 48) and few output channels
                          {2, 27, 96, 1024}, {3, 144, 64, 256}, {4, 16, 64, 256}, {2, 48, 192, 64}, {2, 432, 192, 64}, {3, 128, 12, 64}, {5, 48, 192, 16},
                          // small images of a 3x3 or strided convolution: the kernel gathers from the unfolded matrix [n][(c, r, s)][p]
                          {3, 2304, 256, 16}, {5, 4608, 128, 4}, {2, 72, 64, 16}};
  for (auto& c : convs) { int r = conv_case(c[0], c[1], c[2], c[3]); if (r < 0) ++bad; else taken += r; }
  const int taps[][9] = {{3, 64, 64, 16, 16, 3, 3, 1, 1}, {5, 128, 128, 8, 8, 3, 3, 1, 1}, {9, 64, 128, 4, 4, 3, 3, 1, 1}, {35, 64, 64, 2, 2, 3, 3, 1, 1},
                         {1, 32, 64, 32, 32, 3, 3, 1, 1}, {2, 64, 32, 16, 16, 3, 3, 0, 0}, {2, 64, 64, 8, 8, 5, 5, 2, 2}, {3, 96, 64, 8, 8, 1, 3, 0, 1},
                         {3, 64, 128, 16, 16, 1, 1, 0, 0}};
  int taps_taken = 0;
  for (auto& c : taps) { int r = taps_case(c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8]); if (r < 0) ++bad; else { taken += r; taps_taken += r; } }
  if (taps_taken < 17) { printf("too few tap-loop plans taken (%d)\n", taps_taken); ++bad; }
  for (int ak = 0; ak < 2; ++ak) for (int bk = 0; bk < 2; ++bk) for (int acc = 0; acc < 2; ++acc) {
    int r = gemm_case(160, 96, 72, ak, bk, acc); if (r < 0) ++bad; else taken += r;
    r = gemm_case(128, 256, 2048, ak, bk, acc); if (r < 0) ++bad; else taken += r;
    r = gemm_case(68, 36, 100, ak, bk, acc); if (r < 0) ++bad; else taken += r;                 // row lengths that are no multiple of 32
    r = gemm_case(131, 17, 67, ak, bk, acc); if (r < 0) ++bad; else taken += r;                 // nor of 4
  }
  // 256-wide tiles, as small products have them on a machine of a few SMs: enough of them, and one in two splits
  { int r = gemm_case(250, 508, 520, true, true, true, 4); if (r < 0) ++bad; else taken += r; }
  { int r = gemm_case(128, 244, 3100, false, false, false, 3); if (r < 0) ++bad; else taken += r; }
  const int ragged[][4] = {{2, 64, 72, 100}, {3, 36, 24, 196}, {1, 33, 132, 68}, {2, 40, 64, 132}};
  for (auto& c : ragged) { int r = ragged_case(c[0], c[1], c[2], c[3]); if (r < 0) ++bad; else taken += r; }
  const int any[][11] = {{2, 12, 20, 7, 9, 3, 3, 1, 1, 1, 1}, {3, 40, 72, 11, 7, 3, 3, 1, 1, 2, 2}, {2, 33, 8, 9, 9, 5, 5, 2, 2, 1, 1}, {2, 64, 48, 14, 14, 1, 1, 0, 0, 2, 2},
                         {1, 96, 64, 27, 27, 5, 5, 2, 2, 1, 1}, {5, 8, 136, 5, 13, 3, 2, 0, 1, 2, 1}};
  for (auto& c : any) {
    int r = taps_case(c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8], c[9], c[10]); if (r < 0) ++bad; else taken += r;
  }
  // Pairs of CTAs, as larger layers have them on the real machine: every planner that can choose one, without splits and with, with an odd number of
  // row tiles where the planner allows that (images that a tiled load can leave out; not the im2col mode's), a last half of the columns that is not full.
  const int pair_convs[][5] = {{2, 1024, 256, 128, 2}, {2, 256, 1024, 128, 2}, {3, 2052, 252, 128, 6}, {3, 252, 2052, 128, 6}};
  for (auto& c : pair_convs) { int r = conv_case(c[0], c[1], c[2], c[3], c[4]); if (r < 0) ++bad; else taken += r; }
  const int pair_ragged[][5] = {{1, 1056, 200, 132, 2}, {1, 200, 1056, 132, 2}, {1, 2056, 200, 260, 6}, {1, 200, 2056, 260, 6}};
  for (auto& c : pair_ragged) { int r = ragged_case(c[0], c[1], c[2], c[3], c[4]); if (r < 0) ++bad; else taken += r; }
  // images, channels in and out, size, filter size, padding, stride, SMs
  const int pair_taps[][8] = {{4, 256, 256, 8, 3, 1, 1, 4}, {5, 256, 224, 8, 3, 1, 1, 6}, {5, 224, 256, 8, 3, 1, 1, 6}, {4, 256, 512, 8, 3, 1, 1, 8}, {4, 512, 256, 8, 3, 1, 1, 8}, {3, 196, 148, 9, 3, 1, 1, 2},
                              {3, 196, 252, 17, 3, 1, 2, 2}, {5, 516, 252, 7, 3, 1, 1, 8}, {5, 252, 516, 7, 3, 1, 1, 8}};
  for (auto& c : pair_taps) { int r = taps_case(c[0], c[1], c[2], c[3], c[3], c[4], c[4], c[5], c[5], c[6], c[6], c[7]); if (r < 0) ++bad; else taken += r; }
  { int r = gemm_case(380, 508, 1040, true, true, true, 4); if (r < 0) ++bad; else taken += r; }
  { int r = gemm_case(256, 244, 3100, false, false, false, 6); if (r < 0) ++bad; else taken += r; }
  for (const char* what : {"fwd", "dgrad", "ragged fwd", "ragged dgrad", "taps fwd", "taps dgrad", "im2col fwd", "im2col dgrad"}) {
    const bool im2col = !strncmp(what, "im2col", 6);
    printf("pairs of CTAs, %s: %d plans, %d split, %d with an odd number of row tiles\n", what, pairs[what], split_pairs[what], odd_pairs[what]);
    if (pairs[what] < 2 || !split_pairs[what] || pairs[what] == split_pairs[what] || (im2col ? odd_pairs[what] != 0 : !odd_pairs[what])) ++bad;
  }
  if (pairs["gemm"] < 1 || pairs["padded gemm"] + pairs["gemm"] < 2) { printf("pairs of CTAs: too few products\n"); ++bad; }
  printf("%d plans emulated, %d failures\n", taken, bad);
  return bad ? 1 : (taken >= 140 ? 0 : 2);
}
