// Hand-mirrored host programs for the reference's training apps.
//
// The Scala generator cannot run without a JVM, so each program below is written the way the staged output
// of the corresponding app is structured: parameters allocated first (before the arena mark), then per batch
// upload -> forward -> seed gradient -> backward (reverse order) -> loss read-back -> SGD over every parameter
// tensor -> arena reset.  References:
//   MNIST CNN   src/main/scala/lantern/NIPS18App/MnistCNN.scala:36-60, 168-194 and its shipped output
//               src/out/NIPS18evaluation/evaluationCNN/Lantern/Lantern.cpp
//   ResNet-50   src/main/scala/lantern/PLDI19APP/resnet50FromOnnx.scala:135-214 with the architecture of
//               src/out/PLDI19evaluation/resnet50/pytorch/resnet50.py:55-160 (op mapping ONNXLib.scala:833-1071)
//   SqueezeNet  src/main/scala/lantern/PLDI19APP/squeezenetFromOnnx.scala:111-226 with the architecture of
//               src/out/PLDI19evaluation/squeezenet/pytorch/pytorch_squeeze_cifar10.py:21-92
// The exported C functions carry the prefix given by HOST_FN (ltbh_ for the CUDA library).
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#ifdef __SSE2__
#include <emmintrin.h>
#endif

#include "loader.hpp"
#include "tape.hpp"

#ifndef HOST_FN
#define HOST_FN(name) ltbh_##name
#endif

using namespace lantern_host;

namespace {

// A batch's copy into pinned memory.  The processor never reads the copy back, so it is written with streaming stores, which leave out the
// read of the destination that an ordinary store begins with: 1.6 MB in 69 us, 93 with memcpy.  One thread is enough: the recurrent program
// at batch 256, whose batch that is, takes 124 us a step with this, 150 with memcpy, and 125 with three helper threads, which
// cost a program 0.3 ms at its first step and 0.1 ms at its close.  A small copy stays in cache and the upload reads it from there: 6 KB are on
// the device after 11.5 us (13 with streaming stores), 48 KB after 14.4 (13.1).
constexpr size_t kStreamFrom = 32u << 10;
void copy_to_staging(void* dst, const void* src, size_t bytes) {
#ifdef __SSE2__
  if (bytes >= kStreamFrom && ((uintptr_t)dst & 15) == 0) {
    __m128i* d = (__m128i*)dst; const __m128i* s = (const __m128i*)src;
    for (size_t n = bytes / 64; n > 0; --n, d += 4, s += 4) {
      const __m128i a = _mm_loadu_si128(s), b = _mm_loadu_si128(s + 1), c = _mm_loadu_si128(s + 2), e = _mm_loadu_si128(s + 3);
      _mm_stream_si128(d, a); _mm_stream_si128(d + 1, b); _mm_stream_si128(d + 2, c); _mm_stream_si128(d + 3, e);
    }
    memcpy(d, s, bytes % 64);
    _mm_sfence();                      // in memory before an upload is queued
    return;
  }
#endif
  memcpy(dst, src, bytes);
}
// A batch above this size is copied and uploaded in pieces, each queued as soon as it is in pinned memory, so that the copy of a piece runs
// beside the upload of the one before: 1.6 MB are on the device after 93 us, 108 in one piece.  Smaller pieces cost the host 2 us each.
constexpr size_t kUploadPiece = 512u << 10;

struct ParamDecl { std::vector<int> shape; int init; float scale; int64_t count; int64_t offset; bool state = false; };   // state: a running statistic, not trained (no gradient, not all-reduced)
enum { INIT_ZERO = 0, INIT_RAND = 1, INIT_ONE = 2 };

struct Model {
  virtual ~Model() {}
  std::string name;
  int batch = 0;
  int in_c = 0, in_h = 0, in_w = 0;
  int64_t label_count = 0;     // int32 targets per step (0: one per sample)
  std::vector<ParamDecl> decls;
  float* slab_x = nullptr;   // all parameter tensors, contiguous (each padded to 64 floats)
  float* slab_d = nullptr;   // their gradients, same layout
  int64_t slab_count = 0;
  void* mark = nullptr;
  float* stage_x = nullptr;  // pinned staging for the batch
  int32_t* stage_y = nullptr;
  float* loss_host = nullptr;  // pinned, 1 float
  void* graph[3] = {nullptr, nullptr, nullptr};        // the recorded step: in its general form, and reading staging pair 0 or 1 (1 + slot)
  bool use_graph = false;
  float graph_lr[3] = {0.f, 0.f, 0.f};
  size_t zero_bytes = 0;       // bytes of zero-initialised gradient buffers the largest step so far asked for (0: not known yet)
  bool early_reduce = false;   // this step runs data-parallel with an update: finished gradient ranges are summed during backward
  bool branches = true;        // independent runs of calls (shortcut convolutions) are issued as branch regions
  bool fused_cells = true;     // recursive models: one call per gate (ltb_affine_act) instead of one per operator
  bool whole_tree = true;      // tree-LSTM: the whole tree in one call each way (ltb_tree_fwd) instead of one per node
  bool whole_sequence = true;  // with fused cells: the vanilla RNN's whole unrolled sequence (ltb_rnn_seq_fwd) and a whole tree node (ltb_tree_node_fwd) in one call
  bool resident = false;       // read the batch from dev_x/dev_y instead of uploading it
  float* dev_x = nullptr; int32_t* dev_y = nullptr;
  float* dev_loss = nullptr;   // the loss of the last step, kept outside the arena span that the step resets
  // The classifier's output of the last step (CNN programs: batch x classes), copied out of the arena span that the step
  // resets so that predictions (arg-max per row) can be read afterwards.
  float* dev_logits = nullptr; int64_t logit_count = 0; TR last_logits;
  // Two steps in flight (submit / collect): staging pair p = step & 1; marker p = its upload done, marker 2 + p = its step done.
  bool feeding = false;
  int slot = -1;               // while feeding: the staging pair that the step being issued reads its batch from and leaves its loss in
  int64_t submitted = 0;
  float* feed_x[2] = {nullptr, nullptr}; int32_t* feed_y[2] = {nullptr, nullptr}; float* feed_loss = nullptr;
  float* dstage_x[2] = {nullptr, nullptr}; int32_t* dstage_y[2] = {nullptr, nullptr};   // device side of the two staging pairs (uploads run beside the step before)

  int declare(std::initializer_list<int> shape, int init, float scale = 0.f) {
    ParamDecl d; d.shape.assign(shape.begin(), shape.end()); d.init = init; d.scale = scale;
    d.count = 1; for (int s : d.shape) d.count *= s;
    d.offset = slab_count;
    slab_count += (d.count + 63) / 64 * 64;
    decls.push_back(d);
    return (int)decls.size() - 1;
  }
  TR P(int i) const {
    const ParamDecl& d = decls[i];
    TR t; t.rank = (int)d.shape.size(); for (int k = 0; k < t.rank; ++k) t.shape[k] = d.shape[k];
    t.x = slab_x + d.offset; t.d = slab_d + d.offset; return t;
  }
  // Allocation and initialisation in declaration order; rand() is consumed only by INIT_RAND tensors, in order,
  // after srand(seed) -- the order MnistCNN's generated code draws its weights in.
  void finalize(int seed) {
    slab_x = alloc_zero(slab_count);
    slab_d = alloc_zero(slab_count);
    bool first = true;
    for (auto& d : decls) {
      if (d.init == INIT_RAND) { BK(randinit)(slab_x + d.offset, d.count, d.scale, first ? seed : -1); first = false; }
      else if (d.init == INIT_ONE) BK(fill)(slab_x + d.offset, 1.0f, d.count);
    }
    if (first && seed >= 0) srand((unsigned)seed);
    if (label_count == 0) label_count = batch;
    stage_x = (float*)BK(host_alloc)((size_t)batch * in_c * in_h * in_w * 4);
    stage_y = (int32_t*)BK(host_alloc)((size_t)label_count * 4);
    loss_host = (float*)BK(host_alloc)(4);
    dev_x = alloc_value((int64_t)batch * in_c * in_h * in_w);
    dev_y = (int32_t*)BK(malloc_uninit)((size_t)label_count * 4);
    dev_loss = alloc_value(1);
    for (int p = 0; p < 2; ++p) { dstage_x[p] = alloc_value((int64_t)batch * in_c * in_h * in_w); dstage_y[p] = (int32_t*)BK(malloc_uninit)((size_t)label_count * 4); }
    if (logit_count > 0) dev_logits = alloc_value(logit_count);
    mark = BK(mark)();
  }
  virtual TR forward(Tape& t, const TR& x, const int32_t* y) = 0;
  // What became of the last step: 0, or the code of what kept it from being run, with the reason if it was this program's own (else the
  // library has it).  A step that fails leaves the parameters as they were.
  int status = 0;
  std::string reason;
  void note(int rc) { if (rc && !status) status = rc; }
  int refuse(int rc, const char* why) { status = rc; reason = why; return rc; }
  // Labels that no call may see (null: the labels are fine): they would send a kernel, or the program itself, outside an array.
  virtual const char* bad_labels(const int32_t*) { return nullptr; }
  // Data that a step draws on the host (a dropout mask): into staging block p, and from there to where the step reads it.
  virtual int draw_host_data(int) { return 0; }

  // One training step's device work, in the order of the generated programs.
  int enqueue(float lr, bool update) {
    Tape tape;
    zero_pool_begin(zero_bytes);
    int64_t nin = (int64_t)batch * in_c * in_h * in_w;
    TR x; x.rank = 4; x.shape[0] = batch; x.shape[1] = in_c; x.shape[2] = in_h; x.shape[3] = in_w; x.is_input = true;
    int32_t* y;
    if (slot >= 0) { x.x = dstage_x[slot]; y = dstage_y[slot]; }
    else if (resident) {      // batch already in device memory (measurement of the device-side step alone)
      x.x = dev_x; y = dev_y;
    } else {                  // the generated programs upload every batch: resnet50FromOnnx.scala:173-174
      x.x = alloc_value(nin);
      y = (int32_t*)BK(malloc_uninit)((size_t)label_count * 4);
      BK(h2d)(x.x, stage_x, (size_t)nin * 4);
      BK(h2d)(y, stage_y, (size_t)label_count * 4);
    }
    early_reduce = update && BK(comm_world)() > 1;
    last_logits = TR();
    TR loss = forward(tape, x, y);
    if (status) { zero_pool_end(); BK(reset)(mark); return status; }
    if (dev_logits && last_logits.x && last_logits.count() == logit_count) BK(d2d)(dev_logits, last_logits.x, (size_t)logit_count * 4);
    if (slot < 0) BK(d2d)(dev_loss, loss.x, 4);
    BK(fill)(loss.d, 1.0f, 1);                       // gradR_loss: y.d.setAsOne(), TD.scala:1763-1780
    tape.backward();
    if (slot >= 0) BK(d2h_async)(feed_loss + slot, loss.x, 4);
    else BK(d2h_async)(loss_host, dev_loss, 4);
    if (update && !status) apply_update(lr);
    if (tracing()) dump_trace();
    { const size_t asked = zero_pool_end(); if (asked > zero_bytes) zero_bytes = asked; }   // the largest step so far: a smaller tree leaves part of the block unused
    BK(reset)(mark);
    return status;
  }
  // Data parallelism: pushed on the tape at a point of the forward pass, this fires in the backward pass once every layer
  // after that point is done, i.e. when the gradients of the parameters declared from `first_decl` up to offset `hi` of the
  // slab are final; their all-reduce then overlaps the rest of the backward pass (measured on 2 GPUs: 5.64 -> 5.47 ms per step).
  void reduce_when_final(Tape& t, int first_decl, int64_t hi) {
    if (!early_reduce) return;
    float* d = slab_d + decls[first_decl].offset; const int64_t n = hi - decls[first_decl].offset;
    t.push([=] { BK(allreduce_begin)(d, n); });
  }
  // SGD of the CNN apps (NNModule.scala:265-287: geam x -= lr*d, then d = 0), fused with the gradient all-reduce when the
  // communicator has more than one rank.
  virtual void apply_update(float lr) {
    if (BK(comm_world)() > 1) BK(allreduce_sgd_step)(slab_x, slab_d, lr, slab_count);
    else BK(sgd_step)(slab_x, slab_d, lr, slab_count);
  }
  std::string trace_text;
  // One line per operator output, in forward order (read back before the reset): index, element count, shape, sum|x|,
  // sum|d|, non-zero counts, smallest non-zero |x|, then sum x^2, sum d^2 and eight signed sums of x and of d.  A signed sum
  // is sum_i s_k(i) v_i with s_k(i) = +-1 from a fixed hash of (i, k): for two tensors a, b the mean over k of
  // (S_k(a) - S_k(b))^2 estimates |a - b|^2, so two libraries can be compared tensor by tensor from these few numbers.
  void dump_trace() {
    trace_text.clear();
    std::vector<float> h;
    int idx = 0;
    for (const TR& t : trace_list()) {
      int64_t n = t.count(); h.resize((size_t)n);
      double ax = 0, ad = 0, minx = 1e30, x2 = 0, d2 = 0, px[8] = {0}, pd[8] = {0}; long long nzx = 0, nzd = 0;
      auto signs = [](int64_t i) { uint64_t z = (uint64_t)i + 0x9E3779B97F4A7C15ull; z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull; z = (z ^ (z >> 27)) * 0x94D049BB133111EBull; return z ^ (z >> 31); };
      BK(d2h)(h.data(), t.x, (size_t)n * 4);
      for (int64_t i = 0; i < n; ++i) {
        const double v = h[i], a = std::fabs(v); ax += a; x2 += v * v; if (a != 0) { ++nzx; if (a < minx) minx = a; }
        const uint64_t s = signs(i); for (int k = 0; k < 8; ++k) px[k] += ((s >> k) & 1) ? v : -v;
      }
      if (t.d) {
        BK(d2h)(h.data(), t.d, (size_t)n * 4);
        for (int64_t i = 0; i < n; ++i) {
          const double v = h[i]; ad += std::fabs(v); d2 += v * v; nzd += h[i] != 0;
          const uint64_t s = signs(i); for (int k = 0; k < 8; ++k) pd[k] += ((s >> (8 + k)) & 1) ? v : -v;
        }
      }
      char line[1024];
      int w = snprintf(line, sizeof line, "%d %lld [%d,%d,%d,%d] %.9e %.9e %lld %lld %.3e %.9e %.9e", idx++, (long long)n, t.shape[0], t.shape[1], t.shape[2], t.shape[3], ax, ad, nzx, nzd, minx, x2, d2);
      for (int k = 0; k < 8; ++k) w += snprintf(line + w, sizeof line - w, " %.9e", px[k]);
      for (int k = 0; k < 8; ++k) w += snprintf(line + w, sizeof line - w, " %.9e", pd[k]);
      snprintf(line + w, sizeof line - w, "\n");
      trace_text += line;
    }
    trace_list().clear();
  }
  void load(const float* xh, const int32_t* yh) {
    copy_to_staging(stage_x, xh, (size_t)batch * in_c * in_h * in_w * 4);
    memcpy(stage_y, yh, (size_t)label_count * 4);
  }
  void drop_graphs() { for (void*& rec : graph) if (rec) { BK(graph_destroy)(rec); rec = nullptr; } }
  int step_async(const float* xh, const int32_t* yh, float lr, bool update) {
    status = 0; reason.clear();
    return status = issue_step(xh, yh, lr, update);
  }
  int issue_step(const float* xh, const int32_t* yh, float lr, bool update) {
    if (!resident && xh) {
      if (const char* why = bad_labels(yh)) return refuse(LTB_E_ARG, why);
      load(xh, yh);
    }
    if (!feeding && draw_host_data(0)) return LTB_E_CUDA;
    if (use_graph && update && zero_bytes > 0) {        // the first step runs eagerly: it measures the gradient pool
      void*& rec = graph[1 + slot];
      if (rec && graph_lr[1 + slot] != lr) { BK(graph_destroy)(rec); rec = nullptr; }
      if (!rec) {
        int rc = BK(graph_begin)(); if (rc) return rc;
        rc = enqueue(lr, true);
        rec = BK(graph_end)(); graph_lr[1 + slot] = lr;
        if (!rec) return LTB_E_CUDA;
        if (rc) { BK(graph_destroy)(rec); rec = nullptr; return rc; }
      }
      return BK(graph_launch)(rec);
    }
    return enqueue(lr, update);
  }
  // The loss of this batch, a NaN if the step failed (`status` tells one from the loss of a diverged network).
  float step(const float* xh, const int32_t* yh, float lr, bool update) {
    step_async(xh, yh, lr, update);
    note(BK(sync)());
    return status ? NAN : *loss_host;
  }
  // Training with two steps in flight.  The generated programs upload a batch, run the step and block on the loss copy
  // (resnet50FromOnnx.scala:173-186), so the device idles while the host prepares the next batch.  submit() copies the
  // batch into one of two pinned staging pairs, queues the upload and the step, and returns; collect(k) waits for
  // step k alone.  The staging pair of step k is refilled by step k + 2, after its upload marker has fired.  A step is recorded
  // once per pair: it reads the batch where the upload puts it and leaves its loss in the pair's pinned word.  (One recording
  // for both, with the batch, its labels and the loss copied to and from fixed addresses around it: five more nodes a step,
  // each 2 to 4 us on the device between two kernels: the RNN of one row 90 -> 74 us a step, the MNIST CNN 185 -> 163.  The second recording costs
  // the host as much again as the first, once a program and once a change of the learning rate: 2.4 ms for ResNet-50, 0.9 for SqueezeNet, 0.34 for the
  // MNIST CNN, 0.1 to 0.2 for the RNN, part of it beside the step on the device; five to a hundred steps earn it back.)
  void feed_mode(bool on) {
    if (feeding == on) return;
    drop_graphs();
    if (on && !feed_loss) {
      const size_t xb = (size_t)batch * in_c * in_h * in_w * 4;
      for (int p = 0; p < 2; ++p) { feed_x[p] = (float*)BK(host_alloc)(xb); feed_y[p] = (int32_t*)BK(host_alloc)((size_t)label_count * 4); }
      feed_loss = (float*)BK(host_alloc)(8);
    }
    BK(sync)();
    if (!on && submitted) *loss_host = feed_loss[(submitted - 1) & 1];
    feeding = resident = on;
  }
  // Staging pair for the next submit, free to be written (a loader decodes a batch straight into it).
  int feed_slot(float** x, int32_t** y) {
    feed_mode(true);
    const int p = (int)(submitted & 1);
    if (submitted >= 2) { int rc = BK(marker_wait)(p); if (rc) return rc; }
    *x = feed_x[p]; *y = feed_y[p];
    return 0;
  }
  // xh == nullptr: the caller has filled the pair returned by feed_slot.
  int64_t submit(const float* xh, const int32_t* yh, float lr) {
    float* sx; int32_t* sy;
    status = 0; reason.clear();
    if (feed_slot(&sx, &sy)) return -1;
    if (const char* why = bad_labels(xh ? yh : sy)) { refuse(LTB_E_ARG, why); return -1; }
    const int p = (int)(submitted & 1);
    const size_t xb = (size_t)batch * in_c * in_h * in_w * 4;
    if (draw_host_data(p)) return -1;
    // The upload runs on the copy stream beside the step before it (marker 2 + p: step submitted - 2, the last one that read the
    // device staging pair, is done; marker p: the upload has left the host staging pair); the compute stream then waits for the
    // upload on the device.
    const size_t yb = (size_t)label_count * 4;
    int after = submitted >= 2 ? 2 + p : -1;
    if (xh) {
      memcpy(sy, yh, yb);
      for (size_t at = 0; at < xb; at += kUploadPiece, after = -1) {
        const size_t n = xb - at < kUploadPiece ? xb - at : kUploadPiece;
        copy_to_staging((char*)sx + at, (const char*)xh + at, n);
        if (BK(upload)((char*)dstage_x[p] + at, (const char*)sx + at, n, after)) return -1;
      }
    } else if (BK(upload)(dstage_x[p], sx, xb, after)) return -1;
    if (BK(upload)(dstage_y[p], sy, yb, -1) || BK(upload_marker)(p)) return -1;
    if (BK(stream_wait_marker)(p)) return -1;
    slot = p;
    const int rc = step_async(nullptr, nullptr, lr, true);
    slot = -1;
    if (rc || BK(marker_record)(2 + p)) return -1;
    return submitted++;
  }
  int collect(int64_t k, float* loss) {
    if (k < 0 || k >= submitted || k + 2 < submitted) return LTB_E_ARG;     // only the last two steps keep their loss
    const int p = (int)(k & 1);
    int rc = BK(marker_wait)(2 + p); if (rc) return rc;
    *loss = feed_loss[p];
    return 0;
  }
};

// ------------------------------------------------------------------------------------------------ MNIST CNN
struct Mnist : Model {
  int c1w, c1b, c2w, c2b, l1w, l1b, l2w, l2b;
  // The dropout mask is drawn by the host ahead of the step, in the order Backend.dropout draws it (rand() per element, kept when
  // above the rate, TensorDslCPU.scala:1066-1088), so that the step itself touches the host nowhere and can be recorded (the step
  // issued call by call took 210 us, most of it launches).
  static constexpr float kRate = 0.5f;
  float* mask_host[2] = {nullptr, nullptr}; float* mask_stage[2] = {nullptr, nullptr}; float* mask_dev = nullptr;
  Mnist(int b, int seed) {
    name = "mnist"; batch = b; in_c = 1; in_h = in_w = 28; logit_count = (int64_t)b * 10;
    // Conv2D: uniform(+-sqrt(6/fan_in)) == (rand-0.5)*2*sqrt(6/fan_in), bias 0 (NNModule.scala:128-146);
    // Linear1D: (rand-0.5)/sqrt(in), weight stored [in,out] (NNModule.scala:112-117).
    c1w = declare({10, 1, 5, 5}, INIT_RAND, 2.0f * sqrtf(6.0f / 25.0f));  c1b = declare({10}, INIT_ZERO);
    c2w = declare({20, 10, 5, 5}, INIT_RAND, 2.0f * sqrtf(6.0f / 250.0f)); c2b = declare({20}, INIT_ZERO);
    l1w = declare({320, 50}, INIT_RAND, 1.0f / sqrtf(320.0f)); l1b = declare({50}, INIT_ZERO);
    l2w = declare({50, 10}, INIT_RAND, 1.0f / sqrtf(50.0f));   l2b = declare({10}, INIT_ZERO);
    finalize(seed);
    for (int p = 0; p < 2; ++p) { mask_host[p] = (float*)BK(host_alloc)((size_t)b * 50 * 4); mask_stage[p] = alloc_value((int64_t)b * 50); }
    mask_dev = alloc_value((int64_t)b * 50);
    mark = BK(mark)();                   // allocated after the mark was taken: move the mark above them
  }
  ~Mnist() override { for (int p = 0; p < 2; ++p) BK(host_free)(mask_host[p]); }
  int draw_host_data(int p) override {
    const int64_t n = (int64_t)batch * 50;
    if (!feeding) { int rc = BK(sync)(); if (rc) return rc; }           // the staging block may still be on its way
    const float scale = 1.0f / (1.0f - kRate);
    for (int64_t i = 0; i < n; ++i) mask_host[p][i] = ((float)rand() / RAND_MAX > kRate) ? scale : 0.0f;
    if (!feeding) return BK(h2d)(mask_dev, mask_host[p], (size_t)n * 4);
    // beside the step before, as the batch (Model::submit): staging block p was read for the last time by step submitted - 2
    int rc = BK(upload)(mask_stage[p], mask_host[p], (size_t)n * 4, submitted >= 2 ? 2 + p : -1);
    return rc ? rc : BK(upload_marker)(p);                              // marker p: the whole staging pair has left, mask included
  }
  TR forward(Tape& t, const TR& x, const int32_t* y) override {   // MnistCNN.scala:43-59
    TR b1 = P(c1b), b2 = P(c2b);
    TR s0 = t.conv(x, P(c1w), &b1, 1, 0);
    TR s1 = t.max_pool(t.relu(s0, false), 2, 2);
    TR s2 = t.conv(s1, P(c2w), &b2, 1, 0);
    TR s25 = t.max_pool(t.relu(s2, false), 2, 2);
    TR flat = view(s25, {batch, 320});
    TR s3 = t.dropout_masked(t.plus_bias(t.dot(flat, P(l1w)), P(l1b)), slot >= 0 ? mask_stage[slot] : mask_dev);
    TR out = t.plus_bias(t.dot(s3, P(l2w)), P(l2b));
    last_logits = out;
    return t.sum(t.nll(t.log_softmax(out), y));
  }
};

// ------------------------------------------------------------------------------------------------ min-char-rnn
// Vanilla RNN of NNModule.scala:189-200 (VanillaRNNCell = Linear1D2 + tanh, Linear1D) unrolled by DynamicRNNFix
// (NNModule.scala:240-253) as the app VanillaRNN.scala:187-291 uses it: vocabulary 80 one-hot inputs x[T][B][80],
// hidden 100, T = 20 steps, per step  h = tanh(x_t.W1 + h.W2 + b);  o = h.Wo (+)= bo;  loss += sum(nll(logSoftmax(o), y_t));
// Adagrad lr-as-given, clip 5.  The targets arrive as y[t][b] (the generated code gathers them per step from a
// [b][t] host array, NNModule.scala:246-248; the order of the buffer is this host program's choice).
struct VanillaRnn : Model {
  static constexpr int T = 20;
  const int V, Hd;                  // 80 / 100 for the benchmark configuration; 26 / 50 in the reference's shipped generated program
  int w1, w2, bh, wo, bo;
  float* slab_h = nullptr;          // Adagrad accumulators, same layout as the parameter slab
  VanillaRnn(int b, int seed, int vocab, int hidden) : V(vocab), Hd(hidden) {
    name = "rnn"; batch = b; in_c = T; in_h = 1; in_w = V; label_count = (int64_t)T * b;
    w1 = declare({V, Hd}, INIT_RAND, 1.0f / sqrtf((float)V));   w2 = declare({Hd, Hd}, INIT_RAND, 1.0f / sqrtf((float)Hd));
    bh = declare({Hd}, INIT_ZERO);
    wo = declare({Hd, V}, INIT_RAND, 1.0f / sqrtf((float)Hd));  bo = declare({V}, INIT_ZERO);
    finalize(seed);
    slab_h = alloc_zero(slab_count);   // allocated after the mark was taken: move the mark above it
    mark = BK(mark)();
  }
  TR forward(Tape& t, const TR& x, const int32_t* y) override {
    if (fused_cells && whole_sequence)                 // all T steps in one call (ltb_rnn_seq_fwd / _bwd): 4 launches per sequence
      return t.rnn_sequence(x, y, P(w1), P(w2), P(bh), P(wo), P(bo), T, batch);
    TR h = make({batch, Hd});                          // cell.init: zeros
    BK(fill)(h.x, 0.0f, h.count());
    TR loss = make({1});
    BK(fill)(loss.x, 0.0f, 1);
    for (int s = 0; s < T; ++s) {
      TR xt; xt.rank = 2; xt.shape[0] = batch; xt.shape[1] = V; xt.x = x.x + (int64_t)s * batch * V; xt.is_input = true;
      TR o;
      if (fused_cells) {       // the cell and the output layer as one call each (ltb_affine_act_rows)
        TR w2t = P(w2);
        h = t.affine_act_rows(LTB_TANH, xt, P(w1), &h, &w2t, P(bh));
        o = t.affine_act_rows(-1, h, P(wo), nullptr, nullptr, P(bo));
      } else {
        TR pre = t.binary(LTB_ADD, t.binary(LTB_ADD, t.dot(xt, P(w1)), t.dot(h, P(w2))), P(bh));
        h = t.unary(LTB_TANH, pre);
        o = t.plus_bias(t.dot(h, P(wo)), P(bo));
      }
      loss = t.binary(LTB_ADD, loss, t.sum(t.nll(t.log_softmax(o), y + (int64_t)s * batch)));
    }
    return loss;
  }
  void apply_update(float lr) override {               // NNModule.scala:289-295 -> Backend.adagrad_update (TD.scala:377)
    BK(adagrad_update)(slab_x, slab_d, slab_h, lr, 5.0f, 1, slab_count);
  }
};

// ------------------------------------------------------------------------------------------------ TreeLSTM (sentiment)
// PLDI19APP/SentimentTreeLSTM.scala:67-146: Leaf (3 gates from a 300-d embedding), Node (5 gates from the two children),
// Out (5-way classifier at every node), recursion LOOPTM over the (lch, rch) arrays from node 0, losses added up the
// tree, Adagrad lr-as-given with the default clip 1.0 over the 22 tensors, one tree per step.
// One quirk of the app is kept on purpose: Leaf and Node return ArrayBuffer(hidden, cell) and the caller destructures it
// as ArrayBuffer(cell, hidden) (lines 131 and 135), so the classifier reads the cell state and the children's two states
// reach the parent with their roles exchanged.  This program does exactly the same.
// A step's "labels" carry the tree: y[0] = node count n <= 99, then four arrays with a stride of 99 ints: scores (0..4),
// words (row of the embedding table), left child, right child (-1 = none; node 0 is the root).  The embedding table
// (1000 rows x 300, N(0, 0.1), fixed seed) stands in for the GloVe file the app reads; it is data, not a parameter.
struct TreeLstm : Model {
  static constexpr int E = 300, Hd = 150, O = 5, MAXN = 99, VOCAB = 1000;
  int Wi, bi, Wo, bo, Wu, bu;
  int U0i, U1i, bbi, U00f, U01f, U10f, U11f, bbf, U0o, U1o, bbo, U0u, U1u, bbu;
  int Why, by;
  float* slab_h = nullptr;
  float* table = nullptr;
  struct State { TR loss, first, second; };   // the app's ArrayBuffer(loss, "hidden", "cell") with its exchanged roles
  // pldi19 == false: the earlier NIPS18App/SentimentTreeLSTM.scala:118-170, whose generated program ships under
  // src/out/NIPS18evaluation/evaluationTreeLSTM/Lantern/Lantern.cpp: the same cell without the exchanged roles, and a
  // hand-written Adagrad loop without gradient clipping.
  const bool pldi19;

  TreeLstm(int, int seed, bool pldi19_variant) : pldi19(pldi19_variant) {
    name = "treelstm"; batch = 1; in_c = in_h = in_w = 1; label_count = 1 + 4 * MAXN;
    auto W = [&](int r, int c) { return declare({r, c}, INIT_RAND, 0.01f); };
    auto Z = [&](int n) { return declare({n}, INIT_ZERO); };
    Wi = W(Hd, E); bi = Z(Hd); Wo = W(Hd, E); bo = Z(Hd); Wu = W(Hd, E); bu = Z(Hd);
    U0i = W(Hd, Hd); U1i = W(Hd, Hd); bbi = Z(Hd);
    U00f = W(Hd, Hd); U01f = W(Hd, Hd); U10f = W(Hd, Hd); U11f = W(Hd, Hd); bbf = Z(Hd);
    U0o = W(Hd, Hd); U1o = W(Hd, Hd); bbo = Z(Hd);
    U0u = W(Hd, Hd); U1u = W(Hd, Hd); bbu = Z(Hd);
    Why = W(O, Hd); by = Z(O);
    finalize(seed);
    slab_h = alloc_zero(slab_count);
    table = alloc_value((int64_t)VOCAB * E);
    {
      std::vector<float> h((size_t)VOCAB * E);
      uint64_t st = 0x9E3779B97F4A7C15ull;              // own generator: the weights' rand() stream stays untouched
      auto u01 = [&]() { st = st * 6364136223846793005ull + 1442695040888963407ull; return (double)((st >> 11) + 1) / 9007199254740993.0; };
      for (size_t i = 0; i + 1 < h.size() + 1; i += 2) {
        const double r = std::sqrt(-2.0 * std::log(u01())), a = 6.283185307179586 * u01();
        h[i] = (float)(0.1 * r * std::cos(a)); if (i + 1 < h.size()) h[i + 1] = (float)(0.1 * r * std::sin(a));
      }
      BK(h2d)(table, h.data(), h.size() * 4); BK(sync)();
    }
    mark = BK(mark)();
  }
  // With fused cells (the default) a gate is one call forward and one backward (ltb_affine_act) instead of the five and
  // about eight small kernels of the operator-by-operator form, which is kept for comparison (model_use_fused_cells).
  TR gate(Tape& t, int op, int W0, const TR& a, int W1, const TR& b, int bias) {      // (W0.a plusBias W1.b plusBias bias).op
    if (fused_cells) { TR w1 = P(W1); return t.affine_act(op, P(W0), a, &w1, &b, P(bias)); }
    return t.unary(op, t.plus_bias(t.plus_bias(t.dot(P(W0), a), t.dot(P(W1), b)), P(bias)));
  }
  TR leaf_gate(Tape& t, int op, int W, const TR& e, int bias) {                       // (W.e plusBias bias).op
    if (fused_cells) return t.affine_act(op, P(W), e, nullptr, nullptr, P(bias));
    return t.unary(op, t.plus_bias(t.dot(P(W), e), P(bias)));
  }
  TR out(Tape& t, const TR& in, const int32_t* score) {                              // Out.apply, lines 111-118
    TR pred = fused_cells ? t.affine_act(-1, P(Why), in, nullptr, nullptr, P(by)) : t.plus_bias(t.dot(P(Why), in), P(by));
    return t.nll(t.log_softmax(view(pred, {1, O})), score);
  }
  std::vector<State> known;                  // of the nodes visited so far, for one that is the child of two
  std::vector<char> visited;
  const State& visit(Tape& t, const int32_t* host, const int32_t* dev, int i) {
    if (!visited[i]) { State s = node(t, host, dev, i); known[i] = s; visited[i] = 1; }
    return known[i];
  }
  State node(Tape& t, const int32_t* host, const int32_t* dev, int i) {
    const int32_t *scores = dev + 1, *words = host + 1 + MAXN, *lch = host + 1 + 2 * MAXN, *rch = host + 1 + 3 * MAXN;
    State s;
    if (fused_cells && whole_sequence) {               // the whole node in one call forward and one backward (ltb_tree_node_fwd / _bwd)
      TR none, W[5][2], bias[5];
      Tape::NodeOut o;
      if (lch[i] < 0) {
        TR e; e.rank = 1; e.shape[0] = E; e.x = table + (int64_t)words[i] * E; e.is_input = true;
        W[0][0] = P(Wi); W[3][0] = P(Wo); W[4][0] = P(Wu); bias[0] = P(bi); bias[3] = P(bo); bias[4] = P(bu);
        o = t.tree_node(false, pldi19, e, nullptr, W, bias, nullptr, nullptr, P(Why), P(by), scores + i, nullptr, nullptr);
      } else {
        State l = visit(t, host, dev, lch[i]), r = visit(t, host, dev, rch[i]);
        W[0][0] = P(U0i); W[0][1] = P(U1i); W[1][0] = P(U00f); W[1][1] = P(U01f); W[2][0] = P(U10f); W[2][1] = P(U11f);
        W[3][0] = P(U0o); W[3][1] = P(U1o); W[4][0] = P(U0u); W[4][1] = P(U1u);
        bias[0] = P(bbi); bias[1] = P(bbf); bias[2] = P(bbf); bias[3] = P(bbo); bias[4] = P(bbu);
        o = t.tree_node(true, pldi19, l.first, &r.first, W, bias, &l.second, &r.second, P(Why), P(by), scores + i, &l.loss, &r.loss);
      }
      s.loss = o.loss;
      s.first = pldi19 ? o.cell : o.hidden; s.second = pldi19 ? o.hidden : o.cell;   // the PLDI19 application's exchanged roles
      return s;
    }
    if (lch[i] < 0) {                                                                // leaf, lines 72-85 and 130-133
      TR e; e.rank = 1; e.shape[0] = E; e.x = table + (int64_t)words[i] * E; e.is_input = true;
      TR ig = leaf_gate(t, LTB_SIGMOID, Wi, e, bi);
      TR og = leaf_gate(t, LTB_SIGMOID, Wo, e, bo);
      TR uv = leaf_gate(t, LTB_TANH, Wu, e, bu);
      TR cell, hidden;
      if (fused_cells) t.lstm_cell(ig, uv, nullptr, nullptr, nullptr, nullptr, og, &cell, &hidden);
      else { cell = t.binary(LTB_MUL, ig, uv); hidden = t.binary(LTB_MUL, og, t.unary(LTB_TANH, cell)); }
      if (!pldi19) { s.loss = out(t, hidden, scores + i); s.first = hidden; s.second = cell; return s; }
      // val ArrayBuffer(cell', hidden') = leaf(...): cell' = hidden, hidden' = cell
      s.loss = out(t, /*hidden'*/ cell, scores + i);
      s.first = /*hidden'*/ cell; s.second = /*cell'*/ hidden;
      return s;
    }
    State l = visit(t, host, dev, lch[i]), r = visit(t, host, dev, rch[i]);
    const TR &hl = l.first, &cl = l.second, &hr = r.first, &cr = r.second;           // ArrayBuffer(loss, hiddenl, celll) = l
    TR ig = gate(t, LTB_SIGMOID, U0i, hl, U1i, hr, bbi);
    TR fl = gate(t, LTB_SIGMOID, U00f, hl, U01f, hr, bbf);
    TR fr = gate(t, LTB_SIGMOID, U10f, hl, U11f, hr, bbf);
    TR og = gate(t, LTB_SIGMOID, U0o, hl, U1o, hr, bbo);
    TR uv = gate(t, LTB_TANH, U0u, hl, U1u, hr, bbu);
    TR cell, hidden;
    if (fused_cells) t.lstm_cell(ig, uv, &fl, &cl, &fr, &cr, og, &cell, &hidden);
    else {
      cell = t.plus_bias(t.plus_bias(t.binary(LTB_MUL, ig, uv), t.binary(LTB_MUL, fl, cl)), t.binary(LTB_MUL, fr, cr));
      hidden = t.binary(LTB_MUL, og, t.unary(LTB_TANH, cell));
    }
    if (!pldi19) {        // loss = lossl + lossr + nll, NIPS18App/SentimentTreeLSTM.scala:158
      s.loss = t.binary(LTB_ADD, t.binary(LTB_ADD, l.loss, r.loss), out(t, hidden, scores + i));
      s.first = hidden; s.second = cell;
      return s;
    }
    s.loss = t.plus_bias(t.plus_bias(out(t, /*hidden'*/ cell, scores + i), l.loss), r.loss);
    s.first = cell; s.second = hidden;
    return s;
  }
  // Whether node 0 is the root of a tree of all n nodes, as the whole-tree call takes them.  The labels may also say less (nodes that node 0 does not
  // reach, which have no part in the loss) or more (a node under two parents, whose loss counts twice): such a step goes node by node from node 0.
  static bool is_one_tree(const int32_t* host, int n) {
    const int32_t *lch = host + 1 + 2 * MAXN, *rch = host + 1 + 3 * MAXN;
    int parents[MAXN] = {};
    for (int i = 0; i < n; ++i) if (lch[i] >= 0) { ++parents[lch[i]]; ++parents[rch[i]]; }
    for (int i = 1; i < n; ++i) if (parents[i] != 1) return false;
    return parents[0] == 0;
  }
  // The whole tree in one call each way (ltb_tree_fwd / _bwd): the nodes sorted by height (node 0 is the last), their links uploaded once.
  ltb_tree tree = {};
  std::vector<int32_t> topo;                       // kept until the backward call has been issued
  TR forward_tree(Tape& t, const int32_t* host, int n) {
    const int32_t *scores = host + 1, *words = host + 1 + MAXN, *lch = host + 1 + 2 * MAXN, *rch = host + 1 + 3 * MAXN;
    std::vector<int> height(n, -1), pos(n);
    std::function<int(int)> hgt = [&](int i) -> int {
      if (height[i] >= 0) return height[i];
      if (lch[i] < 0) return height[i] = 0;
      const int a = hgt(lch[i]), b = hgt(rch[i]);
      return height[i] = 1 + (a > b ? a : b);
    };
    int top = 0;
    for (int i = 0; i < n; ++i) { const int h = hgt(i); if (h > top) top = h; }
    topo.assign((size_t)4 * n + top + 2, 0);
    int32_t *left = topo.data(), *right = left + n, *score = right + n, *word = score + n, *first = word + n;
    for (int i = 0; i < n; ++i) ++first[height[i] + 1];
    for (int h = 0; h <= top; ++h) first[h + 1] += first[h];
    { std::vector<int> fill(first, first + top + 1); for (int i = 0; i < n; ++i) pos[i] = fill[height[i]]++; }
    for (int i = 0; i < n; ++i) {
      const int q = pos[i]; const bool inner = lch[i] >= 0;
      left[q] = inner ? pos[lch[i]] : -1; right[q] = inner ? pos[rch[i]] : -1; score[q] = scores[i]; word[q] = words[i];
    }
    tree = ltb_tree{};
    tree.nodes = n; tree.levels = top + 1; tree.hidden = Hd; tree.in_len = E; tree.classes = O; tree.classify_cell = pldi19 ? 1 : 0;
    auto leaf = [&](int slot, int w, int b) { tree.leaf_W[slot] = P(w).x; tree.leaf_dW[slot] = P(w).d; tree.leaf_bias[slot] = P(b).x; tree.leaf_dbias[slot] = P(b).d; };
    auto gate_of = [&](int slot, int w0, int w1, int b) {
      tree.W[slot][0] = P(w0).x; tree.W[slot][1] = P(w1).x; tree.dW[slot][0] = P(w0).d; tree.dW[slot][1] = P(w1).d; tree.bias[slot] = P(b).x; tree.dbias[slot] = P(b).d;
    };
    leaf(0, Wi, bi); leaf(3, Wo, bo); leaf(4, Wu, bu);
    gate_of(0, U0i, U1i, bbi); gate_of(1, U00f, U01f, bbf); gate_of(2, U10f, U11f, bbf); gate_of(3, U0o, U1o, bbo); gate_of(4, U0u, U1u, bbu);
    { const TR w = P(Why), b = P(by); tree.Why = w.x; tree.dWhy = w.d; tree.by = b.x; tree.dby = b.d; }
    tree.table = table;
    const int64_t vstride = LTB_TREE_VALUES(Hd), gstride = LTB_TREE_GRADS(Hd);
    tree.values = alloc_value(n * vstride); tree.grads = alloc_zero(n * gstride);
    int32_t* dev = (int32_t*)BK(malloc_uninit)(topo.size() * 4);
    BK(h2d)(dev, topo.data(), topo.size() * 4);
    tree.topo_host = topo.data(); tree.topo = dev;
    note(BK(tree_fwd)(&tree));
    t.push([this] { note(BK(tree_bwd)(&tree)); });
    TR loss; loss.rank = 1; loss.shape[0] = 1;
    loss.x = tree.values + (n - 1) * vstride + 8 * LTB_TREE_PITCH(Hd) + 32; loss.d = tree.grads + (n - 1) * gstride + 2 * LTB_TREE_PITCH(Hd);
    return loss;
  }
  // Every node, whether node 0 reaches it or not: links inside the arrays and round no circle, scores of the classifier, words of the table.
  const char* bad_labels(const int32_t* host) override {
    const int n = host[0];
    if (n < 1 || n > MAXN) return nullptr;             // an empty step
    const int32_t *scores = host + 1, *words = host + 1 + MAXN, *lch = host + 1 + 2 * MAXN, *rch = host + 1 + 3 * MAXN;
    int parents[MAXN] = {}, top[MAXN], left = 0;
    for (int i = 0; i < n; ++i) {
      if (scores[i] < 0 || scores[i] >= O) return "a score outside the classes";
      if (lch[i] < 0) { if (words[i] < 0 || words[i] >= VOCAB) return "a leaf's word outside the embedding table"; continue; }
      if (lch[i] >= n || rch[i] < 0 || rch[i] >= n) return "a child outside the tree";
      ++parents[lch[i]]; ++parents[rch[i]];
    }
    for (int i = 0; i < n; ++i) if (!parents[i]) top[left++] = i;
    int done = 0;
    while (left > 0) {                                 // parents before children: what never comes up goes round in a circle
      const int i = top[--left]; ++done;
      if (lch[i] >= 0) for (int k : {lch[i], rch[i]}) if (!--parents[k]) top[left++] = k;
    }
    return done == n ? nullptr : "a node that is its own descendant";
  }
  TR forward(Tape& t, const TR&, const int32_t* y) override {
    const int32_t* const host = slot >= 0 ? feed_y[slot] : stage_y;      // y as the host has it
    const int n = host[0];
    if (n < 1 || n > MAXN) { TR z = make({1}); BK(fill)(z.x, 0.0f, 1); return z; }
    if (fused_cells && whole_sequence && whole_tree && is_one_tree(host, n)) return forward_tree(t, host, n);
    known.assign((size_t)n, State()); visited.assign((size_t)n, 0);
    return visit(t, host, y, 0).loss;
  }
  void apply_update(float lr) override { BK(adagrad_update)(slab_x, slab_d, slab_h, lr, pldi19 ? 1.0f : 3.0e38f, 1, slab_count); }
  // Replaces the embedding table (rows x 300 floats, rows <= VOCAB) by the caller's.
  int set_table(const float* host, int rows) {
    if (rows < 1 || rows > VOCAB) return LTB_E_ARG;
    int rc = BK(h2d)(table, host, (size_t)rows * E * 4);
    return rc ? rc : BK(sync)();
  }
};

// ------------------------------------------------------------------------------------------------ ResNet-50 (CIFAR)
struct ResNet50 : Model {
  struct ConvBN { int w, gamma, beta, rmean, rvar; };
  struct Block { ConvBN a, b, c, down; bool has_down; int stride; };
  ConvBN stem; std::vector<Block> blocks; int fcw, fcb;

  ConvBN conv_bn(int cin, int cout, int k) {
    ConvBN cb;
    cb.w = declare({cout, cin, k, k}, INIT_RAND, 2.0f * sqrtf(6.0f / (float)(cin * k * k)));
    cb.gamma = declare({cout}, INIT_ONE); cb.beta = declare({cout}, INIT_ZERO);
    cb.rmean = declare({cout}, INIT_ZERO); cb.rvar = declare({cout}, INIT_ONE);
    decls[cb.rmean].state = decls[cb.rvar].state = true;   // each replica keeps the running statistics of its own batches
    return cb;
  }
  // max_blocks < 16 gives a prefix of the network (stem, max pool, the first max_blocks bottleneck blocks) closed by an
  // average pool over the whole remaining map and the classifier: shallow enough for its TF32 gradients to be compared
  // tightly, made of exactly the layer types and the issue order of the full program.
  ResNet50(int b, int seed, int max_blocks = 16) {
    name = max_blocks < 16 ? "resnet50_prefix" : "resnet50"; batch = b; in_c = 3; in_h = in_w = 32; logit_count = (int64_t)b * 10;
    stem = conv_bn(3, 64, 3);
    int inplanes = 64; const int layers[4] = {3, 4, 6, 3}; const int planes[4] = {64, 128, 256, 512};
    for (int s = 0; s < 4; ++s)
      for (int i = 0; i < layers[s] && (int)blocks.size() < max_blocks; ++i) {
        Block bl; bl.stride = (i == 0 && s > 0) ? 2 : 1;
        bl.a = conv_bn(inplanes, planes[s], 1); bl.b = conv_bn(planes[s], planes[s], 3); bl.c = conv_bn(planes[s], planes[s] * 4, 1);
        bl.has_down = (i == 0);
        if (bl.has_down) bl.down = conv_bn(inplanes, planes[s] * 4, 1);
        inplanes = planes[s] * 4;
        blocks.push_back(bl);
      }
    fcw = declare({10, inplanes}, INIT_RAND, 1.0f / sqrtf((float)inplanes)); fcb = declare({10}, INIT_ZERO);
    finalize(seed);
  }
  TR cbn(Tape& t, const TR& x, const ConvBN& p, int stride, int pad, bool relu) {
    TR y = t.batch_norm(t.conv(x, P(p.w), nullptr, stride, pad), P(p.gamma), P(p.beta), P(p.rmean).x, P(p.rvar).x);
    return relu ? t.relu(y, true) : y;
  }
  TR forward(Tape& t, const TR& x, const int32_t* y) override {
    TR h = t.max_pool(cbn(t, x, stem, 1, 1, true), 2, 2);
    const size_t stage_start[3] = {3, 7, 13};            // first block of stages 2, 3, 4: the slab above each is final when backward gets there
    for (size_t bi = 0; bi < blocks.size(); ++bi) {       // Bottleneck.forward, resnet50.py:72-93
      const Block& bl = blocks[bi];
      for (int k = 0; k < 3 && blocks.size() == 16; ++k)
        if (bi == stage_start[k]) reduce_when_final(t, bl.a.w, k == 2 ? slab_count : decls[blocks[stage_start[k + 1]].a.w].offset);
      // A block with a shortcut convolution has two runs of calls that meet only at the sum: the shortcut (conv + BN) is
      // issued as a branch beside the three conv + BN of the main path.  Backward replays the tape in reverse, so every
      // marker pushes its counterpart: the shortcut's gradients run as a branch from the sum's gradient on, and are joined
      // before the gradient of the block's first convolution, which accumulates into the same input gradient.
      const bool fork = bl.has_down && branches;
      if (fork) BK(branch_mark)();
      TR o = t.conv(h, P(bl.a.w), nullptr, 1, 0);
      if (fork) t.push([] { BK(branch_join)(); });
      o = t.relu(t.batch_norm(o, P(bl.a.gamma), P(bl.a.beta), P(bl.a.rmean).x, P(bl.a.rvar).x), true);
      o = cbn(t, o, bl.b, bl.stride, 1, true);
      o = cbn(t, o, bl.c, 1, 0, false);
      TR res = h;
      if (bl.has_down) {
        if (fork) { BK(branch_begin)(); t.push([] { BK(branch_end)(); }); }
        res = cbn(t, h, bl.down, bl.stride, 0, false);
        if (fork) { BK(branch_end)(); t.push([] { BK(branch_begin)(); }); BK(branch_join)(); t.push([] { BK(branch_mark)(); }); }
      }
      h = t.relu(t.binary(LTB_ADD, o, res), true);
    }
    TR p = t.avg_pool(h, h.shape[2], 1);                                         // 2x2 on the full network's last map
    TR flat = view(p, {batch, h.shape[1]});
    TR logits = t.plus_bias(t.gemm(flat, false, P(fcw), true, 1.0f), P(fcb));   // ONNX Gemm, ONNXLib.scala:956-974
    last_logits = logits;
    return t.mean(t.nll(t.log_softmax(logits), y));                              // resnet50FromOnnx.scala:153-156
  }
};

// ------------------------------------------------------------------------------------------------ SqueezeNet (CIFAR)
struct SqueezeNet : Model {
  struct Conv { int w, b; };
  struct Fire { Conv s, e1, e3; };
  Conv first, last; std::vector<Fire> fires;
  Conv conv(int cin, int cout, int k) {
    Conv c; c.w = declare({cout, cin, k, k}, INIT_RAND, 2.0f * sqrtf(6.0f / (float)(cin * k * k))); c.b = declare({cout}, INIT_ZERO); return c;
  }
  SqueezeNet(int b, int seed) {
    name = "squeezenet"; batch = b; in_c = 3; in_h = in_w = 32; logit_count = (int64_t)b * 10;
    first = conv(3, 96, 3);
    const int cfg[8][4] = {{96, 16, 64, 64}, {128, 16, 64, 64}, {128, 32, 128, 128}, {256, 32, 128, 128},
                           {256, 48, 192, 192}, {384, 48, 192, 192}, {384, 64, 256, 256}, {512, 64, 256, 256}};
    for (auto& c : cfg) { Fire f; f.s = conv(c[0], c[1], 1); f.e1 = conv(c[1], c[2], 1); f.e3 = conv(c[1], c[3], 3); fires.push_back(f); }
    last = conv(512, 10, 4);
    finalize(seed);
  }
  TR cr(Tape& t, const TR& x, const Conv& c, int pad) { TR b = P(c.b); return t.relu(t.conv(x, P(c.w), &b, 1, pad), true); }
  TR fire(Tape& t, const TR& x, const Fire& f) {
    TR s = cr(t, x, f.s, 0);
    return t.concat1(cr(t, s, f.e1, 0), cr(t, s, f.e3, 1));
  }
  TR forward(Tape& t, const TR& x, const int32_t* y) override {
    TR h = t.max_pool(cr(t, x, first, 1), 2, 2);
    for (int i = 0; i < 3; ++i) h = fire(t, h, fires[i]);
    h = t.max_pool(h, 2, 2);
    for (int i = 3; i < 7; ++i) {
      if (i == 4) reduce_when_final(t, fires[4].s.w, slab_count);
      h = fire(t, h, fires[i]);
    }
    h = t.max_pool(h, 2, 2);
    h = fire(t, h, fires[7]);
    TR lb = P(last.b);
    TR logits = view(t.conv(h, P(last.w), &lb, 1, 0), {batch, 10});
    last_logits = logits;
    return t.mean(t.nll(t.log_softmax(logits), y));
  }
};

}  // namespace

extern "C" {

void* HOST_FN(model_create)(const char* name, int batch, int seed) {
  std::string n(name);
  BK(set_fusion)(3);     // generated programs issue every device operation through the library: the one-call look-ahead is safe, and a
                         // gradient buffer has no reader after the operator that absorbs its in-place ReLU gradient (level 2); in the
                         // networks of this file the last batch norm of a residual block is read by the block's sum only (level 3)
  BK(set_filter_cache)(1);   // and they write parameters only through the optimizer, transfer and fill entry points
  if (n == "mnist") return new Mnist(batch, seed);
  if (n == "resnet50") return new ResNet50(batch, seed);
  if (n == "resnet50_prefix") return new ResNet50(batch, seed, 1);        // stem + the first bottleneck block + classifier
  if (n == "squeezenet") return new SqueezeNet(batch, seed);
  if (n == "rnn") return new VanillaRnn(batch, seed, 80, 100);
  if (n == "rnn_26_50") return new VanillaRnn(batch, seed, 26, 50);     // sizes of src/out/NIPS18evaluation/evaluationRNN/Lantern.cpp
  if (n == "treelstm") return new TreeLstm(batch, seed, true);
  if (n == "treelstm_nips18") return new TreeLstm(batch, seed, false);
  return nullptr;
}
void HOST_FN(model_destroy)(void* m) {
  Model* M = (Model*)m;
  M->drop_graphs();
  BK(host_free)(M->stage_x); BK(host_free)(M->stage_y); BK(host_free)(M->loss_host);
  for (int p = 0; p < 2; ++p) { BK(host_free)(M->feed_x[p]); BK(host_free)(M->feed_y[p]); }
  BK(host_free)(M->feed_loss);
  delete M;
}
int HOST_FN(model_num_params)(void* m) { return (int)((Model*)m)->decls.size(); }
int64_t HOST_FN(model_param_count)(void* m, int i) { return ((Model*)m)->decls[i].count; }
int HOST_FN(model_param_is_state)(void* m, int i) { return ((Model*)m)->decls[i].state ? 1 : 0; }   // 1: a batch-norm running statistic
float* HOST_FN(model_param_ptr)(void* m, int i) { Model* M = (Model*)m; return M->slab_x + M->decls[i].offset; }
float* HOST_FN(model_grad_ptr)(void* m, int i) { Model* M = (Model*)m; return M->slab_d + M->decls[i].offset; }
int64_t HOST_FN(model_slab_count)(void* m) { return ((Model*)m)->slab_count; }
float* HOST_FN(model_slab_params)(void* m) { return ((Model*)m)->slab_x; }
float* HOST_FN(model_slab_grads)(void* m) { return ((Model*)m)->slab_d; }
int64_t HOST_FN(model_input_count)(void* m) { Model* M = (Model*)m; return (int64_t)M->batch * M->in_c * M->in_h * M->in_w; }
// TreeLSTM only: load the embedding table (rows x 300) the leaves read.
int HOST_FN(model_set_table)(void* m, const float* host, int rows) {
  TreeLstm* T = dynamic_cast<TreeLstm*>((Model*)m);
  return T ? T->set_table(host, rows) : LTB_E_ARG;
}
int64_t HOST_FN(model_label_count)(void* m) { return ((Model*)m)->label_count; }
// Recursive models: gates as single fused calls (default) or operator by operator, as the reference stages them.
// on: 0 operator by operator, 1 one call per gate / cell, 2 in addition the vanilla RNN's whole sequence and a whole tree node in one call, 3 (default) the
// whole tree.
int HOST_FN(model_use_fused_cells)(void* m, int on) {
  Model* M = (Model*)m;
  M->drop_graphs();
  M->fused_cells = on != 0; M->whole_sequence = on >= 2; M->whole_tree = on >= 3; return 0;
}
// Issue independent runs of calls as branch regions (default) or everything in program order on one stream.
// Large activation gradients declared unset instead of zero-filled (ltb_grad_unset; default on).  Process-wide: it is a property
// of how the tape allocates, not of one model.
int HOST_FN(model_use_deferred_zero)(void*, int on) { deferred_grads() = on != 0; return 0; }
int HOST_FN(model_use_branches)(void* m, int on) {
  Model* M = (Model*)m;
  M->drop_graphs();
  M->branches = on != 0; return 0;
}
// A recorded step can only be replayed when every step issues the same operations: not so for one tree per step.
int HOST_FN(model_use_graph)(void* m, int on) { Model* M = (Model*)m; M->use_graph = on != 0 && M->name != "treelstm"; return 0; }
// Keep one batch resident in device memory; later steps read it there and upload nothing (x_host/y_host are ignored).
int HOST_FN(model_set_resident)(void* m, const float* x_host, const int32_t* y_host) {
  Model* M = (Model*)m;
  M->feed_mode(false);
  M->drop_graphs();
  if (!x_host) { M->resident = false; return 0; }
  M->status = 0; M->reason.clear();
  if (const char* why = M->bad_labels(y_host)) return M->refuse(LTB_E_ARG, why);
  M->load(x_host, y_host);
  BK(h2d)(M->dev_x, M->stage_x, (size_t)M->batch * M->in_c * M->in_h * M->in_w * 4);
  BK(h2d)(M->dev_y, M->stage_y, (size_t)M->label_count * 4);
  BK(sync)();
  M->resident = true;
  return 0;
}
// Blocking step: returns the loss of this batch (a NaN if the step failed: model_status). update=0 leaves the parameter gradients in place for inspection.
float HOST_FN(model_step)(void* m, const float* x_host, const int32_t* y_host, float lr, int update) {
  Model* M = (Model*)m;
  if (M->feeding) M->feed_mode(false);
  return M->step(x_host, y_host, lr, update != 0);
}
// Non-blocking step: the loss is available from model_last_loss after the library's sync.
int HOST_FN(model_step_async)(void* m, const float* x_host, const int32_t* y_host, float lr) {
  Model* M = (Model*)m;
  if (M->feeding) M->feed_mode(false);
  return M->step_async(x_host, y_host, lr, true);
}
// Two steps in flight: submit returns the step's number (or -1) without waiting; collect(k) waits for step k and gives its
// loss.  Only the last two submitted steps can be collected.
int64_t HOST_FN(model_submit)(void* m, const float* x_host, const int32_t* y_host, float lr) { return ((Model*)m)->submit(x_host, y_host, lr); }
// What became of the last step: 0, or a negative code with the reason in buf.  model_step, model_step_async and model_submit set it.
int HOST_FN(model_status)(void* m, char* buf, int len) {
  const Model* M = (Model*)m;
  if (buf && len > 0) { strncpy(buf, M->reason.c_str(), len - 1); buf[len - 1] = 0; if (M->status && M->reason.empty()) BK(last_error)(buf, len); }
  return M->status;
}
int HOST_FN(model_collect)(void* m, int64_t step, float* loss) { return ((Model*)m)->collect(step, loss); }
float HOST_FN(model_last_loss)(void* m) { const Model* M = (Model*)m; return M->feeding && M->submitted ? M->feed_loss[(M->submitted - 1) & 1] : *M->loss_host; }
// The classifier's output of the last step (batch x classes floats); returns the number of floats, 0 for programs without one.
int64_t HOST_FN(model_logits)(void* m, float* host_out) {
  Model* M = (Model*)m;
  if (!M->dev_logits || BK(d2h)(host_out, M->dev_logits, (size_t)M->logit_count * 4)) return 0;
  return M->logit_count;
}

// ---- data and parameter files in the reference's formats (loader.hpp)
void* HOST_FN(loader_open_floats)(const char* data_path, const char* target_path, int64_t floats_per_sample, float mean, float stdev) {
  Loader* L = new Loader;
  L->open_floats(data_path, target_path, floats_per_sample, mean, stdev);
  return L;                                      // a loader that failed to open has length 0 and a message (loader_error)
}
void* HOST_FN(loader_open_cifar)(const char* path, int64_t bytes_per_sample) {
  Loader* L = new Loader;
  L->open_cifar(path, bytes_per_sample);
  return L;
}
const char* HOST_FN(loader_error)(void* l) { return ((Loader*)l)->error.c_str(); }
int64_t HOST_FN(loader_length)(void* l) { Loader* L = (Loader*)l; return L->error.empty() ? L->length : 0; }
int HOST_FN(loader_fill)(void* l, int64_t index, int batch, float* x, int32_t* y) {
  Loader* L = (Loader*)l;
  return L->error.empty() && L->fill(index, batch, x, y) ? 0 : LTB_E_ARG;
}
void HOST_FN(loader_close)(void* l) { Loader* L = (Loader*)l; L->close(); delete L; }
// One pass over the loader's batches (at most max_batches when positive) with two steps in flight: batch i + 1 is decoded
// into pinned staging while the device runs step i.  losses (nullable) receives one value per batch.  Returns the number
// of steps, or a negative error code.
int64_t HOST_FN(model_train_epoch)(void* m, void* l, float lr, float* losses, int64_t max_batches) {
  Model* M = (Model*)m; Loader* L = (Loader*)l;
  if (!L->error.empty() || L->sample_count != (int64_t)M->in_c * M->in_h * M->in_w || M->label_count != M->batch) return LTB_E_ARG;
  int64_t n = L->batches(M->batch);
  if (max_batches > 0 && max_batches < n) n = max_batches;
  int64_t prev = -1;
  for (int64_t i = 0; i < n; ++i) {
    float* sx; int32_t* sy; float loss;
    if (M->feed_slot(&sx, &sy) || !L->fill(i, M->batch, sx, sy)) return LTB_E_STATE;
    const int64_t k = M->submit(nullptr, nullptr, lr);
    if (k < 0) return LTB_E_CUDA;
    if (prev >= 0) { if (M->collect(prev, &loss)) return LTB_E_CUDA; if (losses) losses[i - 1] = loss; }
    prev = k;
  }
  if (prev >= 0) { float loss; if (M->collect(prev, &loss)) return LTB_E_CUDA; if (losses) losses[n - 1] = loss; }
  return n;
}
// Parameter file: every tensor's floats back to back, unpadded, in declaration order (ONNXLib.scala:157-185).
int HOST_FN(model_save_params)(void* m, const char* path) {
  Model* M = (Model*)m;
  std::vector<float> slab((size_t)M->slab_count);
  if (BK(d2h)(slab.data(), M->slab_x, slab.size() * 4)) return LTB_E_CUDA;
  FILE* f = fopen(path, "wb");
  if (!f) return LTB_E_ARG;
  bool ok = true;
  for (const ParamDecl& d : M->decls) ok = ok && fwrite(slab.data() + d.offset, 4, (size_t)d.count, f) == (size_t)d.count;
  return fclose(f) == 0 && ok ? 0 : LTB_E_STATE;
}
int HOST_FN(model_load_params)(void* m, const char* path) {
  Model* M = (Model*)m;
  MappedFile f;
  if (!f.open(path)) return LTB_E_ARG;
  int64_t total = 0;
  for (const ParamDecl& d : M->decls) total += d.count;
  if ((int64_t)(f.bytes / 4) != total || f.bytes % 4) { f.close(); return LTB_E_ARG; }      // not this model's file
  std::vector<float> slab((size_t)M->slab_count, 0.0f);
  const float* src = (const float*)f.data;
  for (const ParamDecl& d : M->decls) { memcpy(slab.data() + d.offset, src, (size_t)d.count * 4); src += d.count; }
  f.close();
  if (BK(sync)() || BK(h2d)(M->slab_x, slab.data(), slab.size() * 4) || BK(sync)()) return LTB_E_CUDA;
  return 0;
}
// Debug: run one step without update and write per-operator checksums (see Model::dump_trace) into buf.
int HOST_FN(model_trace)(void* m, const float* x_host, const int32_t* y_host, char* buf, int len) {
  Model* M = (Model*)m;
  tracing() = true; trace_list().clear();
  BK(set_fusion)(1);     // the trace reads every gradient buffer after the step: masked gradients are written back as the separate calls would
  M->step(x_host, y_host, 0.0f, false);
  BK(set_fusion)(3);
  tracing() = false;
  strncpy(buf, M->trace_text.c_str(), len - 1); buf[len - 1] = 0;
  return (int)M->trace_text.size();
}

}  // extern "C"
