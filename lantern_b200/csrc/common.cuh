// Shared state and helpers of liblantern_b200 (internal; the public contract is include/lantern_b200.h).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <string>

#include "../../include/lantern_b200.h"

namespace ltb {

constexpr int kSMs = 148;             // B200: 2 dies x 74 SMs; grids are sized in multiples of this
constexpr size_t kGranule = 256;      // arena granule (TMA wants 16 B bases/strides; 256 keeps every tensor sector-aligned)

// Look-ahead fusion (ltb_set_fusion): an operation whose result the very next call may finish in the same kernel is held back
// for one call.  BN forward or a same-shape add followed by an in-place ReLU of their result become one kernel; an in-place
// ReLU gradient followed by BN backward or by the add's gradient reading that buffer become one kernel.  A convolution and the
// in-place ReLU of its result share the contraction's epilogue, and a held ReLU gradient joins the bias-gradient pass of the
// convolution backward that reads it.  A log-softmax, the negative log likelihood of its result and the sum (mean) of that are one kernel,
// and so are the seed of the loss's gradient (a fill of one element) and the three gradients.  Any other call
// first issues the held operation on its own, so results never change; only the moment of the launch does.
enum { PEND_NONE = 0, PEND_BN_FWD = 1, PEND_ADD = 2, PEND_RELU_GRAD = 3, PEND_RELU_ADD_GRAD = 4, PEND_BN_ADD = 5, PEND_CONV = 6, PEND_BN_INF = 7, PEND_BN_RELU = 8,
       PEND_LSM = 9, PEND_NLL = 10, PEND_SEED = 11, PEND_SUM_GRAD = 12, PEND_NLL_GRAD = 13 };
struct ConvDims { int N, C, H, W, K, R, S, sh, sw, ph, pw, oH, oW; };
struct Pending {
  int kind = PEND_NONE;
  int64_t n = 0;
  // PEND_BN_FWD
  const float *x = nullptr, *gamma = nullptr, *beta = nullptr;
  float *y = nullptr, *run_mean = nullptr, *run_var = nullptr, *save_mean = nullptr, *save_istd = nullptr;
  int N = 0, C = 0, HW = 0; float eps = 0, momentum = 0;
  // PEND_LSM: y = log softmax of x, N rows of C; PEND_NLL: and out = -y[target].  PEND_SEED: d[0] = value; PEND_SUM_GRAD: and da[0..n) += scale d[0]
  // (seeded: whether the first part is there); PEND_NLL_GRAD: and db[row][target] -= da[row], N rows of C
  const int32_t* target = nullptr; float value = 0, scale = 0; bool seeded = false;
  // PEND_ADD: out = a + b
  const float *a = nullptr, *b = nullptr; float* out = nullptr;
  // PEND_RELU_GRAD: d = relu_y > 0 ? d : 0
  const float* relu_y = nullptr; float* d = nullptr;
  // PEND_RELU_ADD_GRAD (fusion level 2): m = relu_y > 0 ? d : 0; da += m; db += m, held so that the batch-norm backward whose dy is
  // da (or db) reads m straight from d and writes the other destination itself; fa / fb: that destination holds nothing yet
  float *da = nullptr, *db = nullptr; int fa = 0, fb = 0;
  // PEND_CONV: y = conv(x, w) (+ bias)
  const float *w = nullptr, *bias = nullptr; ConvDims dims = {};
  // PEND_BN_RELU: a PEND_BN_FWD or PEND_BN_ADD (`inner`) and the in-place ReLU of its result, held one call further: the convolution that
  // reads the result has its own output cleared and its channels-last copy written by the same kernel (BnExtra)
  int inner = PEND_NONE;
  // PEND_BN_ADD (fusion level 3): the PEND_BN_FWD fields, then out = y + a with y the held batch norm's result; an in-place ReLU of
  // out makes the three one kernel that never writes y
};

struct Context {
  bool inited = false;
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  char* heap = nullptr;
  size_t heap_bytes = 0;
  size_t used = 0;
  size_t top_used = 0;                // bytes taken from the far end of the arena for blocks that live until ltb_reset (step_alloc)
  bool keep_off = false;              // the two ends met once: nothing is kept at the far end any more
  int fatal = 1;
  int last = 0;
  std::string msg;
  int math = LTB_MATH_TF32;
  int64_t launches = 0;
  bool capturing = false;
  int64_t capture_launch_base = 0;
  unsigned* tickets = nullptr;        // two device words, zero between launches: how many CTAs of a launch are done (one for each of the streams a branch region has)
  int* dev_status = nullptr;          // device word set by kernels whose bounded waits run out
  int* host_status = nullptr;         // pinned mirror
  int64_t wait_limit_cycles = 2000000000ll;   // bound of every device-side spin wait (about a second; ltb_set_wait_limit)
  float* scratch = nullptr;           // private workspace for multi-stage reductions
  size_t scratch_bytes = 0;
  int sm_count = kSMs;
  bool profiling = false;             // per-launch CUDA-event timing (ltb_profile)
  bool pdl = true;                    // launches may begin while the kernel before them runs (see pdl_enter)
  const char* label = nullptr;        // optional name override for the next launches
  cudaStream_t side = nullptr;        // second stream: the weight-gradient half of conv backward runs beside the data-gradient half
  cudaStream_t copy = nullptr;        // uploads beside the compute work (ltb_upload)
  cudaEvent_t fork_ev = nullptr, join_ev = nullptr;
  unsigned tune = 0;                  // LTB_TUNE (environment, read by ltb_init): switches single optimisations off for A/B measurements:
                                      // 1 no in-kernel gather, 2 no tap-loop weight-grad from kept copies, 4 no kept copies, 32 deferred zero fill off (ltb_grad_unset fills at once)
  bool deterministic = false;         // split-K sums in a fixed order (clusters, slabs) instead of atomics (ltb_set_deterministic)
  bool filter_cache = false;          // per-tap filter forms kept across calls (ltb_set_filter_cache)
  bool fusion = false;                // look-ahead fusion of BN/add with ReLU (off unless the host opts in)
  bool fusion_single_use = false;     // level 3: a batch-norm result consumed by add + in-place ReLU has no other reader and is not written
  bool fusion_no_writeback = false;   // level 2: an absorbed in-place ReLU gradient is applied on load only (its buffer is dead afterwards)
  Pending pending;
  Pending ahead;                      // a PEND_BN_RELU taken over by the convolution call that is running; issued by its first launch that reads or clears something
  bool side_open = false;             // weight gradients are running on the side stream that no stream has waited for yet (side_join)
  size_t side_base = 0;               // arena mark below the staging blocks held for them
  bool hold_workspace = false;        // while two halves are in flight their staging blocks are released together at the end
  // Branch region (ltb_branch_mark .. ltb_branch_join): a run of calls issued on a third stream beside the caller's.
  cudaStream_t branch = nullptr, trunk = nullptr;
  cudaEvent_t mark_ev = nullptr, branch_done_ev = nullptr;
  bool branch_marked = false, in_branch = false, branch_ended = false;
  // Private workspace of the calling side: while a branch region is open the two streams each get one half.
  float* cur_scratch() const { return in_branch ? scratch + (scratch_bytes / 2) / sizeof(float) : scratch; }
  size_t cur_scratch_bytes() const { return branch_marked ? scratch_bytes / 2 : scratch_bytes; }
};
extern Context g;
// Whether q lies in the part of the arena from p on, the part that ltb_free or ltb_reset gives back.  Memory of the caller's own lies outside
// at any address: a kept copy of such a tensor stays until its source is written or the step ends, a declaration until it is used.
inline bool in_arena_from(const void* q, const void* p) { return q >= p && (const char*)q < g.heap + g.heap_bytes; }

int fail(int code, const char* fmt, ...);
int flush_pending();
int relu_add_grad_issue(const Pending& p);                 // issues the held operation on its own (elementwise.cu)
// issue functions shared by the entry points and the flush (pool_bn.cu / elementwise.cu)
int conv_fwd_issue(const Pending& p, bool relu);           // contract.cu
int bn_inference_issue(const Pending& p, bool relu);
// What a batch norm's kernel does beside its own work for the convolution that follows: clear `zero` (n4 times 16 bytes) and write a
// channels-last copy of the result.
struct ZeroFill { float4* p = nullptr; int64_t n4 = 0; };
struct BnExtra { ZeroFill zero; float* cl = nullptr; };
bool bn_fwd_writes_copy(const Pending& p);                 // whether the kernel that p takes can write the copy
int bn_fwd_issue(const Pending& p, bool relu, const BnExtra& extra = BnExtra());
// A result that the launches of this call add into and that has to be zero before: `p` (null: nothing to clear) is cleared by whichever
// kernel of the call runs first and can, `done` says that one did.
struct Clear { float* p = nullptr; size_t floats = 0; bool done = false; };
ZeroFill take_clear(Clear* c);                             // what a kernel is given to clear (gemm_tc.cu)
// Issues g.ahead, if there is one, with the clearing and the copy; cl: where the channels-last copy goes.
int issue_ahead(Clear* clear = nullptr, float* cl = nullptr);
int add_issue(const float* a, const float* b, float* out, int64_t n, bool relu);
int relu_issue(float* x, int64_t n);
int fill_issue(float* x, float v, int64_t n);
int head_issue(const Pending& p);                          // PEND_LSM, PEND_NLL, PEND_SUM_GRAD, PEND_NLL_GRAD on their own (reduce.cu)
int relu_grad_issue(const float* y, float* d, int64_t n);
// Host waits while a communicator exists: bounded, with NCCL's asynchronous error state polled (comm.cu).
void filter_cache_clear();           // gemm_tc.cu
void filter_cache_drop_from(const void* p);
void cl_cache_clear();               // gemm_tc.cu: kept channels-last copies (they live in step_alloc blocks)
void cl_cache_drop_from(const void* p);
// A block from the far end of the arena that stays until ltb_reset; nullptr when the two ends would meet (context.cu).
void* step_alloc(size_t bytes);
// A call is about to write [p, p + bytes): kept copies and cached filter forms whose source overlaps it are stale (p == nullptr: all of
// them).  Every entry point reports every buffer it writes (LTB_WRITES).
void filter_cache_note_write(const void* p, size_t bytes);
// Gradient buffers declared unset (ltb_grad_unset): logically zero, physically not yet written.
//   grad_take_unset(p, bytes)  true when [p, p + bytes) is exactly one declared block: the caller WRITES its result instead
//                              of adding (the declaration is consumed);
//   grad_settle(p, bytes)      any other use of a block that starts at p: fill it with zeros now (on the current stream).
// Both cost a look-up in a small host table, and nothing at all while no block is declared.
bool grad_take_unset(const void* p, size_t bytes);
int grad_settle(const void* p, size_t bytes);
void grad_unset_drop_from(const void* p);
void grad_unset_clear();
// Weight gradients left running on the side stream after ltb_conv2d_bwd has returned (look-ahead fusion on): nothing but the optimizer
// reads them, so the data-gradient chain does not wait for each.  Every entry point waits for them first (LTB_INITED_NOFLUSH), but for
// the gradient calls that make up the chain, which wait only when one of their buffers meets one that the side stream uses.
//   side_join()               the current stream waits, the staging blocks go back to the arena;
//   side_add(p, bytes, wr)    the side stream reads (or writes) this range;
//   side_check(p, bytes, wr)  the caller is about to read (or write) it: joins if that matters.
int side_join();
void side_add(const void* p, size_t bytes, bool written);
int side_check(const void* p, size_t bytes, bool write);
#define LTB_SIDE_CHECK(ptr, count, write) do { if (::ltb::g.side_open && (ptr)) { int rc_k_ = ::ltb::side_check((ptr), (size_t)(count) * 4, (write)); if (rc_k_) return rc_k_; } } while (0)
void mask_staging_free();             // elementwise.cu
bool comm_active();
int comm_wait_stream(cudaStream_t s, const char* what);
int comm_wait_event(cudaEvent_t ev, const char* what);
void profile_before(const char* name);
void profile_after();

#define LTB_REQUIRE(cond, ...) do { if (!(cond)) return ::ltb::fail(LTB_E_ARG, __VA_ARGS__); } while (0)
// A gradient buffer that was declared unset and is about to be used in any way but as a whole, writable destination: zeros first.
// The entry point writes `count` floats at ptr (null: not asked for): kept copies and cached forms of what was there are stale.
#define LTB_WRITES(ptr, count) do { if (ptr) ::ltb::filter_cache_note_write((ptr), (size_t)(count) * 4); } while (0)
#define LTB_SETTLE(ptr) do { int rc_s_ = ::ltb::grad_settle((ptr), 0); if (rc_s_) return rc_s_; } while (0)
#define LTB_CUDA(call) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) return ::ltb::fail(LTB_E_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); } while (0)
#define LTB_INITED_CHAIN() do { if (!::ltb::g.inited) return ::ltb::fail(LTB_E_STATE, "%s: library not initialised (call ltb_init)", __func__); } while (0)
#define LTB_INITED_NOFLUSH() do { LTB_INITED_CHAIN(); if (::ltb::g.side_open) { int rc_j_ = ::ltb::side_join(); if (rc_j_) return rc_j_; } } while (0)
// Every entry point first issues an operation held back by the look-ahead fusion; the few that may complete it use _NOFLUSH.
#define LTB_INITED() do { LTB_INITED_NOFLUSH(); if (::ltb::g.pending.kind) { int rc_ = ::ltb::flush_pending(); if (rc_) return rc_; } } while (0)

// Quotients by a divisor that is the same for a whole launch: a multiplication and a shift (0 <= n < 2^31; the round-up method of
// Granlund and Montgomery). 
struct FastDiv {
  unsigned mul = 0, shift = 0, d = 1;
  FastDiv() = default;
  explicit FastDiv(int divisor) : d((unsigned)divisor) {
    if (d == 1) return;
    unsigned log = 0; while ((1u << log) < d) ++log;
    mul = (unsigned)(((1ull << (31 + log)) + d - 1) / d); shift = log - 1;
  }
  __device__ __forceinline__ int div(int n) const { return d == 1 ? n : (int)(__umulhi((unsigned)n, mul) >> shift); }
  __device__ __forceinline__ int divmod(int n, int& rem) const { const int q = div(n); rem = n - q * (int)d; return q; }
};

// Programmatic dependent launch: a kernel may be launched, and its CTAs set up, while the kernel before it on the stream still runs.
// Every kernel of this library starts with pdl_enter() (the engine splits it): it lets the next kernel start where there is room for
// it, and waits for the kernels before it to finish, memory included, before it touches global memory.  In a recorded step of small
// kernels the launch latency between neighbours is what this hides: SqueezeNet at batch 64 1.06 -> 0.97 ms, MNIST 0.280 -> 0.225,
// ResNet-50 at batch 8 2.15 -> 2.00.  The batch norms with more CTAs than SMs are launched without it (g.pdl): waiting, their large CTAs
// keep a weight-gradient on the side stream out of the SMs (ResNet-50 at batch 128: 3.87 ms with, 3.81 without).
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() { pdl_launch(); pdl_wait(); }
// The whole grid's share of a ZeroFill.
__device__ __forceinline__ void zero_fill(const ZeroFill& z) {
  if (z.n4 == 0) return;
  const int64_t block = ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x, per = blockDim.x * blockDim.y;
  for (int64_t i = block * per + threadIdx.y * blockDim.x + threadIdx.x; i < z.n4; i += (int64_t)gridDim.x * gridDim.y * gridDim.z * per) z.p[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}
#endif
inline void pdl_attribute(cudaLaunchAttribute& a) { a.id = cudaLaunchAttributeProgrammaticStreamSerialization; a.val.programmaticStreamSerializationAllowed = 1; }

// Every kernel launch of the library goes through this macro so that ltb_kernel_launches() is exact.  While the launch profiler is on
// kernels run strictly one after the other.
#define LTB_LAUNCH(kernel, grid, block, smem, ...)                                           \
  do {                                                                                       \
    cudaLaunchConfig_t cfg_ = {};                                                            \
    cfg_.gridDim = (grid); cfg_.blockDim = (block); cfg_.dynamicSmemBytes = (size_t)(smem); cfg_.stream = ::ltb::g.stream; \
    cudaLaunchAttribute attr_[1];                                                            \
    ::ltb::pdl_attribute(attr_[0]);                                                          \
    cfg_.attrs = attr_; cfg_.numAttrs = ::ltb::g.profiling || !::ltb::g.pdl ? 0 : 1;                          \
    if (::ltb::g.profiling) ::ltb::profile_before(::ltb::g.label ? ::ltb::g.label : #kernel); \
    cudaError_t e_ = cudaLaunchKernelEx(&cfg_, kernel, __VA_ARGS__);                         \
    if (::ltb::g.profiling) ::ltb::profile_after();                                          \
    ++::ltb::g.launches;                                                                     \
    if (e_ != cudaSuccess) return ::ltb::fail(LTB_E_CUDA, "launch of %s failed: %s", #kernel, cudaGetErrorString(e_)); \
  } while (0)

// The same for a launch with a thread-block cluster of `cluster` CTAs along x (grid.x must be a multiple of it).
#define LTB_LAUNCH_CLUSTER(kernel, grid, block, cluster, ...) LTB_LAUNCH_CLUSTER_XZ(kernel, grid, block, cluster, 1, 0, __VA_ARGS__)
#define LTB_LAUNCH_CLUSTER_Z(kernel, grid, block, cluster, smem, ...) LTB_LAUNCH_CLUSTER_XZ(kernel, grid, block, 1, cluster, smem, __VA_ARGS__)    // CTAs along z
#define LTB_LAUNCH_CLUSTER_XZ(kernel, grid, block, cx, cz, smem, ...)                        \
  do {                                                                                       \
    cudaLaunchConfig_t cfg_ = {};                                                            \
    cfg_.gridDim = (grid); cfg_.blockDim = (block); cfg_.dynamicSmemBytes = (size_t)(smem); cfg_.stream = ::ltb::g.stream; \
    cudaLaunchAttribute attr_[2];                                                            \
    ::ltb::pdl_attribute(attr_[1]);                                                          \
    attr_[0].id = cudaLaunchAttributeClusterDimension;                                       \
    attr_[0].val.clusterDim.x = (unsigned)(cx); attr_[0].val.clusterDim.y = 1; attr_[0].val.clusterDim.z = (unsigned)(cz); \
    cfg_.attrs = attr_; cfg_.numAttrs = ::ltb::g.profiling || !::ltb::g.pdl ? 1 : 2;                                                   \
    if (::ltb::g.profiling) ::ltb::profile_before(::ltb::g.label ? ::ltb::g.label : #kernel); \
    cudaError_t e_ = cudaLaunchKernelEx(&cfg_, kernel, __VA_ARGS__);                         \
    if (::ltb::g.profiling) ::ltb::profile_after();                                          \
    ++::ltb::g.launches;                                                                     \
    if (e_ != cudaSuccess) return ::ltb::fail(LTB_E_CUDA, "cluster launch of %s failed: %s", #kernel, cudaGetErrorString(e_)); \
  } while (0)

// While in scope, launches of more CTAs than `most` (the SMs) take no part in programmatic dependent launch (see pdl_enter).
struct PdlUnlessLarge {
  explicit PdlUnlessLarge(int64_t ctas, int64_t most = g.sm_count) { g.pdl = ctas <= most; }
  ~PdlUnlessLarge() { g.pdl = true; }
};
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
// Grid for a grid-stride kernel over `work` thread-items: enough CTAs to cover it, capped at `per_sm` CTAs per SM.
inline int grid_for(int64_t work, int block, int per_sm = 8) {
  int64_t need = ceil_div(work, block);
  int64_t cap = (int64_t)g.sm_count * per_sm;
  if (need < 1) need = 1;
  return (int)(need < cap ? need : cap);
}

}  // namespace ltb
