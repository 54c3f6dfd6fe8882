// C ABI of libb200conv: context, pooled device memory, geometry checks, tensor-map
// construction and the orchestration of the three convolution directions.
#include <dlfcn.h>

#include <algorithm>
#include <chrono>
#include <thread>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <initializer_list>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "internal.h"
#include "staging.h"

using namespace b200;

// ======================================================================================
// context
// ======================================================================================
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

std::mutex g_create_mu;
std::string g_create_err;

}  // namespace

// A captured sequence of calls.  Temporaries that the calls took from the pool while they were
// captured stay reserved for the graph until it is destroyed (the replays use their addresses).
struct b200conv_graph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  std::vector<void*> retained;
  unsigned int* arrivals = nullptr;   // its own counts of slices of cut tiles: a replay may run beside other launches, on another context's stream
  long long launches = 0;   // kernels in the graph
};

// Ring of pinned buffers that host arrays travel through (staging.h): chunks of at most a slot, so
// that the copy of one chunk runs beside the transfer of the one before.
constexpr size_t kRingSlotBytes = 2u << 20;    // 2 MB: 27 us to copy with 8 threads, 41 us on the link
constexpr int kRingSlots = 16;
constexpr size_t kSmallInput = 64u << 10;      // inputs up to this size share one slot and one transfer

// Key of what the context remembers per geometry: a kind and up to 23 integers.  Looked up on every call,
// so it is compared and hashed as integers (text keys cost 1.5 us of the host's 10 us per call).
struct GeoKey {
  int n = 0;
  int v[24];
  GeoKey(std::initializer_list<int> l) {
    for (int x : l) v[n++] = x;
  }
  void add(long long x) { v[n++] = static_cast<int>(x); }
  bool operator==(const GeoKey& o) const { return n == o.n && !memcmp(v, o.v, sizeof(int) * n); }
  std::string text() const {
    std::string t;
    for (int i = 0; i < n; ++i) t += (i ? "." : "") + std::to_string(v[i]);
    return t;
  }
  static bool parse(const char* t, GeoKey* k) {
    k->n = 0;
    while (*t && k->n < 24) {
      char* end;
      k->v[k->n++] = static_cast<int>(strtol(t, &end, 10));
      if (end == t) return false;
      t = *end == '.' ? end + 1 : end;
    }
    return !*t && k->n > 0;
  }
};
struct GeoHash {
  size_t operator()(const GeoKey& k) const {
    uint64_t h = 1469598103934665603ull;
    for (int i = 0; i < k.n; ++i) h = (h ^ static_cast<uint32_t>(k.v[i])) * 1099511628211ull;
    return h ^ (h >> 29);
  }
};
enum { kGeoSlab = 1, kGeoTile, kGeoConv, kGeoWgrad, kGeoSplits, kGeoBalance, kGeoClasses, kGeoRows };      // kinds (first integer of a key)

// Tile of a convolution kernel for one geometry (the result of a search).
struct SlabTile {
  int wt = 0, th = 0, nb = 0, n_acc = 0, slab_bytes = 0;
  int bn = 0, splits = 1;        // accumulator columns, slices of the reduction
  bool row = false;              // slab kernel: whole 128-pixel pieces of one long row (flattened 1x1 layers)
  bool found = false;
};

struct b200conv_ctx {
  int device = 0;
  int num_sms = 148;                         // SMs the persistent kernels spread over (b200conv_set_sm_count)
  int device_sms = 148;
  cudaStream_t stream = nullptr;
  std::mutex mu;
  std::string err;
  int* d_status = nullptr;  // status word of the kernels: h_status as the device sees it
  unsigned int* d_arrivals = nullptr;   // counts of the slices of cut tiles (conv_pair.cu), zero between launches
  volatile int* h_status = nullptr;  // pinned and mapped: written by kernels only when they give up, so that
                                     // a synchronising call reads it without a transfer
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaEvent_t ev_tune0 = nullptr, ev_tune1 = nullptr;   // kernel selection timing
  long long launches = 0;
  const char* last_algo = "none";
  const char* last_variant = "none";        // tensor-core kernel of the last result (timed trials come before it)
  // optional per-kernel timing: an event pair around every launch of our own kernels
  bool prof = false;
  struct ProfRec { int kind; cudaEvent_t a, b; };
  std::vector<ProfRec> prof_recs;
  std::vector<cudaEvent_t> prof_pool;
  EncodeTiledFn encode = nullptr;
  // pooled device memory: free blocks by size, live blocks by address
  std::multimap<size_t, void*> free_blocks;
  std::map<void*, size_t> live;
  size_t pool_bytes = 0;
  void* l2buf = nullptr;
  size_t l2bytes = 0;
  // NCCL (loaded on demand)
  void* nccl_lib = nullptr;
  void* comm = nullptr;
  int nranks = 1, rank = 0;
  float* d_token = nullptr;
  cudaStream_t comm_stream = nullptr;       // collectives that overlap later convolutions
  cudaEvent_t ev_comm_ready = nullptr, ev_comm_done = nullptr;
  cudaStream_t up_stream = nullptr, down_stream = nullptr;   // background copies (PCIe is full duplex)
  cudaEvent_t ev_up = nullptr, ev_down = nullptr;
  bool down_pending = false;
  bool comm_pending = false;
  long long* trace = nullptr;               // debug: phase stamps of the slab kernel
  int diag_c = 0, diag_k = 0;               // during a gradWeights call on merged groups: channels / filters of one of them
  ConvEpilogue epi = default_epilogue();    // epilogue of the forward call in progress
  // forward / gradInputs kernel choice per geometry (true = slab kernel), filled by timing
  std::unordered_map<GeoKey, int, GeoHash> algo_cache;
  // gradWeights split-K slice count per geometry and kernel, chosen by timing
  std::unordered_map<GeoKey, int, GeoHash> split_cache;
  // tiles found by search: the same on every call of a geometry, and the search costs 2 to 30 us
  std::unordered_map<GeoKey, SlabTile, GeoHash> slab_tiles;
  std::unordered_map<GeoKey, SlabTile, GeoHash> pixel_tiles;
  int force_splits = 0;                     // > 0: use this slice count (tests, tuning by hand)
  bool model_only = false;                  // choices that are not remembered yet are the models', not timed (rough comparison)
  bool use_pair = true;                     // 1x1 layers with deep reductions on CTA pairs (gemm_pair.cu)
  bool stack_taps = true;                   // grouped gradWeights of narrow layers: taps as column groups of one MMA
  bool autotune = true;
  // CUDA-graph capture of a sequence of calls (b200conv_graph_*)
  b200conv_graph* capturing = nullptr;
  long long graph_launch_count = 0;
  long long wait_clocks = 4000000000LL;     // bound of device-side waits (about two seconds)
  int comm_timeout_ms = 60000;              // host watchdog of streams that carry collectives
  // pinned ring of the host-pointer calls (made on first use); every such call ends with all slots free
  char* ring = nullptr;
  bool no_ring = false;                     // there is no memory for it
  cudaEvent_t ring_ev[kRingSlots] = {};
  bool ring_busy[kRingSlots] = {};
  int ring_next = 0;
  CopyPool* copy_pool = nullptr;
  std::vector<cudaEvent_t> chunk_ev;        // order a batch's chunks across the upload, compute and download streams
  // packed filters made ahead of time (b200conv_prepack): key -> device buffer and validity
  struct Packed { void* ptr; size_t bytes; bool valid; const void* src; };
  std::map<std::string, Packed> packed;
};

namespace {

int fail(b200conv_ctx* c, int code, const char* fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (c) c->err = buf;
  return code;
}

#define CU_OK(c, expr)                                                                      \
  do {                                                                                      \
    cudaError_t e_ = (expr);                                                                \
    if (e_ != cudaSuccess)                                                                  \
      return fail((c), e_ == cudaErrorMemoryAllocation ? B200CONV_E_NOMEM : B200CONV_E_CUDA, \
                  "%s: %s", #expr, cudaGetErrorString(e_));                                 \
  } while (0)

// Kernel families, for the launch counter and the optional per-kernel timing.
enum { kKConvUmma = 0, kKWgradUmma, kKWgradReduce, kKTranspose, kKPack, kKDirect, kKPool, kKConvReduce, kKCount };
const char* const kKernelNames[kKCount] = {"conv_umma", "wgrad_umma", "wgrad_reduce", "transpose",
                                           "pack", "direct", "pool", "conv_reduce"};

cudaEvent_t prof_event(b200conv_ctx* c) {
  cudaEvent_t e = nullptr;
  if (!c->prof_pool.empty()) {
    e = c->prof_pool.back();
    c->prof_pool.pop_back();
  } else {
    cudaEventCreate(&e);
  }
  return e;
}

#define KLAUNCH(c, kind, expr)                                  \
  do {                                                          \
    cudaEvent_t ea_ = nullptr, eb_ = nullptr;                   \
    const bool prof_ = (c)->prof && !(c)->capturing;            \
    if (prof_) {                                                \
      ea_ = prof_event(c);                                      \
      eb_ = prof_event(c);                                      \
      cudaEventRecord(ea_, (c)->stream);                        \
    }                                                           \
    CU_OK(c, expr);                                             \
    (c)->launches++;                                            \
    if ((c)->capturing) (c)->capturing->launches++;             \
    if (prof_) {                                                \
      cudaEventRecord(eb_, (c)->stream);                        \
      (c)->prof_recs.push_back({kind, ea_, eb_});               \
    }                                                           \
  } while (0)

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
    else prev = -1;
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

// ---- pooled allocator: blocks are recycled without returning to the driver; safe because
// every use is ordered on the context's single stream --------------------------------------
int pool_alloc(b200conv_ctx* c, size_t bytes, void** out) {
  if (bytes == 0) bytes = 256;
  bytes = (bytes + 255) & ~static_cast<size_t>(255);
  auto it = c->free_blocks.lower_bound(bytes);
  if (it != c->free_blocks.end() && it->first <= bytes + bytes / 4 + (1 << 20)) {
    *out = it->second;
    c->live[*out] = it->first;
    c->free_blocks.erase(it);
    return 0;
  }
  void* p = nullptr;
  cudaError_t e = cudaMalloc(&p, bytes);
  if (e != cudaSuccess) {
    // give cached blocks back to the driver and retry once
    cudaGetLastError();
    cudaStreamSynchronize(c->stream);
    for (auto& kv : c->free_blocks) {
      cudaFree(kv.second);
      c->pool_bytes -= kv.first;
    }
    c->free_blocks.clear();
    e = cudaMalloc(&p, bytes);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(c, B200CONV_E_NOMEM, "device allocation of %zu bytes failed: %s", bytes,
                  cudaGetErrorString(e));
    }
  }
  c->pool_bytes += bytes;
  c->live[p] = bytes;
  *out = p;
  return 0;
}

int pool_free(b200conv_ctx* c, void* p) {
  if (!p) return 0;
  auto it = c->live.find(p);
  if (it == c->live.end()) return fail(c, B200CONV_E_INVALID, "free of unknown device pointer %p", p);
  c->free_blocks.insert({it->second, p});
  c->live.erase(it);
  return 0;
}

// Temporaries of one call: returned to the pool when the call ends.
struct Scratch {
  b200conv_ctx* c;
  std::vector<void*> ptrs;
  explicit Scratch(b200conv_ctx* ctx) : c(ctx) {}
  ~Scratch() {
    for (void* p : ptrs) {
      if (c->capturing) c->capturing->retained.push_back(p);   // replays keep using it
      else pool_free(c, p);
    }
  }
  int get(size_t bytes, void** out) {
    int rc = pool_alloc(c, bytes, out);
    if (rc == 0) ptrs.push_back(*out);
    return rc;
  }
};

constexpr int kArrivals = 1024;

int check_status(b200conv_ctx* c) {
  // called after a stream synchronisation
  const int st = *c->h_status;
  if (st != kStatusOk) {
    *c->h_status = 0;
    // a launch that gave up may leave its counts behind
    CU_OK(c, cudaMemsetAsync(c->d_arrivals, 0, kArrivals * sizeof(unsigned int), c->stream));
    if (st == kStatusBadIndex)
      return fail(c, B200CONV_E_CUDA, "a kernel of the range-checked build computed an index outside its buffer "
                  "(the access was skipped); results are invalid");
    return fail(c, B200CONV_E_TIMEOUT, "a device-side wait ran out (status %d); results are invalid", st);
  }
  return 0;
}

// Orders the main stream after a collective that was started on the communication stream.
int join_comm(b200conv_ctx* c) {
  if (c->comm_pending) {
    CU_OK(c, cudaStreamWaitEvent(c->stream, c->ev_comm_done, 0));
    c->comm_pending = false;
  }
  return 0;
}

// Waits for the context's stream.  With a communicator the wait is a host watchdog: a rank whose
// peers have gone would otherwise block for ever inside the collective.  The stream is polled
// together with the communicator's asynchronous error state; on an error, or when the deadline
// passes, the communicator is aborted (its kernels then leave the GPU) and the call fails with
// B200CONV_E_NCCL.  The context stays usable for single-GPU work; a new communicator needs a new
// b200conv_nccl_init on every surviving rank.
int wait_stream(b200conv_ctx* c) {
  if (!c->comm) {
    CU_OK(c, cudaStreamSynchronize(c->stream));
    return 0;
  }
  typedef int (*async_err_fn)(void*, int*);
  typedef int (*abort_fn)(void*);
  async_err_fn get_err = (async_err_fn)dlsym(c->nccl_lib, "ncclCommGetAsyncError");
  abort_fn do_abort = (abort_fn)dlsym(c->nccl_lib, "ncclCommAbort");
  const auto deadline = std::chrono::steady_clock::now() + std::chrono::milliseconds(c->comm_timeout_ms);
  const char* why = nullptr;
  int nccl_state = 0;
  for (;;) {
    cudaError_t q = cudaStreamQuery(c->stream);
    if (q == cudaSuccess) return 0;
    if (q != cudaErrorNotReady) return fail(c, B200CONV_E_CUDA, "cudaStreamQuery: %s", cudaGetErrorString(q));
    if (get_err && get_err(c->comm, &nccl_state) == 0 && nccl_state != 0 && nccl_state != 7) {   // 0 ok, 7 in progress
      why = "the communicator reported an asynchronous error";
      break;
    }
    if (std::chrono::steady_clock::now() > deadline) {
      why = "a collective did not finish before the deadline";
      break;
    }
    std::this_thread::sleep_for(std::chrono::microseconds(20));
  }
  if (do_abort) do_abort(c->comm);
  c->comm = nullptr;
  c->comm_pending = false;
  cudaStreamSynchronize(c->stream);              // the aborted collective's kernels have left by now
  cudaGetLastError();
  return fail(c, B200CONV_E_NCCL, "%s (NCCL state %d, watchdog %d ms): communicator aborted", why, nccl_state,
              c->comm_timeout_ms);
}

int sync_and_check(b200conv_ctx* c) {
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "not allowed while a graph is being captured");
  int rcj = join_comm(c);
  if (rcj) return rcj;
  if ((rcj = wait_stream(c))) return rcj;
  if (c->down_pending) {            // background downloads end after the work they waited for
    CU_OK(c, cudaStreamSynchronize(c->down_stream));
    c->down_pending = false;
  }
  return check_status(c);
}

// ======================================================================================
// geometry
// ======================================================================================
int floordiv(int x, int y) {
  int q = x / y;
  if ((x % y != 0) && ((x < 0) != (y < 0))) --q;
  return q;
}
int pymod(int x, int y) { return x - floordiv(x, y) * y; }

int validate(b200conv_ctx* c, const b200conv_desc* d) {
  if (!d) return fail(c, B200CONV_E_INVALID, "null descriptor");
  if (d->dtype != B200CONV_F32 && d->dtype != B200CONV_F16)
    return fail(c, B200CONV_E_INVALID, "dtype must be float32 or float16");
  if (d->N < 0 || d->C < 0 || d->K < 0 || d->H <= 0 || d->W <= 0 || d->kH <= 0 || d->kW <= 0)
    return fail(c, B200CONV_E_INVALID, "negative or empty dimension");
  if (d->sH < 1 || d->sW < 1 || d->dilH < 1 || d->dilW < 1 || d->groups < 1)
    return fail(c, B200CONV_E_INVALID, "subsample, dilation and groups must be >= 1");
  if (d->padH_l < 0 || d->padH_r < 0 || d->padW_l < 0 || d->padW_r < 0)
    return fail(c, B200CONV_E_INVALID, "pads must be resolved (>= 0)");
  if (d->C % d->groups)
    return fail(c, B200CONV_E_INVALID, "images and kernel must have the same stack size "
                "(channels %d not divisible by groups %d)", d->C, d->groups);
  if (d->K % d->groups)
    return fail(c, B200CONV_E_INVALID, "the number of filters must be divisible by the number of groups");
  const int Ho = floordiv(d->H + d->padH_l + d->padH_r - ((d->kH - 1) * d->dilH + 1), d->sH) + 1;
  const int Wo = floordiv(d->W + d->padW_l + d->padW_r - ((d->kW - 1) * d->dilW + 1), d->sW) + 1;
  if (Ho != d->Ho || Wo != d->Wo || Ho <= 0 || Wo <= 0)
    return fail(c, B200CONV_E_INVALID,
                "shape inconsistency: bottom %d %d %d %d, weight %d %d %d %d, top %d %d %d %d "
                "(expected %d %d %d %d)",
                d->N, d->C, d->H, d->W, d->K, d->C / d->groups, d->kH, d->kW, d->N, d->K, d->Ho,
                d->Wo, d->N, d->K, Ho, Wo);
  return 0;
}

// Pixel tile for a grid of Wt x Ht x N positions holding at most `cap` rows: fewest tiles,
// each tile weighted by the MMA steps it costs (`kk` rows per step); widest box on ties.  even 2: sides that pooling windows do not straddle.
void choose_tile(b200conv_ctx* c, int Wt, int Ht, int N, int cap, int kk, int* bw, int* bh, int* bn, int even = 1) {
  SlabTile& memo = c->pixel_tiles[GeoKey{kGeoTile, Wt, Ht, N, cap, kk, even}];
  if (memo.found) {
    *bw = memo.wt; *bh = memo.th; *bn = memo.nb;
    return;
  }
  long long best = -1;
  *bw = *bh = *bn = 1;
  for (int w = even; w <= std::min(round_up(Wt, even), cap); w += even) {
    for (int h = even; h <= std::min(round_up(Ht, even), cap / w); h += even) {
      const int n = std::max(1, std::min(N, cap / (w * h)));
      const long long tiles = cdiv(Wt, w) * cdiv(Ht, h) * cdiv(N, n);
      const long long cost = tiles * (kk > 0 ? cdiv(w * h * n, kk) : 1);
      if (best < 0 || cost < best || (cost == best && w > *bw)) {
        best = cost;
        *bw = w; *bh = h; *bn = n;
      }
    }
  }
  memo.wt = *bw; memo.th = *bh; memo.nb = *bn;
  memo.found = true;
}

// 5-D channels-last view (c_in_group, group, w, h, n) of a [N][Hs][Ws][Cp] tensor that keeps
// every sH-th row and sW-th column starting at (rh, rw).
int make_view(b200conv_ctx* c, CUtensorMap* m, const void* base, int dtype, int Cg, int groups,
              int Cp, int Ws, int Hs, int N, int rh, int rw, int sH, int sW, int box_c, int bw,
              int bh, int bn, bool swizzle_32b_atoms = false) {
  const size_t es = elem_size(dtype);
  const int W2 = rw < Ws ? (Ws - rw + sW - 1) / sW : 0, H2 = rh < Hs ? (Hs - rh + sH - 1) / sH : 0;
  if (W2 <= 0 || H2 <= 0 || N <= 0 || Cg <= 0) return fail(c, B200CONV_E_INVALID, "empty view");
  cuuint64_t dims[5] = {(cuuint64_t)Cg, (cuuint64_t)groups, (cuuint64_t)W2, (cuuint64_t)H2, (cuuint64_t)N};
  cuuint64_t strides[4] = {(cuuint64_t)(groups > 1 ? Cg : Cp) * es, (cuuint64_t)sW * Cp * es,
                           (cuuint64_t)sH * Ws * Cp * es, (cuuint64_t)Hs * Ws * Cp * es};
  cuuint32_t box[5] = {(cuuint32_t)box_c, 1, (cuuint32_t)bw, (cuuint32_t)bh, (cuuint32_t)bn};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  for (int i = 0; i < 4; ++i)
    if (strides[i] % 16) return fail(c, B200CONV_E_UNSUPPORTED, "view stride %d not 16-byte aligned", i);
  const char* p = static_cast<const char*>(base) + (1LL * rh * Ws + rw) * Cp * es;
  if (reinterpret_cast<uintptr_t>(p) % 16) return fail(c, B200CONV_E_UNSUPPORTED, "view base not 16-byte aligned");
  CUresult r = c->encode(m, dtype == B200CONV_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                         5, const_cast<char*>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         swizzle_32b_atoms ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(c, B200CONV_E_CUDA, "cuTensorMapEncodeTiled(view) failed: %d", (int)r);
  return 0;
}

// Map over packed filters [mats][rows][ldc]: (cols, rows, mats), box (box_c, box_r, 1); with `groups`, mats = taps x
// groups as four dimensions (cols, rows, groups, taps), box (box_c, box_r, 1, box_t), so that a box holds box_t taps of a group.
int make_wmap(b200conv_ctx* c, CUtensorMap* m, const void* base, int dtype, int cols, int rows,
              int mats, int ldc, int box_c, int box_r, int groups = 0, int box_t = 1) {
  const size_t es = elem_size(dtype);
  const int g = std::max(1, groups);
  cuuint64_t dims[4] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)(groups ? g : mats), (cuuint64_t)(mats / g)};
  cuuint64_t strides[3] = {(cuuint64_t)ldc * es, (cuuint64_t)rows * ldc * es, (cuuint64_t)g * rows * ldc * es};
  cuuint32_t box[4] = {(cuuint32_t)box_c, (cuuint32_t)box_r, 1, (cuuint32_t)box_t};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = c->encode(m, dtype == B200CONV_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                         groups ? 4 : 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(c, B200CONV_E_CUDA, "cuTensorMapEncodeTiled(filters) failed: %d", (int)r);
  return 0;
}

// ---- forward-type launch shared by fwd and dgrad ------------------------------------------
struct FwdLikeArgs {
  const void* act;       // channels-last activations [N][Hs][Ws][Cp_in]
  int Hs, Ws, Cin_g, Cp_in;
  const void* wpacked;   // [(tap*groups+g)][n_out][ld_w]
  int ld_w, nmats;
  int n_out, groups, N;  // n_out: output channels per group as stored: a channels-last output of one group
                         // includes its pad channels, so that whole 16-byte pieces leave and no separate
                         // launch has to zero them
  int w_rows;            // rows of a packed filter matrix (the rows up to n_out read as zero)
  int dtype;
  int view_sH, view_sW;  // parity pitch of the activation views
  // Row folding (few input channels): `act` is [N][Hs][fold_Wp][Cp_in] with explicit zero columns;
  // the view's column index is the output column, its innermost extent runs over kW pixels x Cp_in
  // channels (Cin_g is that folded length) and only the filter rows remain as taps.
  // Output classes of the slab kernel (strided gradInputs): class, extent and element offset of each
  struct Class { int W, H; long long off; };
  std::vector<Class> classes;
  std::vector<uint8_t> tap_cls;
  bool fold = false;
  int fold_Wp = 0, fold_sW = 1;
};

// Folded activation view: (folded channel, 1, output column, input row of parity rh, image).
// Consecutive output columns start fold_sW pixels apart, so the rows of the view overlap in memory.
int make_fold_view(b200conv_ctx* c, CUtensorMap* m, const FwdLikeArgs& a, int rh, int sH, int box_c,
                   int bw, int bh, int bn) {
  const size_t es = elem_size(a.dtype);
  const int H2 = rh < a.Hs ? (a.Hs - rh + sH - 1) / sH : 0;
  if (H2 <= 0 || a.N <= 0) return fail(c, B200CONV_E_INVALID, "empty view");
  const size_t pix = (size_t)a.Cp_in * es, row = (size_t)a.fold_Wp * pix;
  cuuint64_t dims[5] = {(cuuint64_t)a.Cin_g, 1, (cuuint64_t)a.Ws, (cuuint64_t)H2, (cuuint64_t)a.N};
  cuuint64_t strides[4] = {row, (cuuint64_t)a.fold_sW * pix, (cuuint64_t)sH * row, (cuuint64_t)a.Hs * row};
  cuuint32_t box[5] = {(cuuint32_t)box_c, 1, (cuuint32_t)bw, (cuuint32_t)bh, (cuuint32_t)bn};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const char* p = static_cast<const char*>(a.act) + (size_t)rh * row;
  CUresult r = c->encode(m, a.dtype == B200CONV_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                         5, const_cast<char*>(p), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(c, B200CONV_E_CUDA, "cuTensorMapEncodeTiled(folded view) failed: %d", (int)r);
  return 0;
}

int make_act_view(b200conv_ctx* c, CUtensorMap* m, const FwdLikeArgs& a, int rh, int rw, int box_c, int bw,
                  int bh, int bn) {
  if (a.fold) return make_fold_view(c, m, a, rh, a.view_sH, box_c, bw, bh, bn);
  return make_view(c, m, a.act, a.dtype, a.Cin_g, a.groups, a.Cp_in, a.Ws, a.Hs, a.N, rh, rw, a.view_sH,
                   a.view_sW, box_c, bw, bh, bn);
}

// One past the last element of `out` that a launch over a Wt x Ht x N pixel grid with these element
// strides may write (what the range-checked build compares every store index with).
long long out_extent(const FwdLikeArgs& a, int Wt, int Ht, long long sn, long long sc, long long sh, long long sw,
                     long long off) {
  return off + (a.N - 1) * sn + (Ht - 1) * sh + (Wt - 1) * sw + (1LL * a.n_out * a.groups - 1) * sc + 1;
}

bool overlap(const void* a, size_t na, const void* b, size_t nb) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
  return x < y + nb && y < x + na;
}

// Kernel variants of a forward / gradInputs launch: the slab kernel (one activation slab per channel block) or
// the per-tap kernel, each with the widest tiles and a whole reduction per tile, or "spread": narrower tiles
// and / or a reduction cut into slices where that occupies more SMs; both also on pairs of CTAs; the
// columns kernel for layers of at most 64 filters, with more than 32 on pairs too.  The
// numbers appear in tuning files.
enum { kConvTap = 0, kConvSlab = 1, kConvSlabSpread = 2, kConvTapSpread = 3, kConvSlabPair = 4, kConvTapPair = 5, kConvCols = 6, kConvColsPair = 7, kConvVariants = 8 };
enum SlabMode { kSlabWide = 0, kSlabSpread, kSlabPair };      // of the slab kernel's tile search

SlabMode slab_mode(int variant) { return variant == kConvSlabSpread ? kSlabSpread : variant == kConvSlabPair ? kSlabPair : kSlabWide; }

// Clocks of an MMA over 128 rows x bn columns x 32 bytes of the reduction: half of the columns, and no less than its operands' reads of
// shared memory, 128 bytes a clock, take.  (MMAs of a tile with fewer filters are narrower, mma_columns(); the searches compare
// tiles as if they were full.)
int mma_clocks(int bn) { return std::max(bn / 2, 32 + bn / 4); }

// Do the MMAs of a pair leave out the columns of a tile that have no filters (mma_columns())?  Each CTA loads half of the columns' filters, always
// by a box of half a tile: with fewer columns the odd CTA's box starts earlier and brings rows that the even CTA has too.  Rows of whole 128-byte
// blocks cost little (a B200, whole tiles -> narrower, 56x56, float32: 128 -> 75 3x3 73 -> 61 us; float16 178 filters 47.0 -> 45.9).  Others reach into a
// line more each, and pay where the MMAs bound the tile: staged stores and not the very shallowest reductions (float32 40 -> 96 at 28x28 30.8 -> 27.2; float16
// 24 -> 192 32.8 -> 35.2), the lanes' stores with 128 columns, or with two rows to a line, from 25 stages on (float16 200 -> 75 51 -> 44, 100 -> 75 5x5 27.6 -> 25.7, 24 -> 75
// 5x5 69.9 -> 69.0, 32 -> 144 5x5 162 -> 151; 72 -> 75 3x3, 18 stages, 65 -> 74; 24 -> 140 5x5 104 -> 119).  The per-tap kernel, bound by L2, gains on whole blocks only (float32
// 128 -> 160 61.8 -> 57.3; 40 -> 160 49.7 -> 52.6, float16 200 -> 192 49.7 -> 53.4).
bool narrow_pair_mmas(const FwdLikeArgs& a, int bn, long long stages, bool per_tap, bool staged) {
  const long long row_bytes = a.ld_w * (long long)elem_size(a.dtype);
  if (row_bytes % 128 == 0) return true;
  if (per_tap) return false;
  return staged ? stages >= 18 || row_bytes >= 96 : stages >= 25 && (bn <= 128 || row_bytes % 64 == 0);
}

// Clocks that splitting the reduction of `items` = tiles x slices work items of rows x bn accumulators adds:
// raw accumulators leave at 32 B/clk per SM, and the reduction kernel costs about 4500 clocks of launch and
// latency plus its reads (48 B/clk per SM from L2).
long long split_clocks(long long items, int rows, int bn, int sms) {
  return 1LL * rows * bn * 4 / 32 + 4500 + items * rows * bn * 4 / (48LL * sms);
}

// Filter taps per stage of the slab kernel's filter ring.  A stage's barriers cost the issuing warp some 50 to 90 clocks of
// tensor time (about 190 when the times below were taken), so a stage holds as many taps as leaves the ring two
// or three stages: with one CTA 12 to 40 KB for narrow tiles and one tap for 128 and 256 filters, whose stages are 16
// and 32 KB already; a pair's CTAs hold half of the filters, so they take three taps of 128 and two of 256.
// Measured (one tap -> several, 64 images, float32 3x3): pairs 256 -> 256 at 56x56 401 -> 340 us, 128 -> 128 at
// 112x112 with pooling 406 -> 341, 64 -> 128 at 112x112 240 -> 201; float16 512 -> 512 at 7x7, 256 images 110 -> 89.
// 32-filter tiles, a filter row -> five taps: 32 groups of 8 channels at 28x28 184 -> 172 us.
int slab_tps(int bn, int ntaps, bool pair) {
  const int most = bn >= 256 ? (pair ? 2 : 1) : bn == 128 ? (pair ? 3 : 1) : bn == 64 ? 5 : 9;
  // a number that divides the taps and has straight-line code in the issuing warp
  for (int t : {9, 5, 4, 3, 2, 1})
    if (t <= most && ntaps % t == 0 && (t > 1 || ntaps == 1 || most == 1)) return t;
  return std::min(most == 9 ? 7 : std::min(most, 4), ntaps);
}
// Filter stages that a tile with the staged epilogue has to keep.
int slab_min_stages(bool pair, int tps) { return tps >= 9 || (pair && tps >= 3) ? 2 : 3; }

// Tile of the slab kernel.  kSlabWide: widest tile that holds the outputs, unsplit; kSlabSpread: the best over the
// tile widths and slice counts as well; kSlabPair: the tile of each CTA of a pair.  `found` is false when nothing fits.
SlabTile find_slab_tile(b200conv_ctx* c, const FwdLikeArgs& a, int ntaps, int Wt, int Ht, int Eh, int Ew, bool tma_layout_ok, SlabMode mode) {
  const bool spread = mode == kSlabSpread, pair = mode == kSlabPair;
  SlabTile& memo = c->slab_tiles[GeoKey{kGeoSlab, a.dtype, a.n_out, a.Cin_g, a.groups, a.N, Wt, Ht, ntaps, Eh, Ew, tma_layout_ok ? 1 : 0,
                                        c->epi.pool, c->num_sms, mode, (int)a.classes.size()}];
  if (memo.bn) return memo;
  const int kBK = a.dtype == B200CONV_F16 ? 64 : 32;
  const int ncls = std::max<int>(1, a.classes.size());
  const int bn_max = std::min(conv_umma_bn(a.n_out), 512 / (ncls == 3 ? 4 : ncls));
  const long long kblocks_n = cdiv(a.Cin_g, kBK);
  const long long es_out = (long long)elem_size(a.dtype);
  long long best_cost = -1, best_work = 0, best_tiles = 0;
  SlabTile best;
  best.bn = bn_max;
  if (pair && (bn_max < 64 || c->num_sms < 2)) { memo = best; return best; }
  const int units = pair ? c->num_sms / 2 : c->num_sms;
  for (int BN = bn_max; BN >= (spread ? 32 : pair ? std::max(64, bn_max / 2) : bn_max); BN /= 2) {
    const int tiles_co = (int)cdiv(a.n_out, BN);
    const int acc_cap = std::min(512 / (BN * ncls), 4);
    const int tps = slab_tps(BN, ntaps, pair);
    const int b_bytes = tps * (pair ? BN / 2 : BN) * 128;
    const long long stages = kblocks_n * cdiv(ntaps, tps);
    // one tile candidate: search the one with the least serial work per SM
    auto consider = [&](int wt, int th, int nb, int n_acc, long long slab_bytes, bool row) {
      const long long tiles = cdiv(Wt, wt) * cdiv(Ht, th) * cdiv(a.N, nb);
      const long long total = (pair ? cdiv(tiles, 2) : tiles) * tiles_co * a.groups;
      // Clocks of the busiest SM: per tile and (tap, channel block) 4 MMAs per accumulator plus
      // 120 clocks of stage hand-over in the issuing thread (slab_tps: 190 once, 50 to 90 since the issue is straight-line
      // code; with 120 or 190 24 layers of 64 to 512 channels get tiles of the same speed); then the accumulators are read
      // out, beside the next tile's MMAs when two accumulator sets fit the 512 TMEM columns.
      // Epilogue: through staged TMA stores when the output is channels-last and the staging
      // buffers fit beside two slabs and two filter stages (about 2500 clocks of latency per tile
      // plus the tile's bytes at the SM's store rate of 32 B/clk), else lane-per-row stores from
      // registers (1200 to 2500 clocks per 128 x 32 block: 16-byte pieces scattered over the pixel rows)
      const long long dense_rows = 1LL * wt * th * nb;
      const int ngr = n_acc == 3 ? 0 : 4 / n_acc;
      const long long stg = (dense_rows * 128 + 1023) / 1024 * 1024;
      const long long min_b = std::min<long long>(slab_min_stages(pair, tps), stages + 1);   // filter stages the staged epilogue insists on
      if (ncls > 1 && (n_acc > acc_cap || n_acc == 3)) return;
      if (c->epi.pool && ((wt | th) & 1)) return;          // pooling windows must not straddle tiles
      const bool tma_fit = tma_layout_ok && ngr > 0 && BN * es_out >= 128 && ngr * stg <= kSlabStageBytes &&
                           (total <= units ? ngr * stg <= 2 * slab_bytes + 2 * b_bytes
                                                : 2 * slab_bytes + min_b * b_bytes + kSlabStageBytes <= kSlabSmemBudget);
      // plus about 1500 clocks per tile for the pipeline to fill again
      // A pair's only accumulator of at most 128 columns is charged 96 clocks: its MMAs follow one another into the same
      // columns, and the search then prefers two accumulators.  With the 64 of mma_clocks(): 512 -> 512 3x3 at 14x14,
      // 128 images, 184.7 -> 234.6 us in float32 and 100 -> 122 in float16; 128 -> 128 at 28x28 float32 63 -> 79.
      const int mma_clk = pair && n_acc * ncls == 1 && BN <= 128 ? 96 : mma_clocks(BN);
      auto mma_part = [&](long long st) { return st * (1LL * std::min(tps, ntaps) * 4 * n_acc * mma_clk + 120) + 1500; };
      const long long whole = 1LL * kblocks_n * (ntaps * 4LL * n_acc * mma_clk + cdiv(ntaps, tps) * 120) + 1500;
      const long long epi_part = tma_fit ? 2500 + ncls * dense_rows * BN * es_out / 32 : 2400LL * n_acc * (BN / 32);
      const long long per_tile = 2 * n_acc * ncls * BN <= 512 ? std::max(whole, epi_part) : whole + epi_part;
      long long cost = cdiv(total, units) * per_tile;
      if (spread) cost += std::min(whole, epi_part);      // the last tile's read-out runs beside nothing (a few tiles per SM only)
      int splits = 1;
      const bool unsplit_ok = (!c->epi.pool && ncls == 1) || tma_fit;     // unsplit, pooling happens in the staged epilogue only
      if (spread && 2 * total <= c->num_sms)
        for (int s = 2; s <= std::min(stages, c->num_sms / total); ++s) {
          const long long cs = mma_part(cdiv(stages, s)) + split_clocks(total * s, 128 * n_acc, BN, c->num_sms);
          if (cs < cost || (s == 2 && !unsplit_ok)) { cost = cs; splits = s; }
        }
      if (splits == 1 && !unsplit_ok) return;
      const long long work = total * n_acc;
      if (best_cost < 0 || cost < best_cost || (cost == best_cost && work < best_work) ||
          (cost == best_cost && work == best_work && tiles < best_tiles)) {
        best_cost = cost; best_work = work; best_tiles = tiles;
        best.wt = wt; best.th = th; best.nb = nb; best.n_acc = n_acc; best.slab_bytes = (int)slab_bytes;
        best.bn = BN; best.splits = splits; best.row = row;
        best.found = true;
      }
    };
    for (int parts = 1; parts <= 16; ++parts) {
      const int wt = (int)cdiv(Wt, parts);
      if (parts > 1 && wt < 8) break;
      const int Ws = wt + Ew;
      if (Ws > 256) continue;
      const int shift_max = Eh * Ws + Ew;
      for (int th = 1; th <= Ht; ++th) {
        const int Hs = th + Eh;
        if (Hs > 256) break;
        const int per_img = Hs * Ws;
        if ((th - 1) * Ws + wt - 1 >= 128 * acc_cap) break;
        for (int nb = 1; nb <= std::min(a.N, 256); ++nb) {
          const long long last = 1LL * (nb - 1) * per_img + (th - 1) * Ws + (wt - 1);
          if (last >= 128LL * acc_cap) break;
          const int n_acc = (int)(last / 128) + 1;
          const long long rows = std::max<long long>(1LL * nb * per_img, 128LL * n_acc + shift_max);
          const long long slab_bytes = (rows * 128 + 1023) / 1024 * 1024;
          if (2 * slab_bytes + 2 * b_bytes > kSlabSmemBudget) break;
          consider(wt, th, nb, n_acc, slab_bytes, false);
        }
      }
    }
    if (Eh == 0 && Ew == 0 && Ht == 1 && a.N == 1 && Wt > 256 && !c->epi.pool && ncls == 1) {
      // one long row of pixels without halo (a flattened 1x1 layer): whole 128-pixel accumulators,
      // as many as still leave room for a second accumulator set
      if (spread || pair) {
        for (int n_acc = 1; n_acc <= (BN >= 256 ? 1 : 2); ++n_acc) consider(128 * n_acc, 1, 1, n_acc, 128 * 128 * n_acc, true);
      } else if (!best.found) {
        best.n_acc = BN >= 256 ? 1 : 2;
        best.wt = 128 * best.n_acc; best.th = best.nb = 1;
        best.slab_bytes = best.wt * 128;
        best.row = best.found = true;
      }
    }
  }
  memo = best;
  return best;
}

// Tile of the per-tap kernel: the pixel box with the fewest tiles; spread: also a narrower accumulator and
// slices of the reduction where that occupies more SMs.
SlabTile tap_tile(b200conv_ctx* c, const FwdLikeArgs& a, int ntaps, int Wt, int Ht, bool spread) {
  SlabTile best;
  choose_tile(c, Wt, Ht, a.N, 128, 0, &best.wt, &best.th, &best.nb, c->epi.pool ? 2 : 1);
  best.bn = conv_umma_bn(a.n_out);
  best.found = true;
  if (!spread) return best;
  const long long tiles = cdiv(Wt, best.wt) * cdiv(Ht, best.th) * cdiv(a.N, best.nb) * a.groups;
  const long long steps = ntaps * cdiv(a.Cin_g, a.dtype == B200CONV_F16 ? 64 : 32);
  const int bn_max = best.bn;
  long long best_cost = -1;
  for (int bn = bn_max; bn >= 32; bn /= 2) {
    const long long total = tiles * cdiv(a.n_out, bn);
    // a stage of the per-tap kernel is never shorter than its two TMA boxes take to issue (about 300 clocks)
    const long long step = std::max(300, 4 * mma_clocks(bn) + 60);
    const long long epi = 2400LL * bn / 32;
    const int most = 2 * total <= c->num_sms ? (int)std::min<long long>(steps, c->num_sms / total) : 1;
    for (int s = 1; s <= most; ++s) {
      const long long cost = s == 1 ? cdiv(total, c->num_sms) * std::max(steps * step, epi) + std::min(steps * step, epi)
                                    : cdiv(steps, s) * step + split_clocks(total * s, 128, bn, c->num_sms);
      if (best_cost < 0 || cost < best_cost) { best_cost = cost; best.bn = bn; best.splits = s; }
    }
  }
  return best;
}

// How a launch of `tiles` pair tiles on `units` pairs is cut: those beyond whole waves get `splits` pairs each.  Where whole tiles follow, the
// slices are added beside their MMAs, at most 8 slices, whose sums take no longer; what remains is the way through memory, some 6000 clocks (512 -> 2048
// 1x1 at 7x7, which would save 2700, took 32 us cut and 25 whole).  Else the raw
// accumulators and the second kernel count in full (split_clocks()).  256 -> 256 3x3 at 14x14, 128 images, float32: 98 tiles on 74 pairs, 24 of
// them cut in three.
struct PairCut { long long tiles; int splits; };
PairCut pair_cut(long long tiles, int units, long long kiters, int bn) {
  const long long rest = tiles % units, step = bn >= 256 ? 512 : 340;       // clocks per stage: MMAs, or 24 KB at 73 B/clk
  const bool beside = tiles > units;
  const long long most = rest ? std::min<long long>({units / rest, kiters, beside ? 8 : kiters}) : 1;
  if (most < 2) return PairCut{0, 1};
  const long long saved = kiters * step - cdiv(kiters, most) * step, cost = beside ? 6400 : split_clocks(2 * rest * most, 128, bn, 2 * units);
  return saved > cost + cost / 4 ? PairCut{rest, (int)most} : PairCut{0, 1};
}

// Slabs of a split launch and the parameters of its reduction that both kernels share.
template <class P>
int split_output(b200conv_ctx* c, Scratch& tmp, P& p, int bn, int rows, ConvReduceParams* q, long long pair_tiles = 0) {
  memset(q, 0, sizeof *q);
  const long long tiles = pair_tiles ? pair_tiles : 1LL * p.tiles_w * p.tiles_h * p.tiles_n * p.groups * p.tiles_co;
  if (tiles > 65535 / 2) return fail(c, B200CONV_E_INVALID, "too many split tiles");
  q->tiles = (int)tiles; q->pair = pair_tiles > 0;
  float* partial;
  const long long elems = (pair_tiles ? 2 : 1) * tiles * p.splits * rows * bn;
  int rc = tmp.get(sizeof(float) * elems, reinterpret_cast<void**>(&partial));
  if (rc) return rc;
  q->partial = p.partial = partial;
  q->partial_elems = p.partial_elems = elems;
  const int pl = p.epi.pool ? 2 : 1;
  q->out_elems = p.out_off + (p.Nimg - 1) * p.out_sn + (p.Ht / pl - 1) * p.out_sh + (p.Wt / pl - 1) * p.out_sw +
                 (1LL * p.n_out * p.groups - 1) * p.out_sc + 1;
  q->status = p.status;
  q->splits = p.splits; q->rows = rows; q->bn_cols = bn;
  q->tiles_w = p.tiles_w; q->tiles_h = p.tiles_h; q->tiles_n = p.tiles_n; q->tiles_co = p.tiles_co; q->groups = p.groups;
  q->Wt = p.Wt; q->Ht = p.Ht; q->Nimg = p.Nimg; q->n_out = p.n_out; q->n_real = p.n_real;
  q->out = p.out; q->bias = p.bias;
  q->out_sn = p.out_sn; q->out_sc = p.out_sc; q->out_sh = p.out_sh; q->out_sw = p.out_sw; q->out_off = p.out_off;
  q->relu = p.relu;
  q->epi = p.epi;
  return 0;
}

// Slab variant (conv_slab.cu) for launches whose taps all read one view.  Returns 0 when it was
// launched, 2 when the geometry does not fit (the caller then uses the per-tap kernel), or an
// error code.
int try_conv_slab(b200conv_ctx* c, const FwdLikeArgs& a, const std::vector<ConvTap>& taps, int rh,
                  int rw, int Wt, int Ht, void* out, long long sn, long long sc, long long sh,
                  long long sw, long long off, const void* bias, int relu, SlabMode mode) {
  if (taps.empty() || (int)taps.size() > kMaxTaps) return 2;
  const int ntap_all = (int)taps.size();
  int dh_min = taps[0].dh, dh_max = taps[0].dh, dw_min = taps[0].dw, dw_max = taps[0].dw;
  for (const ConvTap& t : taps) {
    dh_min = std::min<int>(dh_min, t.dh); dh_max = std::max<int>(dh_max, t.dh);
    dw_min = std::min<int>(dw_min, t.dw); dw_max = std::max<int>(dw_max, t.dw);
  }
  const int Eh = dh_max - dh_min, Ew = dw_max - dw_min;
  const int kBK = a.dtype == B200CONV_F16 ? 64 : 32;
  const long long kblocks_n = cdiv(a.Cin_g, kBK);
  const long long es_out = (long long)elem_size(a.dtype);
  // can the output leave through tiled TMA stores at all (channels-last, whole 128-byte channel rows, aligned)?
  const bool tma_layout_ok = sc == 1 && a.n_out % (int)(128 / es_out) == 0 && !c->epi.residual &&
                             (sw * es_out) % 16 == 0 && (sh * es_out) % 16 == 0 && (sn * es_out) % 16 == 0 &&
                             reinterpret_cast<uintptr_t>(static_cast<const char*>(out) + off * es_out) % 16 == 0;
  const SlabTile tile = find_slab_tile(c, a, ntap_all, Wt, Ht, Eh, Ew, tma_layout_ok, mode);
  if (!tile.found) return 2;
  const bool pair = mode == kSlabPair;
  const int BN = tile.bn, tiles_co = (int)cdiv(a.n_out, BN);
  const int b_rows = pair ? BN / 2 : BN;          // filters a CTA loads
  const int tps = slab_tps(BN, ntap_all, pair), b_bytes = tps * b_rows * 128;
#ifndef B200_PAIR_MIN_KBLOCKS
#define B200_PAIR_MIN_KBLOCKS 4
#endif
  constexpr long long kPairMinKblocks = B200_PAIR_MIN_KBLOCKS;
  // Flattened 1x1 layers with a deep reduction and 256-filter tiles: pairs of CTAs share the filter tile
  // (each loads half of it), which brings the operand traffic from L2 under what an SM can take.
  if (mode == kSlabWide && tile.row && c->use_pair &&
      a.dtype == B200CONV_F16 && BN == 256 && a.n_out % 64 == 0 && a.groups == 1 && !a.fold && taps.size() == 1 &&
      kblocks_n >= kPairMinKblocks && tma_layout_ok && c->num_sms >= 2 && c->epi.beta == 0.f && !c->epi.pool) {
    PairGemmParams q;
    memset(&q, 0, sizeof q);
    int rc = make_act_view(c, &q.view, a, rh, rw, 64, 128, 1, 1);
    if (rc) return rc;
    if ((rc = make_wmap(c, &q.wmap, a.wpacked, a.dtype, a.Cin_g, a.w_rows, a.nmats, a.ld_w, 64, 128))) return rc;
    cuuint64_t dims[4] = {(cuuint64_t)a.n_out, (cuuint64_t)Wt, 1, 1};
    cuuint64_t strides[3] = {(cuuint64_t)(sw * es_out), (cuuint64_t)(sh * es_out), (cuuint64_t)(sn * es_out)};
    cuuint32_t box[4] = {64, 128, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = c->encode(&q.out_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                           const_cast<char*>(static_cast<const char*>(out) + off * es_out), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS) {
      q.kblocks = (int)kblocks_n;
      q.tiles_pix = (int)cdiv(Wt, 256);
      q.tiles_co = (int)cdiv(a.n_out, 256);
      q.by_tiles_co = divisor(q.tiles_co);
      q.pixels = Wt; q.n_out = a.n_out; q.n_real = a.w_rows;
      q.stages = 5;
      q.bias = bias; q.relu = relu; q.epi = c->epi;
      q.status = c->d_status;
      q.wait_clocks = c->wait_clocks;
      c->last_variant = "gemm pair";
      KLAUNCH(c, kKConvUmma, launch_gemm_pair(q, c->num_sms, c->stream));
      return 0;
    }
  }
  SlabConvParams p;
  memset(&p, 0, sizeof p);
  const int b_slab = tile.slab_bytes;
  p.wt = tile.wt; p.th = tile.th; p.nb = tile.nb; p.n_acc = tile.n_acc;
  p.Ws = tile.wt + Ew; p.Hs = tile.th + Eh;
  p.dw_min = dw_min; p.dh_min = dh_min;
  p.slab_bytes = b_slab;
  p.splits = tile.splits;
  p.ncls = std::max<int>(1, a.classes.size());
  p.pair = pair;
  p.tps = tps;
  // Ring depths for `avail` bytes.  Activations come from HBM (the longer latency, and the stream
  // that bounds most layers): the slab ring gets up to 6 buffers once the filter ring holds what
  // one tile consumes (2 to 4 stages); the filter ring then takes what is left, up to 8 stages.
  const int per_tile = (int)std::min<long long>(8, cdiv(kblocks_n * cdiv((long long)taps.size(), tps), tile.splits));
  auto plan_rings = [&](long long avail, int* ss, int* bs) {
    if (2LL * b_slab + 2LL * b_bytes > avail) return false;
    const int fit = (int)std::min<long long>(8, (avail - 2LL * b_slab) / b_bytes);
    // a ring that holds exactly one tile's filters cannot start the next tile's filters before
    // this tile's MMAs are done: shallow reductions get one stage more than a tile consumes
    // (128 -> 512 1x1 forward: 100 -> 70 us with 3 instead of 2 stages)
    int b = std::min(fit, per_tile <= 2 ? per_tile + 1 : std::min(4, per_tile));
    int s_ = (int)std::max<long long>(2, std::min<long long>(6, (avail - 1LL * b * b_bytes) / b_slab));
    // a slab lasts as many stages as a channel block has: beyond two, as many slabs as four stages consume
    s_ = std::min(s_, 2 + (int)cdiv(4, cdiv((long long)taps.size(), tps)));
    b = (int)std::min<long long>(8, (avail - 1LL * s_ * b_slab) / b_bytes);
    *ss = s_; *bs = b;
    return true;
  };
  if (!plan_rings(kSlabSmemBudget, &p.s_stages, &p.b_stages)) return 2;
  if (tile.splits == 1) {
    // TMA-store epilogue: channels-last output whose 128-byte channel chunks never straddle a
    // group, 1/2/4 accumulators (so that the 16 epilogue warps split into equal groups)
    const long long tiles = cdiv(Wt, p.wt) * cdiv(Ht, p.th) * cdiv(a.N, p.nb);
    const long long total = (pair ? cdiv(tiles, 2) : tiles) * tiles_co * a.groups;
    const size_t es = elem_size(a.dtype);
    const long long dense_rows = 1LL * p.wt * p.th * p.nb;
    const int stage_bytes = (int)((dense_rows * 128 + 1023) / 1024 * 1024);
    const int ngroups = p.n_acc == 3 ? 0 : 4 / p.n_acc;
    const char* obase = static_cast<const char*>(out) + off * (long long)es;
    const int row_ch = (int)(128 / es);     // channels of one staged 128-byte row
    bool ok = sc == 1 && a.n_out % row_ch == 0 && BN >= row_ch && ngroups > 0 && !c->epi.residual &&
              ngroups * stage_bytes <= kSlabStageBytes && p.wt <= 256 && p.th <= 256 && p.nb <= 256 &&
              (sw * es) % 16 == 0 && (sh * es) % 16 == 0 && (sn * es) % 16 == 0 &&
              reinterpret_cast<uintptr_t>(obase) % 16 == 0;
    if (ok) {
      if (total <= (pair ? c->num_sms / 2 : c->num_sms)) {
        p.stage_off = 0;                       // one tile per CTA: operands are dead by then
        p.stage_nbuf = std::min(8, (p.s_stages * b_slab + p.b_stages * b_bytes) / stage_bytes) / std::max(1, ngroups) * ngroups;
        ok = p.stage_nbuf >= ngroups;
      } else {
        int ss = 0, bs = 0;
        if (plan_rings(kSlabSmemBudget - kSlabStageBytes, &ss, &bs) && bs >= std::min(slab_min_stages(pair, tps), per_tile + 1)) {
          p.s_stages = ss;
          p.b_stages = bs;
          p.stage_off = ss * b_slab + bs * b_bytes;
          p.stage_reserved = kSlabStageBytes;
          p.stage_nbuf = kSlabStageBytes / stage_bytes / ngroups * ngroups;
        } else {
          ok = false;
        }
      }
    }
    if (c->epi.pool && !ok) return fail(c, B200CONV_E_UNSUPPORTED, "this geometry's epilogue cannot pool");
    if (p.ncls > 1 && !ok) return 2;
    if (ok) {
      const int pl = c->epi.pool ? 2 : 1;       // pooled output: half the rows and columns (strides are the pooled tensor's)
      cuuint64_t strides[3] = {(cuuint64_t)(sw * es), (cuuint64_t)(sh * es), (cuuint64_t)(sn * es)};
      cuuint32_t box[4] = {(cuuint32_t)row_ch, (cuuint32_t)(p.wt / pl), (cuuint32_t)(p.th / pl), (cuuint32_t)p.nb};
      cuuint32_t estr[4] = {1, 1, 1, 1};
      CUresult r = CUDA_SUCCESS;
      for (int q = 0; q < p.ncls && r == CUDA_SUCCESS; ++q) {
        const FwdLikeArgs::Class k = a.classes.empty() ? FwdLikeArgs::Class{Wt, Ht, 0} : a.classes[q];
        cuuint64_t dims[4] = {(cuuint64_t)a.n_out * a.groups, (cuuint64_t)(k.W / pl), (cuuint64_t)(k.H / pl), (cuuint64_t)a.N};
        p.cls_W[q] = k.W; p.cls_H[q] = k.H;
        r = c->encode(&p.out_map[q], a.dtype == B200CONV_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                      4, const_cast<char*>(obase) + k.off * (long long)es, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
      }
      if (r == CUDA_SUCCESS) {
        p.tma_out = 1;
        p.stage_bytes = stage_bytes;
      } else {
        if (c->epi.pool) return fail(c, B200CONV_E_UNSUPPORTED, "this geometry's epilogue cannot pool");
        if (p.ncls > 1) return 2;
        plan_rings(kSlabSmemBudget, &p.s_stages, &p.b_stages);
        p.stage_off = p.stage_reserved = 0;
      }
    } else {
      p.stage_off = p.stage_reserved = 0;
    }
  }
  int rc = make_act_view(c, &p.view, a, rh, rw, kBK, p.Ws, p.Hs, p.nb);
  if (rc) return rc;
  p.tap_boxes = 0;
  for (size_t i = 1; i < taps.size(); ++i) p.tap_boxes |= taps[i].wmat != taps[i - 1].wmat + 1;
  rc = make_wmap(c, &p.wmap, a.wpacked, a.dtype, a.Cin_g, a.w_rows, a.nmats, a.ld_w, kBK, b_rows, a.groups, p.tap_boxes ? 1 : tps);
  if (rc) return rc;
  for (const ConvTap& t : taps) {
    p.tap_wmat[p.ntaps] = t.wmat;
    const int cls = p.ncls > 1 ? a.tap_cls[p.ntaps] : 0;
    const bool adds = p.ncls > 1 && std::find(a.tap_cls.begin(), a.tap_cls.begin() + p.ntaps, cls) != a.tap_cls.begin() + p.ntaps;
    p.tap_issue[p.ntaps] = slab_tap((t.dh - dh_min) * p.Ws + (t.dw - dw_min), cls * BN, adds);
    ++p.ntaps;
  }
  p.kblocks = (int)cdiv(a.Cin_g, kBK);
  p.tap_groups = (int)cdiv(p.ntaps, tps);
  p.groups = a.groups;
  p.Wt = Wt; p.Ht = Ht; p.Nimg = a.N;
  p.tiles_w = (int)cdiv(Wt, p.wt); p.tiles_h = (int)cdiv(Ht, p.th); p.tiles_n = (int)cdiv(a.N, p.nb);
  p.tiles_co = tiles_co;
  p.walk = tile_walk(p.splits, p.tiles_co, p.groups, p.tiles_w, p.tiles_h);
  p.n_out = a.n_out;
  p.n_mma = !pair || narrow_pair_mmas(a, BN, 1LL * p.ntaps * p.kblocks, false, p.tma_out) ? a.n_out : tiles_co * BN;
  p.n_real = a.w_rows;
  p.out = out; p.bias = bias;
  p.out_sn = sn; p.out_sc = sc; p.out_sh = sh; p.out_sw = sw; p.out_off = off;
  p.out_elems = out_extent(a, Wt, Ht, sn, sc, sh, sw, off);
  p.relu = relu;
  p.epi = c->epi;
  p.status = c->d_status;
  p.wait_clocks = c->wait_clocks;
  p.trace = c->trace;
  c->last_variant = p.ncls > 1 ? (pair ? "slab classes pair" : "slab classes") : pair ? "slab pair" : p.splits > 1 ? "slab split" : "slab";
  if (p.splits == 1) {
    KLAUNCH(c, kKConvUmma, launch_conv_slab(p, a.dtype, BN, c->num_sms, c->stream));
    return 0;
  }
  Scratch tmp(c);
  ConvReduceParams q;
  CU_OK(c, load_conv_slab(a.dtype, conv_umma_bn(a.n_out)));
  if ((rc = split_output(c, tmp, p, BN, p.n_acc * 128, &q))) return rc;
  q.Ws = p.Ws; q.Hs = p.Hs; q.wt = p.wt; q.th = p.th; q.nb = p.nb;
  KLAUNCH(c, kKConvUmma, launch_conv_slab(p, a.dtype, BN, c->num_sms, c->stream));
  KLAUNCH(c, kKConvReduce, launch_conv_reduce(q, a.dtype, c->stream));
  return 0;
}

// Columns kernel (conv_cols.cu) for layers of at most 64 filters per group whose taps are a whole grid of rows and columns over one view.
// Returns 0 when it was launched (launch false: when it could be), 2 when the geometry does not fit, or an error code.  d2s_C > 0: the output
// channels are the four classes of a stride-2 gradInputs with that many channels, `out` is the d2s_H x d2s_W gradient, channels-last, 16 bytes
// per pixel.
int try_conv_cols(b200conv_ctx* c, const FwdLikeArgs& a, const std::vector<ConvTap>& taps, int rh, int rw, int Wt, int Ht, void* out, long long sn,
                  long long sc, long long sh, long long sw, long long off, const void* bias, int relu, bool launch, bool pair, int d2s_C = 0,
                  int d2s_H = 0, int d2s_W = 0) {
  const int es = (int)elem_size(a.dtype), kBK = a.dtype == B200CONV_F16 ? 64 : 32;
  if (a.n_out > 64 || a.fold || !a.classes.empty() || c->epi.residual || sc != 1 || taps.size() < 2 || 1LL * Wt * Ht * a.N == 0) return 2;
  if (!d2s_C && (((sw | sh | sn) * es) % 16 || reinterpret_cast<uintptr_t>(static_cast<const char*>(out) + off * es) % 16)) return 2;
  ColsConvParams p;
  memset(&p, 0, sizeof p);
  // the grid: rows of the same dh, kW neighbouring matrices each, the same column offsets in every row
  std::vector<ConvTap> t = taps;
  std::sort(t.begin(), t.end(), [](const ConvTap& x, const ConvTap& y) { return x.wmat < y.wmat; });
  int kW = 0;
  while (kW < (int)t.size() && t[kW].dh == t[0].dh) ++kW;
  if (kW < 2 || kW > kMaxColTaps || t.size() % kW || (int)t.size() / kW > kMaxColTaps) return 2;
  p.kW = kW; p.kH = (int)t.size() / kW;
  p.dh_min = t[0].dh; p.dw_min = t[0].dw;
  int dh_max = t[0].dh, dw_max = t[0].dw;
  for (size_t i = 0; i < t.size(); ++i) {
    const ConvTap &first = t[i / kW * kW], &col = t[i % kW];
    if (t[i].dh != first.dh || t[i].dw != col.dw || t[i].wmat != first.wmat + (int)(i % kW)) return 2;
    p.dh_min = std::min<int>(p.dh_min, t[i].dh); dh_max = std::max<int>(dh_max, t[i].dh);
    p.dw_min = std::min<int>(p.dw_min, t[i].dw); dw_max = std::max<int>(dw_max, t[i].dw);
  }
  const int Eh = dh_max - p.dh_min, Ew = dw_max - p.dw_min;
  p.dil = std::abs(t[1].dw - t[0].dw);
  for (int j = 1; j < kW; ++j)
    if (t[j].dw - t[j - 1].dw != t[1].dw - t[0].dw || p.dil == 0) return 2;
  p.bn = a.n_out <= 16 ? 16 : a.n_out <= 32 ? 32 : 64;
  const int n_cols = kW * p.bn;
  if (pair && (p.bn != 64 || !c->use_pair || c->num_sms < 2)) return 2;
  if (n_cols > 256 || (d2s_C && (d2s_C > 4 || a.n_out > 16))) return 2;
  const bool rightwards = t[1].dw > t[0].dw;
  // a pair's MMAs take the columns of the even CTA's 32 filters first, then those of the other's
  const int step = pair ? p.bn / 2 : p.bn;
  p.pair = pair;
  p.col_first = rightwards ? 0 : (kW - 1) * step;
  p.col_step = rightwards ? step : -step;
  p.chunk_step = pair ? kW * step : 32;
  p.chunk_ch = std::min(32, p.bn);        // 32 at most: the groups of epilogue warps share a tile
  if (!d2s_C && a.groups > 1 && a.n_out % p.chunk_ch) return 2;
  // two accumulators where two sets of them fit 512 columns
  const int even = c->epi.pool ? 2 : 1, most_acc = 4 * n_cols <= 512 && !pair ? 2 : 1;
  const ColsTile tile = cols_tile(Wt, Ht, Eh, Ew, n_cols, most_acc, even);
  if (!tile.found) return 2;
  p.wt = tile.wt; p.th = tile.th; p.pitch = tile.pitch; p.n_acc = tile.n_acc;
  p.Hs = p.th + Eh;
  p.slab_bytes = std::max(p.Hs * p.pitch, 128 * p.n_acc + Eh * p.pitch) * 128;
  p.slab_bytes = (p.slab_bytes + 1023) / 1024 * 1024;
  // groups of epilogue warps: 4 / n_acc, one per chunk of channels, the rest on further tiles with accumulator sets of their own
  const int nchunks = d2s_C ? 1 : (int)cdiv(a.n_out, p.chunk_ch);
  p.step = 4 / p.n_acc / nchunks;
  while (p.step > 2 && p.step * p.n_acc * n_cols > 512) --p.step;
  p.sets = std::max(2, p.step);
  const int ngrp = nchunks * p.step;
  p.stage_bytes = d2s_C ? 0 : (p.wt * p.th * p.chunk_ch * es + 1023) / 1024 * 1024;
  int bufs = 1;
  p.s_stages = p.b_stages = 2;
  auto fits = [&](int s, int b, int f) { return 1LL * s * p.slab_bytes + 1LL * b * p.rps * (pair ? n_cols / 2 : n_cols) * 128 + 1LL * f * ngrp * p.stage_bytes <= kSlabSmemBudget; };
  p.rps = p.kH <= 5 && t.back().wmat == t[0].wmat + (int)t.size() - 1 ? p.kH : 1;      // rows that are neighbours in the packed filters
  if (!fits(2, 2, 1)) p.rps = 1;
  if (!fits(2, 2, 1)) return 2;
  if (!launch) return 0;
  // A CTA whose tiles are all of one group loads the filters once where the ring holds them whole.  For that the CTAs are a multiple of
  // the groups; those left out cost the rest some tiles more.  Groups of 32 channels, 3x3 at 28x28, 64 images, most tiles of a CTA with whole
  // multiples over those without -> time with over without: float32 1.06 0.91 (20 groups), 1.07 0.93 (23), 1.10 0.96 (15), 1.18 1.01 (25), 1.23 1.03 (30);
  // float16, whose filters are half the bytes, 1.02 0.96 (5), 1.06 0.95 (20, merged to 10), 1.07 1.06 (23), 1.10 1.09 (15), 1.18 1.16 (25).
  const int per_tile = (int)cdiv(a.Cin_g, kBK) * (p.kH / p.rps), units = pair ? c->num_sms / 2 : c->num_sms, whole = units / a.groups * a.groups;
  const long long pix_tiles = cdiv(Wt, p.wt) * cdiv(Ht, p.th) * a.N, tiles = (pair ? (pix_tiles + 1) / 2 : pix_tiles) * a.groups;
  p.resident = whole > 0 && per_tile <= kMaxColStages && fits(2, per_tile, 1) && (es == 4 ? 10 * cdiv(tiles, whole) <= 11 * cdiv(tiles, units) : 16 * cdiv(tiles, whole) <= 17 * cdiv(tiles, units));
  if (p.resident) p.b_stages = per_tile;
  for (char step : {'s', 'b', 'f', 'b', 's', 'b', 'b'}) {
    if (step == 'b' && p.resident) continue;
    const int s = p.s_stages + (step == 's'), b = p.b_stages + (step == 'b'), f = step == 'f' ? 2 : bufs;
    if (fits(s, b, f)) { p.s_stages = s; p.b_stages = b; bufs = f; }
  }
  p.stage_nbuf = bufs * ngrp;
  for (int i = 0; i < p.kH; ++i) { p.row_mat[i] = t[i * kW].wmat; p.row_shift[i] = (int16_t)((t[i * kW].dh - p.dh_min) * p.pitch); }
  int rc = make_act_view(c, &p.view, a, rh, rw, kBK, p.pitch, p.Hs, 1);
  if (rc) return rc;
  if ((rc = make_wmap(c, &p.wmap, a.wpacked, a.dtype, a.Cin_g, a.w_rows, a.nmats, a.ld_w, kBK, step, a.groups, p.rps * kW))) return rc;
  if (!d2s_C) {
    const int pl = even;
    cuuint64_t dims[4] = {(cuuint64_t)a.n_out * a.groups, (cuuint64_t)(Wt / pl), (cuuint64_t)(Ht / pl), (cuuint64_t)a.N};
    cuuint64_t strides[3] = {(cuuint64_t)(sw * es), (cuuint64_t)(sh * es), (cuuint64_t)(sn * es)};
    cuuint32_t box[4] = {(cuuint32_t)p.chunk_ch, (cuuint32_t)(p.wt / pl), (cuuint32_t)(p.th / pl), 1}, estr[4] = {1, 1, 1, 1};
    const int row_bytes = p.chunk_ch * es;
    CUresult r = c->encode(&p.out_map, a.dtype == B200CONV_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                           static_cast<char*>(out) + off * es, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           row_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return 2;
  }
  p.kblocks = (int)cdiv(a.Cin_g, kBK);
  p.groups = a.groups;
  p.Wt = Wt; p.Ht = Ht; p.Nimg = a.N;
  p.tiles_w = (int)cdiv(Wt, p.wt); p.tiles_h = (int)cdiv(Ht, p.th);
  p.by_groups = divisor(a.groups); p.by_tiles_w = divisor(p.tiles_w); p.by_tiles_h = divisor(p.tiles_h);
  p.n_out = a.n_out; p.n_real = a.w_rows;
  p.d2s = d2s_C > 0; p.d2s_C = d2s_C; p.d2s_H = d2s_H; p.d2s_W = d2s_W;
  p.out = out;
  p.out_elems = 1LL * a.N * d2s_H * d2s_W * (16 / es);
  p.bias = bias; p.relu = relu; p.epi = c->epi;
  p.status = c->d_status;
  p.wait_clocks = c->wait_clocks;
  c->last_variant = pair ? "columns pair" : "columns";
  KLAUNCH(c, kKConvUmma, launch_conv_cols(p, a.dtype, c->num_sms, c->stream));
  return 0;
}

// Can the per-tap kernel run on pairs of CTAs: staged TMA stores of whole 128-byte channel rows, tiles of at least 128 filters?
bool tap_pair_ok(b200conv_ctx* c, const FwdLikeArgs& a, const void* out, long long sn, long long sc, long long sh, long long sw, long long off) {
  const long long es = (long long)elem_size(a.dtype);
  return c->use_pair && c->num_sms >= 2 && a.n_out > 64 && a.n_out % (int)(128 / es) == 0 && sc == 1 && !c->epi.residual &&
         ((sw | sh | sn) * es) % 16 == 0 && reinterpret_cast<uintptr_t>(static_cast<const char*>(out) + off * es) % 16 == 0;
}

int run_conv_umma_one(b200conv_ctx* c, const FwdLikeArgs& a, const std::vector<ConvTap>& taps_in,
                      const std::vector<std::pair<int, int>>& view_parity, int Wt, int Ht, void* out,
                      long long sn, long long sc, long long sh, long long sw, long long off,
                      const void* bias, int relu, int variant) {
  if (variant == kConvCols || variant == kConvColsPair) {          // (a tuning file may name it for any geometry)
    const int rh = view_parity[0].first, rw = view_parity[0].second;
    const int rc = view_parity.size() == 1 && rh < a.Hs && rw < a.Ws
                       ? try_conv_cols(c, a, taps_in, rh, rw, Wt, Ht, out, sn, sc, sh, sw, off, bias, relu, true, variant == kConvColsPair) : 2;
    if (rc != 2) return rc;
    variant = kConvTap;
  }
  if (variant == kConvSlab || variant == kConvSlabSpread || variant == kConvSlabPair) {
    // the slab kernel reads one view (a tuning file may name it for a geometry with several)
    const bool one_view = view_parity.size() == 1;
    const int rh = view_parity[0].first, rw = view_parity[0].second;
    if (one_view && rh < a.Hs && rw < a.Ws) {
      const int rc = try_conv_slab(c, a, taps_in, rh, rw, Wt, Ht, out, sn, sc, sh, sw, off, bias, relu, slab_mode(variant));
      if (rc != 2) return rc;
    }
    variant = variant == kConvSlabSpread ? kConvTapSpread : kConvTap;
  }
  UmmaConvParams p;
  memset(&p, 0, sizeof p);
  const int kBK = a.dtype == B200CONV_F16 ? 64 : 32;
  const bool pair = variant == kConvTapPair && tap_pair_ok(c, a, out, sn, sc, sh, sw, off);     // (a tuning file may name it for any geometry)
  const SlabTile tile = tap_tile(c, a, (int)taps_in.size(), Wt, Ht, variant == kConvTapSpread);
  p.bw = tile.wt; p.bh = tile.th; p.bn = tile.nb;
  p.splits = tile.splits;
  p.bn_cols = tile.bn;
  // views that exist (non-empty); taps pointing at empty views contribute nothing
  std::vector<int> remap(view_parity.size(), -1);
  int nviews = 0;
  for (size_t v = 0; v < view_parity.size(); ++v) {
    const int rh = view_parity[v].first, rw = view_parity[v].second;
    if (rh >= a.Hs || rw >= a.Ws) continue;
    int rc = make_act_view(c, &p.views[nviews], a, rh, rw, kBK, p.bw, p.bh, p.bn);
    if (rc) return rc;
    remap[v] = nviews++;
  }
  for (const ConvTap& t : taps_in) {
    if (remap[t.view] < 0) continue;
    ConvTap u = t;
    u.view = static_cast<int16_t>(remap[t.view]);
    p.taps[p.ntaps++] = u;
  }
  if (p.ntaps == 0) return 1;  // caller zero-fills
  for (int v = nviews; v < kMaxViews; ++v) p.views[v] = p.views[0];
  p.nviews = nviews;
  const int BN = tile.bn;
  int rc = make_wmap(c, &p.wmap, a.wpacked, a.dtype, a.Cin_g, a.w_rows, a.nmats, a.ld_w, kBK, pair ? BN / 2 : BN);
  if (rc) return rc;
  p.kblocks = static_cast<int>(cdiv(a.Cin_g, kBK));
  p.splits = std::min(p.splits, p.ntaps * p.kblocks);
  p.groups = a.groups;
  p.Wt = Wt; p.Ht = Ht; p.Nimg = a.N;
  p.tiles_w = static_cast<int>(cdiv(Wt, p.bw));
  p.tiles_h = static_cast<int>(cdiv(Ht, p.bh));
  p.tiles_n = static_cast<int>(cdiv(a.N, p.bn));
  p.tiles_co = static_cast<int>(cdiv(a.n_out, BN));
  p.walk = tile_walk(p.splits, p.tiles_co, p.groups, p.tiles_w, p.tiles_h);
  p.n_out = a.n_out;
  p.n_mma = !pair || narrow_pair_mmas(a, BN, 1LL * p.ntaps * p.kblocks, true, true) ? a.n_out : p.tiles_co * BN;
  p.n_real = a.w_rows;
  p.out = out; p.bias = bias;
  p.out_sn = sn; p.out_sc = sc; p.out_sh = sh; p.out_sw = sw; p.out_off = off;
  p.out_elems = out_extent(a, Wt, Ht, sn, sc, sh, sw, off);
  p.relu = relu;
  p.epi = c->epi;
  p.status = c->d_status;
  p.wait_clocks = c->wait_clocks;
  if (pair) {
    const long long es = (long long)elem_size(a.dtype), tiles = cdiv(1LL * p.tiles_w * p.tiles_h * p.tiles_n, 2) * p.groups * p.tiles_co;
    const int pl = c->epi.pool ? 2 : 1;
    cuuint64_t dims[4] = {(cuuint64_t)a.n_out * a.groups, (cuuint64_t)(Wt / pl), (cuuint64_t)(Ht / pl), (cuuint64_t)a.N};
    cuuint64_t strides[3] = {(cuuint64_t)(sw * es), (cuuint64_t)(sh * es), (cuuint64_t)(sn * es)};
    cuuint32_t box[4] = {(cuuint32_t)kBK, (cuuint32_t)(p.bw / pl), (cuuint32_t)(p.bh / pl), (cuuint32_t)p.bn};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = c->encode(&p.out_map, a.dtype == B200CONV_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                           static_cast<char*>(out) + off * es, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS && c->epi.pool) return fail(c, B200CONV_E_UNSUPPORTED, "this geometry's epilogue cannot pool");
    if (r != CUDA_SUCCESS) return run_conv_umma_one(c, a, taps_in, view_parity, Wt, Ht, out, sn, sc, sh, sw, off, bias, relu, kConvTap);
    PairCut cut = pair_cut(tiles, c->num_sms / 2, 1LL * p.ntaps * p.kblocks, BN);
    unsigned int* counts = c->capturing ? c->capturing->arrivals : c->d_arrivals;
    if (cut.tiles >= tiles || 2 * cut.tiles > kArrivals) counts = nullptr;
    if (c->epi.pool && !counts) cut = PairCut{0, 1};                // the pair that adds the slices pools
    p.cut = (int)cut.tiles; p.splits = cut.splits;
    Scratch tmp(c);
    ConvReduceParams q;
    if (p.cut) {
      rc = split_output(c, tmp, p, BN, 128, &q, cut.tiles);
      if (rc && rc != B200CONV_E_NOMEM) return rc;
      if (rc) { p.cut = 0; p.splits = 1; }                        // no memory for the slices: whole reductions need none
      if (p.cut) p.arrivals = counts;
      p.walk.splits = divisor(p.splits);
      q.Ws = q.wt = p.bw; q.Hs = q.th = p.bh; q.nb = p.bn;
    }
    c->last_variant = p.splits > 1 ? "tap pair cut" : "tap pair";
    KLAUNCH(c, kKConvUmma, launch_conv_pair(p, a.dtype, c->num_sms, c->stream));
    if (p.cut && !p.arrivals) KLAUNCH(c, kKConvReduce, launch_conv_reduce(q, a.dtype, c->stream));
    return 0;
  }
  c->last_variant = p.splits > 1 ? "tap split" : "tap";
  if (p.splits == 1) {
    KLAUNCH(c, kKConvUmma, launch_conv_umma(p, a.dtype, c->num_sms, c->stream));
    return 0;
  }
  Scratch tmp(c);
  ConvReduceParams q;
  CU_OK(c, load_conv_umma(a.dtype, conv_umma_bn(a.n_out)));
  if ((rc = split_output(c, tmp, p, BN, 128, &q))) return rc;
  q.Ws = q.wt = p.bw; q.Hs = q.th = p.bh; q.nb = p.bn;
  KLAUNCH(c, kKConvUmma, launch_conv_umma(p, a.dtype, c->num_sms, c->stream));
  KLAUNCH(c, kKConvReduce, launch_conv_reduce(q, a.dtype, c->stream));
  return 0;
}

// Times of `n` variants in milliseconds: run(i) enqueues variant i and returns 0 or a code, which goes to codes[i] and
// leaves ms[i] at -1.  Returns an error of the timing itself.
// Every variant runs twice, the second time between two events (the first loads its code and makes the choices inside
// it); with one exception this decides: variants within a fifth (and the 4 us by which short launches differ between
// events) of the best are timed again in bursts of up to 7 back to back (8 did as well), the way a program issues them, once,
// and once more if they are still within 5 %.  Alone, a kernel of 5 us costs 5 us more and the chained launch hides nothing.
// All variants in two bursts each made the first passes of 32 cases take 200 ms together, this and rough_times() 127.
// `alone` takes the times of the single runs, those of variants that are then out of the running among them.
template <class Run>
int time_variants(b200conv_ctx* c, int n, Run run, float* ms, int* codes, bool rough = false, float* alone = nullptr) {
  if (!c->ev_tune0) {
    CU_OK(c, cudaEventCreate(&c->ev_tune0));
    CU_OK(c, cudaEventCreate(&c->ev_tune1));
  }
  auto timed = [&](int i, int reps, float* m) -> int {
    CU_OK(c, cudaEventRecord(c->ev_tune0, c->stream));
    for (int r = 0; r < reps && !codes[i]; ++r) codes[i] = run(i);
    CU_OK(c, cudaEventRecord(c->ev_tune1, c->stream));
    CU_OK(c, cudaStreamSynchronize(c->stream));
    CU_OK(c, cudaEventElapsedTime(m, c->ev_tune0, c->ev_tune1));
    *m = codes[i] ? -1.f : *m / reps;
    return 0;
  };
  auto best = [&] {
    float b = -1.f;
    for (int i = 0; i < n; ++i)
      if (ms[i] >= 0.f && (b < 0.f || ms[i] < b)) b = ms[i];
    return b;
  };
  for (int i = 0; i < n; ++i) {
    ms[i] = -1.f;
    if ((codes[i] = run(i))) continue;
    if (int rc = timed(i, 1, &ms[i])) return rc;
  }
  if (alone) std::copy(ms, ms + n, alone);
  const float first = best();
  if (first < 0.f || first > 0.5f || rough) return 0;     // long enough for one measurement
  const int reps = std::max(1, std::min(7, (int)(0.14f / std::max(first, 0.001f))));
  float limit = 1.2f * first + 0.004f;
  for (int round = 0; round < 2; ++round) {
    int close = 0;
    for (int i = 0; i < n; ++i) close += ms[i] >= 0.f && ms[i] <= limit;
    if (close < 2) return 0;
    for (int i = 0; i < n; ++i) {
      if (ms[i] < 0.f || ms[i] > limit) { ms[i] = -1.f; continue; }     // out of the running
      float m;
      if (int rc = timed(i, reps, &m)) return rc;
      ms[i] = round && m >= 0.f ? std::min(ms[i], m) : m;
    }
    limit = 1.05f * best();
  }
  return 0;
}

// Rough times of `n` variants that make choices of their own: those are the models' where none is remembered, each
// variant runs twice and the second run counts.  A variant far behind in this comparison is not worth its own timings.
template <class Run>
int rough_times(b200conv_ctx* c, int n, Run run, float* ms, int* codes) {
  c->model_only = true;
  const int rc = time_variants(c, n, run, ms, codes, true);
  c->model_only = false;
  return rc;
}
constexpr float kFarBehind = 1.4f;

// Picks the kernel variant.  All compute the same thing; which one is fastest depends on the layer (halo
// rows wasted by the slab grid against activations fetched once per tap; few tiles per SM against a second
// kernel that adds slices), so the first call of a geometry times the variants that apply with CUDA events
// and the context remembers the winner (the reference's GPU path selects its convolution algorithm the same
// way, theano/gpuarray/opt.py:2144-2222).  While a graph is being captured, or with timing off, the remembered
// choice or the model's is used.
int run_conv_umma(b200conv_ctx* c, const FwdLikeArgs& a, const std::vector<ConvTap>& taps_in,
                  const std::vector<std::pair<int, int>>& view_parity, int Wt, int Ht, void* out,
                  long long sn, long long sc, long long sh, long long sw, long long off,
                  const void* bias, int relu, bool allow_slab = true) {
  if (view_parity.size() != 1) allow_slab = false;
  auto run_one = [&](int variant) -> int {
    if (c->epi.pool && (variant == kConvCols || variant == kConvColsPair)) {
      const int rc = try_conv_cols(c, a, taps_in, view_parity[0].first, view_parity[0].second, Wt, Ht, out, sn, sc, sh, sw, off, bias, relu, true,
                                   variant == kConvColsPair);
      if (rc != 2) return rc;
      variant = kConvSlab;
    }
    if (c->epi.pool && variant == kConvTapPair && tap_pair_ok(c, a, out, sn, sc, sh, sw, off)) {
      const int rc = run_conv_umma_one(c, a, taps_in, view_parity, Wt, Ht, out, sn, sc, sh, sw, off, bias, relu, variant);
      if (rc != B200CONV_E_UNSUPPORTED) return rc;
    }
    if (c->epi.pool) {                // else the slab kernel pools, in its staged epilogue or in the reduction of its slices
      const int rc = try_conv_slab(c, a, taps_in, view_parity[0].first, view_parity[0].second, Wt, Ht, out, sn, sc, sh, sw, off, bias,
                                   relu, slab_mode(variant));
      return rc == 2 ? fail(c, B200CONV_E_UNSUPPORTED, "this geometry's epilogue cannot pool") : rc;
    }
    return run_conv_umma_one(c, a, taps_in, view_parity, Wt, Ht, out, sn, sc, sh, sw, off, bias, relu, variant);
  };
  auto run = [&](int variant) -> int {
    const int rc = run_one(variant);
    // no memory for the slices of a split reduction: whole reductions need none
    if (rc != B200CONV_E_NOMEM || (variant != kConvSlabSpread && variant != kConvTapSpread)) return rc;
    return run_one(variant == kConvSlabSpread ? kConvSlab : kConvTap);
  };
  int tsum = 0;
  for (const ConvTap& t : taps_in) tsum = tsum * 31 + t.dh * 7 + t.dw;
  GeoKey key{kGeoConv, a.dtype, a.N, a.Hs, a.Ws, a.Cin_g, a.n_out, a.groups, Wt, Ht, a.view_sH, a.view_sW, (int)taps_in.size(), tsum};
  key.add(sc);
  key.add(sw);
  const size_t es = elem_size(a.dtype);
  // Outputs that staged stores cannot write, with a residual or, channels-last, off the 16-byte boundaries, have a choice of their own, timed on
  // their first call: the layer's may be a kernel that has no other stores (per-tap pairs, columns), and the lanes' own stores are bound by
  // other things (64 -> 32 3x3 at 112x112, 64 images, float32, with a residual: per-tap 205 us, slab 279; NCHW without: 175, 150).  Where such a call
  // may not be timed, the layer's choice serves, or the best of the others when the layer was timed, which its choice then carries along
  // (choice + kConvVariants * (other + 1)).
  const bool lane_stores = c->epi.residual || (sc == 1 && (((sw | sh | sn) * (long long)es) % 16 ||
                                                           reinterpret_cast<uintptr_t>(static_cast<const char*>(out) + off * (long long)es) % 16));
  GeoKey lane_key = key;
  key.add(c->epi.pool * 4 + (c->use_pair ? 2 : 0) + (allow_slab ? 1 : 0));
  lane_key.add(8 + (c->use_pair ? 2 : 0) + (allow_slab ? 1 : 0));
  const bool tma = sc == 1 && a.n_out % (int)(128 / es) == 0 && !c->epi.residual && (sw * es) % 16 == 0 && (sh * es) % 16 == 0 &&
                   (sn * es) % 16 == 0 && reinterpret_cast<uintptr_t>(static_cast<const char*>(out) + off * (long long)es) % 16 == 0;
  // what cannot pool does not depend on the choice that an earlier call left (a split reduction pools any output)
  if (c->epi.pool && !(allow_slab && tma)) return fail(c, B200CONV_E_UNSUPPORTED, "this geometry's epilogue cannot pool");
  // A launch that adds to its own output (residual == y) must run once: it is not timed, and the choice is left to a
  // later call that may repeat it.
  const size_t out_bytes = es * out_extent(a, Wt, Ht, sn, sc, sh, sw, off);
  const bool in_place = c->epi.residual && overlap(c->epi.residual, out_bytes, out, out_bytes);
  const bool timed = c->autotune && !c->capturing && !c->model_only && !in_place;
  if (c->autotune) {
    auto it = c->algo_cache.find(lane_stores ? lane_key : key);
    if (it != c->algo_cache.end()) return run(it->second % kConvVariants);
    if (lane_stores && !timed && (it = c->algo_cache.find(key)) != c->algo_cache.end()) {
      const int layers = it->second % kConvVariants, lanes = it->second / kConvVariants - 1;
      if (layers <= kConvSlabPair) return run(layers);
      if (lanes >= 0) return run(lanes);
    }
  }
  // the variants that apply, the static preference last
  int cand[kConvVariants], ncand = 0;
  const SlabTile narrow = tap_tile(c, a, (int)taps_in.size(), Wt, Ht, true);
  const bool tap_spread = narrow.splits > 1 || narrow.bn != conv_umma_bn(a.n_out);
  if (!c->epi.pool) {
    cand[ncand++] = kConvTap;
    if (tap_spread) cand[ncand++] = kConvTapSpread;
  }
  const SlabTile t = tap_tile(c, a, (int)taps_in.size(), Wt, Ht, false);
  if (tap_pair_ok(c, a, out, sn, sc, sh, sw, off) &&
      cdiv(cdiv(Wt, t.wt) * cdiv(Ht, t.th) * cdiv(a.N, t.nb), 2) * cdiv(a.n_out, t.bn) * a.groups >= c->num_sms / 4)
    cand[ncand++] = kConvTapPair;
  for (int v = kConvCols; allow_slab && v <= kConvColsPair; ++v)
    if (try_conv_cols(c, a, taps_in, view_parity[0].first, view_parity[0].second, Wt, Ht, out, sn, sc, sh, sw, off, bias, relu, false, v == kConvColsPair) == 0)
      cand[ncand++] = v;
  if (allow_slab) {
    int eh[2] = {0, 0}, ew[2] = {0, 0};
    for (size_t i = 0; i < taps_in.size(); ++i) {
      const ConvTap& t = taps_in[i];
      if (i == 0) { eh[0] = eh[1] = t.dh; ew[0] = ew[1] = t.dw; }
      eh[0] = std::min<int>(eh[0], t.dh); eh[1] = std::max<int>(eh[1], t.dh);
      ew[0] = std::min<int>(ew[0], t.dw); ew[1] = std::max<int>(ew[1], t.dw);
    }
    const SlabTile w = find_slab_tile(c, a, (int)taps_in.size(), Wt, Ht, eh[1] - eh[0], ew[1] - ew[0], tma, kSlabWide);
    const SlabTile n = find_slab_tile(c, a, (int)taps_in.size(), Wt, Ht, eh[1] - eh[0], ew[1] - ew[0], tma, kSlabSpread);
    if (c->epi.pool && !w.found) return fail(c, B200CONV_E_UNSUPPORTED, "this geometry's epilogue cannot pool");
    // pairs of CTAs where at least half of the SMs get work (below, the variants that spread a tile are ahead)
    const SlabTile m = c->use_pair ? find_slab_tile(c, a, (int)taps_in.size(), Wt, Ht, eh[1] - eh[0], ew[1] - ew[0], tma, kSlabPair) : SlabTile();
    const bool pair = m.found && cdiv(cdiv(Wt, m.wt) * cdiv(Ht, m.th) * cdiv(a.N, m.nb), 2) * cdiv(a.n_out, m.bn) * a.groups >= c->num_sms / 4;
    if (w.found) cand[ncand++] = kConvSlab;
    if (n.found && (!w.found || n.splits > 1 || n.bn != w.bn || n.wt != w.wt || n.th != w.th || n.nb != w.nb)) cand[ncand++] = kConvSlabSpread;
    if (pair) cand[ncand++] = kConvSlabPair;
  }
  if (ncand == 0) return fail(c, B200CONV_E_UNSUPPORTED, "this geometry's epilogue cannot pool");
  if (!timed || ncand == 1) return run(cand[ncand - 1]);
  int best = -1, lane_best = -1, codes[kConvVariants];
  float ms[kConvVariants], alone[kConvVariants], best_ms = 0.f, lane_ms = 0.f;
  if (const int rc = time_variants(c, ncand, [&](int i) { return run(cand[i]); }, ms, codes, false, alone)) return rc;
  for (int i = 0; i < ncand; ++i) {
    if (codes[i] && !(codes[i] == B200CONV_E_UNSUPPORTED && c->epi.pool)) return codes[i];
    if (ms[i] >= 0.f && (best < 0 || ms[i] < best_ms)) { best = cand[i]; best_ms = ms[i]; }
    // the best of those that write any output; a single run's time counts where it did not come to bursts
    const float m = ms[i] >= 0.f ? ms[i] : alone[i];
    if (cand[i] <= kConvSlabPair && m >= 0.f && (lane_best < 0 || m < lane_ms)) { lane_best = cand[i]; lane_ms = m; }
  }
  if (best < 0) return fail(c, B200CONV_E_UNSUPPORTED, "this geometry's epilogue cannot pool");
  if (lane_stores) c->algo_cache[lane_key] = best;
  else c->algo_cache[key] = best > kConvSlabPair && lane_best >= 0 ? best + kConvVariants * (lane_best + 1) : best;
  return run(best);     // the last run may have been another variant: leave the output of the chosen one
}

int to_nhwc(b200conv_ctx* c, Scratch& tmp, const void* src, int N, int C, int H, int W, int dtype,
            const void** out) {
  const int Cp = pad_channels(C, dtype);
  void* buf;
  int rc = tmp.get(elem_size(dtype) * (size_t)N * H * W * Cp, &buf);
  if (rc) return rc;
  KLAUNCH(c, kKTranspose, launch_transpose(src, buf, N, C, H * W, H * W, Cp, dtype, c->stream));
  *out = buf;
  return 0;
}

// Row folding applies to ungrouped layers whose whole filter row (kW pixels x padded channels)
// fits one reduction block of the MMA: the 3-channel stems of VGG and ResNet.
bool fold_ok(const b200conv_desc& d) {
  const int kBK = d.dtype == B200CONV_F16 ? 64 : 32;
  const int Cp = pad_channels(d.C, d.dtype);
  return d.groups == 1 && d.dilW == 1 && d.kW > 1 && Cp * d.kW <= kBK && Cp * 2 <= kBK && d.kH <= kMaxTaps &&
         d.sH <= kMaxViews && d.N > 0 && d.C > 0 && d.K > 0;
}
// Padded row length: left pad, the image, and enough zero columns on the right for the last
// output's kBK / Cp pixels.
int fold_width(const b200conv_desc& d) {
  const int kBK = d.dtype == B200CONV_F16 ? 64 : 32;
  const int Cp = pad_channels(d.C, d.dtype);
  return std::max(d.padW_l + d.W + d.padW_r, (d.Wo - 1) * d.sW + kBK / Cp);
}

// Space-to-depth applies to ungrouped stride-2 layers with at most 4 input channels whose filter
// rows span at most kS2dPixels blocks of 2 x 2 pixels: the 7x7 stride-2 stem of ResNet.  t0 / q0:
// first block row / column a filter touches relative to the output position; ntaps: block rows.
bool s2d_ok(const b200conv_desc& d, int* t0, int* ntaps, int* q0) {
  if (d.groups != 1 || d.sH != 2 || d.sW != 2 || d.dilH != 1 || d.dilW != 1) return false;
  if (d.N <= 0 || d.C <= 0 || d.K <= 0 || 4 * d.C > kS2dChannels) return false;
  *t0 = floordiv(-d.padH_l, 2);
  *q0 = floordiv(-d.padW_l, 2);
  *ntaps = floordiv(d.kH - 1 - d.padH_l, 2) - *t0 + 1;
  const int span = floordiv(d.kW - 1 - d.padW_l, 2) - *q0 + 1;
  return span >= 1 && span <= kS2dPixels && *ntaps >= 1 && *ntaps <= kMaxTaps;
}

// A 1x1, stride-1, unpadded convolution on channels-last tensors is a plain matrix product over
// the N*H*W pixels.  Seen as ONE image of one row of N*H*W pixels it tiles into whole 128-pixel
// tiles, where tiles cut from 56x56, 28x28, 14x14 or 7x7 images leave 12 to 25 % of the
// accumulator rows empty.
bool flatten_1x1(const b200conv_desc& d, bool all_nhwc, b200conv_desc* f) {
  if (!all_nhwc || d.kH != 1 || d.kW != 1 || d.sH != 1 || d.sW != 1) return false;
  if (d.padH_l | d.padH_r | d.padW_l | d.padW_r) return false;
  if (d.N == 1 && d.H == 1) return false;       // already one row
  const long long P = 1LL * d.N * d.H * d.W;
  if (P <= 0 || P > (1LL << 30)) return false;
  *f = d;
  f->N = 1; f->H = 1; f->W = (int)P;
  f->Ho = 1; f->Wo = (int)P;
  return true;
}

// ---- filters packed ahead of time ------------------------------------------------------------
std::string pack_key(const void* w, int K, int Cg, int kH, int kW, int groups, int flip, int mode, int ldc, int dtype) {
  char key[160];
  snprintf(key, sizeof key, "%p.%d.%d.%d.%d.%d.%d.%d.%d.%d", w, K, Cg, kH, kW, groups, flip, mode, ldc, dtype);
  return key;
}
// The packed form of `w` if b200conv_prepack made one and the filters have not been reported
// changed since; nullptr otherwise (the caller then packs into scratch memory as usual).
// kScratchFilters among the flags of a direction: `w` is scratch of this call (filters uploaded from the host, merged
// groups), whose address may be that of a bank that was packed ahead of time and has gone since.
constexpr int kScratchFilters = 1 << 30;
void* packed_lookup(b200conv_ctx* c, const void* w, int K, int Cg, int kH, int kW, int groups, int flip, int mode,
                    int ldc, int dtype) {
  if (c->packed.empty()) return nullptr;
  auto it = c->packed.find(pack_key(w, K, Cg, kH, kW, groups, flip, mode, ldc, dtype));
  return it != c->packed.end() && it->second.valid ? it->second.ptr : nullptr;
}
// Which packing the plain (not folded, merged or space-to-depth) forward (mode 0) / gradInputs
// (mode 1) path of a geometry performs; false when that path packs nothing or is not taken.
bool fold_ok(const b200conv_desc& d);
bool s2d_ok(const b200conv_desc& d, int* t0, int* ntaps, int* q0);
bool plain_pack(const b200conv_desc& d, int mode, int* ldc) {
  if (!umma_ok(d) || merge_factor(d) > 1) return false;
  const int Cg = d.C / d.groups, Kg = d.K / d.groups;
  if (mode == 0) {
    int a, b, e;
    if (s2d_ok(d, &a, &b, &e) || fold_ok(d)) return false;
    *ldc = pad_channels(Cg, d.dtype);
    return !(d.kH == 1 && d.kW == 1 && *ldc == Cg);        // a 1x1 bank is read in place
  }
  const int ncls = d.sH * d.sW;
  if (ncls > 1 && d.groups == 1 && ncls * d.C <= 64) return false;   // merged parity classes pack their own form
  *ldc = pad_channels(Kg, d.dtype);
  return true;
}

// ======================================================================================
// the three directions on device pointers
// ======================================================================================
// merge > 1: `d` is a layer whose groups were merged that many at a time, `w` still the bank of its own groups.
int fwd_device(b200conv_ctx* c, const b200conv_desc& d, const void* x, const void* w,
               const void* bias, void* y, int flags, int merge = 1) {
  const int Cg = d.C / d.groups, Kg = d.K / d.groups;
  const size_t es = elem_size(d.dtype);
  const bool out_nhwc = flags & B200CONV_OUT_NHWC, in_nhwc = flags & B200CONV_IN_NHWC;
  const int Kp = pad_channels(d.K, d.dtype);
  if (d.N == 0 || d.K == 0) return 0;
  if (c->epi.pool) {
    if (!out_nhwc || (d.Ho & 1) || (d.Wo & 1) || (flags & B200CONV_FORCE_DIRECT) || c->epi.residual)
      return fail(c, B200CONV_E_UNSUPPORTED, "the pooling epilogue needs a channels-last output with even height and width");
    if (merge_factor(d) > 1 || !umma_ok(d))
      return fail(c, B200CONV_E_UNSUPPORTED, "this geometry's epilogue cannot pool");
  }
  b200conv_desc flat;
  if (!(flags & B200CONV_FORCE_DIRECT) && !c->epi.pool && flatten_1x1(d, in_nhwc && out_nhwc, &flat))
    return fwd_device(c, flat, x, w, bias, y, flags, merge);
  Scratch tmp(c);
  // the direct kernels take the bias as float32; the tensor-core kernels read it in the data type
  const float* bias_f = d.dtype == B200CONV_F32 ? static_cast<const float*>(bias) : nullptr;
  auto convert_bias = [&]() -> int {
    if (!bias || bias_f) return 0;
    float* f;
    int r = tmp.get(sizeof(float) * d.K, reinterpret_cast<void**>(&f));
    if (r) return r;
    KLAUNCH(c, kKPack, launch_convert_bias(bias, f, d.K, d.dtype, c->stream));
    bias_f = f;
    return 0;
  };
  if (bias && out_nhwc && Kp != d.K) {           // the epilogue reads one value per stored channel
    void* padded;
    int rc = tmp.get(es * Kp, &padded);
    if (rc) return rc;
    KLAUNCH(c, kKPack, launch_pad_bias(bias, padded, d.K, Kp, d.dtype, c->stream));
    bias = padded;
  }
  const int mg = (flags & B200CONV_FORCE_DIRECT) || merge > 1 ? 1 : merge_factor(d);
  if (mg > 1) {
    b200conv_desc dm = d;
    dm.groups = d.groups / mg;
    int a, b, e;
    const bool stem = fold_ok(dm) || (!(flags & B200CONV_NO_S2D) && s2d_ok(dm, &a, &b, &e));     // those pack another form
    if (umma_ok(dm) && !stem) return fwd_device(c, dm, x, w, bias, y, flags | kScratchFilters, mg);
    if (umma_ok(dm)) {
      void* wm;
      int rc = tmp.get(es * (size_t)d.K * Cg * mg * d.kH * d.kW, &wm);
      if (rc) return rc;
      KLAUNCH(c, kKPack, launch_merge_groups(w, wm, d.K, Cg, Kg, mg, d.kH * d.kW, 0, d.dtype, c->stream));
      return fwd_device(c, dm, x, wm, bias, y, flags | kScratchFilters);
    }
  }
  const bool use_umma = !(flags & B200CONV_FORCE_DIRECT) && umma_ok(d);
  if (!use_umma) {
    if (flags & B200CONV_FORCE_UMMA) return fail(c, B200CONV_E_UNSUPPORTED, "geometry not covered by the tensor-core kernel");
    if (in_nhwc || out_nhwc) return fail(c, B200CONV_E_UNSUPPORTED, "direct kernels take NCHW tensors only");
    if (int r = convert_bias()) return r;
    KLAUNCH(c, kKDirect, launch_direct_fwd(d, x, w, bias_f, y, (flags & B200CONV_RELU) ? 1 : 0, c->epi, c->stream));
    c->last_algo = "direct";
    return 0;
  }
  const int Cp = pad_channels(d.C, d.dtype);
  int s2_t0 = 0, s2_nt = 0, s2_q0 = 0;
  if (!(flags & B200CONV_NO_S2D) && s2d_ok(d, &s2_t0, &s2_nt, &s2_q0)) {
    // stride 2 with very few channels: 2 x 2 pixel blocks become channels, the layer a stride-1
    // layer with one tap per block row whose reduction runs over kS2dPixels consecutive blocks
    const int win = kS2dPixels * kS2dChannels;
    const int H2 = (d.H + 1) / 2, Wq = d.Wo + kS2dPixels - 1;
    void *xs, *wf;
    int rc = tmp.get(es * (size_t)d.N * H2 * Wq * kS2dChannels, &xs);
    if (rc) return rc;
    KLAUNCH(c, kKTranspose, launch_pad_s2d(x, xs, d.N, d.C, d.H, d.W, Cp, H2, Wq, s2_q0, in_nhwc ? 1 : 0,
                                           d.dtype, c->stream));
    if ((rc = tmp.get(es * (size_t)s2_nt * d.K * win, &wf))) return rc;
    KLAUNCH(c, kKPack, launch_pack_filters_s2d(w, wf, d.K, d.C, d.kH, d.kW, s2_nt, s2_t0, s2_q0, d.padH_l,
                                               d.padW_l, win, d.flip, d.dtype, c->stream));
    std::vector<ConvTap> taps;
    std::vector<std::pair<int, int>> parity(1, {0, 0});
    for (int t = 0; t < s2_nt; ++t) {
      ConvTap tp;
      tp.dh = (int16_t)(t + s2_t0); tp.dw = 0; tp.view = 0; tp.wmat = (int16_t)t;
      taps.push_back(tp);
    }
    FwdLikeArgs a;
    a.act = xs; a.Hs = H2; a.Ws = d.Wo; a.Cin_g = win; a.Cp_in = kS2dChannels;
    a.wpacked = wf; a.ld_w = win; a.nmats = s2_nt;
    a.n_out = out_nhwc ? Kp : d.K; a.w_rows = d.K; a.groups = 1; a.N = d.N; a.dtype = d.dtype;
    a.view_sH = 1; a.view_sW = 1;
    a.fold = true; a.fold_Wp = Wq; a.fold_sW = 1;
    long long sn, sc, sh, sw;
    if (out_nhwc) {
      const int pl = c->epi.pool ? 2 : 1;
      sn = 1LL * (d.Ho / pl) * (d.Wo / pl) * Kp; sc = 1; sh = 1LL * (d.Wo / pl) * Kp; sw = Kp;
    } else {
      sn = 1LL * d.K * d.Ho * d.Wo; sc = 1LL * d.Ho * d.Wo; sh = d.Wo; sw = 1;
    }
    rc = run_conv_umma(c, a, taps, parity, d.Wo, d.Ho, y, sn, sc, sh, sw, 0, bias,
                       (flags & B200CONV_RELU) ? 1 : 0, !(flags & B200CONV_NO_SLAB));
    if (rc == 1) return fail(c, B200CONV_E_CUDA, "internal: empty space-to-depth view");
    c->last_algo = "umma";
    return rc;
  }
  if (fold_ok(d)) {
    // few input channels: one reduction block holds a whole filter row (kW pixels x Cp channels)
    const int kBK = d.dtype == B200CONV_F16 ? 64 : 32;
    const int Wp = fold_width(d);
    void *xp, *wf;
    int rc = tmp.get(es * (size_t)d.N * d.H * Wp * Cp, &xp);
    if (rc) return rc;
    KLAUNCH(c, kKTranspose, launch_pad_fold(x, xp, d.N, d.C, d.H, d.W, Cp, Wp, d.padW_l, in_nhwc ? 1 : 0,
                                            d.dtype, c->stream));
    if ((rc = tmp.get(es * (size_t)d.kH * d.K * kBK, &wf))) return rc;
    KLAUNCH(c, kKPack, launch_pack_filters_fold(w, wf, d.K, d.C, d.kH, d.kW, Cp, kBK, d.flip, d.dtype, c->stream));
    std::vector<ConvTap> taps;
    std::vector<std::pair<int, int>> parity;
    for (int i = 0; i < d.kH; ++i) {
      const int ah = i * d.dilH - d.padH_l, rh = pymod(ah, d.sH);
      int v = -1;
      for (size_t q = 0; q < parity.size(); ++q)
        if (parity[q].first == rh) v = (int)q;
      if (v < 0) { v = (int)parity.size(); parity.push_back({rh, 0}); }
      ConvTap t;
      t.dh = (int16_t)floordiv(ah, d.sH); t.dw = 0; t.view = (int16_t)v; t.wmat = (int16_t)i;
      taps.push_back(t);
    }
    FwdLikeArgs a;
    a.act = xp; a.Hs = d.H; a.Ws = d.Wo; a.Cin_g = kBK; a.Cp_in = Cp;
    a.wpacked = wf; a.ld_w = kBK; a.nmats = d.kH;
    a.n_out = out_nhwc ? Kp : d.K; a.w_rows = d.K; a.groups = 1; a.N = d.N; a.dtype = d.dtype;
    a.view_sH = d.sH; a.view_sW = 1;
    a.fold = true; a.fold_Wp = Wp; a.fold_sW = d.sW;
    long long sn, sc, sh, sw;
    if (out_nhwc) {
      const int pl = c->epi.pool ? 2 : 1;
      sn = 1LL * (d.Ho / pl) * (d.Wo / pl) * Kp; sc = 1; sh = 1LL * (d.Wo / pl) * Kp; sw = Kp;
    } else {
      sn = 1LL * d.K * d.Ho * d.Wo; sc = 1LL * d.Ho * d.Wo; sh = d.Wo; sw = 1;
    }
    rc = run_conv_umma(c, a, taps, parity, d.Wo, d.Ho, y, sn, sc, sh, sw, 0, bias,
                       (flags & B200CONV_RELU) ? 1 : 0, !(flags & B200CONV_NO_SLAB));
    if (rc == 1) return fail(c, B200CONV_E_CUDA, "internal: empty folded view");
    c->last_algo = "umma";
    return rc;
  }
  const void* xin = x;
  if (!in_nhwc) {
    int rc = to_nhwc(c, tmp, x, d.N, d.C, d.H, d.W, d.dtype, &xin);
    if (rc) return rc;
  }
  const int ldw = pad_channels(Cg, d.dtype);
  void* wp;
  int rc = 0;
  if (d.kH == 1 && d.kW == 1 && ldw == Cg && merge == 1 && reinterpret_cast<uintptr_t>(w) % 16 == 0) {
    // a 1x1 filter bank [K][C] already is its packed form (rows = filters, channels contiguous)
    wp = const_cast<void*>(w);
  } else {
    wp = flags & kScratchFilters ? nullptr : packed_lookup(c, w, d.K, Cg, d.kH, d.kW, d.groups, d.flip, 0, ldw, d.dtype);
    if (!wp) {
      rc = tmp.get(es * (size_t)d.kH * d.kW * d.K * ldw, &wp);
      if (rc) return rc;
      KLAUNCH(c, kKPack, launch_pack_filters(pack_job(w, wp, d.K, Cg, d.kH * d.kW, d.groups, d.flip, 0, ldw, merge), d.dtype, c->stream));
    }
  }

  std::vector<ConvTap> taps;
  std::vector<std::pair<int, int>> parity;
  for (int i = 0; i < d.kH; ++i)
    for (int j = 0; j < d.kW; ++j) {
      const int ah = i * d.dilH - d.padH_l, aw = j * d.dilW - d.padW_l;
      const int rh = pymod(ah, d.sH), rw = pymod(aw, d.sW);
      int v = -1;
      for (size_t q = 0; q < parity.size(); ++q)
        if (parity[q].first == rh && parity[q].second == rw) v = (int)q;
      if (v < 0) { v = (int)parity.size(); parity.push_back({rh, rw}); }
      ConvTap t;
      t.dh = (int16_t)floordiv(ah, d.sH); t.dw = (int16_t)floordiv(aw, d.sW);
      t.view = (int16_t)v; t.wmat = (int16_t)(i * d.kW + j);
      taps.push_back(t);
    }
  FwdLikeArgs a;
  a.act = xin; a.Hs = d.H; a.Ws = d.W; a.Cin_g = Cg; a.Cp_in = Cp;
  a.wpacked = wp; a.ld_w = ldw; a.nmats = d.kH * d.kW * d.groups;
  a.n_out = out_nhwc && d.groups == 1 ? Kp : Kg; a.w_rows = Kg; a.groups = d.groups; a.N = d.N; a.dtype = d.dtype;
  a.view_sH = d.sH; a.view_sW = d.sW;
  long long sn, sc, sh, sw;
  if (out_nhwc) {
    const int pl = c->epi.pool ? 2 : 1;
    sn = 1LL * (d.Ho / pl) * (d.Wo / pl) * Kp; sc = 1; sh = 1LL * (d.Wo / pl) * Kp; sw = Kp;
  } else {
    sn = 1LL * d.K * d.Ho * d.Wo; sc = 1LL * d.Ho * d.Wo; sh = d.Wo; sw = 1;
  }
  rc = run_conv_umma(c, a, taps, parity, d.Wo, d.Ho, y, sn, sc, sh, sw, 0, bias,
                     (flags & B200CONV_RELU) ? 1 : 0, !(flags & B200CONV_NO_SLAB));
  if (rc == 1) {  // every tap fell outside the image: conv == 0, only the epilogue remains
    b200conv_desc z = d;
    z.C = 0;
    if (out_nhwc) return fail(c, B200CONV_E_UNSUPPORTED, "degenerate geometry with channels-last output");
    if (int r = convert_bias()) return r;
    KLAUNCH(c, kKDirect, launch_direct_fwd(z, x, w, bias_f, y, (flags & B200CONV_RELU) ? 1 : 0, c->epi, c->stream));
    rc = 0;
  }
  c->last_algo = "umma";
  return rc;
}

int dgrad_device(b200conv_ctx* c, const b200conv_desc& d, const void* w, const void* dy, void* dx,
                 int flags, int merge = 1) {
  const int Cg = d.C / d.groups, Kg = d.K / d.groups;
  const size_t es = elem_size(d.dtype);
  const bool out_nhwc = flags & B200CONV_OUT_NHWC, in_nhwc = flags & B200CONV_IN_NHWC;
  const int Cp = pad_channels(d.C, d.dtype), Kp = pad_channels(d.K, d.dtype);
  if (d.N == 0 || d.C == 0) return 0;
  b200conv_desc flat;
  if (!(flags & B200CONV_FORCE_DIRECT) && flatten_1x1(d, in_nhwc && out_nhwc, &flat))
    return dgrad_device(c, flat, w, dy, dx, flags, merge);
  const size_t dx_bytes = es * (size_t)d.N * d.H * d.W * (out_nhwc ? Cp : d.C);
  const int mg = (flags & B200CONV_FORCE_DIRECT) || merge > 1 ? 1 : merge_factor(d);
  if (mg > 1) {
    b200conv_desc dm = d;
    dm.groups = d.groups / mg;
    const bool classes = d.sH * d.sW > 1 && dm.groups == 1 && d.sH * d.sW * d.C <= 64;            // those pack another form
    if (umma_ok(dm) && !classes) return dgrad_device(c, dm, w, dy, dx, flags | kScratchFilters, mg);
    if (umma_ok(dm)) {
      Scratch tm(c);
      void* wm;
      int rc = tm.get(es * (size_t)d.K * Cg * mg * d.kH * d.kW, &wm);
      if (rc) return rc;
      KLAUNCH(c, kKPack, launch_merge_groups(w, wm, d.K, Cg, Kg, mg, d.kH * d.kW, 0, d.dtype, c->stream));
      return dgrad_device(c, dm, wm, dy, dx, flags | kScratchFilters);
    }
  }
  const bool use_umma = !(flags & B200CONV_FORCE_DIRECT) && umma_ok(d);
  if (!use_umma) {
    if (flags & B200CONV_FORCE_UMMA) return fail(c, B200CONV_E_UNSUPPORTED, "geometry not covered by the tensor-core kernel");
    if (in_nhwc || out_nhwc) return fail(c, B200CONV_E_UNSUPPORTED, "direct kernels take NCHW tensors only");
    KLAUNCH(c, kKDirect, launch_direct_dgrad(d, w, dy, dx, c->stream));
    c->last_algo = "direct";
    return 0;
  }
  Scratch tmp(c);
  const void* gin = dy;
  if (!in_nhwc) {
    int rc = to_nhwc(c, tmp, dy, d.N, d.K, d.Ho, d.Wo, d.dtype, &gin);
    if (rc) return rc;
  }
  const int ldw = pad_channels(Kg, d.dtype);
  int rc;

  // Output pixels split into sH*sW parity classes; class (h0, w0) is a stride-1 problem over
  // the taps with (h0 + padH_l - i*dilH) divisible by sH (same for columns).
  struct Cls { int h0, w0, Ht, Wt; std::vector<ConvTap> taps; };
  std::vector<Cls> classes;
  bool need_zero = out_nhwc && Cp != d.C && d.groups > 1;
  for (int h0 = 0; h0 < d.sH; ++h0)
    for (int w0 = 0; w0 < d.sW; ++w0) {
      Cls k;
      k.h0 = h0; k.w0 = w0;
      k.Ht = h0 < d.H ? (d.H - h0 + d.sH - 1) / d.sH : 0;
      k.Wt = w0 < d.W ? (d.W - w0 + d.sW - 1) / d.sW : 0;
      if (k.Ht == 0 || k.Wt == 0) continue;
      for (int i = 0; i < d.kH; ++i) {
        const int th = h0 + d.padH_l - i * d.dilH;
        if (pymod(th, d.sH)) continue;
        for (int j = 0; j < d.kW; ++j) {
          const int tw = w0 + d.padW_l - j * d.dilW;
          if (pymod(tw, d.sW)) continue;
          ConvTap t;
          t.dh = (int16_t)floordiv(th, d.sH); t.dw = (int16_t)floordiv(tw, d.sW);
          t.view = 0; t.wmat = (int16_t)(i * d.kW + j);
          k.taps.push_back(t);
        }
      }
      if (k.taps.empty()) need_zero = true;
      classes.push_back(k);
    }
  // Few channels and a stride: the classes become channel blocks of ONE stride-1 problem over
  // the union of their tap offsets (a class without a tap at an offset gets a zero filter block
  // there), followed by a depth-to-space pass.  Each class alone would fill a small fraction of
  // an MMA's columns, and the gradient would be read once per class.
  const int ncls = d.sH * d.sW;
  if (ncls > 1 && ncls <= kMaxParityClasses && d.groups == 1 && ncls * d.C <= 64 &&
      (int)classes.size() == ncls && !(flags & B200CONV_NO_MERGE_PARITY)) {
    MergedTapTable tb;
    std::vector<ConvTap> utaps;
    bool fits = true;
    for (size_t k = 0; k < classes.size() && fits; ++k)
      for (const ConvTap& t : classes[k].taps) {
        size_t u = 0;
        while (u < utaps.size() && !(utaps[u].dh == t.dh && utaps[u].dw == t.dw)) ++u;
        if (u == utaps.size()) {
          if (utaps.size() == (size_t)kMaxTaps) { fits = false; break; }
          ConvTap nt = t;
          nt.wmat = (int16_t)u;
          utaps.push_back(nt);
          for (int q = 0; q < kMaxParityClasses; ++q) tb.src[u][q] = -1;
        }
        tb.src[u][classes[k].h0 * d.sW + classes[k].w0] = t.wmat;
      }
    if (!fits) utaps.clear();
    if (!utaps.empty()) {
      const int Ct = pad_channels(ncls * d.C, d.dtype);
      const int nu = (int)utaps.size(), n_out = Ct;      // padded with zero filters: whole 16-byte pieces
      const int Hq = (d.H + d.sH - 1) / d.sH, Wq = (d.W + d.sW - 1) / d.sW;
      // row by row, so that a row's columns are neighbours in the packed filters
      std::sort(utaps.begin(), utaps.end(), [](const ConvTap& x, const ConvTap& y) { return x.dh != y.dh ? x.dh < y.dh : x.dw < y.dw; });
      MergedTapTable sorted;
      for (int u = 0; u < nu; ++u) {
        std::copy(std::begin(tb.src[utaps[u].wmat]), std::end(tb.src[utaps[u].wmat]), std::begin(sorted.src[u]));
        utaps[u].wmat = (int16_t)u;
      }
      tb = sorted;
      void *wp, *merged;
      if ((rc = tmp.get(es * (size_t)nu * n_out * ldw, &wp))) return rc;
      KLAUNCH(c, kKPack, launch_pack_filters_merged(w, wp, d.K, d.C, d.kH, d.kW, d.flip, tb, nu, ncls, n_out,
                                                    ldw, d.dtype, c->stream));
      FwdLikeArgs a;
      a.act = gin; a.Hs = d.Ho; a.Ws = d.Wo; a.Cin_g = Kg; a.Cp_in = Kp;
      a.wpacked = wp; a.ld_w = ldw; a.nmats = nu;
      a.n_out = a.w_rows = n_out; a.groups = 1; a.N = d.N; a.dtype = d.dtype;
      a.view_sH = 1; a.view_sW = 1;
      std::vector<std::pair<int, int>> parity(1, {0, 0});
      // The columns kernel writes the gradient's pixels itself; else the classes go through a tensor of their own and a depth-to-space pass.
      // 64 -> 3 7x7 at 224x224, float16, 256 images 415 -> 143 us, one 13.3 -> 6.7; 32 -> 3 4x4 at 64x64, 2 images 10.1 -> 6.2; float32 688 -> 248,
      // 17.1 -> 7.6 and 10.9 -> 6.0: of nine such layers in both types the columns kernel was slower on none.
      if (d.sH == 2 && d.sW == 2 && out_nhwc && Cp * es == 16 && !(flags & B200CONV_NO_SLAB)) {
        rc = try_conv_cols(c, a, utaps, 0, 0, Wq, Hq, dx, 0, 1, 0, 0, 0, nullptr, 0, true, false, d.C, d.H, d.W);
        if (rc == 0) c->last_algo = "umma";
        if (rc != 2) return rc;
      }
      if ((rc = tmp.get(es * (size_t)d.N * Hq * Wq * Ct, &merged))) return rc;
      rc = run_conv_umma(c, a, utaps, parity, Wq, Hq, merged, 1LL * Hq * Wq * Ct, 1, 1LL * Wq * Ct, Ct, 0,
                         nullptr, 0, !(flags & B200CONV_NO_SLAB));
      if (rc) return rc == 1 ? fail(c, B200CONV_E_CUDA, "internal: empty gradient view") : rc;
      KLAUNCH(c, kKTranspose, launch_depth_to_space(merged, dx, d.N, d.C, d.H, d.W, d.sH, d.sW, Ct, Cp,
                                                    out_nhwc ? 1 : 0, d.dtype, c->stream));
      c->last_algo = "umma";
      return 0;
    }
  }
  void* wp = flags & kScratchFilters ? nullptr : packed_lookup(c, w, d.K, Cg, d.kH, d.kW, d.groups, d.flip, 1, ldw, d.dtype);
  if (!wp) {
    if ((rc = tmp.get(es * (size_t)d.kH * d.kW * d.C * ldw, &wp))) return rc;
    KLAUNCH(c, kKPack, launch_pack_filters(pack_job(w, wp, d.K, Cg, d.kH * d.kW, d.groups, d.flip, 1, ldw, merge), d.dtype, c->stream));
  }
  if (need_zero) CU_OK(c, cudaMemsetAsync(dx, 0, dx_bytes, c->stream));
  FwdLikeArgs a;
  a.act = gin; a.Hs = d.Ho; a.Ws = d.Wo; a.Cin_g = Kg; a.Cp_in = Kp;
  a.wpacked = wp; a.ld_w = ldw; a.nmats = d.kH * d.kW * d.groups;
  a.n_out = out_nhwc && d.groups == 1 ? Cp : Cg; a.w_rows = Cg; a.groups = d.groups; a.N = d.N; a.dtype = d.dtype;
  a.view_sH = 1; a.view_sW = 1;
  std::vector<std::pair<int, int>> parity(1, {0, 0});
  const bool slab_ok = !(flags & B200CONV_NO_SLAB);
  auto each_class = [&]() -> int {
    for (const Cls& k : classes) {
      if (k.taps.empty()) continue;
      long long sn, sc, sh, sw, off;
      if (out_nhwc) {
        sn = 1LL * d.H * d.W * Cp; sc = 1; sh = 1LL * d.sH * d.W * Cp; sw = 1LL * d.sW * Cp;
        off = (1LL * k.h0 * d.W + k.w0) * Cp;
      } else {
        sn = 1LL * d.C * d.H * d.W; sc = 1LL * d.H * d.W; sh = 1LL * d.sH * d.W; sw = d.sW;
        off = 1LL * k.h0 * d.W + k.w0;
      }
      const int r = run_conv_umma(c, a, k.taps, parity, k.Wt, k.Ht, dx, sn, sc, sh, sw, off, nullptr, 0, slab_ok);
      if (r) return r == 1 ? fail(c, B200CONV_E_CUDA, "internal: empty gradient view") : r;
    }
    return 0;
  };
  // All classes from one slab of dy: one launch that reads dy once, its taps grouped by class into accumulators of their
  // own.  Class by class, dy is read ncls times and a class with one tap is a launch that only moves memory
  // (256 images at 56x56 with the packing: 64 <- 128 channels float32 186 -> 134 us, 64 <- 64 float16 96 -> 57; from 128 channels
  // on in float16 both forms are bound by their MMAs and equal).
  const bool full = std::all_of(classes.begin(), classes.end(), [](const Cls& k) { return !k.taps.empty(); });
  if (ncls > 1 && ncls <= kMaxSlabClasses && (int)classes.size() == ncls && full && out_nhwc && slab_ok &&
      !(flags & B200CONV_NO_MERGE_PARITY) && d.kH * d.kW <= kMaxTaps) {
    FwdLikeArgs m = a;
    std::vector<std::pair<ConvTap, int>> all;
    int Wt = 0, Ht = 0;
    for (const Cls& k : classes) {
      for (const ConvTap& t : k.taps) all.push_back({t, (int)m.classes.size()});
      m.classes.push_back({k.Wt, k.Ht, (1LL * k.h0 * d.W + k.w0) * Cp});
      Wt = std::max(Wt, k.Wt); Ht = std::max(Ht, k.Ht);
    }
    // in the order of the packed filters, so that a stage's taps arrive as one box
    std::sort(all.begin(), all.end(), [](const auto& x, const auto& y) { return x.first.wmat < y.first.wmat; });
    std::vector<ConvTap> taps;
    for (auto& t : all) { taps.push_back(t.first); m.tap_cls.push_back((uint8_t)t.second); }
    auto together = [&](SlabMode mode) {
      return try_conv_slab(c, m, taps, 0, 0, Wt, Ht, dx, 1LL * d.H * d.W * Cp, 1, 1LL * d.sH * d.W * Cp, 1LL * d.sW * Cp, 0, nullptr, 0, mode);
    };
    // 0: class by class, 1 / 2: together, on single CTAs / on pairs; timed like the other variants
    auto run = [&](int v) { return v == 0 ? each_class() : together(v == 1 ? kSlabWide : kSlabPair); };
    GeoKey key{kGeoClasses, d.dtype, d.N, d.C, d.H, d.W, d.K, d.kH, d.kW, d.sH, d.sW, d.dilH, d.dilW, d.padH_l, d.padW_l, d.Ho, d.Wo, d.groups,
               c->use_pair ? 1 : 0};
    auto it = c->autotune ? c->algo_cache.find(key) : c->algo_cache.end();
    int choice = it != c->algo_cache.end() ? it->second : -1;
    if (choice < 0 && (!c->autotune || c->capturing)) {
      if ((rc = together(c->use_pair ? kSlabPair : kSlabWide)) == 2 && c->use_pair) rc = together(kSlabWide);
      if (rc != 2) {
        if (rc) return rc;
        c->last_algo = "umma";
        return 0;
      }
      choice = 0;
    }
    if (choice < 0) {
      // class by class makes a choice for each class: those are timed only if it is not far behind with the models'
      float ms[3];
      int codes[3];
      const int n = c->use_pair ? 3 : 2;
      if ((rc = rough_times(c, n, run, ms, codes))) return rc;
      const float together_ms = n > 2 && ms[2] >= 0.f && (ms[1] < 0.f || ms[2] < ms[1]) ? ms[2] : ms[1];
      const int lowest = together_ms >= 0.f && ms[0] > kFarBehind * together_ms ? 1 : 0;
      if ((rc = time_variants(c, n, [&](int v) { return v < lowest ? 2 : run(v); }, ms, codes))) return rc;
      for (int v = 0; v < n; ++v) {
        if (codes[v] && codes[v] != 2) return codes[v];
        if (ms[v] >= 0.f && (choice < 0 || ms[v] < ms[choice])) choice = v;
      }
      if (choice < 0) choice = 0;
      c->algo_cache[key] = choice;
    }
    rc = run(choice);
    if (rc == 2) rc = each_class();          // a choice remembered for another alignment
    if (rc) return rc;
  } else if ((rc = each_class())) {
    return rc;
  }
  c->last_algo = "umma";
  return 0;
}

// Number of split-K slices of a gradWeights launch.  The items (base_items x slices) are spread
// over num_sms persistent CTAs; the launch lasts as long as its busiest CTA: ceil(items / SMs)
// items of ceil(pix_tiles / slices) pixel tiles each, plus `fixed` tiles' worth of per-item
// overhead (pipeline fill, accumulator read-out).  Pick the count that makes that smallest;
// among equals the smallest count (fewer partial slabs to add up).
static long long balanced_splits(long long pix_tiles, long long base_items, int sms, long long cap,
                                 long long fixed) {
  base_items = std::max(1LL, base_items);
  cap = std::max(1LL, std::min(cap, pix_tiles));
  const long long hi = std::min(cap, std::max(1LL, cdiv(3LL * sms, base_items)));
  long long best = 1, best_cost = -1;
  for (long long s = 1; s <= hi; ++s) {
    const long long per = cdiv(pix_tiles, s);
    if (cdiv(pix_tiles, per) != s) continue;
    const long long cost = cdiv(base_items * s, sms) * (per + fixed);
    if (best_cost < 0 || cost < best_cost) { best = s; best_cost = cost; }
  }
  return best;
}

// The same, remembered (the loop above runs up to 444 times).
long long balanced_splits(b200conv_ctx* c, long long pix_tiles, long long base_items, int sms, long long cap, long long fixed) {
  SlabTile& memo = c->pixel_tiles[GeoKey{kGeoBalance, (int)pix_tiles, (int)base_items, sms, (int)cap, (int)fixed}];
  if (!memo.found) {
    memo.wt = (int)balanced_splits(pix_tiles, base_items, sms, cap, fixed);
    memo.found = true;
  }
  return memo.wt;
}

int wgrad_device(b200conv_ctx* c, const b200conv_desc& d, const void* x, const void* dy, void* dw,
                 int flags);

// A slice count the kernels can use near `s`: they cut the pixel tiles into ceil(tiles / s) per slice, and
// every slice must get at least one tile.
int valid_splits(long long pix_tiles, long long s) {
  s = std::max(1LL, std::min(s, pix_tiles));
  return (int)cdiv(pix_tiles, cdiv(pix_tiles, s));
}

// The slice count of a gradWeights launch.  The model's choice `s0` is right about the busiest SM's
// work but knows nothing of the reduction kernel's cost or of L2 effects, so with timing-based
// selection on, the first call of a geometry also times half and twice that count (main kernel plus
// reduction) and the context remembers the fastest; the role the reference's
// GPU back end gives its meta-optimizer (theano/gpuarray/opt.py:2144-2222).  `run(splits, scratch)`
// enqueues the launch.  Returns the count, or a negative error code.
template <class Run>
int pick_splits(b200conv_ctx* c, const GeoKey& key, long long pix_tiles, long long cap, long long base_items, int sms,
                long long fixed, Run run) {
  cap = std::max(1LL, std::min(cap, pix_tiles));
  if (c->force_splits > 0) return valid_splits(pix_tiles, std::min<long long>(c->force_splits, cap));
  if (c->autotune) {
    // whatever call or file the count came from: a slice without a tile would add up what its accumulator held before
    auto it = c->split_cache.find(key);
    if (it != c->split_cache.end()) return valid_splits(pix_tiles, std::min<long long>(it->second, cap));
  }
  const int s0 = (int)balanced_splits(c, pix_tiles, base_items, sms, cap, fixed);
  if (!c->autotune || c->capturing || c->model_only) return s0;
  int cand[3] = {s0, valid_splits(pix_tiles, std::min<long long>(cap, std::max(1, s0 / 2))),
                 valid_splits(pix_tiles, std::min<long long>(cap, 2LL * s0))};
  int n = 1, best = 0, codes[3];
  for (int i = 1; i < 3; ++i)
    if (std::find(cand, cand + n, cand[i]) == cand + n) cand[n++] = cand[i];
  if (n == 1) return c->split_cache[key] = s0;
  float ms[3];
  const int rc = time_variants(c, n, [&](int i) { Scratch trial(c); return run(cand[i], trial); }, ms, codes);
  if (rc) return rc < 0 ? rc : -rc;
  for (int i = 0; i < n; ++i) {
    if (codes[i]) return codes[i] < 0 ? codes[i] : -codes[i];
    if (ms[i] >= 0.f && (ms[best] < 0.f || ms[i] < ms[best])) best = i;
  }
  return c->split_cache[key] = cand[best];
}

// NO_ROWS is part of a choice between kernels: what was chosen without one of them says nothing about calls that allow it.  So is NO_S2D,
// which gives a layer another form.  (ROWS and NO_GROUP decide before a choice is looked up.)
GeoKey wgrad_key(int kind, const b200conv_desc& d, int flags) {
  return GeoKey{kind, d.dtype, d.N, d.C, d.H, d.W, d.K, d.kH, d.kW, d.sH, d.sW, d.dilH, d.dilW, d.padH_l, d.padW_l, d.Ho, d.Wo,
                d.groups, flags & (B200CONV_ATOMIC_SPLITK | (kind == kGeoSplits ? B200CONV_DW_F32 : B200CONV_NO_ROWS | B200CONV_NO_S2D))};
}

// The sums of a gradient (wgrad_exact.cuh); during a call on merged groups `d` is the merged layer, and its groups are the layer's own.
WgradSum wgrad_sum(const b200conv_ctx* c, const b200conv_desc& d, const void* x, bool x_nhwc, const void* dy, bool dy_nhwc) {
  WgradSum s;
  s.x = x; s.dy = dy;
  s.f16 = d.dtype == B200CONV_F16;
  s.Cg = c->diag_c ? c->diag_c : d.C / d.groups;
  s.Kg = c->diag_k ? c->diag_k : d.K / d.groups;
  s.N = d.N; s.H = d.H; s.W = d.W; s.Ho = d.Ho; s.Wo = d.Wo; s.kH = d.kH; s.kW = d.kW;
  s.sH = d.sH; s.sW = d.sW; s.dilH = d.dilH; s.dilW = d.dilW; s.padH = d.padH_l; s.padW = d.padW_l; s.flip = d.flip;
  s.segments = 0;
  s.x_c = x_nhwc ? 1 : 1LL * d.H * d.W;
  s.x_w = x_nhwc ? pad_channels(d.C, d.dtype) : 1;
  s.x_h = s.x_w * d.W;
  s.x_n = x_nhwc ? s.x_h * d.H : s.x_c * d.C;
  s.dy_c = dy_nhwc ? 1 : 1LL * d.Ho * d.Wo;
  s.dy_w = dy_nhwc ? pad_channels(d.K, d.dtype) : 1;
  s.dy_h = s.dy_w * d.Wo;
  s.dy_n = dy_nhwc ? s.dy_h * d.Ho : s.dy_c * d.K;
  return s;
}

// Kernel and form of the layer in the key of a slice count: one layer's forms differ in their pixel tiles.
enum { kSplitsGroups = 0, kSplitsTaps, kSplitsPair, kSplitsRows, kSplitsRowsS2d, kSplitsRowsFold };

// gradWeights with tap groups (wgrad_group.cu).  Returns 0 when launched, 2 when the geometry is
// left to the one-tap-per-item kernel (no two taps share a row offset, or the column span of the
// taps is too wide), or an error code.
int wgrad_grouped(b200conv_ctx* c, const b200conv_desc& d, const void* xin, const void* gin, void* dw,
                  int flags, Scratch& tmp) {
  const int Cg = d.C / d.groups, Kg = d.K / d.groups;
  const int Cp = pad_channels(d.C, d.dtype), Kp = pad_channels(d.K, d.dtype);
  const int atom = d.dtype == B200CONV_F16 ? 64 : 32;
  const bool swz32 = d.dtype == B200CONV_F32;
  struct T { int view, dh, dw, wmat; };
  std::vector<T> taps;
  std::vector<std::pair<int, int>> parity;
  std::vector<int> slot;   // parity index -> tensor map slot or -1 (empty view)
  int nviews = 0;
  bool dropped = false;
  for (int i = 0; i < d.kH; ++i)
    for (int j = 0; j < d.kW; ++j) {
      const int ah = i * d.dilH - d.padH_l, aw = j * d.dilW - d.padW_l;
      const int rh = pymod(ah, d.sH), rw = pymod(aw, d.sW);
      int v = -1;
      for (size_t q = 0; q < parity.size(); ++q)
        if (parity[q].first == rh && parity[q].second == rw) v = (int)q;
      if (v < 0) {
        v = (int)parity.size();
        parity.push_back({rh, rw});
        slot.push_back((rh < d.H && rw < d.W) ? nviews++ : -1);
      }
      if (slot[v] < 0) { dropped = true; continue; }
      const int wi = d.flip ? d.kH - 1 - i : i, wj = d.flip ? d.kW - 1 - j : j;
      taps.push_back({slot[v], floordiv(ah, d.sH), floordiv(aw, d.sW), wi * d.kW + wj});
    }
  if (taps.empty() || (int)taps.size() > kMaxTaps) return 2;
  // column span per view
  int dwmin[kMaxViews], dwmax[kMaxViews];
  for (int v = 0; v < nviews; ++v) { dwmin[v] = 1 << 20; dwmax[v] = -(1 << 20); }
  for (const T& t : taps) {
    dwmin[t.view] = std::min(dwmin[t.view], t.dw);
    dwmax[t.view] = std::max(dwmax[t.view], t.dw);
  }
  int Ew = 0;
  for (int v = 0; v < nviews; ++v) Ew = std::max(Ew, dwmax[v] - dwmin[v]);
  if (Ew > 15 || Ew == 0) return 2;
  std::sort(taps.begin(), taps.end(), [](const T& a, const T& b) {
    if (a.view != b.view) return a.view < b.view;
    if (a.dh != b.dh) return a.dh < b.dh;
    return a.dw < b.dw;
  });
  GroupWgradParams p;
  memset(&p, 0, sizeof p);
  for (size_t i = 0; i < taps.size();) {
    size_t j = i;
    while (j < taps.size() && j - i < 4 && taps[j].view == taps[i].view && taps[j].dh == taps[i].dh) ++j;
    if (p.ngroups >= kMaxTapGroups) return 2;
    p.grp_view[p.ngroups] = (int16_t)taps[i].view;
    p.grp_dh[p.ngroups] = (int16_t)taps[i].dh;
    p.grp_first[p.ngroups] = (int16_t)i;
    p.grp_n[p.ngroups] = (int16_t)(j - i);
    ++p.ngroups;
    i = j;
  }
  for (size_t i = 0; i < taps.size(); ++i) {
    p.tap_off[i] = (int16_t)(taps[i].dw - dwmin[taps[i].view]);
    p.tap_wmat[i] = (int16_t)taps[i].wmat;
  }
  for (int v = 0; v < nviews; ++v) p.view_dwmin[v] = (int16_t)dwmin[v];
  // Layers with at most 64 channels: a tap group becomes one MMA (tf32: one per 32 channels) whose column groups are
  // the taps, if the taps of every group are evenly spaced (stride and dilation decide the spacing; 1 for a plain 3x3 filter)
  if (Cg <= 64 && c->stack_taps) {
    int step = 0;
    bool even = true;
    for (int gi = 0; gi < p.ngroups && even; ++gi)
      for (int q = 1; q < p.grp_n[gi]; ++q) {
        const int dd = p.tap_off[p.grp_first[gi] + q] - p.tap_off[p.grp_first[gi] + q - 1];
        if (dd <= 0 || (step && dd != step)) even = false;
        step = dd;
      }
    if (even && step > 0) p.stack_step = step;
  }
  // pixel box of a stage
  const int kWgradPix = wgrad_pix(d.dtype);
  if ((d.Wo + Ew) * 2 <= kWgradPix || d.Wo + Ew <= kWgradPix) {
    p.Wa = p.Wb = d.Wo + Ew;                       // whole padded rows
    p.wt = d.Wo;
    p.th = std::max(1, std::min(d.Ho, kWgradPix / p.Wa));
    p.nb = p.th == d.Ho ? std::max(1, std::min(d.N, kWgradPix / (p.Wa * p.th))) : 1;
  } else {
    p.th = 1; p.nb = 1;                            // a segment of one output row
    const int parts = (int)cdiv(d.Wo, kWgradPix - Ew);
    p.wt = (int)cdiv(d.Wo, parts);
    p.Wa = p.wt; p.Wb = p.wt + Ew;
  }
  p.rows_a = p.Wa * p.th * p.nb; p.rows_b = p.Wb * p.th * p.nb;
  p.tiles_w = (int)cdiv(d.Wo, p.wt); p.tiles_h = (int)cdiv(d.Ho, p.th); p.tiles_n = (int)cdiv(d.N, p.nb);
  int rc = make_view(c, &p.dy_map, gin, d.dtype, Kg, d.groups, Kp, d.Wo, d.Ho, d.N, 0, 0, 1, 1, atom, p.Wa,
                     p.th, p.nb, swz32);
  if (rc) return rc;
  for (size_t v = 0; v < parity.size(); ++v) {
    if (slot[v] < 0) continue;
    rc = make_view(c, &p.x_views[slot[v]], xin, d.dtype, Cg, d.groups, Cp, d.W, d.H, d.N, parity[v].first,
                   parity[v].second, d.sH, d.sW, atom, p.Wb, p.th, p.nb, swz32);
    if (rc) return rc;
  }
  for (int v = nviews; v < kMaxViews; ++v) p.x_views[v] = p.x_views[0];
  p.nviews = nviews;
  p.groups = d.groups; p.Kg = Kg; p.Cg = Cg;
  p.Wo = d.Wo; p.Ho = d.Ho; p.Nimg = d.N;
  p.ktiles = (int)cdiv(Kg, 128); p.ctiles = (int)cdiv(Cg, 128);
  p.taps_total = d.kH * d.kW;
  const long long pix_tiles = 1LL * p.tiles_w * p.tiles_h * p.tiles_n;
  const long long base_items = 1LL * p.ktiles * p.ctiles * d.groups * p.ngroups;
  p.atomic = (flags & B200CONV_ATOMIC_SPLITK) ? 1 : 0;
  p.diag_c = c->diag_c; p.diag_k = c->diag_k;
  p.status = c->d_status;
  p.wait_clocks = c->wait_clocks;
  p.trace = c->trace;
  const size_t slab_elems = (size_t)p.taps_total * d.K * Cg;
  auto run = [&](int splits, Scratch& sc) -> int {
    p.splits = splits;
    const int slabs = p.atomic ? 1 : p.splits;
    float* partial;
    int r = sc.get(sizeof(float) * slab_elems * slabs, reinterpret_cast<void**>(&partial));
    if (r) return r;
    if (p.atomic || dropped)
      CU_OK(c, cudaMemsetAsync(partial, 0, sizeof(float) * slab_elems * slabs, c->stream));
    p.partial = partial;
    p.partial_elems = (long long)slab_elems * slabs;
    c->last_variant = "wgrad groups";
    KLAUNCH(c, kKWgradUmma, launch_wgrad_group(p, d.dtype, c->num_sms, c->stream));
    WgradSum sum = wgrad_sum(c, d, xin, true, gin, true);
    sum.segments = p.tiles_w > 1 && p.rows_a % (d.dtype == B200CONV_F16 ? 16 : 8);      // zeros fill the last MMA of every segment
    KLAUNCH(c, kKWgradReduce, launch_wgrad_reduce(partial, dw, slabs, p.taps_total, d.K, Cg, Kg, p.diag_c, p.diag_k,
                                                  (flags & B200CONV_DW_F32) ? B200CONV_F32 : d.dtype, sum, c->stream));
    return 0;
  };
  GeoKey skey = wgrad_key(kGeoSplits, d, flags);
  skey.add(kSplitsGroups);
  // accumulators are not double buffered: aim at one item per SM
  const int splits = pick_splits(c, skey, pix_tiles, pix_tiles, base_items, c->num_sms, 6, run);
  if (splits < 0) return splits;
  if ((rc = run(splits, tmp))) return rc;
  c->last_algo = "umma";
  return 0;
}

// The taps of one stride parity class of x: filter rows x filter columns.
struct RowsView {
  std::vector<int> dh, dw;           // offsets of the filter rows / columns in the view's pixels, ascending
  std::vector<int> tap;              // [row][column]
  std::function<int(CUtensorMap*, int, int)> map;      // tensor map with a box of (columns, rows)
};

// The views of a plain layer for wgrad_rows (channels-last x of C channels); `dropped`: taps that read nothing.
std::vector<RowsView> rows_views(b200conv_ctx* c, const b200conv_desc& d, const void* xin, bool* dropped) {
  const int atom = d.dtype == B200CONV_F16 ? 64 : 32;
  std::vector<RowsView> views;
  *dropped = false;
  for (int rh = 0; rh < d.sH; ++rh)
    for (int rw = 0; rw < d.sW; ++rw) {
      std::vector<int> is, js;
      for (int i = 0; i < d.kH; ++i) if (pymod(i * d.dilH - d.padH_l, d.sH) == rh) is.push_back(i);
      for (int j = 0; j < d.kW; ++j) if (pymod(j * d.dilW - d.padW_l, d.sW) == rw) js.push_back(j);
      if (is.empty() || js.empty()) continue;
      if (rh >= d.H || rw >= d.W) { *dropped = true; continue; }
      RowsView v;
      for (int i : is) v.dh.push_back(floordiv(i * d.dilH - d.padH_l, d.sH));
      for (int j : js) v.dw.push_back(floordiv(j * d.dilW - d.padW_l, d.sW));
      for (int i : is)
        for (int j : js) v.tap.push_back((d.flip ? d.kH - 1 - i : i) * d.kW + (d.flip ? d.kW - 1 - j : j));
      v.map = [=](CUtensorMap* m, int bw, int bh) {
        return make_view(c, m, xin, d.dtype, d.C / d.groups, d.groups, pad_channels(d.C, d.dtype), d.W, d.H, d.N, rh, rw, d.sH, d.sW, atom, bw, bh, 1,
                         d.dtype == B200CONV_F32);
      };
      views.push_back(v);
    }
  return views;
}

// gradWeights with the filter's rows and columns inside one MMA (wgrad_rows.cu).  Returns 0 when launched, 2 when the
// layer is not one for it (more filters per group than a swizzle atom holds, uneven taps, rows too wide for a box) or the flags bar it.
// `form`: kSplitsRows, or the form of x that the views are of; `reduce(partial, slabs)` enqueues the kernel that adds the slabs.
template <class Reduce>
int wgrad_rows(b200conv_ctx* c, const b200conv_desc& d, int form, const std::vector<RowsView>& views, int Cg, bool dropped, int taps_total, const void* gin,
               int flags, Scratch& tmp, int diag_c, int diag_k, Reduce reduce) {
  const bool f16 = d.dtype == B200CONV_F16;
  const int atom = f16 ? 64 : 32, kk = f16 ? 16 : 8, copies = 128 / atom, Kg = d.K / d.groups;
  const bool barred = (flags & (B200CONV_NO_ROWS | B200CONV_ATOMIC_SPLITK)) || (flags & (B200CONV_NO_GROUP | B200CONV_ROWS)) == B200CONV_NO_GROUP;
  if (barred || Kg > atom || views.empty() || views.size() > (size_t)kMaxViews) return 2;
  RowsWgradParams p;
  memset(&p, 0, sizeof p);
  p.nviews = (int)views.size();
  p.stack_step = 1;
  int row_step = 0, col_step = 0, taps = 0, span = 0, Ew = 0, n_max = 0, sets_max = 0;
  for (int v = 0; v < p.nviews; ++v) {
    const RowsView& w = views[v];
    const int rows = (int)w.dh.size(), cols = (int)w.dw.size();
    for (int i = 1; i < rows; ++i) { const int st = w.dh[i] - w.dh[i - 1]; if (st <= 0 || (row_step && st != row_step)) return 2; row_step = st; }
    for (int j = 1; j < cols; ++j) { const int st = w.dw[j] - w.dw[j - 1]; if (st <= 0 || (col_step && st != col_step)) return 2; col_step = st; }
    const int sets = (int)cdiv(rows, copies);
    if (sets > kMaxRowSets || cols * atom > 256 || sets * cols * atom > 512 || taps + rows * cols > kMaxTaps) return 2;
    p.view_nt[v] = (int16_t)cols; p.view_sets[v] = (int16_t)sets; p.view_tap0[v] = (int16_t)taps;
    for (int t : w.tap) p.tap_id[taps++] = (int16_t)t;
    for (int j = 0; j < sets; ++j) {
      p.set_first[v][j] = (int16_t)(j * copies);
      p.set_base[v][j] = (int16_t)std::min(rows - 1, j * copies + copies - 1);
    }
    p.view_dh[v] = (int16_t)w.dh[p.set_base[v][0]];
    p.view_dw[v] = (int16_t)w.dw[0];
    p.halo = std::max<int>(p.halo, p.set_base[v][0] * std::max(1, row_step));
    span = std::max<int>(span, w.dh[p.set_base[v][sets - 1]] - w.dh[p.set_base[v][0]]);
    Ew = std::max<int>(Ew, w.dw[cols - 1] - w.dw[0]);
    n_max = std::max(n_max, cols * atom); sets_max = std::max(sets_max, sets);
  }
  if (row_step == 0 || p.halo == 0) return 2;                          // one filter row: nothing to stack
  if (col_step) p.stack_step = col_step;
  p.groups = d.groups; p.Kg = Kg; p.Cg = Cg; p.Nimg = d.N;
  p.ctiles = (int)cdiv(Cg, atom);
  p.taps_total = taps_total;
  // Tile: grid pitch and rows with the least work per image, the larger of the MMAs' clocks and the boxes' bytes at
  // 40 B/clk, and 200 clocks per stage.  Rows are whole (a segment's dy would have to end in zeros).
  SlabTile& memo = c->pixel_tiles[GeoKey{kGeoRows, d.dtype, d.Wo, d.Ho, Ew, span, p.halo, row_step, p.stack_step, n_max, sets_max, p.nviews}];
  auto plan = [&](int P, int th) -> bool {
    p.pitch = P; p.th = th; p.a_step = row_step * P;
    p.rows_a = (th + p.halo) * P; p.rows_b = (th + span) * P;
    if (p.a_step > 2047 || p.rows_a > 1200 || p.rows_b > 1200) return false;
    for (int v = 0; v < p.nviews; ++v)
      for (int j = 0; j < p.view_sets[v]; ++j) p.set_rows[v][j] = (int16_t)((views[v].dh[p.set_base[v][j]] - p.view_dh[v]) * P);
    p.tiles_h = (int)cdiv(d.Ho + p.halo, th);
    return wgrad_rows_ring(&p, d.dtype);
  };
  if (!memo.found) {
    long long best = -1;
    for (int P = d.Wo + Ew; P < d.Wo + Ew + kk && P <= 256; ++P)
      for (int th = 1; th <= d.Ho + p.halo && th + std::max(p.halo, span) <= 256; ++th) {
        if (th * P % kk) continue;
        if (!plan(P, th)) break;
        const long long mma = 1LL * th * P / kk * sets_max * std::max(n_max / 2, 32 + n_max / 4), load = (p.rows_a + p.rows_b) * 128LL / 40;
        const long long cost = p.tiles_h * (std::max(mma, load) + 200 + (p.stages < 3 ? mma / 8 : 0));
        if (best < 0 || cost < best) { best = cost; memo.wt = P; memo.th = th; }
      }
    memo.found = true;
  }
  if (!memo.wt || !plan(memo.wt, memo.th)) return 2;
  int rc = make_view(c, &p.dy_map, gin, d.dtype, Kg, d.groups, pad_channels(d.K, d.dtype), d.Wo, d.Ho, d.N, 0, 0, 1, 1, atom, p.pitch, p.th + p.halo, 1,
                     d.dtype == B200CONV_F32);
  if (rc) return rc;
  for (int v = 0; v < p.nviews; ++v)
    if ((rc = views[v].map(&p.x_views[v], p.pitch, p.th + span))) return rc;
  p.diag_c = diag_c; p.diag_k = diag_k;
  p.status = c->d_status;
  p.wait_clocks = c->wait_clocks;
  const size_t slab_elems = (size_t)taps_total * d.K * Cg;
  auto run = [&](int splits, Scratch& sc) -> int {
    p.splits = splits;
    float* partial;
    int r = sc.get(sizeof(float) * slab_elems * splits, reinterpret_cast<void**>(&partial));
    if (r) return r;
    if (dropped) CU_OK(c, cudaMemsetAsync(partial, 0, sizeof(float) * slab_elems * splits, c->stream));
    p.partial = partial;
    p.partial_elems = (long long)slab_elems * splits;
    c->last_variant = "wgrad rows";
    KLAUNCH(c, kKWgradUmma, launch_wgrad_rows(p, d.dtype, c->num_sms, c->stream));
    return reduce(partial, splits);
  };
  GeoKey skey = wgrad_key(kGeoSplits, d, flags);
  skey.add(form);
  const long long tiles = 1LL * p.tiles_h * d.N;
  const int splits = pick_splits(c, skey, tiles, tiles, 1LL * p.ctiles * d.groups * p.nviews, c->num_sms, 3, run);
  if (splits < 0) return splits;
  if ((rc = run(splits, tmp))) return rc;
  c->last_algo = "umma";
  return 0;
}

// The number of neighbouring groups that fill a swizzle atom of filters and channels (wgrad_rows), 1: none.
int merge_factor_rows(const b200conv_desc& d) {
  const int atom = d.dtype == B200CONV_F16 ? 64 : 32, Cg = d.C / d.groups, Kg = d.K / d.groups;
  int best = 1;
  for (int m = 2; m <= d.groups && Cg * m <= atom && Kg * m <= atom; ++m)
    if (d.groups % m == 0 && umma_ok(merged_groups(d, m))) best = m;
  return best;
}

enum { kWgradTaps = 0, kWgradGroups = 1, kWgradRows = 2 };      // the gradWeights kernels; the numbers appear in tuning files

// Stacked filter rows (true) or one tap per item for the forms of layers with few channels (pixel blocks, folded rows); *timed: too
// close to tell, the first call of a geometry decides.  Replayed as graphs, one tap -> stacked: float32 up to 5000 output pixels
// 7.8 to 10 us, 0.86 to 1.02 times as fast (one of 8 layers 1.25); from there on 9 to 323 us, 0.92 to 2.9 times (500 images 1 -> 20 filters 5x5
// at 28x28 91 -> 32 us).  float16 up to 20000 pixels 7.5 to 11 us, 0.83 to 1.04 times; above 100000 1.13 to 2.1 times (7x7 stride 2, 256 images
// of 224x224 306 -> 178 us); between them 0.88 (the same stem, 2 and 4 images: 12.4 -> 14.2, 14.9 -> 17.0 us) to 1.33.
bool stem_rows(const b200conv_desc& d, bool* timed) {
  const long long pixels = 1LL * d.N * d.Ho * d.Wo;
  *timed = d.dtype == B200CONV_F16 && pixels >= 20000 && pixels < 100000;
  return pixels >= (d.dtype == B200CONV_F16 ? 20000 : 5000);
}

// Stacked filter rows or another kernel, for the layers with two ways to run: timed on the first call of a geometry, or the former
// if `prefer`.  rows() returns 2 where it does not apply; both leave the gradient and take scratch of their own.  Stacked rows
// have the most slices (an item is all taps of a channel tile), up to ten times the other kernels': without memory for them the other runs.
template <class Rows, class Other>
int rows_or(b200conv_ctx* c, const GeoKey& key, int flags, bool timed, bool prefer, Rows rows, Other other) {
  int rc, choice = prefer || (flags & B200CONV_ROWS) ? kWgradRows : kWgradTaps;
  if (timed && c->autotune && !(flags & (B200CONV_ROWS | B200CONV_NO_ROWS | B200CONV_NO_GROUP))) {
    auto it = c->algo_cache.find(key);
    if (it != c->algo_cache.end()) choice = it->second;
    else if (!c->capturing && !c->model_only) {
      float ms[2];
      int codes[2];
      bool two = false, no_memory = false;
      auto run = [&](int v) -> int {
        if (v) return two ? other() : 2;
        const int r = rows();
        no_memory |= r == B200CONV_E_NOMEM;
        two = r != 2 && r != B200CONV_E_NOMEM;
        return two ? r : 2;
      };
      if ((rc = rough_times(c, 2, run, ms, codes))) return rc;
      if (!codes[0] && !codes[1] && std::max(ms[0], ms[1]) <= kFarBehind * std::min(ms[0], ms[1]) && (rc = time_variants(c, 2, run, ms, codes))) return rc;
      for (int code : codes)
        if (code && code != 2) return code;
      choice = ms[0] >= 0.f && (ms[1] < 0.f || ms[0] < ms[1]) ? kWgradRows : kWgradTaps;
      if (!no_memory) c->algo_cache[key] = choice;
    }
  }
  if (choice == kWgradRows && (rc = rows()) != 2 && rc != B200CONV_E_NOMEM) return rc;
  return other();
}

int wgrad_device(b200conv_ctx* c, const b200conv_desc& d, const void* x, const void* dy, void* dw,
                 int flags) {
  const int Cg = d.C / d.groups, Kg = d.K / d.groups;
  const size_t es = elem_size(d.dtype);
  const bool x_nhwc = flags & B200CONV_IN_NHWC, dy_nhwc = flags & B200CONV_IN2_NHWC;
  const size_t dw_elems = (size_t)d.K * Cg * d.kH * d.kW;
  // the gradient is accumulated in float32 whatever the data type; B200CONV_DW_F32 also stores it so
  const int odt = (flags & B200CONV_DW_F32) ? B200CONV_F32 : d.dtype;
  const size_t oes = elem_size(odt);
  if (dw_elems == 0) return 0;
  if (d.N == 0) {
    CU_OK(c, cudaMemsetAsync(dw, 0, oes * dw_elems, c->stream));
    return 0;
  }
  b200conv_desc flat;
  if (!(flags & B200CONV_FORCE_DIRECT) && flatten_1x1(d, x_nhwc && dy_nhwc, &flat))
    return wgrad_device(c, flat, x, dy, dw, flags);
  const int mg = (flags & B200CONV_FORCE_DIRECT) ? 1 : merge_factor_wgrad(d);
  if (mg > 1) {
    b200conv_desc dm = d;
    dm.groups = d.groups / mg;
    int t0, nt, q0;
    if (umma_ok(dm) && !fold_ok(dm) && !s2d_ok(dm, &t0, &nt, &q0)) {
      // gradient of block-diagonal filters, of which only the diagonal blocks are stored and added up
      Scratch tm(c);
      const void *xin = x, *gin = dy;
      int rc;
      if (!x_nhwc && (rc = to_nhwc(c, tm, x, d.N, d.C, d.H, d.W, d.dtype, &xin))) return rc;
      if (!dy_nhwc && (rc = to_nhwc(c, tm, dy, d.N, d.K, d.Ho, d.Wo, d.dtype, &gin))) return rc;
      // groups merged to 128 filters x 128 channels, or to one swizzle atom with the filter's rows stacked (32 groups of 8 x 8 channels
      // 3x3, 256 images of 28 x 28, float32: 180 -> 83 us)
      const int mr = merge_factor_rows(d);
      const b200conv_desc dr = merged_groups(d, mr);
      auto kernel = [&](int v) -> int {
        if (v == 0) {
          c->diag_c = Cg; c->diag_k = Kg;
          const int r = wgrad_device(c, dm, xin, gin, dw, flags | B200CONV_IN_NHWC | B200CONV_IN2_NHWC);
          c->diag_c = c->diag_k = 0;
          return r;
        }
        if (!umma_ok(dr)) return 2;
        bool dropped;
        const std::vector<RowsView> views = rows_views(c, dr, xin, &dropped);
        Scratch trial(c);
        const int dc = mr > 1 ? Cg : 0, dk = mr > 1 ? Kg : 0;
        return wgrad_rows(c, dr, kSplitsRows, views, Cg * mr, dropped, d.kH * d.kW, gin, flags, trial, dc, dk, [&](float* partial, int slabs) {
          KLAUNCH(c, kKWgradReduce, launch_wgrad_reduce(partial, dw, slabs, d.kH * d.kW, d.K, Cg * mr, Kg * mr, dc, dk, odt, wgrad_sum(c, d, xin, true, gin, true), c->stream));
          return 0;
        });
      };
      // untimed: float32 gains at every size (2 to 256 images of 7x7 to 56x56, graphs: 0.99 to 2.1 times as fast), float16 not below 6000
      // pixels (0.72 to 0.95, one of five layers 1.18; above 0.95 to 1.5, one of 11 layers 0.83)
      const bool prefer = d.dtype == B200CONV_F32 || 1LL * d.N * d.Ho * d.Wo >= 6000;
      return rows_or(c, wgrad_key(kGeoWgrad, d, flags), flags, true, prefer, [&] { return kernel(1); }, [&] { return kernel(0); });
    }
    if (umma_ok(dm)) {
      // few channels in all: the row-folded forms, then keep the diagonal blocks
      Scratch tm(c);
      void* dwm;
      int rc = tm.get(oes * dw_elems * mg, &dwm);
      if (rc) return rc;
      if ((rc = wgrad_device(c, dm, x, dy, dwm, flags))) return rc;
      KLAUNCH(c, kKPack, launch_merge_groups(dwm, dw, d.K, Cg, Kg, mg, d.kH * d.kW, 1, odt, c->stream));
      return 0;
    }
  }
  const bool use_umma = !(flags & B200CONV_FORCE_DIRECT) && umma_ok(d);
  if (!use_umma) {
    if (flags & B200CONV_FORCE_UMMA) return fail(c, B200CONV_E_UNSUPPORTED, "geometry not covered by the tensor-core kernel");
    if (x_nhwc || dy_nhwc) return fail(c, B200CONV_E_UNSUPPORTED, "direct kernels take NCHW tensors only");
    if (odt != d.dtype) return fail(c, B200CONV_E_UNSUPPORTED, "direct kernels store the gradient in the data type");
    KLAUNCH(c, kKDirect, launch_direct_wgrad(d, x, dy, dw, c->stream));
    c->last_algo = "direct";
    return 0;
  }
  Scratch tmp(c);
  const void* xin = x;
  const void* gin = dy;
  int rc;
  int s2_t0 = 0, s2_nt = 0, s2_q0 = 0;
  if (!(flags & (B200CONV_NO_S2D | B200CONV_ATOMIC_SPLITK)) && s2d_ok(d, &s2_t0, &s2_nt, &s2_q0)) {
    // stride 2 with very few channels: the x operand is the image with 2 x 2 pixel blocks as
    // channels, kS2dPixels consecutive blocks per reduction pixel; the taps are the block rows a
    // filter touches, and the reduction puts the result back into filter order
    if (!dy_nhwc && (rc = to_nhwc(c, tmp, dy, d.N, d.K, d.Ho, d.Wo, d.dtype, &gin))) return rc;
    const int kBK = d.dtype == B200CONV_F16 ? 64 : 32;
    const int Cp = pad_channels(d.C, d.dtype), Kp = pad_channels(d.K, d.dtype);
    const int win = kS2dPixels * kS2dChannels;
    const int H2 = (d.H + 1) / 2, Wq = d.Wo + kS2dPixels - 1;
    void* xs;
    if ((rc = tmp.get(es * (size_t)d.N * H2 * Wq * kS2dChannels, &xs))) return rc;
    KLAUNCH(c, kKTranspose, launch_pad_s2d(x, xs, d.N, d.C, d.H, d.W, Cp, H2, Wq, s2_q0, x_nhwc ? 1 : 0,
                                           d.dtype, c->stream));
    const WgradSum sum = wgrad_sum(c, d, x, x_nhwc, gin, true);
    // the filter's block rows stacked inside the MMAs where the filters leave room
    auto rows = [&]() -> int {
      RowsView v;
      for (int t = 0; t < s2_nt; ++t) { v.dh.push_back(t + s2_t0); v.tap.push_back(t); }
      v.dw.push_back(0);
      v.map = [&](CUtensorMap* m, int bw, int bh) -> int {
        const size_t pix = (size_t)kS2dChannels * es, row = (size_t)Wq * pix;
        cuuint64_t dims[5] = {(cuuint64_t)win, 1, (cuuint64_t)d.Wo, (cuuint64_t)H2, (cuuint64_t)d.N};
        cuuint64_t strides[4] = {row, pix, row, (cuuint64_t)H2 * row};
        cuuint32_t box[5] = {(cuuint32_t)kBK, 1, (cuuint32_t)bw, (cuuint32_t)bh, 1};
        cuuint32_t estr[5] = {1, 1, 1, 1, 1};
        CUresult r = c->encode(m, d.dtype == B200CONV_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, xs, dims, strides, box, estr,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, d.dtype == B200CONV_F32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        return r == CUDA_SUCCESS ? 0 : fail(c, B200CONV_E_CUDA, "cuTensorMapEncodeTiled(space-to-depth x) failed: %d", (int)r);
      };
      Scratch sc(c);
      return wgrad_rows(c, d, kSplitsRowsS2d, {v}, win, false, s2_nt, gin, flags, sc, 0, 0, [&](float* partial, int slabs) {
        KLAUNCH(c, kKWgradReduce, launch_wgrad_reduce_s2d(partial, dw, slabs, d.K, d.C, d.kH, d.kW, s2_nt, s2_t0, s2_q0, d.padH_l, d.padW_l, win, d.flip, odt, sum, c->stream));
        return 0;
      });
    };
    auto single = [&]() -> int {
      Scratch sc(c);
      UmmaWgradParams p;
      memset(&p, 0, sizeof p);
      const int atom = kBK;
      choose_tile(c, d.Wo, d.Ho, d.N, wgrad_pix(d.dtype), d.dtype == B200CONV_F16 ? 16 : 8, &p.bw, &p.bh, &p.bn);
      const bool swz32 = d.dtype == B200CONV_F32;
      if ((rc = make_view(c, &p.dy_map, gin, d.dtype, d.K, 1, Kp, d.Wo, d.Ho, d.N, 0, 0, 1, 1, atom, p.bw, p.bh,
                          p.bn, swz32)))
        return rc;
      {
        const size_t pix = (size_t)kS2dChannels * es, row = (size_t)Wq * pix;
        cuuint64_t dims[5] = {(cuuint64_t)win, 1, (cuuint64_t)d.Wo, (cuuint64_t)H2, (cuuint64_t)d.N};
        cuuint64_t strides[4] = {row, pix, row, (cuuint64_t)H2 * row};
        cuuint32_t box[5] = {(cuuint32_t)atom, 1, (cuuint32_t)p.bw, (cuuint32_t)p.bh, (cuuint32_t)p.bn};
        cuuint32_t estr[5] = {1, 1, 1, 1, 1};
        CUresult r = c->encode(&p.x_views[0],
                               d.dtype == B200CONV_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                               5, xs, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               swz32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(c, B200CONV_E_CUDA, "cuTensorMapEncodeTiled(space-to-depth x) failed: %d", (int)r);
      }
      for (int v = 1; v < kMaxViews; ++v) p.x_views[v] = p.x_views[0];
      p.nviews = 1;
      for (int t = 0; t < s2_nt; ++t) {
        ConvTap tp;
        tp.dh = (int16_t)(t + s2_t0); tp.dw = 0; tp.view = 0; tp.wmat = (int16_t)t;
        p.taps[p.ntaps++] = tp;
      }
      p.groups = 1; p.Kg = d.K; p.Cg = win;
      p.Wo = d.Wo; p.Ho = d.Ho; p.Nimg = d.N;
      p.tiles_w = (int)cdiv(d.Wo, p.bw); p.tiles_h = (int)cdiv(d.Ho, p.bh); p.tiles_n = (int)cdiv(d.N, p.bn);
      p.ktiles = (int)cdiv(d.K, 128); p.ctiles = 1;
      p.taps_total = s2_nt;
      const long long pix_tiles = 1LL * p.tiles_w * p.tiles_h * p.tiles_n;
      const long long base_items = 1LL * p.ktiles * p.ntaps;
      p.splits = (int)balanced_splits(c, pix_tiles, base_items, c->num_sms, pix_tiles / 4, 2);
      const size_t slab_elems = (size_t)s2_nt * d.K * win;
      float* partial;
      if ((rc = sc.get(sizeof(float) * slab_elems * p.splits, reinterpret_cast<void**>(&partial)))) return rc;
      p.partial = partial;
      p.partial_elems = (long long)slab_elems * p.splits;
      p.status = c->d_status;
      p.wait_clocks = c->wait_clocks;
      p.trace = c->trace;
      c->last_variant = "wgrad tap";
      KLAUNCH(c, kKWgradUmma, launch_wgrad_umma(p, d.dtype, 64, c->num_sms, c->stream));
      KLAUNCH(c, kKWgradReduce, launch_wgrad_reduce_s2d(partial, dw, p.splits, d.K, d.C, d.kH, d.kW, s2_nt, s2_t0,
                                                        s2_q0, d.padH_l, d.padW_l, win, d.flip, odt, sum, c->stream));
      c->last_algo = "umma";
      return 0;
    };
    bool timed;
    const bool stacked = stem_rows(d, &timed);
    return rows_or(c, wgrad_key(kGeoWgrad, d, flags), flags, timed, stacked, rows, single);
  }
  if (fold_ok(d) && !(flags & B200CONV_ATOMIC_SPLITK)) {
    // few input channels: the x operand is the row-folded image (kW pixels x Cp channels per
    // reduction pixel), the taps are the kH filter rows, and the reduction unfolds the result
    if (!dy_nhwc && (rc = to_nhwc(c, tmp, dy, d.N, d.K, d.Ho, d.Wo, d.dtype, &gin))) return rc;
    const int kBK = d.dtype == B200CONV_F16 ? 64 : 32;
    const int Cp = pad_channels(d.C, d.dtype), Kp = pad_channels(d.K, d.dtype);
    const int Wp = fold_width(d);
    void* xp;
    if ((rc = tmp.get(es * (size_t)d.N * d.H * Wp * Cp, &xp))) return rc;
    KLAUNCH(c, kKTranspose, launch_pad_fold(x, xp, d.N, d.C, d.H, d.W, Cp, Wp, d.padW_l, x_nhwc ? 1 : 0,
                                            d.dtype, c->stream));
    const WgradSum sum = wgrad_sum(c, d, x, x_nhwc, gin, true);
    // the filter rows stacked inside the MMAs where the filters leave room
    auto rows = [&]() -> int {
      std::vector<RowsView> views;
      bool dropped = false;
      for (int rh = 0; rh < d.sH; ++rh) {
        RowsView v;
        for (int i = 0; i < d.kH; ++i)
          if (pymod(i * d.dilH - d.padH_l, d.sH) == rh) { v.dh.push_back(floordiv(i * d.dilH - d.padH_l, d.sH)); v.tap.push_back(i); }
        if (v.dh.empty()) continue;
        if (rh >= d.H) { dropped = true; continue; }
        v.dw.push_back(0);
        v.map = [=](CUtensorMap* m, int bw, int bh) -> int {
          const size_t pix = (size_t)Cp * es, row = (size_t)Wp * pix;
          const int H2 = (d.H - rh + d.sH - 1) / d.sH;
          cuuint64_t dims[5] = {(cuuint64_t)kBK, 1, (cuuint64_t)d.Wo, (cuuint64_t)H2, (cuuint64_t)d.N};
          cuuint64_t strides[4] = {row, (cuuint64_t)d.sW * pix, (cuuint64_t)d.sH * row, (cuuint64_t)d.H * row};
          cuuint32_t box[5] = {(cuuint32_t)kBK, 1, (cuuint32_t)bw, (cuuint32_t)bh, 1};
          cuuint32_t estr[5] = {1, 1, 1, 1, 1};
          CUresult r = c->encode(m, d.dtype == B200CONV_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5,
                                 static_cast<char*>(xp) + (size_t)rh * row, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 d.dtype == B200CONV_F32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
          return r == CUDA_SUCCESS ? 0 : fail(c, B200CONV_E_CUDA, "cuTensorMapEncodeTiled(folded x) failed: %d", (int)r);
        };
        views.push_back(v);
      }
      Scratch sc(c);
      return wgrad_rows(c, d, kSplitsRowsFold, views, kBK, dropped, d.kH, gin, flags, sc, 0, 0, [&](float* partial, int slabs) {
        KLAUNCH(c, kKWgradReduce, launch_wgrad_reduce_fold(partial, dw, slabs, d.K, d.C, d.kH, d.kW, Cp, kBK, d.flip, odt, sum, c->stream));
        return 0;
      });
    };
    auto single = [&]() -> int {
      Scratch sc(c);
      FwdLikeArgs a;
      a.act = xp; a.Hs = d.H; a.Ws = d.Wo; a.Cin_g = kBK; a.Cp_in = Cp; a.N = d.N; a.dtype = d.dtype;
      a.groups = 1; a.view_sH = d.sH; a.view_sW = 1;
      a.fold = true; a.fold_Wp = Wp; a.fold_sW = d.sW;
      UmmaWgradParams p;
      memset(&p, 0, sizeof p);
      const int atom = kBK;
      choose_tile(c, d.Wo, d.Ho, d.N, wgrad_pix(d.dtype), d.dtype == B200CONV_F16 ? 16 : 8, &p.bw, &p.bh, &p.bn);
      const bool swz32 = d.dtype == B200CONV_F32;
      if ((rc = make_view(c, &p.dy_map, gin, d.dtype, d.K, 1, Kp, d.Wo, d.Ho, d.N, 0, 0, 1, 1, atom, p.bw, p.bh,
                          p.bn, swz32)))
        return rc;
      int nviews = 0, view_of_parity[kMaxViews];
      for (int q = 0; q < kMaxViews; ++q) view_of_parity[q] = -2;
      bool dropped = false;
      for (int i = 0; i < d.kH; ++i) {
        const int ah = i * d.dilH - d.padH_l, rh = pymod(ah, d.sH);
        if (view_of_parity[rh] == -2) {
          view_of_parity[rh] = -1;
          if (rh < d.H) {
            // the folded view with the 32-byte-atom swizzle gradWeights needs for tf32
            const size_t pix = (size_t)Cp * es, row = (size_t)Wp * pix;
            const int H2 = (d.H - rh + d.sH - 1) / d.sH;
            cuuint64_t dims[5] = {(cuuint64_t)kBK, 1, (cuuint64_t)d.Wo, (cuuint64_t)H2, (cuuint64_t)d.N};
            cuuint64_t strides[4] = {row, (cuuint64_t)d.sW * pix, (cuuint64_t)d.sH * row, (cuuint64_t)d.H * row};
            cuuint32_t box[5] = {(cuuint32_t)atom, 1, (cuuint32_t)p.bw, (cuuint32_t)p.bh, (cuuint32_t)p.bn};
            cuuint32_t estr[5] = {1, 1, 1, 1, 1};
            char* base = static_cast<char*>(xp) + (size_t)rh * row;
            CUresult r = c->encode(&p.x_views[nviews],
                                   d.dtype == B200CONV_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                                   5, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                   swz32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (r != CUDA_SUCCESS) return fail(c, B200CONV_E_CUDA, "cuTensorMapEncodeTiled(folded x) failed: %d", (int)r);
            view_of_parity[rh] = nviews++;
          }
        }
        if (view_of_parity[rh] < 0) { dropped = true; continue; }
        ConvTap t;
        t.dh = (int16_t)floordiv(ah, d.sH); t.dw = 0; t.view = (int16_t)view_of_parity[rh]; t.wmat = (int16_t)i;
        p.taps[p.ntaps++] = t;
      }
      for (int v = nviews; v < kMaxViews; ++v) p.x_views[v] = nviews ? p.x_views[0] : p.dy_map;
      p.nviews = nviews;
      p.groups = 1; p.Kg = d.K; p.Cg = kBK;
      p.Wo = d.Wo; p.Ho = d.Ho; p.Nimg = d.N;
      p.tiles_w = (int)cdiv(d.Wo, p.bw); p.tiles_h = (int)cdiv(d.Ho, p.bh); p.tiles_n = (int)cdiv(d.N, p.bn);
      p.ktiles = (int)cdiv(d.K, 128); p.ctiles = 1;
      p.taps_total = d.kH;
      const long long pix_tiles = 1LL * p.tiles_w * p.tiles_h * p.tiles_n;
      const long long base_items = 1LL * p.ktiles * std::max(1, p.ntaps);
      p.splits = (int)balanced_splits(c, pix_tiles, base_items, c->num_sms, pix_tiles / 4, 2);
      const size_t slab_elems = (size_t)d.kH * d.K * kBK;
      float* partial;
      if ((rc = sc.get(sizeof(float) * slab_elems * p.splits, reinterpret_cast<void**>(&partial)))) return rc;
      if (dropped || p.ntaps == 0)
        CU_OK(c, cudaMemsetAsync(partial, 0, sizeof(float) * slab_elems * p.splits, c->stream));
      p.partial = partial;
      p.partial_elems = (long long)slab_elems * p.splits;
      p.status = c->d_status;
      p.wait_clocks = c->wait_clocks;
      p.trace = c->trace;
      c->last_variant = "wgrad tap";
      if (p.ntaps > 0) KLAUNCH(c, kKWgradUmma, launch_wgrad_umma(p, d.dtype, 64, c->num_sms, c->stream));
      KLAUNCH(c, kKWgradReduce, launch_wgrad_reduce_fold(partial, dw, p.splits, d.K, d.C, d.kH, d.kW, Cp, kBK,
                                                         d.flip, odt, sum, c->stream));
      c->last_algo = "umma";
      return 0;
    };
    bool timed;
    const bool stacked = stem_rows(d, &timed);
    return rows_or(c, wgrad_key(kGeoWgrad, d, flags), flags, timed, stacked, rows, single);
  }
  if (!x_nhwc && (rc = to_nhwc(c, tmp, x, d.N, d.C, d.H, d.W, d.dtype, &xin))) return rc;
  if (!dy_nhwc && (rc = to_nhwc(c, tmp, dy, d.N, d.K, d.Ho, d.Wo, d.dtype, &gin))) return rc;
  const int Cp = pad_channels(d.C, d.dtype), Kp = pad_channels(d.K, d.dtype);

  // Three tensor-core kernels: one tap per work item, tap groups sharing operands, or all taps of narrow layers in one MMA.  As for
  // the forward kernels the first call of a geometry times those that apply and the context remembers the winner.
  auto rows = [&](Scratch& sc) -> int {
    bool dropped;
    const std::vector<RowsView> views = rows_views(c, d, xin, &dropped);
    return wgrad_rows(c, d, kSplitsRows, views, Cg, dropped, d.kH * d.kW, gin, flags, sc, c->diag_c, c->diag_k, [&](float* partial, int slabs) {
      KLAUNCH(c, kKWgradReduce, launch_wgrad_reduce(partial, dw, slabs, d.kH * d.kW, d.K, Cg, Kg, c->diag_c, c->diag_k, odt, wgrad_sum(c, d, xin, true, gin, true), c->stream));
      return 0;
    });
  };
  const GeoKey key = wgrad_key(kGeoWgrad, d, flags);
  // without timings: the one-tap kernel where it runs 256-column MMAs (their issue and TMA
  // budgets are comfortable), tap groups for narrower layers (they read the operands 3x less)
  int choice = (flags & B200CONV_NO_GROUP) || (!c->autotune && Cg >= 256) ? kWgradTaps : kWgradGroups;
  // (2: not for this layer; without memory for its slices the others run, as in rows_or)
  if ((flags & B200CONV_ROWS) && (rc = rows(tmp)) != 2 && rc != B200CONV_E_NOMEM) return rc;
  if (choice == kWgradGroups && c->autotune) {
    auto itc = c->algo_cache.find(key);
    if (itc != c->algo_cache.end()) {
      choice = itc->second;
    } else if (!c->capturing) {
      // own scratch, returned to the pool after each run: the next run then reuses the buffers and its timing
      // holds no allocation
      // The kernels choose a slice count of their own: that is timed only where they are close with the models'.
      const int order[3] = {kWgradRows, kWgradGroups, kWgradTaps};
      float ms[3];
      int codes[3];
      bool others = false, no_memory = false;                 // others: another kernel than the one-tap form applies
      auto kernel = [&](int i) -> int {
        if (order[i] == kWgradTaps) return others ? wgrad_device(c, d, xin, gin, dw, flags | B200CONV_NO_GROUP | B200CONV_IN_NHWC | B200CONV_IN2_NHWC) : 2;
        Scratch trial(c);
        int r = order[i] == kWgradGroups ? wgrad_grouped(c, d, xin, gin, dw, flags, trial) : rows(trial);
        if (order[i] == kWgradRows && r == B200CONV_E_NOMEM) { no_memory = true; r = 2; }
        others |= r != 2;
        return r;
      };
      if ((rc = rough_times(c, 3, kernel, ms, codes))) return rc;
      float least = -1.f;
      for (float m : ms) if (m >= 0.f && (least < 0.f || m < least)) least = m;
      bool far[3];
      int close = 0;
      for (int i = 0; i < 3; ++i) { far[i] = ms[i] < 0.f || ms[i] > kFarBehind * least; close += !far[i]; }
      for (int code : codes)
        if (code && code != 2) return code;
      if (close > 1) {
        if ((rc = time_variants(c, 3, [&](int i) { return far[i] ? 2 : kernel(i); }, ms, codes))) return rc;
        for (int code : codes)
          if (code && code != 2) return code;
      }
      choice = kWgradTaps;
      least = -1.f;
      for (int i = 0; i < 3; ++i)
        if (ms[i] >= 0.f && (least < 0.f || ms[i] < least)) { least = ms[i]; choice = order[i]; }
      if (!no_memory) c->algo_cache[key] = choice;
    }
  }
  if (choice == kWgradRows && (rc = rows(tmp)) != 2 && rc != B200CONV_E_NOMEM) return rc;
  if (choice != kWgradTaps) {
    rc = wgrad_grouped(c, d, xin, gin, dw, flags, tmp);
    if (rc != 2) return rc;     // 2: geometry not covered, use the one-tap-per-item kernel
  }

  UmmaWgradParams p;
  memset(&p, 0, sizeof p);
  const int atom = d.dtype == B200CONV_F16 ? 64 : 32;
  const int kk = d.dtype == B200CONV_F16 ? 16 : 8;
  const int BN = Cg <= 64 ? 64 : Cg <= 128 ? 128 : 256;
  choose_tile(c, d.Wo, d.Ho, d.N, wgrad_pix(d.dtype, BN), kk, &p.bw, &p.bh, &p.bn);
  const bool swz32 = d.dtype == B200CONV_F32;  // MN-major tf32 operands need 32-byte swizzle atoms
  rc = make_view(c, &p.dy_map, gin, d.dtype, Kg, d.groups, Kp, d.Wo, d.Ho, d.N, 0, 0, 1, 1, atom,
                 p.bw, p.bh, p.bn, swz32);
  if (rc) return rc;
  std::vector<std::pair<int, int>> parity;
  std::vector<int> view_of;  // parity index -> tensor map index or -1
  int nviews = 0;
  bool dropped = false;
  for (int i = 0; i < d.kH; ++i)
    for (int j = 0; j < d.kW; ++j) {
      const int ah = i * d.dilH - d.padH_l, aw = j * d.dilW - d.padW_l;
      const int rh = pymod(ah, d.sH), rw = pymod(aw, d.sW);
      int v = -1;
      for (size_t q = 0; q < parity.size(); ++q)
        if (parity[q].first == rh && parity[q].second == rw) v = (int)q;
      if (v < 0) {
        v = (int)parity.size();
        parity.push_back({rh, rw});
        int slot = -1;
        if (rh < d.H && rw < d.W) {
          slot = nviews++;
          rc = make_view(c, &p.x_views[slot], xin, d.dtype, Cg, d.groups, Cp, d.W, d.H, d.N, rh, rw,
                         d.sH, d.sW, atom, p.bw, p.bh, p.bn, swz32);
          if (rc) return rc;
        }
        view_of.push_back(slot);
      }
      if (view_of[v] < 0) { dropped = true; continue; }
      ConvTap t;
      t.dh = (int16_t)floordiv(ah, d.sH); t.dw = (int16_t)floordiv(aw, d.sW);
      t.view = (int16_t)view_of[v];
      const int wi = d.flip ? d.kH - 1 - i : i, wj = d.flip ? d.kW - 1 - j : j;
      t.wmat = (int16_t)(wi * d.kW + wj);
      p.taps[p.ntaps++] = t;
    }
  for (int v = nviews; v < kMaxViews; ++v) p.x_views[v] = nviews ? p.x_views[0] : p.dy_map;
  p.nviews = nviews;
  p.groups = d.groups; p.Kg = Kg; p.Cg = Cg;
  p.Wo = d.Wo; p.Ho = d.Ho; p.Nimg = d.N;
  p.tiles_w = (int)cdiv(d.Wo, p.bw); p.tiles_h = (int)cdiv(d.Ho, p.bh); p.tiles_n = (int)cdiv(d.N, p.bn);
  // 256+ filters and 256+ channels: pairs of CTAs compute 256 x 256 tiles and share the x tile
  const bool pair = c->use_pair && BN == 256 && Kg >= 256 && c->num_sms >= 2;
  p.ktiles = (int)cdiv(Kg, pair ? 256 : 128); p.ctiles = (int)cdiv(Cg, BN);
  p.taps_total = d.kH * d.kW;
  const long long pix_tiles = 1LL * p.tiles_w * p.tiles_h * p.tiles_n;
  const long long base_items = 1LL * p.ktiles * p.ctiles * d.groups * std::max(1, p.ntaps);
  p.atomic = (flags & B200CONV_ATOMIC_SPLITK) ? 1 : 0;
  p.diag_c = c->diag_c; p.diag_k = c->diag_k;
  p.status = c->d_status;
  p.wait_clocks = c->wait_clocks;
  p.trace = c->trace;
  const size_t slab_elems = (size_t)p.taps_total * d.K * Cg;
  auto run = [&](int splits, Scratch& sc) -> int {
    p.splits = splits;
    const int slabs = p.atomic ? 1 : p.splits;
    float* partial;
    int r = sc.get(sizeof(float) * slab_elems * slabs, reinterpret_cast<void**>(&partial));
    if (r) return r;
    if (p.atomic || dropped || p.ntaps == 0)
      CU_OK(c, cudaMemsetAsync(partial, 0, sizeof(float) * slab_elems * slabs, c->stream));
    p.partial = partial;
    p.partial_elems = (long long)slab_elems * slabs;
    c->last_variant = pair ? "wgrad pair" : "wgrad tap";
    if (p.ntaps > 0) {
      if (pair) KLAUNCH(c, kKWgradUmma, launch_wgrad_pair(p, d.dtype, c->num_sms, c->stream));
      else KLAUNCH(c, kKWgradUmma, launch_wgrad_umma(p, d.dtype, BN, c->num_sms, c->stream));
    }
    KLAUNCH(c, kKWgradReduce, launch_wgrad_reduce(partial, dw, slabs, p.taps_total, d.K, Cg, Kg, p.diag_c, p.diag_k, odt, wgrad_sum(c, d, xin, true, gin, true), c->stream));
    return 0;
  };
  GeoKey skey = wgrad_key(kGeoSplits, d, flags);
  skey.add(pair ? kSplitsPair : kSplitsTaps);
  const int splits = pick_splits(c, skey, pix_tiles, std::max(1LL, pix_tiles / 4), base_items, pair ? c->num_sms / 2 : c->num_sms, 2, run);
  if (splits < 0) return splits;
  if ((rc = run(splits, tmp))) return rc;
  c->last_algo = "umma";
  return 0;
}

// ---- host-pointer wrappers: copy in, run, copy out, synchronise ---------------------------
// Makes the ring on first use.  False where the system gives no page-locked memory for it, or with no copy threads
// asked for: pageable arrays then travel at the pace of the driver's own staging.
bool ring_ready(b200conv_ctx* c) {
  if (c->copy_pool || c->no_ring) return c->copy_pool != nullptr;
  const char* env = getenv("B200CONV_COPY_THREADS");
  const int cores = (int)std::thread::hardware_concurrency();
  // 16 MB into pinned memory: 1069 / 615 / 331 / 218 / 237 us with 1 / 2 / 4 / 8 / 12 threads (link: 310 us)
  const int n = env ? atoi(env) : std::min(8, std::max(2, cores / 2));
  void* p = nullptr;
  cudaError_t e = n <= 0 ? cudaErrorMemoryAllocation : cudaHostAlloc(&p, kRingSlotBytes * kRingSlots, cudaHostAllocDefault);
  for (int i = 0; i < kRingSlots && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&c->ring_ev[i], cudaEventDisableTiming);
  if (e != cudaSuccess) {
    if (p) cudaFreeHost(p);
    cudaGetLastError();
    c->no_ring = true;
    return false;
  }
  c->ring = static_cast<char*>(p);
  c->copy_pool = new CopyPool(std::min(n, 16));
  return true;
}

// A free slot of the ring (waits for the transfer that used it last).
int ring_slot(b200conv_ctx* c, int* k) {
  *k = c->ring_next;
  c->ring_next = (c->ring_next + 1) % kRingSlots;
  if (c->ring_busy[*k]) CU_OK(c, cudaEventSynchronize(c->ring_ev[*k]));
  c->ring_busy[*k] = false;
  return 0;
}
int ring_used(b200conv_ctx* c, int k, cudaStream_t s) {
  CU_OK(c, cudaEventRecord(c->ring_ev[k], s));
  c->ring_busy[k] = true;
  return 0;
}

// The next chunk of an array of which `off` of `bytes` have gone: small ones first, so that the link
// starts early, doubling up to a slot (the calls per chunk cost about 4 us).
size_t chunk_bytes(size_t off, size_t bytes) {
  return std::min(bytes - off, std::min(kRingSlotBytes, std::max<size_t>(256u << 10, off)));
}

bool is_pinned(const void* h, size_t bytes) {
  cudaPointerAttributes a, b;
  if (cudaPointerGetAttributes(&a, h) != cudaSuccess ||
      cudaPointerGetAttributes(&b, static_cast<const char*>(h) + bytes - 1) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost && b.type == cudaMemoryTypeHost;
}

// Host array -> device memory on stream s.  The array may be reused when this returns unless it is pinned.
int upload(b200conv_ctx* c, void* d, const void* h, size_t bytes, cudaStream_t s, bool pinned) {
  if (pinned || !ring_ready(c)) {
    CU_OK(c, cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s));
    return 0;
  }
  int rc;
  for (size_t off = 0, n; off < bytes; off += n) {
    n = chunk_bytes(off, bytes);
    int k;
    if ((rc = ring_slot(c, &k))) return rc;
    char* slot = c->ring + kRingSlotBytes * k;
    c->copy_pool->copy(slot, static_cast<const char*>(h) + off, n, true);
    CU_OK(c, cudaMemcpyAsync(static_cast<char*>(d) + off, slot, n, cudaMemcpyHostToDevice, s));
    if ((rc = ring_used(c, k, s))) return rc;
  }
  return 0;
}

// Device memory -> host array on stream s.  A pinned array is complete when the stream is; a pageable
// one when this returns: chunks travel into ring slots, up to half a ring ahead of the copy threads
// that empty them.
int download(b200conv_ctx* c, void* h, const void* d, size_t bytes, cudaStream_t s, bool pinned) {
  if (pinned || !ring_ready(c)) {
    CU_OK(c, cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, s));
    return 0;
  }
  int rc;
  // Large arrays are likely to be fresh memory: while the transfers of a window fly, the threads make its pages present.
  constexpr size_t kTouchFrom = 4u << 20, kTouchWindow = 16u << 20, kLargeArray = 64u << 20;
  size_t touched = bytes >= kTouchFrom ? 0 : bytes;
  constexpr int kAhead = kRingSlots / 2;
  struct { int slot; size_t off, n; } flying[kAhead];
  size_t off = 0;
  int issued = 0;
  for (int taken = 0; off < bytes || taken < issued; ++taken) {
    for (; off < bytes && issued - taken < kAhead; ++issued) {
      auto& f = flying[issued % kAhead];
      f.off = off;
      f.n = chunk_bytes(off, bytes);
      if ((rc = ring_slot(c, &f.slot))) return rc;
      CU_OK(c, cudaMemcpyAsync(c->ring + kRingSlotBytes * f.slot, static_cast<const char*>(d) + off, f.n, cudaMemcpyDeviceToHost, s));
      if ((rc = ring_used(c, f.slot, s))) return rc;
      off += f.n;
    }
    const auto& f = flying[taken % kAhead];
    while (touched < f.off + f.n) {
      const size_t n = std::min(kTouchWindow, bytes - touched);
      c->copy_pool->touch(static_cast<char*>(h) + touched, n);
      touched += n;
    }
    CU_OK(c, cudaEventSynchronize(c->ring_ev[f.slot]));
    c->ring_busy[f.slot] = false;
    c->copy_pool->copy(static_cast<char*>(h) + f.off, c->ring + kRingSlotBytes * f.slot, f.n, false, bytes >= kLargeArray);
  }
  return 0;
}

int copy_streams(b200conv_ctx* c) {
  if (!c->up_stream) {
    CU_OK(c, cudaStreamCreateWithFlags(&c->up_stream, cudaStreamNonBlocking));
    CU_OK(c, cudaStreamCreateWithFlags(&c->down_stream, cudaStreamNonBlocking));
    CU_OK(c, cudaEventCreateWithFlags(&c->ev_up, cudaEventDisableTiming));
    CU_OK(c, cudaEventCreateWithFlags(&c->ev_down, cudaEventDisableTiming));
  }
  return 0;
}

int chunk_event(b200conv_ctx* c, size_t i, cudaEvent_t* e) {
  while (c->chunk_ev.size() <= i) {
    cudaEvent_t n;
    CU_OK(c, cudaEventCreateWithFlags(&n, cudaEventDisableTiming));
    c->chunk_ev.push_back(n);
  }
  *e = c->chunk_ev[i];
  return 0;
}

// The tensors of one host-pointer call.
struct HostIO {
  b200conv_ctx* c;
  Scratch tmp;
  char *group_dev = nullptr, *group_host = nullptr;   // small inputs side by side: one transfer for all
  size_t group_used = 0;
  int group_slot = -1;
  explicit HostIO(b200conv_ctx* ctx) : c(ctx), tmp(ctx) {}
  int out(size_t bytes, void** d) { return tmp.get(bytes, d); }
  // A small input joins the group (start() sends it), a larger one is on its way when this returns.
  int in(const void* h, size_t bytes, void** d) {
    int rc;
    if (bytes <= kSmallInput && ring_ready(c)) {
      if ((rc = small_space(bytes, d))) return rc;
      memcpy(group_host + (static_cast<char*>(*d) - group_dev), h, bytes);
      return 0;
    }
    // the ring turns under a large input, so the slot of a waiting group has to be on its way first
    if ((rc = start()) || (rc = tmp.get(bytes, d))) return rc;
    return bytes ? upload(c, *d, h, bytes, c->stream, is_pinned(h, bytes)) : 0;
  }
  int start() {
    if (!group_dev) return 0;
    if (group_used) {
      CU_OK(c, cudaMemcpyAsync(group_dev, group_host, group_used, cudaMemcpyHostToDevice, c->stream));
      if (int rc = ring_used(c, group_slot, c->stream)) return rc;
    }
    group_dev = group_host = nullptr;
    group_used = 0;
    return 0;
  }
  int back(void* h, const void* d, size_t bytes) {
    return bytes ? download(c, h, d, bytes, c->stream, is_pinned(h, bytes)) : 0;
  }

 private:
  int small_space(size_t bytes, void** d) {
    int rc;
    if (!group_dev) {
      if ((rc = ring_slot(c, &group_slot))) return rc;
      void* p;
      if ((rc = tmp.get(4 * (kSmallInput + 256), &p))) return rc;      // at most four inputs per call
      group_dev = static_cast<char*>(p);
      group_host = c->ring + kRingSlotBytes * group_slot;
    }
    *d = group_dev + group_used;
    group_used += (bytes + 255) & ~static_cast<size_t>(255);
    return 0;
  }
};

// Forward and gradInputs compute every image by itself, so a large batch goes through in chunks of
// images: the upload of one chunk, the kernels of the one before and the download of the one before
// that run side by side (the link carries both directions at once).
struct BatchPlan {
  int chunks, images;      // chunks of `images` images, the last one possibly smaller
};
BatchPlan plan_batch(int N, size_t in_bytes, size_t out_bytes) {
  // chunks of about 4 MB of the larger side (75 us on the link, against 20 to 40 us of launches and
  // transfers' latencies per chunk), at most 8; equal ones where a count near that divides the batch
  // (another batch size is another geometry to choose kernels for)
  const size_t big = std::max(in_bytes, out_bytes);
  const int n = (int)std::min<size_t>(std::min<size_t>(8, N), big / (4u << 20));
  if (n <= 1 || std::min(in_bytes, out_bytes) < (1u << 20)) return {1, N};
  for (int m = n; m > n / 2 && m > 1; --m)
    if (N % m == 0) return {m, N / m};
  const int per = (int)cdiv(N, n);
  return {(int)cdiv(N, per), per};
}

// Runs `compute(images, device input, device output)` over the batch.
template <class Compute>
int run_batch(b200conv_ctx* c, HostIO& io, int N, const void* hin, size_t in_bytes, void* hout, size_t out_bytes,
              Compute compute) {
  int rc;
  void *din, *dout;
  // a result that lies over the input (and not each image over its own): all of the input goes up before any of the
  // result comes down
  const bool over = overlap(hin, in_bytes, hout, out_bytes) && !(hin == hout && in_bytes == out_bytes);
  const BatchPlan bp = over ? BatchPlan{1, N} : plan_batch(N, in_bytes, out_bytes);
  if (bp.chunks == 1) {
    if ((rc = io.in(hin, in_bytes, &din)) || (rc = io.out(out_bytes, &dout)) || (rc = io.start())) return rc;
    if ((rc = compute(N, din, dout))) return rc;
    return io.back(hout, dout, out_bytes);
  }
  if ((rc = io.start()) || (rc = copy_streams(c)) || (rc = io.out(in_bytes, &din)) || (rc = io.out(out_bytes, &dout))) return rc;
  const bool pin_in = is_pinned(hin, in_bytes), pin_out = is_pinned(hout, out_bytes);
  const size_t in1 = in_bytes / N, out1 = out_bytes / N;
  // the buffers come from the pool of the main stream: what still uses them there goes first
  CU_OK(c, cudaEventRecord(c->ev_up, c->stream));
  CU_OK(c, cudaStreamWaitEvent(c->up_stream, c->ev_up, 0));
  // An error leaves the loop with transfers in flight: they are waited for before the buffers go back.
  auto step = [&](int i) -> int {
    const int a = i * bp.images, b = std::min(N, a + bp.images);
    cudaEvent_t up, done;
    int r;
    if ((r = chunk_event(c, 2 * i, &up)) || (r = chunk_event(c, 2 * i + 1, &done))) return r;
    if ((r = upload(c, static_cast<char*>(din) + in1 * a, static_cast<const char*>(hin) + in1 * a, in1 * (b - a), c->up_stream, pin_in))) return r;
    CU_OK(c, cudaEventRecord(up, c->up_stream));
    CU_OK(c, cudaStreamWaitEvent(c->stream, up, 0));
    if ((r = compute(b - a, static_cast<char*>(din) + in1 * a, static_cast<char*>(dout) + out1 * a))) return r;
    CU_OK(c, cudaEventRecord(done, c->stream));
    CU_OK(c, cudaStreamWaitEvent(c->down_stream, done, 0));
    return 0;
  };
  auto fetch = [&](int i) -> int {
    const int a = i * bp.images, b = std::min(N, a + bp.images);
    return download(c, static_cast<char*>(hout) + out1 * a, static_cast<const char*>(dout) + out1 * a, out1 * (b - a), c->down_stream, pin_out);
  };
  // a pageable result is copied out by the host, one chunk behind, so that it does not hold up the uploads
  for (int i = 0; i < bp.chunks && !rc; ++i) {
    rc = step(i);
    if (!rc && pin_out) rc = fetch(i);
    if (!rc && !pin_out && i > 0) rc = fetch(i - 1);
  }
  if (!rc && !pin_out) rc = fetch(bp.chunks - 1);
  cudaStreamSynchronize(c->up_stream);
  cudaStreamSynchronize(c->down_stream);
  return rc;
}

}  // namespace

// ======================================================================================
// exported functions
// ======================================================================================
extern "C" {

const char* b200conv_version(void) { return "b200conv 0.1 (sm_100a)"; }

int b200conv_create_error(char* buf, size_t n) {
  std::lock_guard<std::mutex> g(g_create_mu);
  if (buf && n) {
    strncpy(buf, g_create_err.c_str(), n - 1);
    buf[n - 1] = 0;
  }
  return (int)g_create_err.size();
}

int b200conv_create(int device, b200conv_ctx** out) {
  std::lock_guard<std::mutex> g(g_create_mu);
  if (!out) return B200CONV_E_INVALID;
  *out = nullptr;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0) {
    g_create_err = std::string("no CUDA device: ") + cudaGetErrorString(e);
    cudaGetLastError();
    return B200CONV_E_CUDA;
  }
  if (device < 0 || device >= ndev) {
    g_create_err = "device index out of range";
    return B200CONV_E_INVALID;
  }
  cudaDeviceProp prop;
  cudaGetDeviceProperties(&prop, device);
  if (prop.major != 10) {
    g_create_err = "device is not compute capability 10.x (this library is built for sm_100a only)";
    return B200CONV_E_UNSUPPORTED;
  }
  DeviceGuard dg(device);
  b200conv_ctx* c = new b200conv_ctx();
  c->device = device;
  c->num_sms = c->device_sms = prop.multiProcessorCount;
  void* hs = nullptr;
  bool ok = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) == cudaSuccess &&
            cudaHostAlloc(&hs, sizeof(int), cudaHostAllocMapped) == cudaSuccess &&
            cudaHostGetDevicePointer(reinterpret_cast<void**>(&c->d_status), hs, 0) == cudaSuccess &&
            cudaMalloc(reinterpret_cast<void**>(&c->d_arrivals), kArrivals * sizeof(unsigned int)) == cudaSuccess &&
            cudaMemsetAsync(c->d_arrivals, 0, kArrivals * sizeof(unsigned int), c->stream) == cudaSuccess &&      // a non-blocking stream waits for no other
            cudaEventCreate(&c->ev0) == cudaSuccess && cudaEventCreate(&c->ev1) == cudaSuccess;
  if (ok) {
    c->h_status = static_cast<volatile int*>(hs);
    *c->h_status = 0;
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qr;
    ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) == cudaSuccess &&
         qr == cudaDriverEntryPointSuccess && fn;
    c->encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  if (!ok) {
    g_create_err = std::string("context setup failed: ") + cudaGetErrorString(cudaGetLastError());
    delete c;
    return B200CONV_E_CUDA;
  }
  *out = c;
  return 0;
}

void b200conv_destroy(b200conv_ctx* c) {
  if (!c) return;
  DeviceGuard dg(c->device);
  cudaStreamSynchronize(c->stream);
  b200conv_nccl_destroy(c);
  for (auto& kv : c->free_blocks) cudaFree(kv.second);
  for (auto& kv : c->live) cudaFree(kv.first);
  if (c->l2buf) cudaFree(c->l2buf);
  if (c->d_token) cudaFree(c->d_token);
  if (c->up_stream) {
    cudaStreamDestroy(c->up_stream);
    cudaStreamDestroy(c->down_stream);
    cudaEventDestroy(c->ev_up);
    cudaEventDestroy(c->ev_down);
  }
  if (c->comm_stream) {
    cudaStreamDestroy(c->comm_stream);
    cudaEventDestroy(c->ev_comm_ready);
    cudaEventDestroy(c->ev_comm_done);
  }
  delete c->copy_pool;
  if (c->ring) cudaFreeHost(c->ring);
  for (cudaEvent_t e : c->ring_ev)
    if (e) cudaEventDestroy(e);
  for (cudaEvent_t e : c->chunk_ev) cudaEventDestroy(e);
  cudaFreeHost(const_cast<int*>(c->h_status));
  cudaFree(c->d_arrivals);
  for (auto& r : c->prof_recs) { cudaEventDestroy(r.a); cudaEventDestroy(r.b); }
  for (auto& e : c->prof_pool) cudaEventDestroy(e);
  cudaEventDestroy(c->ev0);
  cudaEventDestroy(c->ev1);
  if (c->ev_tune0) { cudaEventDestroy(c->ev_tune0); cudaEventDestroy(c->ev_tune1); }
  cudaStreamDestroy(c->stream);
  delete c;
}

int b200conv_last_error(b200conv_ctx* c, char* buf, size_t n) {
  if (!c) return 0;
  std::lock_guard<std::mutex> g(c->mu);
  if (buf && n) {
    strncpy(buf, c->err.c_str(), n - 1);
    buf[n - 1] = 0;
  }
  return (int)c->err.size();
}

int b200conv_padded_channels(int C, int dtype) { return pad_channels(C, dtype); }

// Resets the context's forward epilogue when a call returns, whichever way.
struct EpilogueScope {
  b200conv_ctx* c;
  EpilogueScope(b200conv_ctx* ctx, const ConvEpilogue& e) : c(ctx) { c->epi = e; }
  ~EpilogueScope() { c->epi = default_epilogue(); }
};

static int fwd_call(b200conv_ctx* c, const b200conv_desc* d, const void* x, const void* w, const void* bias,
                    const void* residual, void* y, ConvEpilogue epi, int flags) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  int rc = validate(c, d);
  if (rc) return rc;
  epi.pool = (flags & B200CONV_POOL2X2) ? 1 : 0;
  if (!(flags & B200CONV_HOST_PTRS)) {
    epi.residual = residual;
    EpilogueScope scope(c, epi);
    return fwd_device(c, *d, x, w, bias, y, flags);
  }
  if (epi.pool) return fail(c, B200CONV_E_UNSUPPORTED, "the pooling epilogue takes channels-last device tensors");
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "host-pointer calls cannot be captured in a graph");
  if (flags & (B200CONV_IN_NHWC | B200CONV_OUT_NHWC))
    return fail(c, B200CONV_E_INVALID, "host tensors are NCHW");
  const size_t es = elem_size(d->dtype);
  const size_t nx = es * (size_t)d->N * d->C * d->H * d->W, nw = es * (size_t)d->K * (d->C / d->groups) * d->kH * d->kW,
               ny = es * (size_t)d->N * d->K * d->Ho * d->Wo;
  HostIO io(c);
  void *dw_, *db_ = nullptr, *dr_ = nullptr;
  if ((rc = io.in(w, nw, &dw_))) return rc;
  if (bias && (rc = io.in(bias, es * d->K, &db_))) return rc;
  if (residual && (rc = io.in(residual, ny, &dr_))) return rc;
  const char* res = static_cast<const char*>(dr_);
  rc = run_batch(c, io, d->N, x, nx, y, ny, [&](int images, const void* xin, void* yout) {
    b200conv_desc part = *d;
    part.N = images;
    epi.residual = res;
    if (res && images) res += ny / d->N * images;
    EpilogueScope scope(c, epi);
    return fwd_device(c, part, xin, dw_, db_, yout, (flags & ~B200CONV_HOST_PTRS) | kScratchFilters);
  });
  if (rc) return rc;
  return sync_and_check(c);
}

int b200conv_fwd(b200conv_ctx* c, const b200conv_desc* d, const void* x, const void* w,
                 const void* bias, void* y, int flags) {
  return fwd_call(c, d, x, w, bias, nullptr, y, default_epilogue(), flags);
}

int b200conv_fwd_epilogue(b200conv_ctx* c, const b200conv_desc* d, const void* x, const void* w,
                          const void* bias, const void* residual, void* y, float alpha, float beta,
                          float slope, int flags) {
  ConvEpilogue e = default_epilogue();
  e.alpha = alpha;
  e.beta = residual ? beta : 0.f;
  e.lin = 0.5f * (1.f + slope);
  e.abs = 0.5f * (1.f - slope);
  return fwd_call(c, d, x, w, bias, residual, y, e, flags);
}

int b200conv_dgrad(b200conv_ctx* c, const b200conv_desc* d, const void* w, const void* dy, void* dx,
                   int flags) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  int rc = validate(c, d);
  if (rc) return rc;
  if (!(flags & B200CONV_HOST_PTRS)) return dgrad_device(c, *d, w, dy, dx, flags);
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "host-pointer calls cannot be captured in a graph");
  if (flags & (B200CONV_IN_NHWC | B200CONV_OUT_NHWC))
    return fail(c, B200CONV_E_INVALID, "host tensors are NCHW");
  const size_t es = elem_size(d->dtype);
  const size_t nx = es * (size_t)d->N * d->C * d->H * d->W, nw = es * (size_t)d->K * (d->C / d->groups) * d->kH * d->kW,
               ny = es * (size_t)d->N * d->K * d->Ho * d->Wo;
  HostIO io(c);
  void* dw_;
  if ((rc = io.in(w, nw, &dw_))) return rc;
  rc = run_batch(c, io, d->N, dy, ny, dx, nx, [&](int images, const void* dyin, void* dxout) {
    b200conv_desc part = *d;
    part.N = images;
    return dgrad_device(c, part, dw_, dyin, dxout, (flags & ~B200CONV_HOST_PTRS) | kScratchFilters);
  });
  if (rc) return rc;
  return sync_and_check(c);
}

int b200conv_wgrad(b200conv_ctx* c, const b200conv_desc* d, const void* x, const void* dy, void* dw,
                   int flags) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  int rc = validate(c, d);
  if (rc) return rc;
  if (!(flags & B200CONV_HOST_PTRS)) return wgrad_device(c, *d, x, dy, dw, flags);
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "host-pointer calls cannot be captured in a graph");
  if (flags & (B200CONV_IN_NHWC | B200CONV_IN2_NHWC))
    return fail(c, B200CONV_E_INVALID, "host tensors are NCHW");
  const size_t es = elem_size(d->dtype);
  const size_t nx = es * (size_t)d->N * d->C * d->H * d->W, nw = es * (size_t)d->K * (d->C / d->groups) * d->kH * d->kW,
               ny = es * (size_t)d->N * d->K * d->Ho * d->Wo;
  HostIO io(c);
  void *dx_, *dy_, *dw_;
  const size_t nw_out = (flags & B200CONV_DW_F32) ? nw / es * sizeof(float) : nw;
  if ((rc = io.in(x, nx, &dx_)) || (rc = io.in(dy, ny, &dy_)) || (rc = io.out(nw_out, &dw_)) || (rc = io.start())) return rc;
  if ((rc = wgrad_device(c, *d, dx_, dy_, dw_, flags & ~B200CONV_HOST_PTRS))) return rc;
  if ((rc = io.back(dw, dw_, nw_out))) return rc;
  return sync_and_check(c);
}

int b200conv_maxpool2x2(b200conv_ctx* c, const void* x, void* y, int N, int C, int H, int W,
                        int dtype, int flags) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (N < 0 || C < 0 || H < 2 || W < 2) return fail(c, B200CONV_E_INVALID, "pool needs H, W >= 2");
  const size_t es = elem_size(dtype);
  const int nhwc = (flags & B200CONV_IN_NHWC) ? 1 : 0, Cp = pad_channels(C, dtype);
  if (!(flags & B200CONV_HOST_PTRS)) {
    KLAUNCH(c, kKPool, launch_maxpool2x2(x, y, N, C, H, W, nhwc, Cp, dtype, c->stream));
    return 0;
  }
  if (nhwc) return fail(c, B200CONV_E_INVALID, "host tensors are NCHW");
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "host-pointer calls cannot be captured in a graph");
  HostIO io(c);
  void *dx_, *dy_;
  int rc;
  const size_t nx = es * (size_t)N * C * H * W, ny = es * (size_t)N * C * (H / 2) * (W / 2);
  if ((rc = io.in(x, nx, &dx_)) || (rc = io.out(ny, &dy_)) || (rc = io.start())) return rc;
  KLAUNCH(c, kKPool, launch_maxpool2x2(dx_, dy_, N, C, H, W, 0, Cp, dtype, c->stream));
  if ((rc = io.back(y, dy_, ny))) return rc;
  return sync_and_check(c);
}

int b200conv_maxpool2x2_grad(b200conv_ctx* c, const void* x, const void* y, const void* gy, void* gx,
                             int N, int C, int H, int W, int dtype, int flags) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (N < 0 || C < 0 || H < 2 || W < 2) return fail(c, B200CONV_E_INVALID, "pool needs H, W >= 2");
  const size_t es = elem_size(dtype);
  const int nhwc = (flags & B200CONV_IN_NHWC) ? 1 : 0, Cp = pad_channels(C, dtype);
  if (!(flags & B200CONV_HOST_PTRS)) {
    KLAUNCH(c, kKPool, launch_maxpool2x2_grad(x, y, gy, gx, N, C, H, W, nhwc, Cp, dtype, c->stream));
    return 0;
  }
  if (nhwc) return fail(c, B200CONV_E_INVALID, "host tensors are NCHW");
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "host-pointer calls cannot be captured in a graph");
  HostIO io(c);
  void *dx_, *dy_, *dgy_, *dgx_;
  int rc;
  const size_t nx = es * (size_t)N * C * H * W, ny = es * (size_t)N * C * (H / 2) * (W / 2);
  if ((rc = io.in(x, nx, &dx_)) || (rc = io.in(y, ny, &dy_)) || (rc = io.in(gy, ny, &dgy_)) ||
      (rc = io.out(nx, &dgx_)) || (rc = io.start()))
    return rc;
  KLAUNCH(c, kKPool, launch_maxpool2x2_grad(dx_, dy_, dgy_, dgx_, N, C, H, W, 0, Cp, dtype, c->stream));
  if ((rc = io.back(gx, dgx_, nx))) return rc;
  return sync_and_check(c);
}

int b200conv_elementwise(b200conv_ctx* c, int op, const void* a, const void* b, void* out, long long pixels, int C,
                         int b_kind, float scalar, int dtype) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (op < 0 || op >= kEwCount || b_kind < 0 || b_kind > 3 || pixels < 0 || C < 0 ||
      (dtype != B200CONV_F32 && dtype != B200CONV_F16))
    return fail(c, B200CONV_E_INVALID, "bad element-wise operation");
  if ((b_kind == 0 || b_kind == 2) && !b) return fail(c, B200CONV_E_INVALID, "second operand missing");
  if (pixels == 0 || C == 0) return 0;
  const int Cp = pad_channels(C, dtype);
  Scratch tmp(c);
  float* chan = nullptr;
  if (b_kind == 2) {                       // the per-channel operand as Cp float32 values
    int rc = tmp.get(sizeof(float) * Cp, reinterpret_cast<void**>(&chan));
    if (rc) return rc;
    CU_OK(c, cudaMemsetAsync(chan, 0, sizeof(float) * Cp, c->stream));
    KLAUNCH(c, kKPack, launch_convert_bias(b, chan, C, dtype, c->stream));
  }
  KLAUNCH(c, kKTranspose, launch_elementwise(a, b_kind == 0 ? b : nullptr, chan, out, pixels * Cp, C, Cp, op, b_kind,
                                             scalar, dtype, c->stream));
  return 0;
}

int b200conv_channel_sum(b200conv_ctx* c, const void* x, void* out, long long pixels, int C, int dtype) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (pixels < 0 || C <= 0 || (dtype != B200CONV_F32 && dtype != B200CONV_F16))
    return fail(c, B200CONV_E_INVALID, "bad channel sum");
  const int Cp = pad_channels(C, dtype);
  Scratch tmp(c);
  float* partial = nullptr;
  int rc = tmp.get(sizeof(float) * Cp * channel_sum_blocks(pixels), reinterpret_cast<void**>(&partial));
  if (rc) return rc;
  KLAUNCH(c, kKTranspose, launch_channel_sum(x, partial, out, pixels, C, Cp, dtype, c->stream));
  return 0;
}

int b200conv_malloc(b200conv_ctx* c, size_t bytes, void** dptr) {
  if (!c || !dptr) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  return pool_alloc(c, bytes, dptr);
}
int b200conv_free(b200conv_ctx* c, void* dptr) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  // the block's next user is not the filter bank that was packed from it
  auto it = c->live.find(dptr);
  if (it != c->live.end()) {
    const char *lo = static_cast<const char*>(dptr), *hi = lo + it->second;
    for (auto& kv : c->packed)
      if (kv.second.src >= lo && kv.second.src < hi) kv.second.valid = false;
  }
  return pool_free(c, dptr);
}
int b200conv_host_alloc(b200conv_ctx* c, size_t bytes, void** hptr) {
  if (!c || !hptr) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  cudaError_t e = cudaHostAlloc(hptr, bytes ? bytes : 1, cudaHostAllocDefault);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(c, B200CONV_E_NOMEM, "pinned allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
  }
  return 0;
}
int b200conv_host_free(b200conv_ctx* c, void* hptr) {
  if (!c) return cudaFreeHost(hptr) == cudaSuccess ? 0 : B200CONV_E_CUDA;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  CU_OK(c, cudaFreeHost(hptr));
  return 0;
}
int b200conv_memcpy_h2d(b200conv_ctx* c, void* dst, const void* src, size_t bytes) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (bytes) CU_OK(c, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, c->stream));
  return 0;
}
int b200conv_memcpy_d2h(b200conv_ctx* c, void* dst, const void* src, size_t bytes) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (bytes) CU_OK(c, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
  return 0;
}
int b200conv_memset(b200conv_ctx* c, void* dst, int value, size_t bytes) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (bytes) CU_OK(c, cudaMemsetAsync(dst, value, bytes, c->stream));
  return 0;
}
int b200conv_memcpy_h2d_bg(b200conv_ctx* c, void* dst, const void* src, size_t bytes) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "not allowed while a graph is being captured");
  int rc = copy_streams(c);
  if (rc) return rc;
  if (bytes) CU_OK(c, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, c->up_stream));
  return 0;
}

int b200conv_join_uploads(b200conv_ctx* c) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "not allowed while a graph is being captured");
  if (!c->up_stream) return 0;
  CU_OK(c, cudaEventRecord(c->ev_up, c->up_stream));
  CU_OK(c, cudaStreamWaitEvent(c->stream, c->ev_up, 0));
  return 0;
}

int b200conv_memcpy_d2h_bg(b200conv_ctx* c, void* dst, const void* src, size_t bytes) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "not allowed while a graph is being captured");
  int rc = copy_streams(c);
  if (rc) return rc;
  CU_OK(c, cudaEventRecord(c->ev_down, c->stream));
  CU_OK(c, cudaStreamWaitEvent(c->down_stream, c->ev_down, 0));
  if (bytes) CU_OK(c, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->down_stream));
  c->down_pending = true;
  return 0;
}

int b200conv_sync(b200conv_ctx* c) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  return sync_and_check(c);
}

int b200conv_nchw_to_nhwc(b200conv_ctx* c, const void* src, void* dst, int N, int C, int H, int W,
                          int dtype) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  KLAUNCH(c, kKTranspose, launch_transpose(src, dst, N, C, H * W, H * W, pad_channels(C, dtype), dtype, c->stream));
  return 0;
}
int b200conv_nhwc_to_nchw(b200conv_ctx* c, const void* src, void* dst, int N, int C, int H, int W,
                          int dtype) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  KLAUNCH(c, kKTranspose, launch_transpose(src, dst, N, H * W, C, pad_channels(C, dtype), H * W, dtype, c->stream));
  return 0;
}

int b200conv_timer_start(b200conv_ctx* c) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  CU_OK(c, cudaEventRecord(c->ev0, c->stream));
  return 0;
}
int b200conv_timer_stop(b200conv_ctx* c, float* ms) {
  if (!c || !ms) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  int rc = join_comm(c);
  if (rc) return rc;
  CU_OK(c, cudaEventRecord(c->ev1, c->stream));
  rc = sync_and_check(c);
  if (rc) return rc;
  CU_OK(c, cudaEventElapsedTime(ms, c->ev0, c->ev1));
  return 0;
}
long long b200conv_launch_count(b200conv_ctx* c) { return c ? c->launches : 0; }

// ---- CUDA graphs: record a sequence of device-pointer calls once, replay it with one launch ---
int b200conv_graph_begin(b200conv_ctx* c) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "a graph is already being captured");
  int rc = join_comm(c);
  if (rc) return rc;
  // without memory for the counts of its own the graph's cut tiles are summed by a second kernel
  void* counts = nullptr;
  if (pool_alloc(c, kArrivals * sizeof(unsigned int), &counts) == 0) {
    const cudaError_t e = cudaMemsetAsync(counts, 0, kArrivals * sizeof(unsigned int), c->stream);
    rc = e == cudaSuccess ? wait_stream(c) : fail(c, B200CONV_E_CUDA, "clearing a graph's counts failed: %s", cudaGetErrorString(e));
    if (rc) {                                            // they are zero for a replay on any stream, or there is no graph
      pool_free(c, counts);
      return rc;
    }
  }
  CU_OK(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeRelaxed));
  c->capturing = new b200conv_graph();
  c->capturing->arrivals = static_cast<unsigned int*>(counts);
  if (counts) c->capturing->retained.push_back(counts);
  return 0;
}

int b200conv_graph_end(b200conv_ctx* c, b200conv_graph** out) {
  if (!c || !out) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (!c->capturing) return fail(c, B200CONV_E_INVALID, "no graph is being captured");
  b200conv_graph* gr = c->capturing;
  int rc = join_comm(c);      // a collective started inside the capture joins before it ends
  c->capturing = nullptr;
  cudaError_t e = cudaStreamEndCapture(c->stream, &gr->graph);
  if (e == cudaSuccess && rc == 0) e = cudaGraphInstantiate(&gr->exec, gr->graph, 0);
  if (e != cudaSuccess || rc) {
    cudaGetLastError();
    for (void* p : gr->retained) pool_free(c, p);
    if (gr->graph) cudaGraphDestroy(gr->graph);
    delete gr;
    return rc ? rc : fail(c, B200CONV_E_CUDA, "graph capture failed: %s", cudaGetErrorString(e));
  }
  *out = gr;
  return 0;
}

int b200conv_graph_launch(b200conv_ctx* c, b200conv_graph* gr) {
  if (!c || !gr || !gr->exec) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "not allowed while a graph is being captured");
  CU_OK(c, cudaGraphLaunch(gr->exec, c->stream));
  c->launches += gr->launches;
  return 0;
}

int b200conv_graph_destroy(b200conv_ctx* c, b200conv_graph* gr) {
  if (!c || !gr) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  cudaStreamSynchronize(c->stream);
  if (gr->exec) cudaGraphExecDestroy(gr->exec);
  if (gr->graph) cudaGraphDestroy(gr->graph);
  for (void* p : gr->retained) pool_free(c, p);
  delete gr;
  return 0;
}

int b200conv_prepack(b200conv_ctx* c, int count, const b200conv_desc* descs, const void* const* filters,
                     int directions) {
  if (!c || count < 0 || (count && (!descs || !filters))) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  PackBatch batch[2];                       // one per data type
  int nblocks[2] = {0, 0};
  batch[0].njobs = batch[1].njobs = 0;
  auto flush = [&](int t) -> int {
    if (batch[t].njobs) KLAUNCH(c, kKPack, launch_pack_filters_batch(batch[t], nblocks[t], t, c->stream));
    batch[t].njobs = 0;
    nblocks[t] = 0;
    return 0;
  };
  for (int i = 0; i < count; ++i) {
    int rc = validate(c, &descs[i]);
    if (rc) return rc;
    b200conv_desc d = descs[i];
    if (!filters[i] || d.N == 0 || d.C == 0 || d.K == 0) continue;
    b200conv_desc flat;
    if (flatten_1x1(d, true, &flat)) d = flat;         // the geometry the channels-last calls will see
    const int Cg = d.C / d.groups;
    for (int mode = 0; mode < 2; ++mode) {
      int ldc = 0;
      if (!(directions & (1 << mode)) || !plain_pack(d, mode, &ldc)) continue;
      const std::string key = pack_key(filters[i], d.K, Cg, d.kH, d.kW, d.groups, d.flip, mode, ldc, d.dtype);
      const size_t rows = mode == 0 ? (size_t)d.K : (size_t)d.C;
      const size_t bytes = elem_size(d.dtype) * (size_t)d.kH * d.kW * rows * ldc;
      auto it = c->packed.find(key);
      if (it == c->packed.end()) {
        void* p = nullptr;
        if ((rc = pool_alloc(c, bytes, &p))) return rc;
        it = c->packed.insert({key, b200conv_ctx::Packed{p, bytes, false, filters[i]}}).first;
      }
      const int t = d.dtype == B200CONV_F16 ? 1 : 0;
      if (batch[t].njobs == kPackBatchJobs && (rc = flush(t))) return rc;
      PackJob& j = batch[t].jobs[batch[t].njobs++];
      j = pack_job(filters[i], it->second.ptr, d.K, Cg, d.kH * d.kW, d.groups, d.flip, mode, ldc);
      j.first_block = nblocks[t];
      nblocks[t] += plan_pack(&j, d.dtype, kPackBlocks / std::max(1, count));
      it->second.valid = true;
    }
  }
  int rc = flush(0);
  if (rc) return rc;
  return flush(1);
}

int b200conv_filters_changed(b200conv_ctx* c, const void* w) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  for (auto& kv : c->packed)
    if (!w || kv.second.src == w) kv.second.valid = false;
  return 0;
}

int b200conv_set_autotune(b200conv_ctx* c, int enable) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  c->autotune = enable != 0;
  return 0;
}

int b200conv_memory_info(b200conv_ctx* c, size_t* pool_bytes, size_t* device_free_bytes) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (pool_bytes) *pool_bytes = c->pool_bytes;
  if (device_free_bytes) {
    size_t total = 0;
    CU_OK(c, cudaMemGetInfo(device_free_bytes, &total));
  }
  return 0;
}

int b200conv_set_wait_limit(b200conv_ctx* c, long long clocks) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  if (clocks < 1000) return fail(c, B200CONV_E_INVALID, "wait limit must be at least 1000 clocks");
  c->wait_clocks = clocks;
  return 0;
}

int b200conv_selftest_wait(b200conv_ctx* c) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (c->capturing) return fail(c, B200CONV_E_INVALID, "not allowed while a graph is being captured");
  CU_OK(c, launch_wait_selftest(c->d_status, c->d_arrivals, kArrivals, c->wait_clocks, c->stream));
  return sync_and_check(c);
}

int b200conv_set_pair_kernels(b200conv_ctx* c, int enable) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  c->use_pair = enable != 0;
  c->algo_cache.clear();
  return 0;
}

int b200conv_set_stacked_taps(b200conv_ctx* c, int enable) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  c->stack_taps = enable != 0;
  c->algo_cache.clear();
  c->split_cache.clear();
  return 0;
}

int b200conv_set_splits(b200conv_ctx* c, int splits) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  if (splits < 0) return fail(c, B200CONV_E_INVALID, "slice count must be >= 0 (0 = chosen by the library)");
  c->force_splits = splits;
  return 0;
}

// The tuning file: a header line naming the device the choices were timed on and the kernels, then one line per
// choice.  Choices made on another device model, SM count or set of kernels are not loaded.
// kTuningKernels goes up with each change of the kernels after which earlier timings or the numbers of choices no longer hold.
// 2: three gradWeights kernels to choose from where there were two, float32 pairs behind the one-tap choice.  (Files before it
// have no such number.)
// 3: the per-tap kernel on pairs, with and without cut tiles; the columns kernel, on one CTA and on pairs.
constexpr int kTuningKernels = 3;
static std::string tuning_header(b200conv_ctx* c) {
  cudaDeviceProp prop;
  cudaGetDeviceProperties(&prop, c->device);
  std::string name = prop.name;
  for (char& ch : name)
    if (ch == ' ') ch = '_';
  return "b200conv-tuning 1 " + name + " " + std::to_string(c->num_sms) + " kernels " + std::to_string(kTuningKernels);
}

int b200conv_tuning_save(b200conv_ctx* c, const char* path) {
  if (!c || !path) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  FILE* f = fopen(path, "w");
  if (!f) return fail(c, B200CONV_E_INVALID, "cannot write %s", path);
  fprintf(f, "%s\n", tuning_header(c).c_str());
  for (auto& kv : c->algo_cache) fprintf(f, "a %s %d\n", kv.first.text().c_str(), kv.second);
  for (auto& kv : c->split_cache) fprintf(f, "s %s %d\n", kv.first.text().c_str(), kv.second);
  fclose(f);
  return 0;
}

int b200conv_tuning_load(b200conv_ctx* c, const char* path, int* loaded) {
  if (!c || !path) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (loaded) *loaded = 0;
  FILE* f = fopen(path, "r");
  if (!f) return fail(c, B200CONV_E_INVALID, "cannot read %s", path);
  char line[512];
  int n = 0;
  bool ok = fgets(line, sizeof line, f) != nullptr;
  if (ok) {
    std::string head = line;
    while (!head.empty() && (head.back() == '\n' || head.back() == '\r')) head.pop_back();
    ok = head == tuning_header(c);
  }
  if (!ok) {
    fclose(f);
    return fail(c, B200CONV_E_INVALID, "%s was not written for this device, SM count and version of the kernels", path);
  }
  while (fgets(line, sizeof line, f)) {
    char kind = 0, text[400];
    int val = 0;
    GeoKey key{};
    if (sscanf(line, "%c %399s %d", &kind, text, &val) != 3 || !GeoKey::parse(text, &key)) continue;
    // keys of another form (older files) are passed over
    const bool known = kind == 'a' ? (key.v[0] == kGeoConv && key.n == 17) || ((key.v[0] == kGeoWgrad || key.v[0] == kGeoClasses) && key.n == 19)
                                   : key.v[0] == kGeoSplits && key.n == 20;
    if (!known) continue;
    if (kind == 'a' && val >= 0 && val < (key.v[0] == kGeoConv ? kConvVariants * (kConvSlabPair + 2) : kConvVariants)) { c->algo_cache[key] = val; ++n; }
    else if (kind == 's' && val >= 1) { c->split_cache[key] = val; ++n; }
  }
  fclose(f);
  if (loaded) *loaded = n;
  return 0;
}

int b200conv_debug_trace(b200conv_ctx* c, void* dbuf) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  c->trace = static_cast<long long*>(dbuf);
  return 0;
}

int b200conv_kernel_timing(b200conv_ctx* c, int enable) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  CU_OK(c, cudaStreamSynchronize(c->stream));
  for (auto& r : c->prof_recs) {
    c->prof_pool.push_back(r.a);
    c->prof_pool.push_back(r.b);
  }
  c->prof_recs.clear();
  c->prof = enable != 0;
  return 0;
}

int b200conv_kernel_time(b200conv_ctx* c, const char* name, float* total_ms, int* launches) {
  if (!c || !name || !total_ms || !launches) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  int kind = -1;
  for (int k = 0; k < kKCount; ++k)
    if (!strcmp(name, kKernelNames[k])) kind = k;
  if (kind < 0) return fail(c, B200CONV_E_INVALID, "unknown kernel family '%s'", name);
  CU_OK(c, cudaStreamSynchronize(c->stream));
  float sum = 0.f;
  int n = 0;
  for (auto& r : c->prof_recs) {
    if (r.kind != kind) continue;
    float ms = 0.f;
    CU_OK(c, cudaEventElapsedTime(&ms, r.a, r.b));
    sum += ms;
    ++n;
  }
  *total_ms = sum;
  *launches = n;
  return 0;
}
const char* b200conv_last_algo(b200conv_ctx* c) { return c ? c->last_algo : "none"; }
const char* b200conv_last_variant(b200conv_ctx* c) { return c ? c->last_variant : "none"; }

int b200conv_flush_l2(b200conv_ctx* c) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (!c->l2buf) {
    c->l2bytes = 256u << 20;  // twice the 126 MB L2
    cudaError_t e = cudaMalloc(&c->l2buf, c->l2bytes);
    if (e != cudaSuccess) {
      cudaGetLastError();
      c->l2buf = nullptr;
      return fail(c, B200CONV_E_NOMEM, "L2 flush buffer: %s", cudaGetErrorString(e));
    }
  }
  CU_OK(c, launch_fill_l2(c->l2buf, c->l2bytes, c->stream));
  return 0;
}

// ---- NCCL through dlopen: no link-time dependency, nothing loaded unless asked for ---------
typedef struct { char internal[128]; } nccl_uid;
typedef int (*nccl_get_uid_fn)(nccl_uid*);
typedef int (*nccl_init_rank_fn)(void**, int, nccl_uid, int);
typedef int (*nccl_allreduce_fn)(const void*, void*, size_t, int, int, void*, cudaStream_t);
typedef int (*nccl_destroy_fn)(void*);
typedef const char* (*nccl_errstr_fn)(int);

static int nccl_load(b200conv_ctx* c) {
  if (c->nccl_lib) return 0;
  // B200CONV_NCCL_LIB names another library with NCCL's entry points (tests use a stand-in whose
  // collectives fail or stall on the host, so that the watchdog can be exercised without a fault)
  const char* names[] = {getenv("B200CONV_NCCL_LIB"), "libnccl.so.2", "libnccl.so"};
  for (const char* n : names) {
    if (!n || !*n) continue;
    c->nccl_lib = dlopen(n, RTLD_NOW | RTLD_GLOBAL);
    if (c->nccl_lib) break;
  }
  if (!c->nccl_lib) return fail(c, B200CONV_E_NCCL, "cannot load libnccl.so.2: %s", dlerror());
  return 0;
}
static int nccl_fail(b200conv_ctx* c, const char* what, int code) {
  nccl_errstr_fn es = (nccl_errstr_fn)dlsym(c->nccl_lib, "ncclGetErrorString");
  return fail(c, B200CONV_E_NCCL, "%s failed: %s", what, es ? es(code) : "?");
}

int b200conv_nccl_unique_id(b200conv_ctx* c, void* id128) {
  if (!c || !id128) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  int rc = nccl_load(c);
  if (rc) return rc;
  nccl_get_uid_fn f = (nccl_get_uid_fn)dlsym(c->nccl_lib, "ncclGetUniqueId");
  if (!f) return fail(c, B200CONV_E_NCCL, "ncclGetUniqueId not found");
  int r = f(static_cast<nccl_uid*>(id128));
  return r ? nccl_fail(c, "ncclGetUniqueId", r) : 0;
}

int b200conv_nccl_init(b200conv_ctx* c, int nranks, int rank, const void* id128) {
  if (!c || !id128 || nranks < 1 || rank < 0 || rank >= nranks) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  int rc = nccl_load(c);
  if (rc) return rc;
  nccl_init_rank_fn f = (nccl_init_rank_fn)dlsym(c->nccl_lib, "ncclCommInitRank");
  if (!f) return fail(c, B200CONV_E_NCCL, "ncclCommInitRank not found");
  nccl_uid id;
  memcpy(&id, id128, sizeof id);
  int r = f(&c->comm, nranks, id, rank);
  if (r) return nccl_fail(c, "ncclCommInitRank", r);
  c->nranks = nranks;
  c->rank = rank;
  if (!c->d_token) CU_OK(c, cudaMalloc(&c->d_token, sizeof(float)));
  CU_OK(c, cudaMemsetAsync(c->d_token, 0, sizeof(float), c->stream));
  return 0;
}

int b200conv_allreduce_sum(b200conv_ctx* c, void* dbuf, size_t count, int dtype) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (!c->comm) return c->nranks == 1 ? 0 : fail(c, B200CONV_E_NCCL, "communicator not initialised (or aborted)");
  nccl_allreduce_fn f = (nccl_allreduce_fn)dlsym(c->nccl_lib, "ncclAllReduce");
  if (!f) return fail(c, B200CONV_E_NCCL, "ncclAllReduce not found");
  // ncclFloat16 = 6, ncclFloat32 = 7, ncclSum = 0
  int r = f(dbuf, dbuf, count, dtype == B200CONV_F16 ? 6 : 7, 0, c->comm, c->stream);
  return r ? nccl_fail(c, "ncclAllReduce", r) : 0;
}

int b200conv_allreduce_sum_async(b200conv_ctx* c, void* dbuf, size_t count, int dtype) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  if (!c->comm) return c->nranks == 1 ? 0 : fail(c, B200CONV_E_NCCL, "communicator not initialised (or aborted)");
  nccl_allreduce_fn f = (nccl_allreduce_fn)dlsym(c->nccl_lib, "ncclAllReduce");
  if (!f) return fail(c, B200CONV_E_NCCL, "ncclAllReduce not found");
  if (!c->comm_stream) {
    CU_OK(c, cudaStreamCreateWithFlags(&c->comm_stream, cudaStreamNonBlocking));
    CU_OK(c, cudaEventCreateWithFlags(&c->ev_comm_ready, cudaEventDisableTiming));
    CU_OK(c, cudaEventCreateWithFlags(&c->ev_comm_done, cudaEventDisableTiming));
  }
  // Collectives queue up on the communication stream in the order they are issued; the main
  // stream only joins the last of them (b200conv_comm_wait and friends).
  CU_OK(c, cudaEventRecord(c->ev_comm_ready, c->stream));
  CU_OK(c, cudaStreamWaitEvent(c->comm_stream, c->ev_comm_ready, 0));
  int r = f(dbuf, dbuf, count, dtype == B200CONV_F16 ? 6 : 7, 0, c->comm, c->comm_stream);
  if (r) return nccl_fail(c, "ncclAllReduce", r);
  CU_OK(c, cudaEventRecord(c->ev_comm_done, c->comm_stream));
  c->comm_pending = true;
  return 0;
}

int b200conv_set_sm_count(b200conv_ctx* c, int sms) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  if (sms < 1 || sms > c->device_sms)
    return fail(c, B200CONV_E_INVALID, "SM count must be between 1 and %d", c->device_sms);
  c->num_sms = sms;
  c->algo_cache.clear();            // kernel choices were timed for another SM count
  c->split_cache.clear();
  return 0;
}

int b200conv_set_comm_timeout(b200conv_ctx* c, int milliseconds) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  if (milliseconds < 1) return fail(c, B200CONV_E_INVALID, "timeout must be at least 1 ms");
  c->comm_timeout_ms = milliseconds;
  return 0;
}

int b200conv_comm_wait(b200conv_ctx* c) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  return join_comm(c);
}

int b200conv_barrier(b200conv_ctx* c) {
  if (!c) return B200CONV_E_INVALID;
  if (c->comm) {
    int rc = b200conv_allreduce_sum(c, c->d_token, 1, B200CONV_F32);
    if (rc) return rc;
  }
  return b200conv_sync(c);
}

int b200conv_nccl_destroy(b200conv_ctx* c) {
  if (!c || !c->comm) return 0;
  nccl_destroy_fn f = (nccl_destroy_fn)dlsym(c->nccl_lib, "ncclCommDestroy");
  if (f) f(c->comm);
  c->comm = nullptr;
  c->nranks = 1;
  return 0;
}

}  // extern "C"

// ======================================================================================
// gradWeights for callers that must not allocate
// ======================================================================================
// The split-K slabs of the filter gradient normally come from the context's pooled device
// memory, which may call cudaMalloc.  This variant keeps them in a fixed array that is part
// of the library image instead, so the call itself allocates nothing.
namespace {

constexpr size_t kStaticScratchBytes = 32u << 20;   // 32 MiB, resident on every GPU that loads the library
static __device__ __align__(256) unsigned char g_wgrad_scratch[kStaticScratchBytes];

constexpr int kMaxStaticDevices = 64;
std::mutex g_static_mu;
void* g_static_scratch_addr[kMaxStaticDevices];  // device address of g_wgrad_scratch, per device

// In host code `g_wgrad_scratch` is only a handle for the runtime, not a device address; the
// address on the current device has to be asked for.  Done once per device.
int static_scratch_address(b200conv_ctx* c, float** out) {
  std::lock_guard<std::mutex> g(g_static_mu);
  if (c->device < 0 || c->device >= kMaxStaticDevices)
    return fail(c, B200CONV_E_UNSUPPORTED, "device index %d beyond the static scratch table", c->device);
  if (!g_static_scratch_addr[c->device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_wgrad_scratch);
    if (e != cudaSuccess || !p) {
      cudaGetLastError();
      return fail(c, B200CONV_E_CUDA, "cudaGetSymbolAddress(static scratch): %s", cudaGetErrorString(e));
    }
    g_static_scratch_addr[c->device] = p;
  }
  *out = static_cast<float*>(g_static_scratch_addr[c->device]);
  return 0;
}

}  // namespace

extern "C" int b200conv_wgrad_static(b200conv_ctx* c, const b200conv_desc* dp, const void* x,
                                     const void* dy, void* dw, int flags) {
  if (!c) return B200CONV_E_INVALID;
  std::lock_guard<std::mutex> g(c->mu);
  DeviceGuard dg(c->device);
  int rc = validate(c, dp);
  if (rc) return rc;
  const b200conv_desc& d = *dp;
  if (flags & (B200CONV_HOST_PTRS | B200CONV_FORCE_DIRECT))
    return fail(c, B200CONV_E_INVALID, "wgrad_static takes channels-last device tensors only");
  const int Cg = d.C / d.groups, Kg = d.K / d.groups;
  const size_t es = elem_size(d.dtype);
  const size_t dw_elems = (size_t)d.K * Cg * d.kH * d.kW;
  if (dw_elems == 0) return 0;
  if (d.N == 0) {
    CU_OK(c, cudaMemsetAsync(dw, 0, es * dw_elems, c->stream));
    return 0;
  }
  if (!umma_ok(d))
    return fail(c, B200CONV_E_UNSUPPORTED, "wgrad_static covers the tensor-core geometries only");
  const size_t slab_bytes = sizeof(float) * (size_t)d.kH * d.kW * d.K * Cg;
  if (slab_bytes > kStaticScratchBytes)
    return fail(c, B200CONV_E_INVALID,
                "filter gradient needs %zu bytes of scratch per split-K slice; the static scratch "
                "holds %zu bytes (use b200conv_wgrad)", slab_bytes, kStaticScratchBytes);
  float* scratch = nullptr;
  if ((rc = static_scratch_address(c, &scratch))) return rc;

  const int Cp = pad_channels(d.C, d.dtype), Kp = pad_channels(d.K, d.dtype);
  UmmaWgradParams p;
  memset(&p, 0, sizeof p);
  const int atom = d.dtype == B200CONV_F16 ? 64 : 32;
  const int kk = d.dtype == B200CONV_F16 ? 16 : 8;
  const bool swz32 = d.dtype == B200CONV_F32;
  const int BN = Cg <= 64 ? 64 : Cg <= 128 ? 128 : 256;
  choose_tile(c, d.Wo, d.Ho, d.N, wgrad_pix(d.dtype, BN), kk, &p.bw, &p.bh, &p.bn);
  if ((rc = make_view(c, &p.dy_map, dy, d.dtype, Kg, d.groups, Kp, d.Wo, d.Ho, d.N, 0, 0, 1, 1, atom,
                      p.bw, p.bh, p.bn, swz32)))
    return rc;
  int nviews = 0;
  int view_slot[kMaxViews];
  int par_h[kMaxViews], par_w[kMaxViews], npar = 0;
  bool dropped = false;
  for (int i = 0; i < d.kH; ++i)
    for (int j = 0; j < d.kW; ++j) {
      const int ah = i * d.dilH - d.padH_l, aw = j * d.dilW - d.padW_l;
      const int rh = pymod(ah, d.sH), rw = pymod(aw, d.sW);
      int v = -1;
      for (int q = 0; q < npar; ++q)
        if (par_h[q] == rh && par_w[q] == rw) v = q;
      if (v < 0) {
        v = npar++;
        par_h[v] = rh; par_w[v] = rw;
        view_slot[v] = -1;
        if (rh < d.H && rw < d.W) {
          view_slot[v] = nviews++;
          if ((rc = make_view(c, &p.x_views[view_slot[v]], x, d.dtype, Cg, d.groups, Cp, d.W, d.H, d.N,
                              rh, rw, d.sH, d.sW, atom, p.bw, p.bh, p.bn, swz32)))
            return rc;
        }
      }
      if (view_slot[v] < 0) { dropped = true; continue; }
      ConvTap t;
      t.dh = (int16_t)floordiv(ah, d.sH); t.dw = (int16_t)floordiv(aw, d.sW);
      t.view = (int16_t)view_slot[v];
      const int wi = d.flip ? d.kH - 1 - i : i, wj = d.flip ? d.kW - 1 - j : j;
      t.wmat = (int16_t)(wi * d.kW + wj);
      p.taps[p.ntaps++] = t;
    }
  for (int v = nviews; v < kMaxViews; ++v) p.x_views[v] = nviews ? p.x_views[0] : p.dy_map;
  p.nviews = nviews;
  p.groups = d.groups; p.Kg = Kg; p.Cg = Cg;
  p.Wo = d.Wo; p.Ho = d.Ho; p.Nimg = d.N;
  p.tiles_w = (int)cdiv(d.Wo, p.bw); p.tiles_h = (int)cdiv(d.Ho, p.bh); p.tiles_n = (int)cdiv(d.N, p.bn);
  p.ktiles = (int)cdiv(Kg, 128); p.ctiles = (int)cdiv(Cg, BN);
  p.taps_total = d.kH * d.kW;
  const long long pix_tiles = 1LL * p.tiles_w * p.tiles_h * p.tiles_n;
  const long long base_items = 1LL * p.ktiles * p.ctiles * d.groups * std::max(1, p.ntaps);
  p.splits = (int)balanced_splits(c, pix_tiles, base_items, c->num_sms,
                                  std::min<long long>(pix_tiles / 4, (long long)(kStaticScratchBytes / slab_bytes)), 2);
  p.atomic = (flags & B200CONV_ATOMIC_SPLITK) ? 1 : 0;
  const int slabs = p.atomic ? 1 : p.splits;
  // the array keeps whatever the previous call left: clear what this call adds into or skips
  if (p.atomic || dropped || p.ntaps == 0)
    CU_OK(c, cudaMemsetAsync(scratch, 0, slab_bytes * slabs, c->stream));
  p.partial = scratch;
  p.partial_elems = (long long)(slab_bytes / sizeof(float)) * slabs;
  p.status = c->d_status;
  p.wait_clocks = c->wait_clocks;
  c->last_variant = "wgrad tap";
  if (p.ntaps > 0) KLAUNCH(c, kKWgradUmma, launch_wgrad_umma(p, d.dtype, BN, c->num_sms, c->stream));
  KLAUNCH(c, kKWgradReduce, launch_wgrad_reduce(scratch, dw, slabs, p.taps_total, d.K, Cg, Kg, 0, 0,
                                                (flags & B200CONV_DW_F32) ? B200CONV_F32 : d.dtype, wgrad_sum(c, d, x, true, dy, true), c->stream));
  c->last_algo = "umma";
  return 0;
}
