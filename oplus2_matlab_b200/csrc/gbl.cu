// gbl.cu -- host side of global reductions: device scratch, result slots,
// and delivery into the caller's variables.
//
// Semantics kept from the reference CUDA back-end (airfoil/update_kernel.cu:
// 116-169, jac1/update_kernel.cu:94-141): OP_INC adds the device sum to the
// host value, OP_MAX / OP_MIN combine with it; the variable holds the result
// when the loop call returns.  In deferred mode the device results wait in
// slots until op2b_sync / op_fetch_data, so no call blocks.

#include <string.h>

#include <algorithm>
#include <atomic>
#include <thread>

#include "launch.cuh"
#include "loops.h"
#include "reduce.cuh"
#include "seq_sum.cuh"

namespace op2b {

namespace {
constexpr int kSlots = 4096;
struct RedState {
  char *dev = nullptr;  // [2 x kMaxRedBlocks x 8] partials | tickets (256 B)
  // result slots in mapped pinned host memory: the last block of a reduction
  // stores the result where the host reads it, so delivery needs no copy
  char *host = nullptr;
  unsigned *flags = nullptr;  // one per slot, in the same memory
  unsigned flag_seq = 0;      // the last number given to a flag
  int next_slot = 0;
  int graph_slots = 0;  // slots baked into captured graphs stay reserved
  void *seq = nullptr;
  size_t seq_bytes = 0;
};
RedState &rs() {
  static RedState s;
  return s;
}
size_t off_ticket() { return 2 * (size_t)kMaxRedBlocks * 8; }
size_t off_slots() { return off_ticket() + 256; }

void ensure_red() {
  RedState &S = rs();
  if (S.dev) return;
  size_t bytes = off_slots();
  S.dev = (char *)dev_alloc(bytes);
  OP2B_CUDA(cudaMemset(S.dev, 0, bytes));
  OP2B_CUDA(cudaHostAlloc((void **)&S.host, (size_t)kSlots * 12, cudaHostAllocMapped));
  memset(S.host, 0, (size_t)kSlots * 12);
  S.flags = (unsigned *)(S.host + (size_t)kSlots * 8);
}

template <class T>
void combine(char *host, const T v, op_access acc, bool assign) {
  T *h = (T *)host;
  switch (acc) {
    case OP_INC: *h = assign ? v : (T)(*h + v); break;
    case OP_MAX: *h = (*h > v) ? *h : v; break;
    case OP_MIN: *h = (*h < v) ? *h : v; break;
    default: break;
  }
}

// The request's result is in host memory once its flag says so, which is
// before an event behind the kernel would be seen (eager iteration at 7k cells
// 41.5 -> 35.1 us, at 720k 62.9 -> 54.4, relieved kernels included).  A look at
// the stream from time to time ends the wait when the work behind it failed.
bool wait_flag(const GblRequest &r) {
  volatile unsigned *f = rs().flags + r.flag_slot;
  static const char *yield = getenv("OP2B_SYNC_YIELD");
  for (unsigned n = 1; *f != r.seq; n++) {
    if (yield && yield[0] == '1') std::this_thread::yield();
    if (n & 0x3fff) continue;
    const cudaError_t e = cudaStreamQuery(rt().stream);
    if (e == cudaErrorNotReady) continue;
    if (e == cudaSuccess && *f == r.seq) break;
    cuda_fail(e == cudaSuccess ? cudaErrorUnknown : e, "global reduction", __FILE__, __LINE__);
    return false;
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  return true;
}

void deliver(const std::vector<GblRequest> &reqs) {
  RedState &S = rs();
  if (reqs.empty()) return;
  red_tail_flush();
  bool sync = false;
  for (auto &r : reqs) sync = sync || !r.seq;
  if (sync) OP2B_CUDA(cudaStreamSynchronize(rt().stream));  // the slots are host memory
  for (auto &r : reqs) {
    if (r.seq && !wait_flag(r)) return;
    const char *p = S.host + (size_t)r.slot * 8;
    if (r.type == GBL_F64) combine<double>(r.host, *(const double *)p, r.acc, r.assign);
    else combine<float>(r.host, *(const float *)p, r.acc, r.assign);
  }
}

std::vector<GblRequest> &pending() {
  static std::vector<GblRequest> v;
  return v;
}

// with no result outstanding, every slot a captured graph does not hold is free
void free_slots() {
  if (pending().empty()) rs().next_slot = rs().graph_slots;
}

struct Tail {  // red_tail_leave
  bool on = false, captured = false;
  int type = 0, n = 0, slot = 0, slot_max = -1, ticket_arg = 0, nparams = 0;
  unsigned seq = 0;
  cudaGraphNode_t node = nullptr;
};
Tail g_tail;
std::vector<Tail> g_tail_patches;

template <class T>
RedTail<T> tail_of(const Tail &t) {
  RedState &S = rs();
  RedTail<T> r;
  r.sums = (const T *)S.dev;
  r.maxs = t.slot_max >= 0 ? (const T *)(S.dev + (size_t)kMaxRedBlocks * 8) : nullptr;
  r.sum = (T *)(S.host + (size_t)t.slot * 8);
  r.max = t.slot_max >= 0 ? (T *)(S.host + (size_t)t.slot_max * 8) : nullptr;
  r.flag = t.seq ? S.flags + t.slot : nullptr;
  r.seq = t.seq;
  r.n = t.n;
  return r;
}

template <class T>
__global__ void __launch_bounds__(256) k_red_tail(RedTail<T> t) {
  pdl_wait();
  pdl_trigger();
  red_tail_fold(t);
}

}  // namespace

unsigned red_flag(int slot, unsigned **flag) {
  *flag = nullptr;
  if (rt().gbl_deferred) return 0;
  RedState &S = rs();
  if (++S.flag_seq == 0) ++S.flag_seq;
  *flag = S.flags + slot;
  return S.flag_seq;
}

bool red_tail_wanted(bool tail_next) {
  return tuning("red_tail", 1) && (rt().gbl_deferred ? rt().own_capture : tail_next);
}

unsigned red_tail_leave(int type, int n, int slot, int slot_max, int ticket_arg, int nparams) {
  Tail t;
  t.on = true;
  t.type = type;
  t.n = n;
  t.slot = slot;
  t.slot_max = slot_max;
  t.ticket_arg = ticket_arg;
  t.nparams = nparams;
  unsigned *flag;
  t.seq = red_flag(slot, &flag);
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  const cudaGraphNode_t *deps = nullptr;
  const cudaGraphEdgeData *edges = nullptr;
  size_t nd = 0;
  if (rt().own_capture &&
      cudaStreamGetCaptureInfo_v3(rt().stream, &st, nullptr, nullptr, &deps, &edges, &nd) ==
          cudaSuccess &&
      st == cudaStreamCaptureStatusActive) {
    t.captured = true;
    cudaGraphNodeType kind;
    if (nd == 1 && cudaGraphNodeGetType(deps[0], &kind) == cudaSuccess &&
        kind == cudaGraphNodeTypeKernel)
      t.node = deps[0];
  }
  cudaGetLastError();
  g_tail = t;
  return t.seq;
}

template <class T>
RedTail<T> red_tail_take() {
  if (g_tail.on && g_tail.type == (sizeof(T) == 8 ? GBL_F64 : GBL_F32)) {
    g_tail.on = false;
    return tail_of<T>(g_tail);
  }
  RedTail<T> none;
  memset(&none, 0, sizeof none);
  return none;
}
template RedTail<float> red_tail_take<float>();
template RedTail<double> red_tail_take<double>();

void red_tail_flush() {
  if (!g_tail.on) return;
  g_tail.on = false;
  if (g_tail.captured && g_tail.node) {  // that kernel folds its partials itself
    g_tail_patches.push_back(g_tail);
    return;
  }
  if (g_tail.type == GBL_F64)
    launch_pdl(k_red_tail<double>, 1, 256, 0, rt().stream, tail_of<double>(g_tail));
  else
    launch_pdl(k_red_tail<float>, 1, 256, 0, rt().stream, tail_of<float>(g_tail));
}

void red_tail_patch_captured() {
  for (Tail &t : g_tail_patches) {
    cudaKernelNodeParams kp;
    OP2B_CUDA(cudaGraphKernelNodeGetParams(t.node, &kp));
    if (error_pending()) break;
    std::vector<void *> args(kp.kernelParams, kp.kernelParams + t.nparams);
    unsigned *ticket = red_ticket();
    args[t.ticket_arg] = &ticket;
    kp.kernelParams = args.data();
    kp.extra = nullptr;
    OP2B_CUDA(cudaGraphKernelNodeSetParams(t.node, &kp));
  }
  g_tail_patches.clear();
}

void red_tail_drop_captured() {
  g_tail_patches.clear();
  if (g_tail.captured) g_tail.on = false;
}

// every reduction asks for its partials before it is launched: those of the
// one before it are folded by then
void *red_partials(int i) {
  ensure_red();
  red_tail_flush();
  return rs().dev + (size_t)i * kMaxRedBlocks * 8;
}

unsigned *red_ticket() {
  ensure_red();
  return (unsigned *)(rs().dev + off_ticket());
}

void *red_slot_ptr(int slot) {
  ensure_red();
  return rs().host + (size_t)slot * 8;  // a mapped host address (unified addressing)
}

int red_new_slot() {
  ensure_red();
  RedState &S = rs();
  if (S.next_slot >= kSlots) {
    deliver_deferred();  // frees every slot not held by a captured graph
    S.next_slot = S.graph_slots ? S.graph_slots : 0;
    if (S.next_slot >= kSlots) {
      fail(-1, "op2b error: global reduction slots exhausted by captured graphs\n");
      S.next_slot = 0;
    }
  }
  return S.next_slot++;
}

// the values, then seq_sum's tables: a sum, two pairs and a binade per tile of
// values (at least 4 bytes each), two pairs per run
static size_t seq_table_offset(size_t bytes) { return (bytes + 255) & ~(size_t)255; }

void *red_seq_buffer(size_t bytes) {
  RedState &S = rs();
  if (bytes > S.seq_bytes) {
    OP2B_CUDA(cudaStreamSynchronize(rt().stream));
    dev_free(S.seq);
    S.seq = dev_alloc(seq_table_offset(bytes) +
                      (bytes / 4 / kSeqTile + 2) *
                          (sizeof(double) + (1 + kSeqRuns) * sizeof(SeqTwo<double>) + 8));
    S.seq_bytes = S.seq ? bytes : 0;
  }
  return S.seq;
}

template <class T>
unsigned seq_sum(const T *v, long long n, T init, T *out, const int *order, int w, int slot) {
  unsigned *flag;
  const unsigned seq = red_flag(slot, &flag);
  const int ntile = (int)std::max(1LL, (n + kSeqTile - 1) / kSeqTile);
  char *tab = (char *)v + seq_table_offset(sizeof(T) * (size_t)n);
  double *tsum = (double *)tab;
  SeqTwo<T> *tiles = (SeqTwo<T> *)(tsum + ntile), *runs = tiles + ntile;
  int *binade = (int *)(runs + (size_t)ntile * kSeqRuns);
  const SeqVals<T> a{v, n, order, w};
  cudaStream_t s = rt().stream;
  launch_pdl(k_seq_tile_sums<T>, ntile, kSeqThreads, 0, s, a, tsum);
  launch_pdl(k_seq_fold<T>, ntile, kSeqThreads, 0, s, a, init, ntile, (const double *)tsum, tiles,
             runs, binade, red_ticket() + 1, out, flag, seq);
  return seq;
}
template unsigned seq_sum<float>(const float *, long long, float, float *, const int *, int, int);
template unsigned seq_sum<double>(const double *, long long, double, double *, const int *, int,
                                  int);

int red_grid(long long n, int threads) {
  long long want = (n + threads - 1) / threads;
  long long cap = (long long)rt().num_sms * 4;
  if (cap > kMaxRedBlocks) cap = kMaxRedBlocks;
  if (want < 1) want = 1;
  return (int)(want < cap ? want : cap);
}

void red_finish(const std::vector<GblRequest> &reqs) {
  if (reqs.empty()) return;
  if (rt().gbl_deferred) {
    for (auto &r : reqs) pending().push_back(r);
    return;
  }
  deliver(reqs);
  free_slots();
}

void red_finish_after(cudaEvent_t done, const std::vector<GblRequest> &reqs) {
  if (reqs.empty()) return;
  RedState &S = rs();
  bool event = false;
  for (auto &r : reqs) event = event || !r.seq;
  if (event) OP2B_CUDA(cudaEventSynchronize(done));  // the slots are host memory
  for (auto &r : reqs) {
    if (r.seq && !wait_flag(r)) return;
    const char *p = S.host + (size_t)r.slot * 8;
    if (r.type == GBL_F64) combine<double>(r.host, *(const double *)p, r.acc, r.assign);
    else combine<float>(r.host, *(const float *)p, r.acc, r.assign);
  }
  free_slots();
}

size_t red_pending_count() { return pending().size(); }

std::vector<GblRequest> red_take_pending_since(size_t mark) {
  std::vector<GblRequest> &p = pending();
  std::vector<GblRequest> out;
  if (mark < p.size()) {
    out.assign(p.begin() + mark, p.end());
    p.resize(mark);
  }
  return out;
}

void red_replace_pending(const std::vector<GblRequest> &reqs) {
  std::vector<GblRequest> &p = pending();
  std::vector<GblRequest> keep;
  for (auto &r : p) {
    bool same = false;
    for (auto &q : reqs) same = same || (q.slot == r.slot);
    if (!same) keep.push_back(r);
  }
  keep.insert(keep.end(), reqs.begin(), reqs.end());
  p.swap(keep);
}

void deliver_deferred() {
  if (pending().empty()) return;
  std::vector<GblRequest> v;
  v.swap(pending());
  deliver(v);
  free_slots();
}

void red_reserve_for_graph() { rs().graph_slots = std::max(rs().graph_slots, rs().next_slot); }

}  // namespace op2b

extern "C" int op2b_set_gbl_deferred(int on) {
  op2b::flush_pending();
  op2b::Runtime &R = op2b::rt();
  int old = R.gbl_deferred;
  if (old && !on) op2b::deliver_deferred();
  R.gbl_deferred = on != 0;
  return old;
}
