// reduce.cuh -- device side of global reductions (op_arg_gbl with OP_INC /
// OP_MIN / OP_MAX).
//
// The reference reduces with a shared-memory tree whose last 32 steps rely on
// warp-synchronous execution (common/op_lib.cu:268-332), a pattern that is
// undefined under independent thread scheduling (sm_70 and later), then sums
// 200 block partials on the host.  Here:
//   TREE: each thread folds its elements in ascending order, lanes combine with
//         __shfl_down_sync in a fixed pattern, warps through shared memory,
//         blocks write a partial, and the last block to finish (atomic ticket)
//         folds the partials in index order.  The grid is a function of the
//         set size only, so results are bit-reproducible run to run.
//   SEQ:  the loop writes each contribution to a scratch array in element
//         order and seq_sum (seq_sum.cuh) adds them to the caller's initial
//         value in that order -- op_seq.h's result, bit for bit.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace op2b {

struct OpSum {
  template <class T>
  __device__ __forceinline__ T operator()(T a, T b) const { return a + b; }
};
// MAX(a, b) of common/op_lib_core.h:167 with a = running value
struct OpMax {
  template <class T>
  __device__ __forceinline__ T operator()(T a, T b) const { return (a > b) ? a : b; }
};
struct OpMin {
  template <class T>
  __device__ __forceinline__ T operator()(T a, T b) const { return (a < b) ? a : b; }
};

template <class T, class Op>
__device__ __forceinline__ T warp_fold(T v, Op op) {
  for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// Block fold; result valid in thread 0.  Uses `ws` (>= 32 entries).
template <class T, class Op>
__device__ __forceinline__ T block_fold(T v, T identity, Op op, T *ws) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_fold(v, op);
  __syncthreads();
  if (lane == 0) ws[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = lane < nw ? ws[lane] : identity;
    v = warp_fold(v, op);
  }
  return v;
}

// Per-call device storage of one reduction: block partials and the result.
template <class T>
struct RedSlot {
  T *partials;         // [gridDim.x]
  T *result;           // final value (no host seed applied)
  // the first reduction's: set to seq once every result is in host memory,
  // for a host that waits for it (null: nobody does)
  unsigned *flag = nullptr, seq = 0;
};

// Finish up to two reductions of one kernel: write block partials, and let
// the last block fold them in index order.  `ticket` must be 0 on entry and
// is reset to 0 by the last block.
template <class T, class Op0, class Op1, int N>
__device__ __forceinline__ void grid_finish(const T (&v)[N], const T (&identity)[N], Op0 op0,
                                            Op1 op1, RedSlot<T> (&slot)[N], unsigned *ticket) {
  __shared__ T ws[32];
  __shared__ bool last;
#pragma unroll
  for (int i = 0; i < N; i++) {
    T b = i == 0 ? block_fold(v[i], identity[i], op0, ws) : block_fold(v[i], identity[i], op1, ws);
    if (threadIdx.x == 0) slot[i].partials[blockIdx.x] = b;
  }
  // thread 0 wrote the partials: it alone fences them before taking a ticket
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int i = 0; i < N; i++) {
    T x = identity[i];
    for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) {
      T p = __ldcg(slot[i].partials + k);
      x = i == 0 ? op0(x, p) : op1(x, p);
    }
    x = i == 0 ? block_fold(x, identity[i], op0, ws) : block_fold(x, identity[i], op1, ws);
    if (threadIdx.x == 0) *slot[i].result = x;
  }
  if (threadIdx.x == 0) {
    *ticket = 0u;
    if (slot[0].flag) {
      __threadfence_system();
      *reinterpret_cast<volatile unsigned *>(slot[0].flag) = slot[0].seq;
    }
  }
}

// a kernel whose partials the next kernel folds (RedTail) writes them only
template <class T, class Op0, class Op1, int N>
__device__ __forceinline__ void grid_leave(const T (&v)[N], const T (&identity)[N], Op0 op0,
                                           Op1 op1, RedSlot<T> (&slot)[N]) {
  __shared__ T ws[32];
#pragma unroll
  for (int i = 0; i < N; i++) {
    T b = i == 0 ? block_fold(v[i], identity[i], op0, ws) : block_fold(v[i], identity[i], op1, ws);
    if (threadIdx.x == 0) slot[i].partials[blockIdx.x] = b;
  }
}

// The end of a reduction left to another kernel: the block partials of one
// or two reductions (a sum, and a maximum) that a kernel has written and not
// folded.  Folding them in that kernel's last block keeps the next kernel
// waiting for a chain of fence, ticket, loads and a store to host memory
// (2 us at the end of every res_calc chain: 47.2 -> 45.2 us a captured
// iteration of 720k FP32 cells with one of its two chains relieved, 14.4 -> 12.4
// at 7k); a CTA of the next kernel does it while the others work.  flag, when
// not null, is set to seq once the results are in host memory, for a host that
// waits for them.
template <class T>
struct RedTail {
  const T *sums, *maxs;  // [n]; maxs may be null
  T *sum, *max;
  unsigned *flag, seq;
  int n;  // 0: nothing to do
};

// by all threads of a block
template <class T>
__device__ __forceinline__ void red_tail_fold(const RedTail<T> &t) {
  __shared__ T ws[32];
  const T low = -static_cast<T>(INFINITY);
  T x = T(0), y = low;
  for (int k0 = threadIdx.x; k0 < t.n; k0 += 4 * blockDim.x) {
    T a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {  // the loads of a round together
      const int k = k0 + i * blockDim.x;
      a[i] = k < t.n ? __ldcg(t.sums + k) : T(0);
      b[i] = t.maxs && k < t.n ? __ldcg(t.maxs + k) : low;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      x += a[i];
      y = OpMax()(y, b[i]);
    }
  }
  x = block_fold(x, T(0), OpSum(), ws);
  if (t.maxs) y = block_fold(y, low, OpMax(), ws);
  if (threadIdx.x == 0) {
    *t.sum = x;
    if (t.maxs) *t.max = y;
    if (t.flag) {
      __threadfence_system();
      *reinterpret_cast<volatile unsigned *>(t.flag) = t.seq;
    }
  }
}

}  // namespace op2b
