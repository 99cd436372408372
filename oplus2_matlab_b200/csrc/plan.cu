// plan.cu -- execution plans built on the device.
//
// 1. The reference's op_plan (common/op_lib_core.c:627-1089), reproduced
//    array for array: contiguous blocks, per-block sorted distinct indirect
//    targets (ind_maps) with short block-local indices (loc_maps), greedy
//    thread colouring in element order and greedy block colouring in block
//    order, both in passes of 32 colours, and blkmap grouped by colour.  The
//    O(N log N) part (gather, sort, dedupe, inverse) runs one CTA per block
//    and indirect dataset; the thread colouring runs one CTA per block; the
//    block colouring is the reference's sequential greedy over blocks, run by
//    one CTA on the blocks' conflicts, which are found in parallel.  All of it
//    is integer work with one exact answer, so the result equals op_plan_core.
// 2. A validator for any plan: the reference's op_plan_check
//    (op_lib_core.c:469-620) plus the colouring checks it leaves out.
// 3. The owner-computes ("gather") plan used by the GATHER strategy: per
//    incremented element, its contributions in ascending (element, slot)
//    order, i.e. the order in which op_seq.h applies them.

#include <limits.h>
#include <stdlib.h>

#include <algorithm>
#include <cstring>
#include <thread>

#include "host_threads.h"
#include "plan.h"

namespace op2b {

constexpr int kMaxArgs = 24;

struct ArgMaps {
  const int *map[kMaxArgs];
  int dim[kMaxArgs];
  int idx[kMaxArgs];
};

struct PlanParams {
  ArgMaps am;
  int nargs, ninds, set_size, bsize, nblocks, cls;
  int ind_first[kMaxArgs];  // first position in ind_args of ind m
  int ind_k[kMaxArgs];      // number of args of ind m
  int ind_args[kMaxArgs];   // args grouped by ind, in argument order
  int ind_P[kMaxArgs];      // sort size (power of two >= k*bsize)
  int ind_size[kMaxArgs];   // dat bytes per element for ind m
  int ind_dim[kMaxArgs];    // dat dim for ind m
  int ind_same[kMaxArgs];   // the first ind whose args go through the same maps as m's
  int arg_same[kMaxArgs];   // the first arg of the same map and index
  int arg_ind[kMaxArgs];    // ind of arg a, or -1
  long long tmp_off[kMaxArgs];
  // OP_INC slots (thread / block colouring): arg and its ind
  int ninc;
  int inc_arg[kMaxArgs];
  int inc_ind[kMaxArgs];
  int inc_mbase[kMaxArgs];  // per INC slot: offset of its ind's masks in smem
  int mask_words;           // total mask words per block in smem
};

__device__ __forceinline__ int map_at(const ArgMaps &am, int a, int e) {
  return am.map[a][am.idx[a] + (size_t)e * am.dim[a]];
}

// block-wide exclusive scan of one int per thread (blockDim.x <= 1024)
__device__ int block_excl_scan(int v, int *total) {
  __shared__ int warp_sums[32];
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  int nw = (blockDim.x + 31) >> 5;
  if (warp == 0) {
    int w = lane < nw ? warp_sums[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    warp_sums[lane] = w;  // inclusive
  }
  __syncthreads();
  int excl = x - v + (warp > 0 ? warp_sums[warp - 1] : 0);
  if (total) *total = warp_sums[nw - 1];
  __syncthreads();
  return excl;
}

// P a power of two >= 64.  Exchanges over at most 32 places stay inside the 64
// places of one warp's 32 pairs, so only the wider ones need the CTA's barrier
// (10 of 55 steps for 1024 values)
__device__ void bitonic_sort(int *s, int P) {
  for (int k = 2; k <= P; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = threadIdx.x; t < P / 2; t += blockDim.x) {
        const int i = 2 * t - (t & (j - 1));
        const int a = s[i], b = s[i + j];
        if ((a > b) == ((i & k) == 0)) {
          s[i] = b;
          s[i + j] = a;
        }
      }
      // the next step's reach: j / 2, or k after the last step of this k
      const int reach = j > 1 ? j >> 1 : k;
      if (j > 32 || reach > 32) __syncthreads();
      else __syncwarp();
    }
  __syncthreads();
}

// one CTA per (block b, indirect dataset m): gather the targets of all args
// of m over the block's elements, sort, deduplicate
// (common/op_lib_core.c:781-803)
__global__ void k_block_unique(PlanParams pp, int *ind_sizes, int *tmp) {
  extern __shared__ int s[];
  const int b = blockIdx.x, m = blockIdx.y;
  const int e0 = b * pp.bsize;
  const int bs = min(pp.bsize, pp.set_size - e0);
  const int k = pp.ind_k[m];
  const int K = k * bs;
  if (pp.ind_same[m] != m) return;  // computed with that one
  int P = 64;
  while (P < K) P <<= 1;
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    int v = INT_MAX;
    if (i < K) {
      int a = pp.ind_args[pp.ind_first[m] + i / bs];
      v = map_at(pp.am, a, e0 + i % bs);
    }
    s[i] = v;
  }
  __syncthreads();
  bitonic_sort(s, P);
  int *out = tmp + pp.tmp_off[m] + (long long)b * k * pp.bsize;
  int base = 0;
  for (int r = 0; r < K; r += blockDim.x) {
    int i = r + threadIdx.x;
    int f = (i < K) && (i == 0 || s[i] != s[i - 1]);
    int tot;
    int pos = block_excl_scan(f, &tot);
    if (f) out[base + pos] = s[i];
    base += tot;
  }
  for (int i = threadIdx.x; i < pp.ninds; i += blockDim.x)
    if (pp.ind_same[i] == m) ind_sizes[i + b * pp.ninds] = base;
}

// exclusive scan of ind_sizes over blocks, per indirect dataset
// (common/op_lib_core.c:822-834)
__global__ void k_scan_blocks(int nblocks, int ninds, const int *ind_sizes, int *ind_offs,
                              int *nindirect) {
  const int m = blockIdx.x;
  int run = 0;
  for (int c = 0; c < nblocks; c += blockDim.x) {
    int b = c + threadIdx.x;
    int v = b < nblocks ? ind_sizes[m + b * ninds] : 0;
    int tot;
    int x = block_excl_scan(v, &tot);
    if (b < nblocks) ind_offs[m + b * ninds] = run + x;
    run += tot;
  }
  if (threadIdx.x == 0) nindirect[m] = run;
}

struct IndOut {
  int *ind_maps[kMaxArgs];
  short *loc_maps[kMaxArgs];
};

// place the block's distinct targets in ind_maps, renumber each arg's targets
// to block-local indices (common/op_lib_core.c:807-820), and count the cache
// lines the reference's byte model charges (common/op_lib_core.c:1010-1040)
__global__ void k_block_locmaps(PlanParams pp, IndOut io, const int *ind_sizes,
                                const int *ind_offs, const int *tmp, long long *lines,
                                long long *lines3) {
  extern __shared__ int list[];
  const int b = blockIdx.x, m = blockIdx.y;
  const int e0 = b * pp.bsize;
  const int bs = min(pp.bsize, pp.set_size - e0);
  const int k = pp.ind_k[m];
  const int nu = ind_sizes[m + b * pp.ninds];
  const int off = ind_offs[m + b * pp.ninds];
  const int *src = tmp + pp.tmp_off[m] + (long long)b * k * pp.bsize;
  for (int u = threadIdx.x; u < nu; u += blockDim.x) {
    int t = src[u];
    list[u] = t;
    io.ind_maps[m][off + u] = t;
  }
  __syncthreads();
  // the local indices of this ind's args, and of the args of later inds that
  // go through the same maps (their CTAs have none to find)
  if (pp.ind_same[m] == m)
    for (int i = threadIdx.x; i < k * bs; i += blockDim.x) {
      const int j = i / bs;
      const int e = e0 + i - j * bs;
      const int v = map_at(pp.am, pp.ind_args[pp.ind_first[m] + j], e);
      int lo = 0, hi = nu;  // lower_bound
      while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (list[mid] < v) lo = mid + 1; else hi = mid;
      }
      for (int c = m; c < pp.ninds; c++)
        if (pp.ind_same[c] == m) io.loc_maps[pp.ind_args[pp.ind_first[c] + j]][e] = (short)lo;
    }
  // cache lines: element u starts a new line unless its first line is the
  // previous element's last line
  const long long sz = pp.ind_size[m], cls = pp.cls, cls3 = (long long)pp.ind_dim[m] * pp.cls;
  long long my = 0, my3 = 0;
  for (int u = threadIdx.x; u < nu; u += blockDim.x) {
    long long t = list[u];
    long long a = (t * sz) / cls, z = ((t + 1) * sz - 1) / cls;
    long long prev = u > 0 ? (((long long)list[u - 1] + 1) * sz - 1) / cls : -1;
    my += (a > prev ? 1 : 0) + (z - a);
    long long a3 = (t * sz) / cls3, z3 = ((t + 1) * sz - 1) / cls3;
    long long prev3 = u > 0 ? (((long long)list[u - 1] + 1) * sz - 1) / cls3 : -1;
    my3 += (a3 > prev3 ? 1 : 0) + (z3 - a3);
  }
  for (int o = 16; o > 0; o >>= 1) {
    my += __shfl_down_sync(0xffffffffu, my, o);
    my3 += __shfl_down_sync(0xffffffffu, my3, o);
  }
  __shared__ long long red[2][32];
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = my;
    red[1][threadIdx.x >> 5] = my3;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long s = 0, s3 = 0;
    for (int w = 0; w < (int)(blockDim.x + 31) / 32; w++) {
      s += red[0][w];
      s3 += red[1][w];
    }
    lines[m + b * pp.ninds] = s;
    lines3[m + b * pp.ninds] = s3;
  }
}

// greedy thread colouring of one block in element order, 32 colours per
// pass (common/op_lib_core.c:839-880).  The loop is sequential by definition;
// one thread runs it on block-local masks in shared memory.
__global__ void k_thread_colour(PlanParams pp, IndOut io, const int *ind_sizes, int *thrcol,
                                int *nthrcol) {
  extern __shared__ unsigned smem[];
  const int b = blockIdx.x;
  const int e0 = b * pp.bsize;
  const int bs = min(pp.bsize, pp.set_size - e0);
  unsigned *masks = smem;
  unsigned short *locs = (unsigned short *)(smem + pp.mask_words);
  int *col = (int *)(smem + pp.mask_words + (pp.ninc * pp.bsize + 1) / 2);
  for (int i = threadIdx.x; i < pp.ninc * bs; i += blockDim.x) {
    int sl = i / bs, e = i % bs;
    locs[sl * bs + e] = (unsigned short)io.loc_maps[pp.inc_arg[sl]][e0 + e];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < pp.mask_words; i += blockDim.x) masks[i] = 0u;
  for (int e = threadIdx.x; e < bs; e += blockDim.x) col[e] = -1;
  __syncthreads();
  if (threadIdx.x == 0) {
    int base = 0, ncol = 0, again = 0;
    if (pp.ninc == 2) {
      // the first pass of a loop with two increments, the usual case: the
      // next element's places are read while this one's masks are on their way
      unsigned *ma = masks + pp.inc_mbase[0], *mb = masks + pp.inc_mbase[1];
      const unsigned short *la = locs, *lb = locs + bs;
      int ia = la[0], ib = lb[0];
      for (int e = 0; e < bs; e++) {
        const int i = ia, j = ib;
        const unsigned xa = ma[i], xb = mb[j];
        if (e + 1 < bs) {
          ia = la[e + 1];
          ib = lb[e + 1];
        }
        const int c = __ffs(~(xa | xb)) - 1;
        if (c < 0) {
          again = 1;
          continue;
        }
        col[e] = c;
        ncol = max(ncol, c + 1);
        ma[i] = xa | 1u << c;
        if (ma + i == mb + j) continue;  // the same target twice
        mb[j] = xb | 1u << c;
      }
      base = 32;
    } else {
      again = 1;
    }
    while (again) {
      again = 0;
      for (int sl = 0; sl < pp.ninc; sl++) {
        int nu = ind_sizes[pp.inc_ind[sl] + b * pp.ninds];
        for (int u = 0; u < nu; u++) masks[pp.inc_mbase[sl] + u] = 0u;
      }
      for (int e = 0; e < bs; e++) {
        if (col[e] != -1) continue;
        unsigned mask = 0;
        for (int sl = 0; sl < pp.ninc; sl++) mask |= masks[pp.inc_mbase[sl] + locs[sl * bs + e]];
        int c = __ffs(~mask) - 1;
        if (c < 0) {
          again = 1;
          continue;
        }
        col[e] = base + c;
        ncol = max(ncol, base + c + 1);
        for (int sl = 0; sl < pp.ninc; sl++) masks[pp.inc_mbase[sl] + locs[sl * bs + e]] |= 1u << c;
      }
      base += 32;
    }
    nthrcol[b] = ncol;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < bs; e += blockDim.x) thrcol[e0 + e] = col[e];
}

struct IncWork {
  unsigned *work[kMaxArgs];  // per INC slot: mask array of its ind (aliases allowed)
  int wsize[kMaxArgs];
};

// greedy block colouring in block order, 32 colours per pass, then blocks
// grouped by colour (common/op_lib_core.c:892-965).  One CTA: blocks are
// visited in order as the reference does; each block's target masks are
// ORed and set by all threads in parallel.
__global__ void k_block_colour(PlanParams pp, IncWork iw, int nwork, unsigned *const *work_arrays,
                               const int *work_sizes, int *blk_col, int *blkmap, int *ncolblk,
                               int *ncolors_out) {
  __shared__ unsigned s_mask[32];
  __shared__ int s_again, s_col;
  const int tid = threadIdx.x;
  for (int b = tid; b < pp.nblocks; b += blockDim.x) blk_col[b] = -1;
  int base = 0, ncolors = 0;
  if (tid == 0) s_again = 1;
  __syncthreads();
  while (s_again) {
    __syncthreads();
    if (tid == 0) s_again = 0;
    for (int w = 0; w < nwork; w++)
      for (int t = tid; t < work_sizes[w]; t += blockDim.x) work_arrays[w][t] = 0u;
    __syncthreads();
    for (int b = 0; b < pp.nblocks; b++) {
      if (blk_col[b] != -1) continue;
      const int e0 = b * pp.bsize;
      const int bs = min(pp.bsize, pp.set_size - e0);
      unsigned mask = 0;
      for (int i = tid; i < pp.ninc * bs; i += blockDim.x) {
        int sl = i / bs;
        int t = map_at(pp.am, pp.inc_arg[sl], e0 + i % bs);
        mask |= iw.work[sl][t];
      }
      mask = __reduce_or_sync(0xffffffffu, mask);
      if ((tid & 31) == 0) s_mask[tid >> 5] = mask;
      __syncthreads();
      if (tid == 0) {
        unsigned mm = 0;
        for (int w = 0; w < (int)(blockDim.x + 31) / 32; w++) mm |= s_mask[w];
        int c = __ffs(~mm) - 1;
        s_col = c;
        if (c < 0) s_again = 1;
        else blk_col[b] = base + c;
      }
      __syncthreads();
      int c = s_col;
      if (c >= 0) {
        ncolors = max(ncolors, base + c + 1);
        for (int i = tid; i < pp.ninc * bs; i += blockDim.x) {
          int sl = i / bs;
          int t = map_at(pp.am, pp.inc_arg[sl], e0 + i % bs);
          atomicOr(&iw.work[sl][t], 1u << c);
        }
      }
      __syncthreads();
    }
    base += 32;
    __syncthreads();
  }
  // blocks of each colour in block order (counting sort, stable)
  int start = 0;
  for (int c = 0; c < ncolors; c++) {
    for (int r = 0; r < pp.nblocks; r += blockDim.x) {
      int b = r + tid;
      int f = (b < pp.nblocks) && blk_col[b] == c;
      int tot;
      int pos = block_excl_scan(f, &tot);
      if (f) blkmap[start + pos] = b;
      start += tot;
      if (tid == 0) ncolblk[c] += tot;
    }
  }
  if (tid == 0) *ncolors_out = ncolors;
}

// ---- the same colouring from the blocks' conflicts --------------------------
// A block's colour is the lowest that no earlier block sharing a target with
// it has (the passes of 32 colours come to the same).  The conflicts are
// found in parallel -- per target the blocks that increment it, per pair of
// them a bit in a triangular matrix -- and only the greedy itself goes block
// after block, over neighbours and colours in shared memory instead of the
// masks of every target of the block in global memory: 3.4 -> 0.24 ms for
// 1,586 blocks of 512 edges, 10.6 -> 0.85 ms for 5,620 of 256 (0.15 us a
// block: a chain of shared loads, a warp reduction and a store), and some
// 0.06 ms to find the conflicts.
constexpr int kColourBlocks = 16384;  // blocks the matrix (32 MB) is built for
constexpr int kColourRow = 64;        // earlier neighbours of a block, for the one-warp greedy
constexpr int kColourLong = 32;       // blocks of a target paired by one thread

struct ColourSlots {  // the INC arguments; targets of distinct inds apart
  const int *map[kMaxArgs];
  int dim[kMaxArgs], idx[kMaxArgs], base[kMaxArgs];
  int n;
};

// one (argument, element) after another: its target
__device__ __forceinline__ int colour_target(const ColourSlots &cs, long long i, int nelem,
                                             int &e) {
  const int sl = (int)(i / nelem);
  e = (int)(i - (long long)sl * nelem);
  return cs.base[sl] + cs.map[sl][cs.idx[sl] + (size_t)e * cs.dim[sl]];
}

__global__ void k_colour_count(ColourSlots cs, int nelem, int *cnt) {
  const long long n = (long long)cs.n * nelem;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    int e;
    atomicAdd(cnt + colour_target(cs, i, nelem, e), 1);
  }
}

__global__ void k_colour_scatter(ColourSlots cs, int nelem, int bsize, int *end,
                                 unsigned short *blocks) {
  const long long n = (long long)cs.n * nelem;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    int e;
    const int t = colour_target(cs, i, nelem, e);
    blocks[atomicAdd(end + t, 1)] = (unsigned short)(e / bsize);
  }
}

__device__ __forceinline__ void colour_conflict(unsigned *adj, int words, int a, int b) {
  if (a == b) return;
  const int hi = max(a, b), lo = min(a, b);
  unsigned *w = adj + (size_t)hi * words + (lo >> 5);
  if (*w >> (lo & 31) & 1) return;  // bits are only ever set
  atomicOr(w, 1u << (lo & 31));
}

// end[t]: where target t's blocks end, and the next target's begin
__global__ void k_colour_pairs(int ntarget, const int *end, const unsigned short *blocks,
                               unsigned *adj, int words, int *long_targets, int *nlong) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntarget; t += gridDim.x * blockDim.x) {
    const int k0 = t ? end[t - 1] : 0, k1 = end[t];
    if (k1 - k0 > kColourLong) {
      long_targets[atomicAdd(nlong, 1)] = t;
      continue;
    }
    for (int i = k0 + 1; i < k1; i++)
      for (int j = k0; j < i; j++) colour_conflict(adj, words, blocks[i], blocks[j]);
  }
}

// a target of many blocks: the set of them, then every row of the set
__global__ void k_colour_long(const int *end, const unsigned short *blocks, unsigned *adj,
                              int words, int nb, const int *long_targets, const int *nlong) {
  __shared__ unsigned set[kColourBlocks / 32];
  for (int l = blockIdx.x; l < *nlong; l += gridDim.x) {
    const int t = long_targets[l];
    for (int w = threadIdx.x; w < words; w += blockDim.x) set[w] = 0u;
    __syncthreads();
    for (int i = (t ? end[t - 1] : 0) + threadIdx.x; i < end[t]; i += blockDim.x)
      atomicOr(set + (blocks[i] >> 5), 1u << (blocks[i] & 31));
    __syncthreads();
    for (int w = threadIdx.x; w < words; w += blockDim.x) {
      if (set[w] == 0u) continue;
      for (int b = w << 5; b < nb; b++) {
        if (!(set[b >> 5] >> (b & 31) & 1)) continue;
        const unsigned m = b >> 5 == w ? set[w] & ((1u << (b & 31)) - 1) : set[w];
        if (m) atomicOr(adj + (size_t)b * words + w, m);
      }
    }
    __syncthreads();
  }
}

// each row as a list of its first kColourRow neighbours, one warp per row, and
// the longest row
__global__ void k_colour_rows(int nb, int words, const unsigned *adj, unsigned short *list,
                              int *count, int *longest) {
  const int lane = threadIdx.x & 31;
  for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nb;
       b += (gridDim.x * blockDim.x) >> 5) {
    int n = 0;
    for (int w0 = 0; w0 <= b >> 5; w0 += 32) {
      unsigned bits = w0 + lane <= b >> 5 ? adj[(size_t)b * words + w0 + lane] : 0u;
      int at = __popc(bits);
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += y;
      }
      const int all = __shfl_sync(0xffffffffu, at, 31);
      at += n - __popc(bits);
      n += all;
      for (; bits && at < kColourRow; bits &= bits - 1)
        list[(size_t)b * kColourRow + at++] =
            (unsigned short)((w0 + lane) * 32 + __ffs(bits) - 1);
    }
    if (lane == 0) {
      count[b] = n;
      if (n > *longest) atomicMax(longest, n);
    }
  }
}

// blocks grouped by colour, in block order: rank[b] = earlier blocks of its
// colour.  By all threads of the greedy's CTA; cnt: blocks of each colour
__device__ void colour_place(int nb, int ncolors, const unsigned short *col, int *cnt,
                             const unsigned short *rank, int *blk_col, int *blkmap, int *ncolblk,
                             int *ncolors_out) {
  const int tid = threadIdx.x;
  __syncthreads();
  int run = 0;
  for (int c0 = 0; c0 < ncolors; c0 += blockDim.x) {
    const int c = c0 + tid, v = c < ncolors ? cnt[c] : 0;
    int tot;
    const int x = block_excl_scan(v, &tot);
    if (c < ncolors) {
      ncolblk[c] = v;
      cnt[c] = run + x;
    }
    run += tot;
  }
  __syncthreads();
  for (int b = tid; b < nb; b += blockDim.x) {
    blk_col[b] = col[b];
    blkmap[cnt[col[b]] + rank[b]] = b;
  }
  if (tid == 0) *ncolors_out = ncolors;
}

// the greedy when every row fits a list: one warp colours, the CTA brings the
// next 32 rows
__global__ void __launch_bounds__(256)
    k_colour_narrow(int nb, const unsigned short *__restrict__ list, const int *__restrict__ count,
                    const int *longest, int *blk_col, int *blkmap, int *ncolblk,
                    int *ncolors_out) {
  extern __shared__ int colour_smem[];
  int *cnt = colour_smem;
  unsigned short *col = (unsigned short *)(cnt + nb), *rank = col + nb;
  __shared__ unsigned rows[2][32][kColourRow / 2];
  __shared__ int len[2][32];
  __shared__ int s_ncolors;
  if (*longest > kColourRow) return;
  const int tid = threadIdx.x, lane = tid & 31;
  auto stage = [&](int b0, int buf, int first) {  // by the threads from `first` on
    for (int i = tid - first; i < 32 * (kColourRow / 2); i += 256 - first) {
      const int r = i / (kColourRow / 2), k = i % (kColourRow / 2);
      if (b0 + r < nb)
        rows[buf][r][k] =
            __ldg(reinterpret_cast<const unsigned *>(list + (size_t)(b0 + r) * kColourRow) + k);
    }
    if (tid >= first && tid < first + 32)
      len[buf][tid - first] = b0 + tid - first < nb ? __ldg(count + b0 + tid - first) : 0;
  };
  for (int b = tid; b < nb; b += 256) cnt[b] = 0;
  stage(0, 0, 0);
  int ncolors = 0;
  for (int b0 = 0, buf = 0; b0 < nb; b0 += 32, buf ^= 1) {
    __syncthreads();
    if (tid >= 32) {
      if (b0 + 32 < nb) stage(b0 + 32, buf ^ 1, 32);
      continue;
    }
    // a row's neighbours and their colours are read while the row before it
    // is coloured; that row's own colour is put in by hand
    const int nr = min(32, nb - b0);
    int ia, ib, ca, cb, mine = 0;
    auto read = [&](int r) {
      const unsigned pair = rows[buf][r][lane];  // neighbours 2 lane and 2 lane + 1
      const int n = len[buf][r];
      ia = 2 * lane < n ? (int)(pair & 0xffffu) : -1;
      ib = 2 * lane + 1 < n ? (int)(pair >> 16) : -1;
      ca = ia >= 0 ? (int)col[ia] : -1;
      cb = ib >= 0 ? (int)col[ib] : -1;
    };
    read(0);
    for (int r = 0; r < nr; r++) {
      const int b = b0 + r, xa = ca, xb = cb;
      if (r + 1 < nr) read(r + 1);
      int c = 0;
      for (int base = 0;; base += 32) {
        unsigned mask = 0;
        if (xa >= base && xa < base + 32) mask |= 1u << (xa - base);
        if (xb >= base && xb < base + 32) mask |= 1u << (xb - base);
        mask = __reduce_or_sync(0xffffffffu, mask);
        if (mask != ~0u) {
          c = base + __ffs(~mask) - 1;
          break;
        }
      }
      if (lane == 0) col[b] = (unsigned short)c;
      __syncwarp();
      if (ia == b) ca = c;
      if (ib == b) cb = c;
      if (lane == r) mine = c;
      ncolors = max(ncolors, c + 1);
    }
    // ranks of the 32 blocks among those of their colour
    const unsigned same = __match_any_sync(0xffffffffu, lane < nr ? mine : -1 - lane);
    const unsigned before = same & ((1u << lane) - 1);
    if (lane < nr) rank[b0 + lane] = (unsigned short)(cnt[mine] + __popc(before));
    __syncwarp();
    if (lane < nr && before == 0) cnt[mine] += __popc(same);
    __syncwarp();
  }
  if (tid == 0) s_ncolors = ncolors;
  __syncthreads();
  colour_place(nb, s_ncolors, col, cnt, rank, blk_col, blkmap, ncolblk, ncolors_out);
}

// the greedy for wide rows (a numbering without locality): all threads read a
// row, half a word each; seen[c] = the last block that has a neighbour of
// colour c
__global__ void __launch_bounds__(1024)
    k_colour_wide(int nb, int words, const unsigned *__restrict__ adj, const int *longest,
                  int *blk_col, int *blkmap, int *ncolblk, int *ncolors_out) {
  extern __shared__ int colour_smem[];
  int *cnt = colour_smem, *seen = cnt + nb;
  unsigned short *col = (unsigned short *)(seen + nb + 1), *rank = col + nb;
  __shared__ int s_first[2];
  if (*longest <= kColourRow) return;
  const int tid = threadIdx.x, halves = 2 * words;  // at most 1024
  for (int b = tid; b < nb; b += 1024) cnt[b] = 0;
  for (int b = tid; b <= nb; b += 1024) seen[b] = -1;
  if (tid < 2) s_first[tid] = nb;
  int ncolors = 0;
  unsigned next = tid < halves ? __ldg(adj + (tid >> 1)) : 0u;
  __syncthreads();
  for (int b = 0; b < nb; b++) {
    unsigned bits = next >> (16 * (tid & 1)) & 0xffffu;
    if (b + 1 < nb && tid < halves) next = __ldg(adj + (size_t)(b + 1) * words + (tid >> 1));
    while (bits) {
      const int j = tid * 16 + __ffs(bits) - 1;
      bits &= bits - 1;
      seen[col[j]] = b;
    }
    __syncthreads();
    // the first colour not seen; ncolors itself never is
    for (int c0 = 0; c0 <= ncolors; c0 += 1024) {
      const bool free_c = c0 + tid <= ncolors && seen[c0 + tid] != b;
      const unsigned m = __ballot_sync(0xffffffffu, free_c);
      if (m && (tid & 31) == 0) atomicMin(&s_first[b & 1], c0 + tid + __ffs(m) - 1);
    }
    __syncthreads();
    const int c = s_first[b & 1];
    ncolors = max(ncolors, c + 1);
    if (tid == 0) {
      col[b] = (unsigned short)c;
      rank[b] = (unsigned short)cnt[c]++;
      s_first[(b & 1) ^ 1] = nb;
    }
    __syncthreads();
  }
  colour_place(nb, ncolors, col, cnt, rank, blk_col, blkmap, ncolblk, ncolors_out);
}

// ----------------------------------------------------------- validation --

__global__ void k_check_locmaps(PlanParams pp, IndOut io, const int *ind_sizes,
                                const int *ind_offs, unsigned long long *err) {
  long long n = (long long)pp.nargs * pp.set_size;
  unsigned long long bad = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    int a = (int)(i / pp.set_size), e = (int)(i % pp.set_size);
    int m = pp.arg_ind[a];
    if (io.loc_maps[a] == nullptr || m < 0) continue;
    int b = e / pp.bsize;
    int loc = io.loc_maps[a][e];
    if (loc < 0 || loc >= ind_sizes[m + b * pp.ninds]) {
      bad++;
      continue;
    }
    int g = io.ind_maps[m][ind_offs[m + b * pp.ninds] + loc];
    bad += (g != map_at(pp.am, a, e));
  }
  if (bad) atomicAdd(err, bad);
}

__global__ void k_check_indmaps(PlanParams pp, IndOut io, const int *ind_sizes,
                                const int *ind_offs, const int *to_sizes,
                                unsigned long long *err) {
  const int b = blockIdx.x, m = blockIdx.y;
  const int nu = ind_sizes[m + b * pp.ninds], off = ind_offs[m + b * pp.ninds];
  unsigned long long bad = 0;
  if (threadIdx.x == 0 && b > 0)
    bad += (off != ind_offs[m + (b - 1) * pp.ninds] + ind_sizes[m + (b - 1) * pp.ninds]);
  if (threadIdx.x == 0 && b == 0) bad += (off != 0);
  for (int u = threadIdx.x; u < nu; u += blockDim.x) {
    int t = io.ind_maps[m][off + u];
    if (u > 0) bad += (t <= io.ind_maps[m][off + u - 1]);
    bad += (t < 0 || t >= to_sizes[m]);
  }
  if (bad) atomicAdd(err, bad);
}

// no two elements of one block with the same thread colour touch one
// OP_INC target
__global__ void k_check_thread_colours(PlanParams pp, IndOut io, const int *ind_sizes,
                                       const int *thrcol, const int *nthrcol,
                                       unsigned long long *err) {
  extern __shared__ int own[];
  const int b = blockIdx.x;
  const int e0 = b * pp.bsize;
  const int bs = min(pp.bsize, pp.set_size - e0);
  const int nc = nthrcol[b];
  unsigned long long bad = 0;
  for (int e = threadIdx.x; e < bs; e += blockDim.x) {
    int c = thrcol[e0 + e];
    bad += (c < 0 || c >= nc);
  }
  for (int c = 0; c < nc; c++) {
    for (int w = threadIdx.x; w < pp.mask_words; w += blockDim.x) own[w] = -1;
    __syncthreads();
    for (int e = threadIdx.x; e < bs; e += blockDim.x) {
      if (thrcol[e0 + e] != c) continue;
      for (int sl = 0; sl < pp.ninc; sl++) {
        int loc = io.loc_maps[pp.inc_arg[sl]][e0 + e];
        int old = atomicCAS(&own[pp.inc_mbase[sl] + loc], -1, e);
        bad += (old != -1 && old != e);
      }
    }
    __syncthreads();
  }
  if (bad) atomicAdd(err, bad);
}

// no two blocks of the same block colour touch one OP_INC target
__global__ void k_check_block_colours(PlanParams pp, IncWork iw, const int *blkmap, int first,
                                      int nblk, unsigned long long *err) {
  unsigned long long bad = 0;
  for (int k = blockIdx.x; k < nblk; k += gridDim.x) {
    int b = blkmap[first + k];
    int e0 = b * pp.bsize, bs = min(pp.bsize, pp.set_size - e0);
    for (int i = threadIdx.x; i < pp.ninc * bs; i += blockDim.x) {
      int sl = i / bs;
      int t = map_at(pp.am, pp.inc_arg[sl], e0 + i % bs);
      int old = atomicCAS((int *)&iw.work[sl][t], -1, b);
      bad += (old != -1 && old != b);
    }
  }
  if (bad) atomicAdd(err, bad);
}

__global__ void k_check_blocks(PlanParams pp, const int *blkmap, const int *offset,
                               const int *nelems, int *seen, unsigned long long *err) {
  unsigned long long bad = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < pp.nblocks;
       i += gridDim.x * blockDim.x) {
    int b = blkmap[i];
    if (b < 0 || b >= pp.nblocks) bad++;
    else if (atomicAdd(&seen[b], 1) != 0) bad++;
    bad += (offset[i] != i * pp.bsize);
    bad += (nelems[i] != min(pp.bsize, pp.set_size - i * pp.bsize));
  }
  if (bad) atomicAdd(err, bad);
}

// ------------------------------------------------------------------ scan --

// a chunk of kScanChunk values per CTA of 1024, eight consecutive ones per thread
constexpr int kScanChunk = 8192;
__global__ void __launch_bounds__(1024) k_scan_chunks(const int *in, int *out, int n, int *sums) {
  const long long i0 = (long long)blockIdx.x * kScanChunk + threadIdx.x * 8;
  int v[8], own = 0;
  const bool whole = i0 + 8 <= n && ((uintptr_t)in & 15) == 0 && ((uintptr_t)out & 15) == 0;
  if (whole) {
    const int4 a = reinterpret_cast<const int4 *>(in + i0)[0];
    const int4 b = reinterpret_cast<const int4 *>(in + i0)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = i0 + k < n ? in[i0 + k] : 0;
  }
#pragma unroll
  for (int k = 0; k < 8; k++) own += v[k];
  int total;
  int run = block_excl_scan(own, &total);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int x = v[k];
    v[k] = run;
    run += x;
  }
  if (whole) {
    reinterpret_cast<int4 *>(out + i0)[0] = make_int4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<int4 *>(out + i0)[1] = make_int4(v[4], v[5], v[6], v[7]);
  } else {
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (i0 + k < n) out[i0 + k] = v[k];
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void k_scan_add(int *out, int n, const int *offs, int chunk) {
  int add = offs[blockIdx.x];
  int c0 = blockIdx.x * chunk;
  for (int r = threadIdx.x; r < chunk; r += blockDim.x) {
    int i = c0 + r;
    if (i < n) out[i] += add;
  }
}

void exclusive_scan_nosync(const int *d_in, int *d_out, int n, cudaStream_t s) {
  const int chunk = kScanChunk;
  const int nch = (n + chunk - 1) / chunk;
  if (n <= 0) return;
  int *sums = nullptr;
  OP2B_CUDA(pool_malloc_async((void **)&sums, sizeof(int) * (nch + 1), s));
  k_scan_chunks<<<nch, 1024, 0, s>>>(d_in, d_out, n, sums);
  if (nch > 1) {
    exclusive_scan_nosync(sums, sums, nch, s);
    k_scan_add<<<nch, 1024, 0, s>>>(d_out, n, sums, chunk);
  }
  OP2B_CUDA(cudaFreeAsync(sums, s));
}

long long exclusive_scan(const int *d_in, int *d_out, int n, cudaStream_t s) {
  const int chunk = kScanChunk;
  int nch = (n + chunk - 1) / chunk;
  if (n <= 0) return 0;
  int *sums = nullptr;
  OP2B_CUDA(pool_malloc_async((void **)&sums, sizeof(int) * (nch + 1), s));
  k_scan_chunks<<<nch, 1024, 0, s>>>(d_in, d_out, n, sums);
  if (nch > 1) {
    exclusive_scan(sums, sums, nch, s);
    k_scan_add<<<nch, 1024, 0, s>>>(d_out, n, sums, chunk);
  }
  // total = last exclusive value + last input
  int last_out = 0, last_in = 0;
  OP2B_CUDA(cudaMemcpyAsync(&last_out, d_out + n - 1, sizeof(int), cudaMemcpyDeviceToHost, s));
  OP2B_CUDA(cudaMemcpyAsync(&last_in, d_in + n - 1, sizeof(int), cudaMemcpyDeviceToHost, s));
  OP2B_CUDA(cudaFreeAsync(sums, s));
  OP2B_CUDA(cudaStreamSynchronize(s));
  return (long long)last_out + last_in;
}

// ------------------------------------------------------------- builders --

static std::vector<std::unique_ptr<DevPlan>> g_plans;
static std::vector<std::unique_ptr<GatherPlan>> g_gather;

static bool fill_params(PlanParams &pp, const DevPlan &p, std::vector<int> &to_sizes) {
  memset(&pp, 0, sizeof pp);
  if (p.nargs > kMaxArgs || p.ninds > kMaxArgs) return false;
  pp.nargs = p.nargs;
  pp.ninds = p.ninds;
  pp.set_size = p.set->size;
  pp.bsize = p.bsize;
  pp.nblocks = p.nblocks;
  pp.cls = OP_cache_line_size > 0 ? OP_cache_line_size : 128;
  for (int a = 0; a < p.nargs; a++) {
    pp.arg_ind[a] = p.inds[a];
    if (p.maps[a]) {
      pp.am.map[a] = map_dev(p.maps[a]);
      pp.am.dim[a] = p.maps[a]->dim;
      pp.am.idx[a] = p.idxs[a];
    }
  }
  int pos = 0;
  to_sizes.assign(p.ninds, 0);
  for (int m = 0; m < p.ninds; m++) {
    pp.ind_first[m] = pos;
    for (int a = 0; a < p.nargs; a++)
      if (p.inds[a] == m) {
        if (!p.maps[a]) return false;
        pp.ind_args[pos++] = a;
        if (pp.ind_k[m] == 0) {
          pp.ind_size[m] = p.dats[a]->size;
          pp.ind_dim[m] = p.dats[a]->dim;
          to_sizes[m] = p.maps[a]->to->size;
        }
        pp.ind_k[m]++;
      }
    if (pp.ind_k[m] == 0) return false;
  }
  long long off = 0;
  for (int m = 0; m < p.ninds; m++) {
    pp.tmp_off[m] = off;
    off += (long long)pp.ind_k[m] * p.bsize * p.nblocks;
    int P = 64;
    while (P < pp.ind_k[m] * p.bsize) P <<= 1;
    pp.ind_P[m] = P;
  }
  // q, adt and res of airfoil's res_calc all go through pecell: their distinct
  // targets and local indices are found once
  for (int a = 0; a < p.nargs; a++) {
    pp.arg_same[a] = a;
    for (int c = 0; c < a && pp.arg_same[a] == a; c++)
      if (p.inds[a] >= 0 && p.inds[c] >= 0 && p.maps[c] == p.maps[a] && p.idxs[c] == p.idxs[a])
        pp.arg_same[a] = c;
  }
  for (int m = 0; m < p.ninds; m++) {
    pp.ind_same[m] = m;
    for (int c = 0; c < m && pp.ind_same[m] == m; c++) {
      bool same = pp.ind_k[c] == pp.ind_k[m];
      for (int i = 0; i < pp.ind_k[m] && same; i++)
        same = pp.arg_same[pp.ind_args[pp.ind_first[c] + i]] ==
               pp.arg_same[pp.ind_args[pp.ind_first[m] + i]];
      if (same) pp.ind_same[m] = c;
    }
    pp.tmp_off[m] = pp.tmp_off[pp.ind_same[m]];
  }
  // INC slots and their mask areas (one area per distinct ind)
  int mbase_of_ind[kMaxArgs];
  for (int m = 0; m < kMaxArgs; m++) mbase_of_ind[m] = -1;
  int words = 0;
  for (int a = 0; a < p.nargs; a++)
    if (p.inds[a] >= 0 && p.accs[a] == OP_INC) {
      int m = p.inds[a];
      if (mbase_of_ind[m] < 0) {
        mbase_of_ind[m] = words;
        words += pp.ind_k[m] * p.bsize;
      }
      pp.inc_arg[pp.ninc] = a;
      pp.inc_ind[pp.ninc] = m;
      pp.inc_mbase[pp.ninc] = mbase_of_ind[m];
      pp.ninc++;
    }
  pp.mask_words = words;
  return true;
}

static size_t smem_optin() {
  static int v = -1;
  if (v < 0) {
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, rt().device);
    if (v <= 0) v = 48 * 1024;
  }
  return (size_t)v;
}

// allow a kernel the largest dynamic shared memory the device offers, less
// what the kernel declares statically
template <class K>
static size_t allow_smem(K kernel) {
  cudaFuncAttributes fa;
  OP2B_CUDA(cudaFuncGetAttributes(&fa, kernel));
  size_t dyn = smem_optin() - fa.sharedSizeBytes;
  OP2B_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
  return dyn;
}

// block colours, blkmap and the blocks per colour from the conflicts of the
// blocks; false for more blocks (or targets) than that is built for
static bool colour_blocks(const DevPlan &p, const PlanParams &pp, const std::vector<int> &to_sizes,
                          int *d_ncolblk, int *d_ncolors, cudaStream_t s) {
  const int nb = p.nblocks, n = p.set->size, words = (nb + 31) / 32;
  if (nb > kColourBlocks) return false;
  ColourSlots cs;
  memset(&cs, 0, sizeof cs);
  long long nt = 0;
  std::vector<int> base(kMaxArgs, -1);
  for (int sl = 0; sl < pp.ninc; sl++) {
    const int m = pp.inc_ind[sl], a = pp.inc_arg[sl];
    if (base[m] < 0) {
      base[m] = (int)nt;
      nt += to_sizes[m];
    }
    cs.map[sl] = pp.am.map[a];
    cs.dim[sl] = pp.am.dim[a];
    cs.idx[sl] = pp.am.idx[a];
    cs.base[sl] = base[m];
    cs.n = sl + 1;
  }
  const long long nent = (long long)pp.ninc * n;
  if (nt >= (1LL << 31) - 1 || nent >= (1LL << 31) - 1) return false;
  // adjacency | longest row, number of long targets | per target: blocks' end
  // | long targets | row lengths | rows | blocks
  const size_t adj_bytes = sizeof(unsigned) * (size_t)nb * words;
  const size_t ntz = (size_t)std::max(1LL, nt);
  char *mem = nullptr;
  const size_t bytes =
      adj_bytes + sizeof(int) * (2 + 2 * ntz + nb) +
      sizeof(unsigned short) * ((size_t)nb * kColourRow + (size_t)std::max(1LL, nent));
  if (pool_malloc_async((void **)&mem, bytes, s) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  unsigned *adj = (unsigned *)mem;
  int *longest = (int *)(mem + adj_bytes), *nlong = longest + 1, *end = longest + 2;
  int *longs = end + ntz, *count = longs + ntz;
  unsigned short *list = (unsigned short *)(count + nb), *blocks = list + (size_t)nb * kColourRow;
  OP2B_CUDA(cudaMemsetAsync(mem, 0, adj_bytes + 2 * sizeof(int) + sizeof(int) * ntz, s));
  if (pp.ninc) {
    const int grid = rt().num_sms * 8;
    k_colour_count<<<grid, 256, 0, s>>>(cs, n, end);
    exclusive_scan_nosync(end, end, (int)nt, s);
    k_colour_scatter<<<grid, 256, 0, s>>>(cs, n, p.bsize, end, blocks);
    k_colour_pairs<<<grid, 256, 0, s>>>((int)nt, end, blocks, adj, words, longs, nlong);
    k_colour_long<<<rt().num_sms, 256, 0, s>>>(end, blocks, adj, words, nb, longs, nlong);
  }
  k_colour_rows<<<std::min(rt().num_sms * 8, (nb + 7) / 8), 256, 0, s>>>(nb, words, adj, list,
                                                                        count, longest);
  allow_smem(k_colour_narrow);
  allow_smem(k_colour_wide);
  k_colour_narrow<<<1, 256, 8 * (size_t)nb, s>>>(nb, list, count, longest, p.d_blkcol,
                                                 p.d_blkmap, d_ncolblk, d_ncolors);
  k_colour_wide<<<1, 1024, 12 * (size_t)nb + 4, s>>>(nb, words, adj, longest, p.d_blkcol,
                                                     p.d_blkmap, d_ncolblk, d_ncolors);
  OP2B_CUDA(cudaFreeAsync(mem, s));
  return true;
}

// the same for any number of blocks: a block's colour from the masks of its
// targets, one block after another
static void colour_blocks_by_targets(const DevPlan &p, const PlanParams &pp,
                                     const std::vector<int> &to_sizes, int *d_ncolblk,
                                     int *d_ncolors, cudaStream_t s) {
  IncWork iw;  // one mask array per distinct INC ind
  memset(&iw, 0, sizeof iw);
  std::vector<unsigned *> warr;
  std::vector<int> wsz;
  std::vector<int> ind_w(kMaxArgs, -1);
  for (int sl = 0; sl < pp.ninc; sl++) {
    int m = pp.inc_ind[sl];
    if (ind_w[m] < 0) {
      unsigned *w = nullptr;
      OP2B_CUDA(pool_malloc_async((void **)&w, sizeof(unsigned) * (size_t)to_sizes[m], s));
      ind_w[m] = (int)warr.size();
      warr.push_back(w);
      wsz.push_back(to_sizes[m]);
    }
    iw.work[sl] = warr[ind_w[m]];
    iw.wsize[sl] = to_sizes[m];
  }
  unsigned **d_warr = nullptr;
  int *d_wsz = nullptr;
  int nw = (int)warr.size();
  OP2B_CUDA(pool_malloc_async((void **)&d_warr, sizeof(unsigned *) * (nw ? nw : 1), s));
  OP2B_CUDA(pool_malloc_async((void **)&d_wsz, sizeof(int) * (nw ? nw : 1), s));
  if (nw) {
    OP2B_CUDA(cudaMemcpyAsync(d_warr, warr.data(), sizeof(unsigned *) * nw, cudaMemcpyHostToDevice, s));
    OP2B_CUDA(cudaMemcpyAsync(d_wsz, wsz.data(), sizeof(int) * nw, cudaMemcpyHostToDevice, s));
  }
  k_block_colour<<<1, 1024, 0, s>>>(pp, iw, nw, d_warr, d_wsz, p.d_blkcol, p.d_blkmap, d_ncolblk,
                                    d_ncolors);
  OP2B_CUDA(cudaStreamSynchronize(s));  // the host tables have been read
  for (void *w : warr) OP2B_CUDA(cudaFreeAsync(w, s));
  OP2B_CUDA(cudaFreeAsync(d_warr, s));
  OP2B_CUDA(cudaFreeAsync(d_wsz, s));
}

static void build_plan(DevPlan &p) {
  Runtime &R = rt();
  cudaStream_t s = R.stream;
  const int n = p.set->size;
  // block size from the reference's 48 KB shared-memory budget
  // (common/op_lib_core.c:663-673)
  int maxbytes = 0;
  for (int a = 0; a < p.nargs; a++)
    if (p.inds[a] >= 0) maxbytes += p.dats[a]->size;
  p.bsize = p.part_size;
  if (p.bsize == 0) p.bsize = maxbytes > 0 ? (48 * 1024 / (64 * maxbytes)) * 64 : 512;
  if (p.bsize <= 0) {
    fail(-1, "op_plan error -- invalid block size for kernel %s\n", p.name.c_str());
    return;
  }
  p.nblocks = (n - 1) / p.bsize + 1;

  PlanParams pp;
  std::vector<int> to_sizes;
  if (!fill_params(pp, p, to_sizes)) {
    fail(-1, "op_plan error -- unsupported argument layout for kernel %s\n", p.name.c_str());
    return;
  }
  const size_t optin = smem_optin() - 1024;  // headroom for static shared memory
  for (int m = 0; m < p.ninds; m++)
    if ((size_t)pp.ind_P[m] * sizeof(int) > optin || pp.ind_k[m] * p.bsize > 32767) {
      fail(-1,
           "op_plan error -- block size %d too large for kernel %s (block-local indices "
           "are 16-bit and each block's targets are sorted in shared memory)\n",
           p.bsize, p.name.c_str());
      return;
    }

  const int nb = p.nblocks, ni = p.ninds;
  p.d_nthrcol = (int *)dev_alloc(sizeof(int) * nb);
  p.d_thrcol = (int *)dev_alloc(sizeof(int) * (size_t)n);
  p.d_offset = (int *)dev_alloc(sizeof(int) * nb);
  p.d_nelems = (int *)dev_alloc(sizeof(int) * nb);
  p.d_ind_offs = (int *)dev_alloc(sizeof(int) * (size_t)nb * (ni ? ni : 1));
  p.d_ind_sizes = (int *)dev_alloc(sizeof(int) * (size_t)nb * (ni ? ni : 1));
  p.d_blkmap = (int *)dev_alloc(sizeof(int) * nb);
  p.d_blkcol = (int *)dev_alloc(sizeof(int) * nb);
  p.d_ind_maps.assign(ni, nullptr);
  p.d_loc_maps.assign(p.nargs, nullptr);
  for (int a = 0; a < p.nargs; a++)
    if (p.inds[a] >= 0) p.d_loc_maps[a] = (short *)dev_alloc(sizeof(short) * (size_t)n);

  // offsets and sizes of the contiguous blocks (common/op_lib_core.c:768-773)
  std::vector<int> off(nb), nel(nb);
  for (int b = 0; b < nb; b++) {
    off[b] = b * p.bsize;
    nel[b] = std::min(p.bsize, n - b * p.bsize);
  }
  OP2B_CUDA(cudaMemcpyAsync(p.d_offset, off.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, s));
  OP2B_CUDA(cudaMemcpyAsync(p.d_nelems, nel.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, s));

  long long tmp_total = 0;
  for (int m = 0; m < ni; m++) tmp_total += (long long)pp.ind_k[m] * p.bsize * nb;
  int *tmp = nullptr, *d_nind = nullptr;
  long long *d_lines = nullptr, *d_lines3 = nullptr;
  OP2B_CUDA(pool_malloc_async((void **)&tmp, sizeof(int) * (tmp_total ? tmp_total : 1), s));
  OP2B_CUDA(pool_malloc_async((void **)&d_nind, sizeof(int) * (ni ? ni : 1), s));
  OP2B_CUDA(pool_malloc_async((void **)&d_lines, sizeof(long long) * nb * (ni ? ni : 1), s));
  OP2B_CUDA(pool_malloc_async((void **)&d_lines3, sizeof(long long) * nb * (ni ? ni : 1), s));

  IndOut io;
  memset(&io, 0, sizeof io);
  for (int a = 0; a < p.nargs; a++) io.loc_maps[a] = p.d_loc_maps[a];

  p.nindirect.assign(ni, 0);
  if (ni > 0) {
    int maxP = 0;
    for (int m = 0; m < ni; m++) maxP = std::max(maxP, pp.ind_P[m]);
    size_t sm = sizeof(int) * (size_t)maxP;
    allow_smem(k_block_unique);
    k_block_unique<<<dim3(nb, ni), std::min(1024, std::max(32, maxP / 2)), sm, s>>>(
        pp, p.d_ind_sizes, tmp);
    k_scan_blocks<<<ni, 1024, 0, s>>>(nb, ni, p.d_ind_sizes, p.d_ind_offs, d_nind);
    OP2B_CUDA(cudaMemcpyAsync(p.nindirect.data(), d_nind, sizeof(int) * ni,
                              cudaMemcpyDeviceToHost, s));
    OP2B_CUDA(cudaStreamSynchronize(s));
    for (int m = 0; m < ni; m++) {
      p.d_ind_maps[m] = (int *)dev_alloc(sizeof(int) * (size_t)std::max(1, p.nindirect[m]));
      io.ind_maps[m] = p.d_ind_maps[m];
    }
    int maxk = 0;
    for (int m = 0; m < ni; m++) maxk = std::max(maxk, pp.ind_k[m]);
    size_t sm2 = sizeof(int) * (size_t)maxk * p.bsize;
    allow_smem(k_block_locmaps);
    k_block_locmaps<<<dim3(nb, ni), 512, sm2, s>>>(pp, io, p.d_ind_sizes, p.d_ind_offs, tmp,
                                                   d_lines, d_lines3);
  }

  // thread colouring
  size_t sm3 = sizeof(unsigned) * pp.mask_words + sizeof(unsigned short) * (pp.ninc * p.bsize + 2) +
               sizeof(int) * p.bsize;
  if (sm3 > optin) {
    fail(-1, "op_plan error -- block size %d too large to colour kernel %s\n", p.bsize,
         p.name.c_str());
    return;
  }
  allow_smem(k_thread_colour);
  k_thread_colour<<<nb, 128, sm3, s>>>(pp, io, p.d_ind_sizes, p.d_thrcol, p.d_nthrcol);

  int *d_ncolblk = nullptr, *d_ncolors = nullptr;
  OP2B_CUDA(pool_malloc_async((void **)&d_ncolblk, sizeof(int) * nb, s));
  OP2B_CUDA(pool_malloc_async((void **)&d_ncolors, sizeof(int), s));
  OP2B_CUDA(cudaMemsetAsync(d_ncolblk, 0, sizeof(int) * nb, s));
  if (!colour_blocks(p, pp, to_sizes, d_ncolblk, d_ncolors, s))
    colour_blocks_by_targets(p, pp, to_sizes, d_ncolblk, d_ncolors, s);

  // back to the host: the small per-block tables for nshared and the byte
  // models, the colour counts for the launch loop
  std::vector<int> ind_sizes((size_t)nb * ni);
  std::vector<long long> lines((size_t)nb * ni), lines3((size_t)nb * ni);
  int ncolors = 0;
  p.nthrcol_h.assign(nb, 0);
  if (ni) {
    OP2B_CUDA(cudaMemcpyAsync(ind_sizes.data(), p.d_ind_sizes, sizeof(int) * nb * ni,
                              cudaMemcpyDeviceToHost, s));
    OP2B_CUDA(cudaMemcpyAsync(lines.data(), d_lines, sizeof(long long) * nb * ni,
                              cudaMemcpyDeviceToHost, s));
    OP2B_CUDA(cudaMemcpyAsync(lines3.data(), d_lines3, sizeof(long long) * nb * ni,
                              cudaMemcpyDeviceToHost, s));
  }
  OP2B_CUDA(cudaMemcpyAsync(p.nthrcol_h.data(), p.d_nthrcol, sizeof(int) * nb,
                            cudaMemcpyDeviceToHost, s));
  OP2B_CUDA(cudaMemcpyAsync(&ncolors, d_ncolors, sizeof(int), cudaMemcpyDeviceToHost, s));
  OP2B_CUDA(cudaStreamSynchronize(s));
  p.ncolors = ncolors;
  p.ncolblk.assign(std::max(1, ncolors), 0);
  OP2B_CUDA(cudaMemcpy(p.ncolblk.data(), d_ncolblk, sizeof(int) * std::max(1, ncolors),
                       cudaMemcpyDeviceToHost));
  p.colstart.assign(ncolors + 1, 0);
  for (int c = 0; c < ncolors; c++) p.colstart[c + 1] = p.colstart[c] + p.ncolblk[c];

  OP2B_CUDA(cudaFreeAsync(d_ncolblk, s));
  OP2B_CUDA(cudaFreeAsync(d_ncolors, s));
  OP2B_CUDA(cudaFreeAsync(tmp, s));
  OP2B_CUDA(cudaFreeAsync(d_nind, s));
  OP2B_CUDA(cudaFreeAsync(d_lines, s));
  OP2B_CUDA(cudaFreeAsync(d_lines3, s));

  // shared memory requirement (common/op_lib_core.c:972-985)
  p.nshared = 0;
  double total_shared = 0;
  for (int b = 0; b < nb; b++) {
    int nbytes = 0;
    for (int m = 0; m < ni; m++) nbytes += ROUND_UP(ind_sizes[m + (size_t)b * ni] * pp.ind_size[m]);
    p.nshared = std::max(p.nshared, nbytes);
    total_shared += nbytes;
  }
  // byte models (common/op_lib_core.c:989-1056), exact integer sums
  double t1 = 0, t2 = 0, t3 = 0;
  const double cls = pp.cls;
  for (int b = 0; b < nb; b++) {
    for (int a = 0; a < p.nargs; a++) {
      if (p.inds[a] < 0) {
        double fac = p.accs[a] == OP_READ ? 1.0 : 2.0;
        if (p.dats[a]) {
          double v = fac * nel[b] * p.dats[a]->size;
          t1 += v; t2 += v; t3 += v;
        }
      } else {
        double v = (double)nel[b] * sizeof(short);
        t1 += v; t2 += v; t3 += v;
      }
    }
    for (int m = 0; m < ni; m++) {
      int a = pp.ind_args[pp.ind_first[m]];
      double fac = p.accs[a] == OP_READ ? 1.0 : 2.0;
      double isz = ind_sizes[m + (size_t)b * ni];
      t1 += fac * isz * pp.ind_size[m];
      t2 += fac * (double)lines[m + (size_t)b * ni] * cls;
      t3 += fac * (double)lines3[m + (size_t)b * ni] * pp.ind_dim[m] * cls;
      double fac2 = p.accs[a] == OP_RW ? 2.0 : 1.0;
      t1 += fac2 * isz * sizeof(int);
      t2 += fac2 * isz * sizeof(int);
      t3 += fac2 * isz * sizeof(int);
    }
  }
  p.transfer = t1;
  p.transfer2 = t2;
  p.transfer3 = t3;
  long long tc = 0;
  for (int b = 0; b < nb; b++) {
    tc += p.nthrcol_h[b];
    p.max_thread_colours = std::max(p.max_thread_colours, p.nthrcol_h[b]);
  }
  p.avg_thread_colours = (float)tc / nb;

  if (OP_diags > 1) {
    printf(" number of blocks       = %d \n", nb);
    printf(" number of block colors = %d \n", p.ncolors);
    printf(" maximum block size     = %d \n", p.bsize);
    printf(" average thread colors  = %.2f \n", p.avg_thread_colours);
    printf(" shared memory required = %.2f KB \n", p.nshared / 1024.0f);
    printf(" average data reuse     = %.2f \n", maxbytes * (n / total_shared));
    printf(" data transfer (used)   = %.2f MB \n", p.transfer / (1024.0f * 1024.0f));
    printf(" data transfer (total)  = %.2f MB \n", p.transfer2 / (1024.0f * 1024.0f));
    printf(" SoA/AoS transfer ratio = %.2f \n\n", p.transfer3 / p.transfer2);
  }
}

static void fill_pub(DevPlan &p) {
  op_plan &o = p.pub;
  memset(&o, 0, sizeof o);
  o.name = p.name.c_str();
  o.set = p.set;
  o.nargs = p.nargs;
  o.ninds = p.ninds;
  o.part_size = p.part_size;
  o.maps = p.maps.data();
  o.dats = p.dats.data();
  o.idxs = p.idxs.data();
  o.accs = p.accs.data();
  o.nthrcol = p.d_nthrcol;
  o.thrcol = p.d_thrcol;
  o.offset = p.d_offset;
  p.pub_ind_maps = p.d_ind_maps;
  p.pub_loc_maps = p.d_loc_maps;
  o.ind_maps = p.pub_ind_maps.data();
  o.ind_offs = p.d_ind_offs;
  o.ind_sizes = p.d_ind_sizes;
  o.nindirect = p.nindirect.data();
  o.loc_maps = p.pub_loc_maps.data();
  o.nblocks = p.nblocks;
  o.nelems = p.d_nelems;
  o.ncolors = p.ncolors;
  o.ncolblk = p.ncolblk.data();
  o.blkmap = p.d_blkmap;
  o.nshared = p.nshared;
  o.transfer = (float)p.transfer;
  o.transfer2 = (float)p.transfer2;
  o.count = p.count;
}

DevPlan *get_plan(char const *name, op_set set, int part_size, int nargs, const op_arg *args,
                  int ninds, const int *inds) {
  // cache lookup (common/op_lib_core.c:632-659)
  for (auto &up : g_plans) {
    DevPlan &p = *up;
    if (p.name != name || p.set != set || p.nargs != nargs || p.ninds != ninds ||
        p.part_size != part_size)
      continue;
    bool match = true;
    for (int m = 0; m < nargs && match; m++)
      match = args[m].dat == p.dats[m] && args[m].map == p.maps[m] && args[m].idx == p.idxs[m] &&
              args[m].acc == p.accs[m];
    if (match) {
      if (OP_diags > 3) printf(" old execution plan #%d\n", (int)(&up - &g_plans[0]));
      p.count++;
      p.pub.count = p.count;
      return &p;
    }
  }
  if (OP_diags > 1) printf(" new execution plan #%d for kernel %s\n", (int)g_plans.size(), name);
  std::unique_ptr<DevPlan> up(new DevPlan());
  DevPlan &p = *up;
  p.name = name;
  p.set = set;
  p.part_size = part_size;
  p.nargs = nargs;
  p.ninds = ninds;
  for (int m = 0; m < nargs; m++) {
    p.dats.push_back(args[m].dat);
    p.maps.push_back(args[m].map);
    p.idxs.push_back(args[m].idx);
    p.accs.push_back(args[m].acc);
    p.inds.push_back(inds[m]);
  }
  p.count = 1;
  ensure_cuda();
  build_plan(p);
  if (error_pending()) return nullptr;
  fill_pub(p);
  g_plans.push_back(std::move(up));
  OP_plan_index = (int)g_plans.size();
  return g_plans.back().get();
}

void plan_unused(DevPlan *p) {
  p->count--;
  p->pub.count = p->count;
}

long validate_plan(const DevPlan &p) {
  Runtime &R = rt();
  cudaStream_t s = R.stream;
  PlanParams pp;
  std::vector<int> to_sizes;
  if (!fill_params(pp, p, to_sizes)) return 1;
  unsigned long long *err = nullptr;
  int *d_to = nullptr, *seen = nullptr;
  OP2B_CUDA(pool_malloc_async((void **)&err, sizeof(unsigned long long), s));
  OP2B_CUDA(cudaMemsetAsync(err, 0, sizeof(unsigned long long), s));
  OP2B_CUDA(pool_malloc_async((void **)&d_to, sizeof(int) * (p.ninds ? p.ninds : 1), s));
  if (p.ninds)
    OP2B_CUDA(cudaMemcpyAsync(d_to, to_sizes.data(), sizeof(int) * p.ninds,
                              cudaMemcpyHostToDevice, s));
  OP2B_CUDA(pool_malloc_async((void **)&seen, sizeof(int) * p.nblocks, s));
  OP2B_CUDA(cudaMemsetAsync(seen, 0, sizeof(int) * p.nblocks, s));
  IndOut io;
  memset(&io, 0, sizeof io);
  for (int m = 0; m < p.ninds; m++) io.ind_maps[m] = p.d_ind_maps[m];
  for (int a = 0; a < p.nargs; a++) io.loc_maps[a] = p.d_loc_maps[a];

  k_check_blocks<<<64, 256, 0, s>>>(pp, p.d_blkmap, p.d_offset, p.d_nelems, seen, err);
  if (p.ninds) {
    k_check_indmaps<<<dim3(p.nblocks, p.ninds), 256, 0, s>>>(pp, io, p.d_ind_sizes,
                                                             p.d_ind_offs, d_to, err);
    k_check_locmaps<<<592, 256, 0, s>>>(pp, io, p.d_ind_sizes, p.d_ind_offs, err);
  }
  size_t sm = sizeof(int) * (pp.mask_words ? pp.mask_words : 1);
  allow_smem(k_check_thread_colours);
  k_check_thread_colours<<<p.nblocks, 256, sm, s>>>(pp, io, p.d_ind_sizes, p.d_thrcol,
                                                    p.d_nthrcol, err);
  // block colours: one pass per colour over its blocks, owner arrays reset
  IncWork iw;
  memset(&iw, 0, sizeof iw);
  std::vector<unsigned *> owners;
  std::vector<int> ind_w(kMaxArgs, -1), osz;
  for (int sl = 0; sl < pp.ninc; sl++) {
    int m = pp.inc_ind[sl];
    if (ind_w[m] < 0) {
      unsigned *w = nullptr;
      OP2B_CUDA(pool_malloc_async((void **)&w, sizeof(int) * (size_t)to_sizes[m], s));
      ind_w[m] = (int)owners.size();
      owners.push_back(w);
      osz.push_back(to_sizes[m]);
    }
    iw.work[sl] = owners[ind_w[m]];
  }
  for (int c = 0; c < p.ncolors; c++) {
    for (size_t w = 0; w < owners.size(); w++)
      OP2B_CUDA(cudaMemsetAsync(owners[w], 0xff, sizeof(int) * (size_t)osz[w], s));
    if (pp.ninc && p.ncolblk[c] > 0)
      k_check_block_colours<<<std::min(p.ncolblk[c], 4096), 256, 0, s>>>(
          pp, iw, p.d_blkmap, p.colstart[c], p.ncolblk[c], err);
  }
  unsigned long long h = 0;
  OP2B_CUDA(cudaMemcpyAsync(&h, err, sizeof h, cudaMemcpyDeviceToHost, s));
  for (unsigned *w : owners) OP2B_CUDA(cudaFreeAsync(w, s));
  OP2B_CUDA(cudaFreeAsync(err, s));
  OP2B_CUDA(cudaFreeAsync(d_to, s));
  OP2B_CUDA(cudaFreeAsync(seen, s));
  OP2B_CUDA(cudaStreamSynchronize(s));
  // block count / colour count consistency (common/op_lib_core.c:476-492)
  long nblock = 0;
  for (int c = 0; c < p.ncolors; c++) nblock += p.ncolblk[c];
  if (nblock != p.nblocks) h++;
  return (long)h;
}

// ------------------------------------------------------------ gather plan --

struct SlotMaps {
  const int *map[kMaxArgs];
  int dim[kMaxArgs];
  int idx[kMaxArgs];
};

__global__ void k_gather_count(SlotMaps sm, int nslots, int n, int *cnt) {
  long long tot = (long long)n * nslots;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot;
       i += (long long)gridDim.x * blockDim.x) {
    int e = (int)(i / nslots), sl = (int)(i % nslots);
    int t = sm.map[sl][sm.idx[sl] + (size_t)e * sm.dim[sl]];
    atomicAdd(&cnt[t], 1);
  }
}

__global__ void k_flags(const int *cnt, int n, int *flags) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    flags[i] = cnt[i] > 0;
}

__global__ void k_compact_active(const int *cnt, const int *pos, int n, int *active,
                                 int *acnt) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (cnt[i] > 0) {
      active[pos[i]] = i;
      acnt[pos[i]] = cnt[i];
    }
}

__global__ void k_gather_scatter(SlotMaps sm, int nslots, int n, const int *slot_of_target,
                                 int *cursor, int *keys) {
  long long tot = (long long)n * nslots;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot;
       i += (long long)gridDim.x * blockDim.x) {
    int e = (int)(i / nslots), sl = (int)(i % nslots);
    int t = sm.map[sl][sm.idx[sl] + (size_t)e * sm.dim[sl]];
    int r = slot_of_target ? slot_of_target[t] : t;
    int p = atomicAdd(&cursor[r], 1);
    keys[p] = (int)i;  // i == e * nslots + sl
  }
}

// rows are short on meshes; insertion-sort each row, one thread per row,
// and leave rows longer than 64 to the CTA sorter below
__global__ void k_sort_rows(const int *row, int nrows, int *keys, int *long_rows, int *nlong,
                            int *maxlen) {
  int mx = 0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += gridDim.x * blockDim.x) {
    int a = row[r], b = row[r + 1];
    mx = max(mx, b - a);
    if (b - a > 64) {
      long_rows[atomicAdd(nlong, 1)] = r;
      continue;
    }
    for (int i = a + 1; i < b; i++) {
      int v = keys[i], j = i - 1;
      while (j >= a && keys[j] > v) {
        keys[j + 1] = keys[j];
        j--;
      }
      keys[j + 1] = v;
    }
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0 && mx > 0) atomicMax(maxlen, mx);
}

// tile_first[b] = first row r with row[r] >= kTile * b (lower bound), for
// b = 0..ntiles; row has nrows + 1 non-decreasing entries
__global__ void k_tile_first(const int *row, int nrows, int ntiles, int *tile_first) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b <= ntiles; b += gridDim.x * blockDim.x) {
    long long want = (long long)kTile * b;
    int lo = 0, hi = nrows;
    while (lo < hi) {
      int mid = (lo + hi) >> 1;
      if (row[mid] < want) lo = mid + 1; else hi = mid;
    }
    tile_first[b] = b == ntiles ? nrows : lo;
  }
}

__global__ void k_sort_long_rows(const int *row, const int *long_rows, int *keys) {
  extern __shared__ int s[];
  int r = long_rows[blockIdx.x];
  int a = row[r], len = row[r + 1] - a;
  int P = 1;
  while (P < len) P <<= 1;
  for (int i = threadIdx.x; i < P; i += blockDim.x) s[i] = i < len ? keys[a + i] : INT_MAX;
  __syncthreads();
  bitonic_sort(s, P);
  for (int i = threadIdx.x; i < len; i += blockDim.x) keys[a + i] = s[i];
}

// key = element * nslots + slot -> perm[element] * nslots + slot
__global__ void k_keys_through(int *keys, long long n, int nslots, const int *perm) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int k = keys[i];
    keys[i] = perm[k / nslots] * nslots + k % nslots;
  }
}

GatherPlan *get_gather_plan(op_set set, const op_arg *args, const std::vector<int> &slots,
                            Make make) {
  bool unsuited = false;
  for (auto &up : g_gather) {
    GatherPlan &g = *up;
    if (g.set != set || g.nslots != (int)slots.size() || g.dat != args[slots[0]].dat) continue;
    bool match = true;
    for (int k = 0; k < g.nslots && match; k++)
      match = g.maps[k] == args[slots[k]].map && g.idxs[k] == args[slots[k]].idx;
    if (match && !g.unsuited) return &g;
    unsuited = unsuited || match;
  }
  if (make == Make::kFind || (make == Make::kTry && unsuited)) return nullptr;
  Runtime &R = rt();
  cudaStream_t s = R.stream;
  std::unique_ptr<GatherPlan> up(new GatherPlan());
  GatherPlan &g = *up;
  g.set = set;
  g.dat = args[slots[0]].dat;
  g.nslots = (int)slots.size();
  g.ntarget = g.dat->set->size;
  SlotMaps sm;
  memset(&sm, 0, sizeof sm);
  if (g.nslots > kMaxArgs) {
    fail(-1, "op2b error -- too many OP_INC arguments on one dataset\n");
    return nullptr;
  }
  for (int k = 0; k < g.nslots; k++) {
    const op_arg &a = args[slots[k]];
    g.maps.push_back(a.map);
    g.idxs.push_back(a.idx);
    sm.map[k] = map_dev(a.map);
    sm.dim[k] = a.map->dim;
    sm.idx[k] = a.idx;
  }
  const int n = set->size, T = g.ntarget;
  const long long nkeys = (long long)n * g.nslots;
  int *mem = nullptr;  // scratch
  auto give_up = [&]() -> GatherPlan * {
    if (mem) OP2B_CUDA(cudaFreeAsync(mem, s));
    dev_free(g.d_active);
    dev_free(g.d_row);
    dev_free(g.d_keys);
    g.d_active = g.d_row = g.d_keys = nullptr;
    if (make == Make::kTry) {
      g.unsuited = true;
      g_gather.push_back(std::move(up));
    }
    return nullptr;
  };
  auto keep = [&](size_t ints) {
    return (int *)(make == Make::kTry ? dev_try_alloc(sizeof(int) * ints)
                                      : dev_alloc(sizeof(int) * ints));
  };
  if (nkeys > INT_MAX) {
    if (make != Make::kTry) fail(-1, "op2b error -- loop too large for 32-bit gather keys\n");
    return give_up();
  }
  // parts on 16-byte boundaries: the scans read and write four values at once
  const size_t Tz = ((size_t)T + 3) / 4 * 4;
  const cudaError_t room = pool_malloc_async((void **)&mem, sizeof(int) * (6 * Tz + 6), s);
  if (room != cudaSuccess) {
    mem = nullptr;
    cudaGetLastError();
    if (make != Make::kTry) OP2B_CUDA(room);
    return give_up();
  }
  int *cnt = mem, *flags = cnt + Tz, *pos = flags + Tz, *acnt = pos + Tz, *cursor = acnt + Tz;
  int *long_rows = cursor + Tz + 4, *nlong = long_rows + Tz, *maxlen = nlong + 1;
  OP2B_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * T, s));
  const int grid = R.num_sms * 8;
  k_gather_count<<<grid, 256, 0, s>>>(sm, g.nslots, n, cnt);
  k_flags<<<grid, 256, 0, s>>>(cnt, T, flags);
  g.nactive = (int)exclusive_scan(flags, pos, T, s);
  int *rowcnt = cnt;
  const int *slot_of_target = nullptr;
  if (g.nactive < T) {
    g.d_active = keep(std::max(1, g.nactive));
    if (!g.d_active) return give_up();
    k_compact_active<<<grid, 256, 0, s>>>(cnt, pos, T, g.d_active, acnt);
    rowcnt = acnt;
    slot_of_target = pos;
  }
  g.d_row = keep((size_t)g.nactive + 1);
  g.d_keys = keep((size_t)std::max(1LL, nkeys));
  if (!g.d_row || !g.d_keys) return give_up();
  long long total = g.nactive ? exclusive_scan(rowcnt, g.d_row, g.nactive, s) : 0;
  int tot32 = (int)total;
  OP2B_CUDA(cudaMemcpyAsync(g.d_row + g.nactive, &tot32, sizeof(int), cudaMemcpyHostToDevice, s));
  OP2B_CUDA(cudaMemcpyAsync(cursor, g.d_row, sizeof(int) * ((size_t)g.nactive + 1),
                            cudaMemcpyDeviceToDevice, s));
  k_gather_scatter<<<grid, 256, 0, s>>>(sm, g.nslots, n, slot_of_target, cursor, g.d_keys);
  // renumbered loop set: order each row by the app's element numbers (the
  // order of op_seq.h), then turn the keys back into device numbers below
  const int *to_orig = perm_new2old_dev(set), *to_dev = perm_old2new_dev(set);
  if (to_orig && nkeys)
    k_keys_through<<<grid, 256, 0, s>>>(g.d_keys, nkeys, g.nslots, to_orig);
  OP2B_CUDA(cudaMemsetAsync(nlong, 0, sizeof(int) * 2, s));
  k_sort_rows<<<grid, 256, 0, s>>>(g.d_row, g.nactive, g.d_keys, long_rows, nlong, maxlen);
  int h[2] = {0, 0};
  OP2B_CUDA(cudaMemcpyAsync(h, nlong, sizeof h, cudaMemcpyDeviceToHost, s));
  OP2B_CUDA(cudaStreamSynchronize(s));
  g.max_row = h[1];
  if (make == Make::kTry && g.max_row > kMaxSlotWidth) return give_up();
  g.nkeys = total;
  g.ntiles = (int)((total + kTile - 1) / kTile);
  g.d_tile_first = keep((size_t)g.ntiles + 1);
  if (!g.d_tile_first) return give_up();
  k_tile_first<<<(g.ntiles + 256) / 256, 256, 0, s>>>(g.d_row, g.nactive, g.ntiles, g.d_tile_first);
  if (h[0] > 0) {
    int P = 1;
    while (P < g.max_row) P <<= 1;
    if ((size_t)P * sizeof(int) > smem_optin()) {
      fail(-1, "op2b error -- a target has %d contributions, too many to order on chip\n",
           g.max_row);
      dev_free(g.d_tile_first);
      return give_up();
    }
    allow_smem(k_sort_long_rows);
    k_sort_long_rows<<<h[0], 1024, sizeof(int) * P, s>>>(g.d_row, long_rows, g.d_keys);
  }
  if (to_dev && nkeys) k_keys_through<<<grid, 256, 0, s>>>(g.d_keys, nkeys, g.nslots, to_dev);
  OP2B_CUDA(cudaFreeAsync(mem, s));
  OP2B_CUDA(cudaStreamSynchronize(s));
  g_gather.push_back(std::move(up));
  return g_gather.back().get();
}

// ------------------------------------------------------------- slot plan --

// contributions per target of plan a (cnt = row length) and then of b
__global__ void k_ell_count(int nrows, const int *active, const int *row, int *cnt) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nrows; t += gridDim.x * blockDim.x)
    cnt[active ? active[t] : t] += row[t + 1] - row[t];
}

// write plan a's entries (its CSR keys are already edge << 1 | slot), or
// plan b's ((na + key) << 1) after a's; cnt is the fill level per target
__global__ void k_ell_fill(int nrows, const int *active, const int *row, const int *keys,
                           int width, int offset, int shift, int *cnt, int *ell) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nrows; t += gridDim.x * blockDim.x) {
    const int c = active ? active[t] : t;
    const int k0 = row[t], k1 = row[t + 1], base = cnt[c];
    for (int k = k0; k < k1; k++)
      ell[(size_t)c * width + base + (k - k0)] = (offset + keys[k]) << shift;
    cnt[c] = base + k1 - k0;
  }
}

__global__ void k_max_int(const int *v, int n, int *out) {
  int m = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    m = max(m, v[i]);
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__global__ void k_fill_int(int *p, size_t n, int v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    p[i] = v;
}

// lines that the gathers of the two increments' targets touch (16-byte records,
// eight lanes together) and that the lane before does not, in a sample of
// chunks of kOrderChunk elements (chunks blockIdx.x * step)
constexpr int kOrderChunk = 1024;
// Fewer elements than these keep their order: what they read is then about what
// one SM's L1 holds.  An iteration of a scrambled mesh in coordinate order against
// its own: 2.5k cells 8.45 and 8.45 us, 5.2k 8.95 and 9.14, 10.5k (21k edges) 9.29
// and 9.48, 21k 9.99 and 11.56; making the order takes 100 us.
constexpr int kOrderLeast = 16 * kOrderChunk;
__global__ void __launch_bounds__(kOrderChunk)
    k_target_lines(int step, int n, SlotMaps sm, int *lines) {
  const int t = threadIdx.x, e = blockIdx.x * step * kOrderChunk + t;
  int k = 0;
  if (e < n)
    for (int s = 0; s < 2; s++) {
      const int *m = sm.map[s] + sm.idx[s] + (size_t)e * sm.dim[s];
      k += t % 8 == 0 || m[0] >> 3 != m[-sm.dim[s]] >> 3;
    }
  k = __reduce_add_sync(0xffffffffu, k);
  if ((t & 31) == 0) atomicAdd(lines, k);
}

static std::vector<std::unique_ptr<SlotPlan>> g_slot_plans;

SlotPlan *get_slot_plan(const GatherPlan *a, const GatherPlan *b, Make make) {
  for (auto it = g_slot_plans.begin(); it != g_slot_plans.end(); ++it) {
    SlotPlan *p = it->get();
    if (p->a != a || p->b != b) continue;
    if (make != Make::kBuild) return p->width > 0 && !p->no_room ? p : nullptr;
    if (p->width > 0 || !p->no_room) return p->width > 0 ? p : nullptr;
    g_slot_plans.erase(it);  // there was no room before
    break;
  }
  if (make == Make::kFind) return nullptr;
  std::unique_ptr<SlotPlan> up(new SlotPlan());
  SlotPlan &p = *up;
  p.a = a;
  p.b = b;
  p.ntarget = a->ntarget;
  p.na = a->set->size;
  p.nb = b ? b->set->size : 0;
  const bool shape = a->nslots == 2 && (!b || (b->nslots == 1 && b->ntarget == a->ntarget)) &&
                     (long long)p.na + p.nb + 1 < (1LL << 30);
  if (shape && a->nactive > 0) {
    cudaStream_t s = rt().stream;
    const int grid = rt().num_sms * 8;
    int *cnt = nullptr;
    const cudaError_t room =
        pool_malloc_async((void **)&cnt, sizeof(int) * ((size_t)p.ntarget + 2), s);
    if (room != cudaSuccess) {
      cudaGetLastError();
      if (make == Make::kBuild) OP2B_CUDA(room);
      p.no_room = true;
      g_slot_plans.push_back(std::move(up));
      return nullptr;
    }
    int *mx = cnt + p.ntarget;  // the longest list, the sample's lines
    OP2B_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * ((size_t)p.ntarget + 2), s));
    k_ell_count<<<grid, 256, 0, s>>>(a->nactive, a->d_active, a->d_row, cnt);
    if (b && b->nactive) k_ell_count<<<grid, 256, 0, s>>>(b->nactive, b->d_active, b->d_row, cnt);
    k_max_int<<<grid, 256, 0, s>>>(cnt, p.ntarget, mx);
    // at most 128 chunks: three quarters of the targets on a line of their own is
    // no locality (a mesh numbered along its rows has a quarter)
    SlotMaps sm;
    for (int i = 0; i < 2; i++) {
      sm.map[i] = map_dev(a->maps[i]);
      sm.dim[i] = a->maps[i]->dim;
      sm.idx[i] = a->idxs[i];
    }
    const int nchunk = (p.na + kOrderChunk - 1) / kOrderChunk, step = (nchunk + 127) / 128;
    const int nsample = (nchunk + step - 1) / step;
    if (p.na >= kOrderLeast)
      k_target_lines<<<nsample, kOrderChunk, 0, s>>>(step, p.na, sm, mx + 1);
    int wl[2] = {0, 0};
    OP2B_CUDA(cudaMemcpyAsync(wl, mx, sizeof wl, cudaMemcpyDeviceToHost, s));
    OP2B_CUDA(cudaStreamSynchronize(s));
    const int w = wl[0];
    p.scattered = 2LL * wl[1] > 3LL * std::min((long long)nsample * kOrderChunk, (long long)p.na);
    const long long nkeys = a->nkeys + (b ? b->nkeys : 0);
    if (w >= 1 && w <= kMaxSlotWidth && (long long)w * p.ntarget <= 2 * nkeys + p.ntarget) {
      p.width = w;
      const size_t n = (size_t)w * p.ntarget;
      p.d_ell = (int *)(make == Make::kTry ? dev_try_alloc(sizeof(int) * n)
                                           : dev_alloc(sizeof(int) * n));
      if (!p.d_ell) {
        p.width = 0;
        p.no_room = true;
      } else {
        k_fill_int<<<grid, 256, 0, s>>>(p.d_ell, n, (p.na + p.nb) << 1);
        OP2B_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * (size_t)p.ntarget, s));
        k_ell_fill<<<grid, 256, 0, s>>>(a->nactive, a->d_active, a->d_row, a->d_keys, w, 0, 0,
                                        cnt, p.d_ell);
        if (b && b->nactive)
          k_ell_fill<<<grid, 256, 0, s>>>(b->nactive, b->d_active, b->d_row, b->d_keys, w, p.na,
                                          1, cnt, p.d_ell);
      }
    }
    OP2B_CUDA(cudaFreeAsync(cnt, s));
    OP2B_CUDA(cudaStreamSynchronize(s));
  }
  g_slot_plans.push_back(std::move(up));
  SlotPlan *r = g_slot_plans.back().get();
  return r->width > 0 ? r : nullptr;
}

struct ColouredLoop {  // one loop of get_coloured_lists
  int bsize, nt;
  const int *blkcol, *thrcol;
};

// sort a target's entries by what a block kernel does before what else
__global__ void k_coloured_lists(int ntarget, int W, int na, int nb, const int *__restrict__ ell,
                                 const int *__restrict__ places, ColouredLoop A, ColouredLoop B,
                                 int *__restrict__ out) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ntarget; c += gridDim.x * blockDim.x) {
    // loop and block colour | strip, thread colour | entry
    unsigned hi[kMaxSlotWidth];
    unsigned long long lo[kMaxSlotWidth];
    int k[kMaxSlotWidth], n = 0;
    for (int j = 0; j < W; j++) {
      const int x = ell[(size_t)c * W + j], i = x >> 1;
      if (i >= na + nb) continue;  // padding
      const bool b = i >= na;
      const ColouredLoop &L = b ? B : A;
      const int e = b ? i - na : i, blk = e / L.bsize;
      const unsigned h = (b ? 1u << 31 : 0u) | (unsigned)L.blkcol[blk];
      const unsigned long long l =
          (unsigned long long)((e - blk * L.bsize) / L.nt) << 32 | (unsigned)L.thrcol[e] << 1 |
          (x & 1);
      int m = n++;
      const int v = places[(size_t)c * W + j];  // the same entry, where its value is
      for (; m > 0 && (hi[m - 1] > h || (hi[m - 1] == h && lo[m - 1] > l)); m--) {
        hi[m] = hi[m - 1];
        lo[m] = lo[m - 1];
        k[m] = k[m - 1];
      }
      hi[m] = h;
      lo[m] = l;
      k[m] = v;
    }
    for (int j = 0; j < W; j++)
      out[(size_t)c * W + j] =
          j < n ? (k[j] >> 1) << 2 | (j + 1 == n || hi[j + 1] != hi[j] ? 2 : 0) | (k[j] & 1) : -1;
  }
}

const int *get_coloured_lists(SlotPlan *sp, const SlotPlan::Order *o, const DevPlan *p, int nt,
                              const DevPlan *pb, int nbt) {
  for (auto &c : sp->coloured)
    if (c.o == o && c.p == p && c.pb == pb && c.nt == nt && c.nbt == nbt) return c.d_ell;
  if ((long long)sp->na + sp->nb + 1 >= (1LL << 29) || stream_capturing()) return nullptr;
  SlotPlan::Coloured c{p, pb, o, nt, nbt, nullptr};
  c.d_ell = (int *)dev_try_alloc(sizeof(int) * (size_t)sp->width * sp->ntarget);
  if (!c.d_ell) {
    sp->no_room = true;
    return nullptr;
  }
  const ColouredLoop A{p->bsize, nt, p->d_blkcol, p->d_thrcol};
  const ColouredLoop B{pb ? pb->bsize : 1, nbt, pb ? pb->d_blkcol : nullptr,
                       pb ? pb->d_thrcol : nullptr};
  k_coloured_lists<<<rt().num_sms * 8, 256, 0, rt().stream>>>(sp->ntarget, sp->width, sp->na,
                                                              sp->nb, sp->d_ell,
                                                              o ? o->d_ell : sp->d_ell, A, B,
                                                              c.d_ell);
  rt().plan_queued = true;
  sp->coloured.push_back(c);
  return c.d_ell;
}

// ------------------------------------------------------------ flux order --
// A numbering without locality makes every gather of the flux pass a sector of
// its own: 192 bytes an edge besides its 32, and each cell and node fetched for
// every edge it is on.  The nodes' coordinates then order the edges: strips of
// equal numbers of edges along the first coordinate, each by the second, so
// that a CTA's edges share cells and nodes, which L1 keeps.  The values lie in v
// in the pass's order and the lists say where: every cell still adds the same
// values in the same order.  (Coordinates are a guess -- res_calc's first
// dataset, two reals per node -- and the order is dropped when a sample of it
// is no better.)  A captured iteration of scrambled meshes: 720k FP32 cells 126 ->
// 92 us, 2.88M 674 -> 471, 405k FP64 102 -> 81.  Making it takes about 0.5 ms of
// kernels at 5.8M edges and 200 MB, whose mapping takes longer where the pool has
// not got it: flux_order says from which pass on that pays.
// A counting sort: the strips by a histogram of the first coordinate in 65,536
// steps, then one bin per strip and step of the second.  Edges of one bin lie in
// any order; the sums do not depend on it.
// Edges of a numbering with locality stay as they are.  Sorted by the distance
// between their cells inside chunks of 1024, so that a warp's lanes step through
// both cells together, they touch a tenth fewer lines, which gave 2% at 720k
// FP32 and 3 to 5% in FP64, but made a program's first iterations 6% slower.
constexpr int kCoordSteps = 65536;

// the lists with the edges' places (entry = index << 1 | negate), or lists and
// rows of the loop's order where the sample in cells (distinct cells in the new
// order, in the old) is not a quarter smaller
__global__ void k_order_lists(size_t n, int na, const int *__restrict__ ell,
                              const int *__restrict__ pos,
                              const unsigned long long *__restrict__ cells,
                              const int2 *__restrict__ edge, const int2 *__restrict__ cell,
                              int4 *__restrict__ rows, int *__restrict__ out) {
  const bool good = 4 * cells[0] < 3 * cells[1];  // as flux_orders has it
  const size_t i0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = i0; i < n; i += stride) {
    const int k = ell[i];
    out[i] = good && (k >> 1) < na ? pos[k >> 1] << 1 | (k & 1) : k;
  }
  if (good) return;
  for (size_t e = i0; e < (size_t)na; e += stride) {
    const int2 m = edge[e], c = cell[e];
    rows[e] = make_int4(m.x, m.y, c.x, c.y);
  }
}

// distinct cells on a chunk's edges
__global__ void __launch_bounds__(kOrderChunk)
    k_chunk_cells(int step, int na, const int2 *__restrict__ cell, const int4 *__restrict__ rows,
                  unsigned long long *cells) {
  __shared__ int key[2 * kOrderChunk];
  const int t = threadIdx.x, e = blockIdx.x * step * kOrderChunk + t;
  int2 c = make_int2(INT_MAX, INT_MAX);
  if (e < na) c = cell ? cell[e] : make_int2(rows[e].z, rows[e].w);
  key[t] = c.x;
  key[t + kOrderChunk] = c.y;
  __syncthreads();
  bitonic_sort(key, 2 * kOrderChunk);
  int n = 0;
  for (int i = t; i < 2 * kOrderChunk; i += kOrderChunk)
    n += __syncthreads_count(key[i] != INT_MAX && (i == 0 || key[i] != key[i - 1]));
  if (t == 0) atomicAdd(cells, (unsigned long long)n);
}

// an order of floats as unsigned integers; what is not finite counts as 0
__device__ __forceinline__ unsigned coord_key(float f) {
  const unsigned u = __float_as_uint(isfinite(f) ? f : 0.0f);
  return u >> 31 ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float coord_of(unsigned k) {
  return __uint_as_float(k >> 31 ? k & 0x7fffffffu : ~k);
}

template <class T>
__global__ void k_coord_bounds(int n, const T *__restrict__ x, unsigned *lo, unsigned *hi) {
  unsigned a[2] = {~0u, ~0u}, b[2] = {0u, 0u};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int d = 0; d < 2; d++) {
      const unsigned k = coord_key((float)x[2 * (size_t)i + d]);
      a[d] = min(a[d], k);
      b[d] = max(b[d], k);
    }
  for (int d = 0; d < 2; d++) {
    a[d] = __reduce_min_sync(0xffffffffu, a[d]);
    b[d] = __reduce_max_sync(0xffffffffu, b[d]);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(lo + d, a[d]);
      atomicMax(hi + d, b[d]);
    }
  }
}

template <class T>
__device__ __forceinline__ int coord_step(const T *x, int node, int d, const unsigned *lo,
                                          const unsigned *hi) {
  const float l = coord_of(lo[d]), h = coord_of(hi[d]);
  const float f = coord_of(coord_key((float)x[2 * (size_t)node + d]));
  const float s = h > l ? (f - l) / (h - l) * kCoordSteps : 0.0f;
  return max(0, min(kCoordSteps - 1, (int)s));
}

// steps[e]: both coordinates' steps of the edge's first node
template <class T>
__global__ void k_strip_hist(int na, const int2 *__restrict__ edge, const T *__restrict__ x,
                             const unsigned *lo, const unsigned *hi, unsigned *__restrict__ steps,
                             int *hist) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < na; e += gridDim.x * blockDim.x) {
    const int node = edge[e].x, sx = coord_step(x, node, 0, lo, hi);
    steps[e] = (unsigned)sx << 16 | (unsigned)coord_step(x, node, 1, lo, hi);
    atomicAdd(hist + sx, 1);
  }
}

// before[s]: edges whose first coordinate lies in an earlier step than s.  The
// edge's bin takes the place of its steps
__global__ void k_bin_hist(int na, int nstrip, const int *__restrict__ before, unsigned *steps,
                           int *bins) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < na; e += gridDim.x * blockDim.x) {
    const unsigned s = steps[e];
    const unsigned strip = (unsigned)((long long)before[s >> 16] * nstrip / na);
    steps[e] = strip * kCoordSteps + (s & 0xffffu);
    atomicAdd(bins + steps[e], 1);
  }
}

__global__ void k_bin_place(int na, const int2 *__restrict__ edge, const int2 *__restrict__ cell,
                            const unsigned *__restrict__ bin, int *bins, int4 *__restrict__ rows,
                            int *__restrict__ pos) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < na; e += gridDim.x * blockDim.x) {
    const int p = atomicAdd(bins + bin[e], 1);
    const int2 n = edge[e], c = cell[e];
    rows[p] = make_int4(n.x, n.y, c.x, c.y);
    pos[e] = p;
  }
}

// the coordinate order of all edges into rows and pos (queued)
template <class T>
static bool coord_order(int na, int nnode, const int2 *edge, const int2 *cell, const T *x,
                        int4 *rows, int *pos, cudaStream_t s) {
  int nstrip = 1;
  while ((long long)(nstrip + 1) * (nstrip + 1) * kOrderChunk <= na && nstrip < 1024) nstrip++;
  const size_t nbin = (size_t)nstrip * kCoordSteps;
  int *mem = nullptr;  // bounds (lo 2, hi 2) | first coordinate's histogram | bins | steps
  const size_t words = 4 + kCoordSteps + nbin + (size_t)na;
  if (pool_malloc_async((void **)&mem, sizeof(int) * words, s) != cudaSuccess) return false;
  unsigned *lo = (unsigned *)mem, *hi = lo + 2;
  int *hist = mem + 4, *bins = hist + kCoordSteps;
  unsigned *steps = (unsigned *)(bins + nbin);
  OP2B_CUDA(cudaMemsetAsync(lo, 0xff, 2 * sizeof(int), s));
  OP2B_CUDA(cudaMemsetAsync(hi, 0, sizeof(int) * (2 + kCoordSteps + nbin), s));
  const int grid = rt().num_sms * 8;
  k_coord_bounds<T><<<grid, 256, 0, s>>>(nnode, x, lo, hi);
  k_strip_hist<T><<<grid, 256, 0, s>>>(na, edge, x, lo, hi, steps, hist);
  exclusive_scan_nosync(hist, hist, kCoordSteps, s);
  k_bin_hist<<<grid, 256, 0, s>>>(na, nstrip, hist, steps, bins);
  exclusive_scan_nosync(bins, bins, (int)nbin, s);
  k_bin_place<<<grid, 256, 0, s>>>(na, edge, cell, steps, bins, rows, pos);
  OP2B_CUDA(cudaFreeAsync(mem, s));
  return true;
}

static void make_flux_order(SlotPlan *sp, SlotPlan::Order *o) {
  cudaStream_t s = rt().stream;
  const op_dat x = o->x;
  const int na = sp->na, nchunk = (na + kOrderChunk - 1) / kOrderChunk;
  const int2 *edge = reinterpret_cast<const int2 *>(map_dev(o->mx));
  const int2 *cell = reinterpret_cast<const int2 *>(map_dev(o->mq));
  const size_t nlist = (size_t)sp->width * sp->ntarget;
  o->tried = true;
  // rows | cells | lists
  o->d_rows = (int4 *)dev_try_alloc(sizeof(int4) * ((size_t)na + 1) + sizeof(int) * nlist);
  int *mem = nullptr;  // the edges' places
  bool good = o->d_rows &&
              pool_malloc_async((void **)&mem, sizeof(int) * (size_t)na, s) == cudaSuccess;
  if (good) {
    const int nnode = x->set->size;
    good = strcmp(x->type, "double") == 0
               ? coord_order(na, nnode, edge, cell, (const double *)x->data_d, o->d_rows, mem, s)
               : coord_order(na, nnode, edge, cell, (const float *)x->data_d, o->d_rows, mem, s);
  }
  if (good) {
    unsigned long long *cells = o->d_cells = (unsigned long long *)(o->d_rows + na);
    o->d_ell = (int *)(o->d_rows + na + 1);
    const int step = (nchunk + 127) / 128, nsample = (nchunk + step - 1) / step;
    OP2B_CUDA(cudaMemsetAsync(cells, 0, 2 * sizeof *cells, s));
    k_chunk_cells<<<nsample, kOrderChunk, 0, s>>>(step, na, nullptr, o->d_rows, cells);
    k_chunk_cells<<<nsample, kOrderChunk, 0, s>>>(step, na, cell, nullptr, cells + 1);
    k_order_lists<<<rt().num_sms * 8, 256, 0, s>>>(nlist, na, sp->d_ell, mem, cells, edge, cell,
                                                   o->d_rows, o->d_ell);
    rt().plan_queued = true;
  } else {
    cudaGetLastError();
    dev_free(o->d_rows);
    o->d_rows = nullptr;
  }
  if (mem) OP2B_CUDA(cudaFreeAsync(mem, s));
  if (!o->d_rows) return;
  const std::vector<SlotPlan::Coloured> had = sp->coloured;
  for (const auto &c : had)
    if (!c.o) get_coloured_lists(sp, o, c.p, c.nt, c.pb, c.nbt);
}

const SlotPlan::Order *get_flux_order(SlotPlan *sp, op_map mx, op_map mq, op_dat x,
                                      long long after) {
  if (!sp->scattered) return nullptr;
  SlotPlan::Order *o = nullptr;
  for (auto &p : sp->orders)
    if (p->mx == mx && p->mq == mq) o = p.get();
  if (o && (o->d_rows || o->tried)) return o->d_rows ? o : nullptr;
  if (after < 0 || stream_capturing()) return nullptr;
  if (!o) {
    sp->orders.emplace_back(new SlotPlan::Order());
    o = sp->orders.back().get();
    o->mx = mx;
    o->mq = mq;
  }
  o->x = x;
  if (o->passes++ < after) return nullptr;
  make_flux_order(sp, o);
  return o->d_rows ? o : nullptr;
}

int flux_orders(int *kept) {
  int n = 0, k = 0;
  if (kept) *kept = 0;
  if (stream_capturing()) return -1;
  for (auto &sp : g_slot_plans)
    for (auto &o : sp->orders) {
      if (!o->d_rows) continue;
      unsigned long long c[2] = {0, 0};
      OP2B_CUDA(cudaMemcpyAsync(c, o->d_cells, sizeof c, cudaMemcpyDeviceToHost, rt().stream));
      OP2B_CUDA(cudaStreamSynchronize(rt().stream));
      n++;
      k += 4 * c[0] < 3 * c[1];
    }
  if (kept) *kept = k;
  return n;
}

void make_flux_orders() {
  if (stream_capturing()) return;
  bool made = false;
  for (auto &sp : g_slot_plans)
    for (auto &o : sp->orders)
      if (!o->d_rows && !o->tried) {
        make_flux_order(sp.get(), o.get());
        made = true;
      }
  if (!made) return;
  // the launch behind, which would have to come after these (plan_queued), may be
  // recorded and not run: the host waits instead
  OP2B_CUDA(cudaStreamSynchronize(rt().stream));
  rt().plan_queued = false;
}

}  // namespace op2b

using namespace op2b;

void op2b_release_plans() {
  for (auto &up : g_slot_plans) {
    release_chain_sched(up.get());
    release_tile_plan(up.get());
    dev_free(up->d_ell);
    dev_free(up->d_buf);
    for (auto &c : up->coloured) dev_free(c.d_ell);
    for (auto &o : up->orders) dev_free(o->d_rows);
  }
  g_slot_plans.clear();
  for (auto &up : g_plans) {
    DevPlan &p = *up;
    dev_free(p.d_nthrcol); dev_free(p.d_thrcol); dev_free(p.d_offset); dev_free(p.d_nelems);
    dev_free(p.d_ind_offs); dev_free(p.d_ind_sizes); dev_free(p.d_blkmap);
    dev_free(p.d_blkcol);
    for (int *q : p.d_ind_maps) dev_free(q);
    for (short *q : p.d_loc_maps) dev_free(q);
  }
  g_plans.clear();
  for (auto &up : g_gather) {
    dev_free(up->d_row); dev_free(up->d_keys); dev_free(up->d_active);
    dev_free(up->d_tile_first);
    dev_free(up->d_contrib);
  }
  g_gather.clear();
  extern void op2b_release_host_plans();
  op2b_release_host_plans();
  OP_plan_index = 0;
}

// host copies made by op_plan_core: the plan and the one allocation that holds
// its arrays
struct HostPlan {
  op_plan *o;
  void *slab;
};
static std::vector<HostPlan> g_host_plans;

void op2b_release_host_plans() {
  for (HostPlan &h : g_host_plans) {
    free(h.o->ind_maps);
    free(h.o->loc_maps);
    free(h.slab);
    delete h.o;
  }
  g_host_plans.clear();
}

// One allocation for all arrays of a plan.  They are 24 MB for a mesh of 400k
// cells, which the copies would touch for the first time page by page in the
// driver (10 of the 13.5 ms of op_plan_core on a host where a fault takes
// 1.7 us): up to 8 threads touch them first, and a program that builds one
// plan after another gets memory from the heap that it has touched before,
// which separate arrays, each given back to the system, never do.
static void *plan_slab(size_t bytes) {
  char *p = (char *)malloc(bytes ? bytes : 1);
  const size_t nt = std::min<size_t>(8, std::max(1u, std::thread::hardware_concurrency()));
  if (!p || bytes < ((size_t)4 << 20) || nt < 2) return p;
  on_threads(nt, [p, bytes, nt](size_t t) {
    for (size_t i = bytes / nt * t; i < bytes / nt * (t + 1); i += 4096)
      static_cast<volatile char *>(p)[i] = 0;
  });
  return p;
}

extern "C" {

int op2b_flux_orders(int *kept) {
  op2b::flush_pending();
  if (kept) *kept = 0;
  return rt().cuda_ready ? flux_orders(kept) : 0;
}

op_plan *op_plan_get(char const *name, op_set set, int part_size, int nargs, op_arg *args,
                     int ninds, int *inds) {
  DevPlan *p = get_plan(name, set, part_size, nargs, args, ninds, inds);
  return p ? &p->pub : nullptr;
}

// common/op_lib_core.c:627: the same plan, with every array in host memory
op_plan *op_plan_core(char const *name, op_set set, int part_size, int nargs, op_arg *args,
                      int ninds, int *inds) {
  DevPlan *p = get_plan(name, set, part_size, nargs, args, ninds, inds);
  if (!p) return nullptr;
  for (HostPlan &h : g_host_plans)
    if (h.o->name == p->pub.name && h.o->set == set && h.o->part_size == part_size &&
        h.o->dats == p->pub.dats) {
      h.o->count = p->count;
      return h.o;
    }
  cudaStream_t s = rt().stream;
  const int nb = p->nblocks, n = set->size, ni = p->ninds;
  std::unique_ptr<op_plan> o(new op_plan(p->pub));
  // every array's place in the slab, then the copies
  struct Part {
    void **host;
    const void *dev;
    size_t bytes, at;
  };
  std::vector<Part> parts;
  size_t total = 0;
  auto part = [&](void **host, const void *dev, size_t bytes) {
    parts.push_back(Part{host, dev, bytes, total});
    total += (bytes + 63) & ~(size_t)63;
  };
  const size_t word = sizeof(int);
  o->ind_maps = (int **)calloc(ni ? ni : 1, sizeof(int *));
  o->loc_maps = (short **)calloc(p->nargs ? p->nargs : 1, sizeof(short *));
  part((void **)&o->nthrcol, p->d_nthrcol, word * nb);
  part((void **)&o->thrcol, p->d_thrcol, word * (size_t)n);
  part((void **)&o->offset, p->d_offset, word * nb);
  part((void **)&o->nelems, p->d_nelems, word * nb);
  part((void **)&o->ind_offs, p->d_ind_offs, word * (size_t)nb * ni);
  part((void **)&o->ind_sizes, p->d_ind_sizes, word * (size_t)nb * ni);
  part((void **)&o->blkmap, p->d_blkmap, word * nb);
  for (int m = 0; m < ni; m++)
    part((void **)&o->ind_maps[m], p->d_ind_maps[m], word * (size_t)p->nindirect[m]);
  for (int a = 0; a < p->nargs; a++)
    if (p->d_loc_maps[a])
      part((void **)&o->loc_maps[a], p->d_loc_maps[a], sizeof(short) * (size_t)n);
  part((void **)&o->nindirect, nullptr, word * (size_t)std::max(1, ni));
  part((void **)&o->ncolblk, nullptr, word * (size_t)std::max(1, p->ncolors));
  char *slab = (char *)plan_slab(total);
  if (!slab || !o->ind_maps || !o->loc_maps) {
    free(slab);
    free(o->ind_maps);
    free(o->loc_maps);
    fail(-1, "op_plan_core error -- cannot allocate %zu bytes for the plan of %s\n", total, name);
    return nullptr;
  }
  for (Part &q : parts) {
    *q.host = slab + q.at;
    if (q.dev && q.bytes)
      OP2B_CUDA(cudaMemcpyAsync(slab + q.at, q.dev, q.bytes, cudaMemcpyDeviceToHost, s));
  }
  for (int m = 0; m < ni; m++) o->nindirect[m] = p->nindirect[m];
  for (int c = 0; c < p->ncolors; c++) o->ncolblk[c] = p->ncolblk[c];
  OP2B_CUDA(cudaStreamSynchronize(s));
  g_host_plans.push_back(HostPlan{o.get(), slab});
  return o.release();
}

long op2b_plan_validate(char const *name, op_set set, int part_size, int nargs, op_arg *args,
                        int ninds, int *inds) {
  DevPlan *p = get_plan(name, set, part_size, nargs, args, ninds, inds);
  if (!p) return -1;
  return validate_plan(*p);
}

}  // extern "C"
