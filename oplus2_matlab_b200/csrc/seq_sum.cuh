// seq_sum.cuh -- (((init + v[0]) + v[1]) + ...) + v[n-1] in floating point,
// one rounding per addition in element order as op_seq.h adds, in parallel.
//
// Rounded addition is not associative, but inside one binade of the running
// sum it is integer arithmetic: with s = S * ulp, 2^MANT <= S < 2^(MANT+1),
// adding x >= 0 gives S + floor(x/ulp), plus one when the rest is above half
// an ulp, or is exactly half and the result would be odd.  What one element
// adds thus depends on s only through its binade and the parity of S, and a
// run of elements is a pair (d0, d1): what it adds to an even and to an odd
// S.  Pairs compose associatively, so they are scanned in parallel; a run is
// valid as long as S stays below 2^(MANT+1) at its end (S never falls).  The
// few elements at which the sum enters the next binade are added natively.
// The first (subnormal) binade has the ulp of the second, so zero and
// subnormal sums need no case of their own.
//
// Two launches: k_seq_tile_sums sums every tile of kSeqTile values in
// double; k_seq_fold predicts from those sums the binade the running sum has
// at each tile, reduces the tile and each run of kSeqRun values in it to
// pairs, in that binade and the next, and one warp of its last CTA walks the
// tiles in order, 32 pairs a step.  Where the sum enters the next binade it
// walks the tile's runs, adds the values of the run in question natively and
// goes on in the other pairs.  A run that has no pair for the sum's binade
// is added natively too; a negative value, an infinity or a negative running
// sum ends the walk and the rest is added one by one.  The result is the
// serial sum's, bit for bit, for every input.
//
// Bound: the walk's dependent steps (1-1.5 us for each of some 15 to 25 binade
// changes of airfoil's rms) and reading the values twice.  720k values (180k
// cells): 3.8 ms added one after another by one warp, about 50 us so (FP64
// about 90: 64-bit pairs, which spill at the 64 registers of 1024 threads).
#pragma once

#include <cuda_runtime.h>

#include <cstring>

namespace op2b {

constexpr int kSeqThreads = 1024;
constexpr int kSeqPer = 4;  // consecutive values per thread
constexpr int kSeqTile = kSeqThreads * kSeqPer;
constexpr int kSeqRun = 32 * kSeqPer;         // the values of a warp
constexpr int kSeqRuns = kSeqTile / kSeqRun;  // per tile
constexpr int kSeqPage = 1024;  // tiles whose pairs the walk finds in shared memory
constexpr int kSeqHead = 8 * kSeqRun;  // added natively first: the binade changes often there
static_assert(kSeqRuns == 32, "one lane per run");

template <class T>
struct SeqBits;
template <>
struct SeqBits<float> {
  typedef unsigned U;
  typedef int D;
  static constexpr int MANT = 23, EMAX = 255;
  static constexpr D BIG = 1 << 28;
};
template <>
struct SeqBits<double> {
  typedef unsigned long long U;
  typedef long long D;
  static constexpr int MANT = 52, EMAX = 2047;
  static constexpr D BIG = 1LL << 60;
};

template <class T>
struct SeqPair {
  typename SeqBits<T>::D d0, d1;
};

// a tile or a run: its pair in the binade predicted for the tile, and in the
// next
template <class T>
struct SeqTwo {
  SeqPair<T> p[2];
};

template <class T>
__host__ __device__ __forceinline__ typename SeqBits<T>::U seq_bits(T x) {
  typename SeqBits<T>::U u;
  memcpy(&u, &x, sizeof u);
  return u;
}

// s = S * ulp of binade E; false for a set sign bit, an infinity or a NaN
template <class T>
__host__ __device__ __forceinline__ bool seq_split(T s, int &E, typename SeqBits<T>::D &S) {
  typedef SeqBits<T> B;
  const typename B::U u = seq_bits(s), one = 1;
  if (u >> (8 * sizeof(T) - 1)) return false;
  const int e = (int)(u >> B::MANT);
  if (e == B::EMAX) return false;
  S = (typename B::D)(u & ((one << B::MANT) - 1)) + (e ? (typename B::D)(one << B::MANT) : 0);
  E = e ? e : 1;
  return true;
}

template <class T>
__host__ __device__ __forceinline__ T seq_join(int E, typename SeqBits<T>::D S) {
  const typename SeqBits<T>::U u =
      ((typename SeqBits<T>::U)(E - 1) << SeqBits<T>::MANT) + (typename SeqBits<T>::U)S;
  T x;
  memcpy(&x, &u, sizeof x);
  return x;
}

// the pair p followed by the value x, for sums in binade E
template <class T>
__host__ __device__ __forceinline__ void seq_add(SeqPair<T> &p, T x, int E) {
  typedef SeqBits<T> B;
  typedef typename B::U U;
  typedef typename B::D D;
  const U u = seq_bits(x), one = 1;
  D m;
  int e;
  if (!seq_split(x, e, m)) {
    if ((u << 1) == 0) return;  // -0 adds nothing to a sum that is not negative
    p.d0 = p.d1 = B::BIG;
    return;
  }
  const int sh = E - e;
  D fl = 0, up = 0;
  bool tie = false;
  if (sh <= 0) {
    fl = sh < -1 ? B::BIG : m << -sh;  // a normal m shifted by two ends the binade
  } else if (sh <= B::MANT + 1) {
    fl = m >> sh;
    const U rest = (U)m & ((one << sh) - 1), half = one << (sh - 1);
    up = rest > half;
    tie = rest == half;
  }
  const D a0 = fl + (tie ? ((p.d0 + fl) & 1) : up);
  const D a1 = fl + (tie ? ((p.d1 + 1 + fl) & 1) : up);
  p.d0 = p.d0 + a0 < B::BIG ? p.d0 + a0 : B::BIG;
  p.d1 = p.d1 + a1 < B::BIG ? p.d1 + a1 : B::BIG;
}

// run a followed by run b
template <class T>
__host__ __device__ __forceinline__ SeqPair<T> seq_then(SeqPair<T> a, SeqPair<T> b) {
  typedef typename SeqBits<T>::D D;
  const D x = a.d0 + ((a.d0 & 1) ? b.d1 : b.d0), y = a.d1 + ((a.d1 & 1) ? b.d0 : b.d1);
  return SeqPair<T>{x < SeqBits<T>::BIG ? x : SeqBits<T>::BIG,
                    y < SeqBits<T>::BIG ? y : SeqBits<T>::BIG};
}

// the values of the sum: value j is v[j], or, for a renumbered set,
// component j % w of the element the app numbers j / w, stored at
// order[j / w]
template <class T>
struct SeqVals {
  const T *v;
  long long n;
  const int *order;
  int w;
};

#ifdef __CUDACC__

template <class T>
__device__ __forceinline__ T seq_at(const SeqVals<T> &a, long long j) {
  return a.order ? a.v[(long long)a.w * a.order[j / a.w] + j % a.w] : a.v[j];
}

// this thread's values of tile t, zeros past the end (v is 256-byte aligned
// and a thread's values are 16 or 32 bytes of it)
template <class T>
__device__ __forceinline__ void seq_load(const SeqVals<T> &a, int t, T (&x)[kSeqPer]) {
  const long long j = (long long)t * kSeqTile + threadIdx.x * kSeqPer;
  if (!a.order && j + kSeqPer <= a.n) {
    const int4 *p = reinterpret_cast<const int4 *>(a.v + j);
    int4 w[sizeof(x) / sizeof(int4)];
#pragma unroll
    for (int k = 0; k < (int)(sizeof(x) / sizeof(int4)); k++) w[k] = __ldg(p + k);
    memcpy(x, w, sizeof x);
  } else {
#pragma unroll
    for (int k = 0; k < kSeqPer; k++) x[k] = j + k < a.n ? seq_at(a, j + k) : T(0);
  }
}

template <class T>
__device__ __forceinline__ SeqPair<T> seq_shfl_up(SeqPair<T> p, int o) {
  return SeqPair<T>{__shfl_up_sync(0xffffffffu, p.d0, o), __shfl_up_sync(0xffffffffu, p.d1, o)};
}

// inclusive scan of the lanes' pairs in lane order
template <class T>
__device__ __forceinline__ SeqPair<T> seq_warp_scan(SeqPair<T> p) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const SeqPair<T> q = seq_shfl_up(p, o);
    if (lane >= o) p = seq_then(q, p);
  }
  return p;
}

__device__ __forceinline__ double seq_block_sum(double x, double *ws) {
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = x;
  __syncthreads();
  double y = 0;
  for (int w = 0; w < kSeqThreads / 32; w++) y += ws[w];
  return y;
}

template <class T>
__global__ void __launch_bounds__(kSeqThreads) k_seq_tile_sums(SeqVals<T> a, double *tsum) {
  __shared__ double ws[kSeqThreads / 32];
  pdl_wait();
  pdl_trigger();
  T x[kSeqPer];
  seq_load(a, blockIdx.x, x);
  double d = 0;
#pragma unroll
  for (int k = 0; k < kSeqPer; k++) d += (double)x[k];
  d = seq_block_sum(d, ws);
  if (threadIdx.x == 0) tsum[blockIdx.x] = d;
}

// as many leading lanes' pairs as keep the sum S of binade E inside it
// (a lane past `n` adds nothing); S moves over them
template <class T>
__device__ __forceinline__ int seq_step(const SeqPair<T> &lanes, typename SeqBits<T>::D &S) {
  typedef typename SeqBits<T>::D D;
  constexpr D LIM = (D)2 << SeqBits<T>::MANT;
  const SeqPair<T> p = seq_warp_scan(lanes);
  const D d = (S & 1) ? p.d1 : p.d0;
  const unsigned over = __ballot_sync(0xffffffffu, S + d >= LIM);
  const int good = over ? __ffs(over) - 1 : 32;
  const D step = __shfl_sync(0xffffffffu, d, good > 0 ? good - 1 : 0);
  if (good > 0) S += step;
  return good;
}

// s + x[0] + ... + x[m - 1] in order, by one thread (x: shared memory, 16-byte
// aligned); the next 16 values are on their way while 16 are added
template <class T>
__device__ __forceinline__ T seq_native(T s, const T *x, int m) {
  constexpr int NV = 16 * (int)sizeof(T) / 16;
  auto load = [&](int k, T(&y)[16]) {
    int4 w[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) w[i] = reinterpret_cast<const int4 *>(x + k)[i];
    memcpy(y, w, sizeof y);
  };
  T y[16], next[16];
  int k = 0;
  if (m >= 16) load(0, next);
  for (; k + 16 <= m; k += 16) {
#pragma unroll
    for (int i = 0; i < 16; i++) y[i] = next[i];
    if (k + 32 <= m) load(k + 16, next);
#pragma unroll
    for (int i = 0; i < 16; i++) s = s + y[i];
  }
  for (; k < m; k++) s = s + x[k];
  return s;
}

template <class T>
__global__ void __launch_bounds__(kSeqThreads)
    k_seq_fold(SeqVals<T> a, T init, int ntile, const double *__restrict__ tsum, SeqTwo<T> *tiles,
               SeqTwo<T> *runs, int *binade, unsigned *ticket, T *out, unsigned *flag,
               unsigned flag_seq) {
  typedef SeqBits<T> B;
  typedef typename B::D D;
  __shared__ double ws[kSeqThreads / 32];
  __shared__ SeqTwo<T> page[kSeqPage];
  __shared__ int pbin[kSeqPage];
  __shared__ __align__(16) T vals[kSeqHead];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31;
  T x[kSeqPer];
  pdl_wait();
  pdl_trigger();
  // ---- this CTA's tile and runs as pairs.  The binade is that of a sum
  // 1.5% below the one of the tile sums, so that the two cover the rounding
  // the serial sum may have gathered either way
  {
    seq_load(a, blockIdx.x, x);
    double d = 0;
    for (int t = tid; t < (int)blockIdx.x; t += kSeqThreads) d += tsum[t];
    d = seq_block_sum(d, ws) + (double)init;
    int E = 0;
    D S;
    if (!seq_split((T)(d * 0.985), E, S)) E = 0;  // no pairs: the walk adds natively
    SeqTwo<T> r;
#pragma unroll
    for (int b = 0; b < 2; b++) {
      SeqPair<T> p{0, 0};
      if (E)
#pragma unroll
        for (int k = 0; k < kSeqPer; k++) seq_add(p, x[k], E + b);
      r.p[b] = seq_warp_scan(p);
    }
    if (lane == 31) {
      runs[(size_t)blockIdx.x * kSeqRuns + (tid >> 5)] = r;
      page[tid >> 5] = r;
      __threadfence();
    }
    __syncthreads();
    if (tid < 32) {
      r.p[0] = seq_warp_scan(page[tid].p[0]);
      r.p[1] = seq_warp_scan(page[tid].p[1]);
      if (tid == 31) {
        tiles[blockIdx.x] = r;
        binade[blockIdx.x] = E;
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
      }
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // ---- the last CTA: the head's values and the tiles' pairs into shared
  // memory, then one warp walks
  if (tid < kSeqPage && tid < ntile) {
#pragma unroll
    for (int b = 0; b < 2; b++)
      page[tid].p[b] =
          SeqPair<T>{__ldcg(&tiles[tid].p[b].d0), __ldcg(&tiles[tid].p[b].d1)};
    pbin[tid] = __ldcg(binade + tid);
  }
  seq_load(a, 0, x);
#pragma unroll
  for (int k = 0; k < kSeqPer; k++)
    if (tid * kSeqPer + k < kSeqHead) vals[tid * kSeqPer + k] = x[k];
  __syncthreads();
  if (tid >= 32) return;
  auto pick = [](const SeqTwo<T> &r, int b, int E) {
    return b && E == b ? r.p[0] : b && E == b + 1 ? r.p[1] : SeqPair<T>{B::BIG, B::BIG};
  };
  auto global = [&](const SeqTwo<T> *r) {
    SeqTwo<T> y;
#pragma unroll
    for (int b = 0; b < 2; b++)
      y.p[b] = SeqPair<T>{__ldcg(&r->p[b].d0), __ldcg(&r->p[b].d1)};
    return y;
  };
  // values of run `r` of tile t, 4 per lane
  auto load_run = [&](int t, int r, T(&y)[kSeqPer]) {
    const long long j = (long long)t * kSeqTile + r * kSeqRun + lane * kSeqPer;
#pragma unroll
    for (int k = 0; k < kSeqPer; k++) y[k] = j + k < a.n ? seq_at(a, j + k) : T(0);
  };
  auto add_run = [&](T s, const T(&y)[kSeqPer]) {  // by lane 0, for all lanes
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kSeqPer; k++) vals[lane * kSeqPer + k] = y[k];
    __syncwarp();
    if (lane == 0) s = seq_native(s, vals, kSeqRun);
    return __shfl_sync(0xffffffffu, s, 0);
  };
  T s = init;
  if (lane == 0) s = seq_native(s, vals, (int)(a.n < kSeqHead ? a.n : kSeqHead));
  s = __shfl_sync(0xffffffffu, s, 0);
  int t = 0, run = kSeqHead / kSeqRun, E;  // the values before run `run` of tile t are in s
  D S;
  bool plain = true;
  while (t < ntile && (plain = seq_split(s, E, S))) {
    if (run == 0) {  // whole tiles
      int good = 32;
      while (t < ntile && good == 32) {
        const int k = t + lane;
        SeqPair<T> p{0, 0};
        if (k < ntile) {
          if (k < kSeqPage) p = pick(page[k], pbin[k], E);
          else p = pick(global(tiles + k), __ldcg(binade + k), E);
        }
        good = seq_step<T>(p, S);
        t += good;
      }
      s = seq_join<T>(E, S);
      if (t >= ntile) break;
    }
    // tile t by runs, up to one that has to be added natively
    const int b = t < kSeqPage ? pbin[t] : __ldcg(binade + t);
    const SeqTwo<T> r = global(runs + (size_t)t * kSeqRuns + lane);
    while (run < kSeqRuns && (plain = seq_split(s, E, S))) {
      const int good = seq_step<T>(lane < run ? SeqPair<T>{0, 0} : pick(r, b, E), S);
      s = seq_join<T>(E, S);
      if (good < kSeqRuns) {
        T y[kSeqPer];
        load_run(t, good, y);
        s = add_run(s, y);
      }
      run = good + 1;
    }
    if (run < kSeqRuns) break;  // not plain
    run = 0;
    t++;
  }
  if (!plain && s == s) {  // a NaN stays one; else one by one from run `run` of tile t
    T y[kSeqPer], next[kSeqPer];
    load_run(t, run, next);
    while (t < ntile) {
#pragma unroll
      for (int k = 0; k < kSeqPer; k++) y[k] = next[k];
      if (++run == kSeqRuns) {
        run = 0;
        t++;
      }
      load_run(t, run, next);  // zeros past the end
      s = add_run(s, y);
    }
  }
  if (lane == 0) {
    *out = s;
    *ticket = 0u;
    if (flag) {  // the host polls it: 2 to 2.5 us sooner than an event after the kernel
      __threadfence_system();
      *reinterpret_cast<volatile unsigned *>(flag) = flag_seq;
    }
  }
}

#endif

}  // namespace op2b
