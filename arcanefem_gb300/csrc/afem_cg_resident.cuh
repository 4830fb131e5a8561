// Conjugate gradients in one launch, for systems whose vectors fit the
// register files: a cooperative grid of at most one block per SM, every
// thread owning up to K rows for the whole solve.
//
// What bounds the launches per iteration of the general path is not the work
// but the gaps: at 66 k rows an iteration took 17.4 us in three kernels,
// against 1.9 us of FP64 issue.  Here
//   * x, r, D^-1, p, q of a thread's rows stay in registers (for K > 4 only
//     r, D^-1 and q do), so that an iteration's vector updates move nothing;
//   * the matrix sits in shared memory as 32-row slices, as many of a block's
//     as fit (12 B an entry: 2.8 M entries on the chip); the others are read
//     from the sliced copy in global memory, or from the CSR rows;
//   * only the direction (FP64) or z (FP32) goes through global memory, since
//     other blocks gather it;
//   * the blocks meet in all-to-all exchanges: a block publishes its partial
//     sum and the exchange's number in one 16-byte slot, and each block polls
//     all slots and adds them.  Every block takes the same decisions, results
//     are deterministic, and no exchange pays an atomic's queue or a second
//     trip for a flag;
//   * the sums are made in fixed point (below): in FP64 each of an iteration's
//     two sums is a chain of 20 dependent additions and a division, 3700 of an
//     iteration's 19900 cycles (256^2 triangles; 9.7 -> 8.6 ms a solve).
// Every poll is bounded; one that runs out sets *err and ends all blocks.  (A
// system small enough for one cluster of blocks has no polls: it meets at the
// hardware's cluster barrier, Grid with CL.)
#pragma once
#include "afem_krylov.cuh"

namespace afem {

// Of the failure-detection test (kernels with TEST): how long a poll goes on, and the block that leaves before its
// first exchange.  A limit at run time in the solves themselves cost 2 % at 256^2 triangles and 5 % at 40^3 elasticity.
struct ResWaits {
  int spins, stall;
};
template <class Args>
struct WithWaits : Args {
  ResWaits waits;
};
template <bool TEST, class Args>
using ResArgs = std::conditional_t<TEST, WithWaits<Args>, Args>;

struct CgState {
  double rz, rr, pq, alpha, beta, bnorm2, tol2, pad0;
  int done, iter, status, max_iter;
  unsigned int ticket[4];
};

constexpr int kResThreads = 512;
constexpr int kResWarps = kResThreads / 32;
constexpr int kResMaxRows = 6;                 // rows a thread owns at most
constexpr int kResSpins = 4000000;             // polls of a wait, about 2 s
constexpr int kResCluster = 8;                 // blocks of a system small enough for one cluster
constexpr int kResGrid = 256;                   // blocks at most
constexpr int kSlotBuffers = 4;                // exchanges whose slots are kept apart
constexpr int kSlotStride = 8;                  // slots of 16 B a cache line of its own apart
constexpr size_t kResSmem = 226 * 1024;        // dynamic shared memory of a block

// Sums in fixed point.  Each partial sum becomes a 96-bit integer in units of
// 2^(E - 69), E the exponent of the sum's last value, in five 22-bit limbs that
// a warp adds in one instruction each (redux); integers add exactly, so the
// order does not matter, and the total is rounded once.  Its error is that of
// the conversions, half a unit a thread, against an FP64 tree's half ulp of
// the running sums.  A partial sum of 2^(E + 9) or more (or not finite), or a
// total below 2^(E - 4), sends that exchange to FP64 sums; so does a missing E.
constexpr int kLimbs = 5, kLimbBits = 22;
constexpr int kNoExponent = 1 << 20;

__device__ __forceinline__ int sum_exponent(double total) {
  const int e = (__double2hiint(total) >> 20 & 0x7ff) - 1023;
  return abs(e) <= 900 ? e : kNoExponent;
}

// e: biased as a double's, m: significand of up to 53 bits, 0 for a zero, s: 0 or -1
__device__ __forceinline__ bool to_limbs(int e, unsigned long long m, int s, int E, int (&l)[kLimbs]) {
  int p = e - E - 1006;   // place of the significand's last bit
  if (p < 0) {
    m = p > -54 ? (m + (1ull << (-p - 1))) >> -p : 0ull;
    p = 0;
  }
  const bool ok = e - 1023 - E <= 8;
  if (!ok) p = 0;
  const unsigned long long lo = m << p, hi = p ? m >> (64 - p) : 0ull;
  constexpr int mask = (1 << kLimbBits) - 1;
  const int u[kLimbs] = {(int)lo & mask, (int)(lo >> 22) & mask, (int)(lo >> 44 | hi << 20) & mask, (int)(hi >> 2) & mask,
                         (int)(hi >> 24)};
#pragma unroll
  for (int k = 0; k < kLimbs; ++k) l[k] = (u[k] ^ s) - s;
  return ok;
}
__device__ __forceinline__ bool to_limbs(double v, int E, int (&l)[kLimbs]) {
  const int h = __double2hiint(v), e = h >> 20 & 0x7ff;
  const unsigned long long m = (unsigned long long)((h & 0xfffff) | 0x100000) << 32 | (unsigned)__double2loint(v);
  return to_limbs(e, e ? m : 0ull, h >> 31, E, l);
}
// Subnormal numbers take part: an FP32 sum of tiny terms is made of them long before its total leaves FP32's range.
__device__ __forceinline__ bool to_limbs(float v, int E, int (&l)[kLimbs]) {
  const int b = __float_as_int(v), e = b >> 23 & 0xff;
  const unsigned long long m = (unsigned long long)((b & 0x7fffff) | (e ? 0x800000 : 0)) << 29;
  return to_limbs(e == 255 ? 2047 : max(e, 1) + 896, m, b >> 31, E, l);
}

__device__ __forceinline__ __int128 from_limbs(const int (&l)[kLimbs]) {
  return (__int128)((long long)l[0] + ((long long)l[1] << 22)) +
         ((__int128)((long long)l[2] + ((long long)l[3] << 22)) << 44) + ((__int128)l[4] << 88);
}

__device__ __forceinline__ double fixed_to_double(__int128 t, int E) {
  if (t == 0) return 0.0;
  const bool neg = t < 0;
  unsigned __int128 m = neg ? -(unsigned __int128)t : (unsigned __int128)t;
  const unsigned long long top = (unsigned long long)(m >> 64);
  const int z = top ? __clzll((long long)top) : 64 + __clzll((long long)(unsigned long long)m);
  m <<= z;
  const unsigned long long lead = (unsigned long long)(m >> 64) | ((unsigned long long)m != 0);   // sticky
  const double d = __ull2double_rn(lead);   // exponent 63 or 64
  const int h = (__double2hiint(d) + (64 - z + E - 69) * (1 << 20)) | (neg ? (int)0x80000000 : 0);
  return __hiloint2double(h, __double2loint(d));
}

// Block sums of V values a thread in FP64; value v's ends in the lanes of warp v.
// GB300 takes as long for a warp's FP64 instruction however many lanes take
// part, so the sums go through shared memory with full warps first.
template <int V, class T>
__device__ __forceinline__ double res_block_sum(const T (&v)[V], double* sh) {
  constexpr int B = kResThreads, W = 128 / V;   // four warps add, 128 / V threads per value
  const int t = threadIdx.x;
#pragma unroll
  for (int j = 0; j < V; ++j) sh[j * B + t] = (double)v[j];
  __syncthreads();
  double s = 0.0;
  if (t < 128) {
    const double* p = sh + (t / W) * B + t % W;
    s = p[0];
#pragma unroll
    for (int m = 1; m < B / W; ++m) s += p[m * W];
  }
  __syncthreads();
  if (t < 128) sh[t] = s;
  __syncthreads();
  if (t < 32 * V) {
    const double* p = sh + (t >> 5) * W + (t & 31);
    s = p[0];
#pragma unroll
    for (int m = 1; m < W / 32; ++m) s += p[m * 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  __syncthreads();   // meet() writes sh
  return s;
}

// The blocks' exchanges.  A sum's exchange waits for every block, a barrier
// only for the blocks whose rows this one gathers, and no two barriers follow
// each other: a block can be two exchanges ahead of another's polling, never
// three, so slots are kept apart for four.  FENCE:
// what the block's threads wrote before is visible to every block afterwards
// (a release before the put, an acquire after the polls).
// CL: the grid is one cluster.  Every warp then writes its sum into every
// block's shared memory (by way of a block's sum 45^2 triangles took 1.17 ms,
// now 1.09) and the cluster's barrier stands for the polls and the fences (an
// exchange through L2 takes 1400 to 2500 cycles among 5 blocks; res_plan has
// the solves' times).  That barrier needs no bound: every block takes the same
// branches, decided from the same totals.
template <bool CL, bool TEST>
struct Grid {
  ulonglong2* slots;          // [4 exchanges][2 values][gridDim.x] lines, zero at the launch; CL: shared, [2][2][8][16]
  double* sh;                 // shared, res_scratch(gridDim.x) doubles
  int* err;
  int spins;                  // polls of a wait in a TEST
  unsigned long long epoch = 0;

  // CL: {lo, hi} as the slot `sub` of value w of this block in every block of the cluster, lane i in block i
  __device__ __forceinline__ void spread(int w, int sub, unsigned long long lo, unsigned long long hi) {
    const unsigned lane = threadIdx.x & 31;
    if (lane < gridDim.x) {
      const unsigned at = (unsigned)__cvta_generic_to_shared(
          slots + (((epoch & 1) * 2 + w) * kResCluster + blockIdx.x) * kResWarps + sub);
      asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\t"
                   "st.shared::cluster.v2.u64 [a], {%2, %3};\n\t}"
                   :: "r"(at), "r"(lane), "l"(lo), "l"(hi) : "memory");
    }
  }
  // slot i of value w, counted over the blocks' kResWarps each
  __device__ __forceinline__ ulonglong2 spread_slot(int w, int i) const {
    const volatile unsigned long long* q = reinterpret_cast<const volatile unsigned long long*>(
        slots + ((epoch & 1) * 2 + w) * kResCluster * kResWarps + i);
    return make_ulonglong2(q[0], q[1]);
  }

  // Publish the values that threads 0 (and 32 for the second) of the block hold, poll everyone's into sh.
  // Returns false in every thread if a wait ran out.  Ends with a block barrier.
  template <int V>
  __device__ __forceinline__ bool meet(double v) {
    ++epoch;
    const int nb = gridDim.x;
    if constexpr (CL) {   // every lane of warp j holds value j
      const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
      if (w < V) spread(w, 0, __double_as_longlong(v), 0);
      cluster_sync();
      if (w < V && lane < nb) sh[w * nb + lane] = __longlong_as_double(spread_slot(w, lane * kResWarps).x);
      __syncthreads();
      return true;
    }
    ulonglong2* at = slots + (epoch % kSlotBuffers) * 2 * nb * kSlotStride;
    if (threadIdx.x < 32 * V && (threadIdx.x & 31) == 0)
      slot_put(at + ((threadIdx.x >> 5) * nb + blockIdx.x) * kSlotStride, __double_as_longlong(v), epoch);
    int bad = 0;
    for (int i = threadIdx.x; i < V * nb; i += kResThreads) {
      ulonglong2 s;
      if (!poll(at + i * kSlotStride, &s)) bad = 1;
      sh[i] = __longlong_as_double(s.x);
    }
    return __syncthreads_or(bad) == 0;
  }

  // What the blocks marked in `need` wrote before is visible to this one after.  Waiting for these alone instead of
  // all of them: 256^2 triangles 8.63 -> 8.13 ms, 600^2 41.8 -> 40.5; no change for a shuffled numbering, which
  // marks every block.
  __device__ __forceinline__ bool barrier(const uint8_t* need) {
    if constexpr (CL) {
      cluster_sync();
      return true;
    }
    ++epoch;
    const int nb = gridDim.x;
    ulonglong2* at = slots + (epoch % kSlotBuffers) * 2 * nb * kSlotStride;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      slot_put(at + blockIdx.x * kSlotStride, 0, epoch);
    }
    int bad = 0;
    if (threadIdx.x < nb && need[threadIdx.x]) {   // the pollers acquire for the block
      ulonglong2 s;
      if (!poll(at + threadIdx.x * kSlotStride, &s)) bad = 1;
      __threadfence();
    }
    return __syncthreads_or(bad) == 0;
  }

  __device__ __forceinline__ bool poll(const ulonglong2* s, ulonglong2* got) {
    *got = slot_get(s);
    for (int n = 0; (unsigned)got->y != (unsigned)epoch; *got = slot_get(s))
      if (++n >= (TEST ? spins : kResSpins) || ((n & 1023) == 0 && *(volatile int*)err)) {
        atomicCAS(err, 0, (int)AFEM_ERR_TIMEOUT);
        return false;
      }
    return true;
  }

  // The grid's V sums of v in each of the block's threads: done(j, total) in lane 0 of warp j < V (again, with FP64
  // sums, where those in fixed point cannot be used), and total[j] for all.  Returns false in every thread if a
  // wait ran out.  Ends with a block barrier.
  template <int V, bool FENCE, class T, class F>
  __device__ __forceinline__ bool sum(const T (&v)[V], const int (&E)[V], double* total, int* slow, F&& done) {
    constexpr int W = kResWarps, P = W / V;   // warps, warps that poll a sum's slots
    int (*part)[kLimbs + 1] = reinterpret_cast<int (*)[kLimbs + 1]>(sh);   // [V * W], the last word: taking part
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nb = gridDim.x;
    bool ok = true;
    // a slot's words from limbs and back; the high word's lowest value stands for one that cannot take part
    auto word = [&](const __int128 t) {
      return (unsigned long long)(ok ? (unsigned)(t >> 64) : 0x80000000u) << 32 | (unsigned)epoch;
    };
    auto take = [](const ulonglong2 got, int (&l)[kLimbs], int& in) {
      const int hi = (int)(got.y >> 32);
      constexpr int mask = (1 << kLimbBits) - 1;
      if ((unsigned)hi == 0x80000000u) in = 0;
      l[0] += (int)got.x & mask;
      l[1] += (int)(got.x >> 22) & mask;
      l[2] += (int)((got.x >> 44) | ((unsigned long long)(unsigned)hi << 20)) & mask;
      l[3] += (hi >> 2) & mask;
      l[4] += hi >> 24;
    };
    if constexpr (CL) ++epoch;
#pragma unroll
    for (int j = 0; j < V; ++j) {
      int l[kLimbs] = {};
      ok &= E[j] != kNoExponent;
      if (E[j] != kNoExponent) ok &= to_limbs(v[j], E[j], l);
#pragma unroll
      for (int k = 0; k < kLimbs; ++k) {
        l[k] = __reduce_add_sync(0xffffffffu, l[k]);
        if (!CL && lane == 0) part[j * W + w][k] = l[k];
      }
      if constexpr (CL) {   // every warp's sum straight to all blocks
        ok = __all_sync(0xffffffffu, ok);
        const __int128 t = from_limbs(l);
        spread(j, w, (unsigned long long)t, word(t));
      }
    }
    int bad = 0;
    if constexpr (CL) {
      cluster_sync();
    } else {
      ok = __syncthreads_and(ok);
      ++epoch;
      ulonglong2* at = slots + (epoch % kSlotBuffers) * 2 * nb * kSlotStride;
      if (w < V) {
        int l[kLimbs];
#pragma unroll
        for (int k = 0; k < kLimbs; ++k) l[k] = __reduce_add_sync(0xffffffffu, lane < W ? part[w * W + lane][k] : 0);
        if (lane == 0) {
          const __int128 t = from_limbs(l);
          if constexpr (FENCE) __threadfence();
          slot_put(at + (w * nb + blockIdx.x) * kSlotStride, (unsigned long long)t, word(t));
        }
      }
      __syncthreads();   // part is read
      const int j = w / P;
      int l[kLimbs] = {}, in = 1;
      for (int i = (w - j * P) * 32 + lane; i < nb; i += P * 32) {
        ulonglong2 got;
        if (!poll(at + (j * nb + i) * kSlotStride, &got)) bad = 1;
        take(got, l, in);
      }
      if constexpr (FENCE)
        if ((w - j * P) * 32 < nb) __threadfence();   // the pollers acquire for the block
#pragma unroll
      for (int k = 0; k < kLimbs; ++k) l[k] = __reduce_add_sync(0xffffffffu, l[k]);
      in = __all_sync(0xffffffffu, in);
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < kLimbs; ++k) part[w][k] = l[k];
        part[w][kLimbs] = in;
      }
      if (__syncthreads_or(bad)) return false;
    }
    if (w < V) {
      int l[kLimbs] = {}, in = 1;
      if constexpr (CL) {
        for (int i = lane; i < nb * W; i += 32) take(spread_slot(w, i), l, in);
      } else if (lane < P) {
#pragma unroll
        for (int k = 0; k < kLimbs; ++k) l[k] = part[w * P + lane][k];
        in = part[w * P + lane][kLimbs];
      }
#pragma unroll
      for (int k = 0; k < kLimbs; ++k) l[k] = __reduce_add_sync(0xffffffffu, l[k]);
      ok = __all_sync(0xffffffffu, in);
      const int e0 = V == 1 || w == 0 ? E[0] : E[V - 1];
      const double t = ok ? fixed_to_double(from_limbs(l), e0) : 0.0;
      if (lane == 0) {
        const bool no = !ok || (__double2hiint(t) >> 20 & 0x7ff) - 1023 < e0 - 4;
        total[w] = t;
        slow[w] = no;
        if (!no) done(w, t);
      }
    }
    __syncthreads();
    if (slow[0] || slow[V - 1]) {   // the same in every block
      const double b = res_block_sum<V>(v, sh);
      if (!meet<V>(b)) return false;
      if (w < V) {
        const double t = this->total(w);
        if (lane == 0) {
          total[w] = t;
          done(w, t);
        }
      }
      __syncthreads();
    }
    return true;
  }

  // total of sh[v * gridDim.x ..] for the warp v that calls it, in every lane
  __device__ __forceinline__ double total(int v) const {
    const int nb = gridDim.x, lane = threadIdx.x & 31;
    double s = 0.0;
    for (int i = lane; i < nb; i += 32) s += sh[v * nb + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  }
};

inline size_t res_scratch_doubles(unsigned grid) { return std::max<size_t>(2 * kResThreads, 2 * grid); }

struct ResCtl {
  double total[2], alpha, beta;
  int slow[2];
  int done, status;
};

// The slices of a block's rows that its shared memory holds, filled from the
// CSR rows (a negative column is an unused slot and becomes a zero weight on
// the row itself, as past the end of a row).
template <class T>
struct ResMatrix {
  int32_t* off;    // [slices + 1] first step of each slice
  T* vals;
  int32_t* cols;
  int steps;       // steps of 32 entries that fit

  __device__ __forceinline__ bool resident(int s) const { return off[s + 1] <= steps; }

  // off[] from the row lengths; every thread calls it
  __device__ __forceinline__ void offsets(int nslice, int r0, int r1, const int32_t* __restrict__ rp) {
    for (int s = threadIdx.x >> 5; s < nslice; s += kResThreads / 32) {
      const int row = r0 + 32 * s + (threadIdx.x & 31);
      const int len = row < r1 ? __ldg(rp + row + 1) - __ldg(rp + row) : 0;
      const int m = __reduce_max_sync(0xffffffffu, len);
      if ((threadIdx.x & 31) == 0) off[s + 1] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      off[0] = 0;
      for (int s = 0; s < nslice; ++s) off[s + 1] += off[s];
    }
    __syncthreads();
  }
  __device__ __forceinline__ void fill(int s, int row, int r1, const int32_t* __restrict__ rp,
                                       const int32_t* __restrict__ gcols, const double* __restrict__ gvals) {
    const int m = off[s + 1] - off[s], at = 32 * off[s] + (threadIdx.x & 31);
    const int32_t b = row < r1 ? __ldg(rp + row) : 0, e = row < r1 ? __ldg(rp + row + 1) : 0;
    for (int k = 0; k < m; ++k) {
      const int32_t c = b + k < e ? __ldg(gcols + b + k) : -1;
      cols[at + 32 * k] = c >= 0 ? c : (row < r1 ? row : 0);
      vals[at + 32 * k] = c >= 0 ? (T)__ldg(gvals + b + k) : T(0);
    }
  }
};

// Sum of a row's products in CSR order.  x is written by other blocks between
// the exchanges: plain loads, not the read-only path.  STEP: entries of a row
// are that many apart.
// A chunk's gathers are issued with the next chunk's columns and values, so
// that a row pays one memory latency a chunk.
constexpr int kResChunk = 8;
template <int STEP, bool SHARED, class T>
__device__ __forceinline__ T res_row_dot(const int32_t* c, const T* a, int m, const T* x) {
  T acc = T(0);
  int32_t cc[kResChunk];
  T aa[kResChunk];
  auto load = [&](int k) {
#pragma unroll
    for (int u = 0; u < kResChunk; ++u) {
      const int e = (k + u < m ? k + u : 0) * STEP;
      cc[u] = SHARED ? c[e] : __ldg(c + e);
      aa[u] = SHARED ? a[e] : __ldg(a + e);
    }
  };
  if (m > 0) load(0);
  for (int k = 0; k < m; k += kResChunk) {
    T xx[kResChunk], av[kResChunk];
#pragma unroll
    for (int u = 0; u < kResChunk; ++u) {
      xx[u] = x[cc[u]];
      av[u] = aa[u];
    }
    if (k + kResChunk < m) load(k + kResChunk);
#pragma unroll
    for (int u = 0; u < kResChunk; ++u)
      if (k + u < m) acc = fma(av[u], xx[u], acc);
  }
  return acc;
}
// straight from the CSR row (slices that do not fit where no sliced copy was made)
__device__ __forceinline__ double res_row_dot_csr(int row, const int32_t* __restrict__ rp,
                                                  const int32_t* __restrict__ cols, const double* __restrict__ vals,
                                                  const double* x) {
  double acc = 0.0;
  const int32_t e = __ldg(rp + row + 1);
  for (int32_t k = __ldg(rp + row); k < e; ++k) {
    const int32_t c = __ldg(cols + k);
    if (c >= 0) acc = fma(__ldg(vals + k), x[c], acc);
  }
  return acc;
}

// FP64 CG, up to `iters` iterations: the arithmetic of k_cg_spmv_sl,
// k_cg_update and k_cg_dir row by row; the dot products' partial sums are
// per thread, block and grid.  x, r, p carry the state in and out (with st),
// so that a long solve is a few launches.
struct CgResident {
  int n, rows_pb, iters, steps;          // rows of a block (a multiple of 32), steps of shared memory
  const int32_t *rp, *cols;              // CSR
  const double* vals;
  const int32_t *soff, *scols;           // sliced copy, or null
  const double* svals;
  const double* dinv;                    // or null
  const uint8_t* skip;                   // or null
  double *x, *r, *p;
  ulonglong2* slots;
  int* err;
  CgState* st;
};

template <int K, bool CL, bool TEST = false>
__global__ void __launch_bounds__(kResThreads, 1) k_cg_resident(const ResArgs<TEST, CgResident> a) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ ResCtl ctl;
  __shared__ int32_t soff_sh[K * kResThreads / 32 + 1];
  if (((volatile CgState*)a.st)->done) return;
  if constexpr (TEST)
    if ((int)blockIdx.x == a.waits.stall) return;
  static_assert(!(CL && TEST), "the cluster's barrier has no bound: no block may stay away");
  const int nb = gridDim.x, lane = threadIdx.x & 31;
  __shared__ ulonglong2 cluster_slots[CL ? 4 * kResCluster * kResWarps : 1];
  if constexpr (CL) cluster_sync();   // every block runs before one writes into another
  Grid<CL, TEST> grid;
  grid.slots = CL ? cluster_slots : a.slots;
  grid.sh = reinterpret_cast<double*>(dyn);
  grid.err = a.err;
  if constexpr (TEST) grid.spins = a.waits.spins;
  ResMatrix<double> mat;
  mat.off = soff_sh;
  mat.vals = grid.sh + (2 * kResThreads > 2 * nb ? 2 * kResThreads : 2 * nb);
  mat.cols = reinterpret_cast<int32_t*>(mat.vals + 32 * (size_t)a.steps);
  mat.steps = a.steps;
  const int r0 = blockIdx.x * a.rows_pb, r1 = min(a.n, r0 + a.rows_pb);
  mat.offsets(a.rows_pb / 32, r0, r1, a.rp);
  // the blocks whose p this one's rows gather
  __shared__ uint8_t need[kResGrid];
  if constexpr (!CL) {
    if (threadIdx.x < kResGrid) need[threadIdx.x] = 0;
    __syncthreads();
    for (int row = r0 + (int)threadIdx.x; row < r1; row += kResThreads)
      for (int32_t k = __ldg(a.rp + row); k < __ldg(a.rp + row + 1); ++k) {
        const int32_t c = __ldg(a.cols + k);
        if (c >= 0) need[c / a.rows_pb] = 1;
      }
  }

  constexpr bool kAll = K <= 4;          // x and p in registers too
  double r[K], d[K], q[K], x[kAll ? K : 1], p[kAll ? K : 1];
  unsigned counted = 0;                  // bit k: the row enters the stop test's norm
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = k * kResThreads + threadIdx.x, row = r0 + i;
    r[k] = d[k] = q[k] = 0.0;
    if constexpr (kAll) x[k] = p[k] = 0.0;
    if (i < a.rows_pb && mat.resident(i >> 5)) mat.fill(i >> 5, row, r1, a.rp, a.cols, a.vals);
    if (i < a.rows_pb && row < r1) {
      r[k] = a.r[row];
      d[k] = a.dinv ? __ldg(a.dinv + row) : 1.0;
      if constexpr (kAll) {
        x[k] = a.x[row];
        p[k] = a.p[row];
      }
      if (!(a.skip && a.skip[row])) counted |= 1u << k;
    }
  }
  __syncthreads();
  double rz = a.st->rz;
  const double tol2 = a.st->tol2;
  const int max_iter = a.st->max_iter, iter0 = a.st->iter;
  int epq = kNoExponent, erz = sum_exponent(rz), err = sum_exponent(a.st->rr);   // of the sums' last values
  int it = 0;
  for (;;) {
    // q = A p ; <p, q> -> alpha
    double pq[1] = {0.0};
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = k * kResThreads + threadIdx.x, row = r0 + i;
      if (i < a.rows_pb) {
        const int s = i >> 5, m = mat.off[s + 1] - mat.off[s];   // 0 past the matrix's last slice
        if (mat.resident(s) || m == 0)
          q[k] = res_row_dot<32, true>(mat.cols + 32 * mat.off[s] + lane, mat.vals + 32 * mat.off[s] + lane, m, a.p);
        else if (a.scols) {
          const int64_t at = (int64_t)kSlice * __ldg(a.soff + (row >> 5)) + lane;
          q[k] = res_row_dot<kSlice, false>(a.scols + at, a.svals + at, m, a.p);
        } else if (row < r1)
          q[k] = res_row_dot_csr(row, a.rp, a.cols, a.vals, a.p);
        if (row < r1) pq[0] += (kAll ? p[kAll ? k : 0] : a.p[row]) * q[k];
      }
    }
    if (!grid.template sum<1, false>(pq, {epq}, ctl.total, ctl.slow, [&](int, double t) {
          const bool ok = t > 0.0 && isfinite(t);
          ctl.alpha = ok ? quotient(rz, t) : 0.0;
          ctl.status = ok ? AFEM_OK : AFEM_ERR_BREAKDOWN;
          ctl.done = !ok;
        }))
      return;
    epq = sum_exponent(ctl.total[0]);
    if (ctl.done) break;
    // x += alpha p ; r -= alpha q ; z = D^-1 r ; <r, z>, <r, r> -> beta, stop test
    const double alpha = ctl.alpha;
    double rs[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = k * kResThreads + threadIdx.x, row = r0 + i;
      if (i < a.rows_pb && row < r1) {
        if constexpr (kAll) x[k] += alpha * p[k];
        else a.x[row] += alpha * a.p[row];
        r[k] = r[k] - alpha * q[k];
        q[k] = d[k] * r[k];
        rs[0] += r[k] * q[k];
        if (counted >> k & 1) rs[1] += r[k] * r[k];
      }
    }
    ++it;
    if (!grid.template sum<2, false>(rs, {erz, err}, ctl.total, ctl.slow, [&](int j, double t) {
          if (j == 0) {
            ctl.beta = quotient(t, rz);
            return;
          }
          ctl.done = !isfinite(t) || t <= tol2 || iter0 + it >= max_iter;
          ctl.status = !isfinite(t) ? AFEM_ERR_BREAKDOWN
                                    : t > tol2 && iter0 + it >= max_iter ? AFEM_ERR_NOT_CONVERGED : AFEM_OK;
        }))
      return;
    rz = ctl.total[0];
    erz = sum_exponent(rz);
    err = sum_exponent(ctl.total[1]);
    if (ctl.done) break;
    // p = z + beta p
    const double beta = ctl.beta;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int i = k * kResThreads + threadIdx.x, row = r0 + i;
      if (i < a.rows_pb && row < r1) {
        const double pn = q[k] + beta * (kAll ? p[kAll ? k : 0] : a.p[row]);
        if constexpr (kAll) p[k] = pn;
        a.p[row] = pn;
      }
    }
    if (it == a.iters) break;
    if (!grid.barrier(need)) return;
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = k * kResThreads + threadIdx.x, row = r0 + i;
    if (i < a.rows_pb && row < r1) {
      a.r[row] = r[k];
      if constexpr (kAll) a.x[row] = x[k];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.st->rz = rz;
    if (it > 0) a.st->rr = ctl.total[1];
    a.st->iter = iter0 + it;
    a.st->status = ctl.status;
    a.st->done = ctl.done;
  }
}

// A 3x3-block matrix in FP32 as k_cgf_spmv_b3s reads it: slices of 32 block
// rows, one column index and nine value planes a step.
struct ResMatrix3 {
  int32_t* off;
  float* vals;
  int32_t* cols;
  int steps;

  __device__ __forceinline__ bool resident(int s) const { return off[s + 1] <= steps; }
  __device__ __forceinline__ void offsets(int nslice, int I0, int I1, const int32_t* __restrict__ rp) {
    for (int s = threadIdx.x >> 5; s < nslice; s += kResThreads / 32) {
      const int I = I0 + 32 * s + (threadIdx.x & 31);
      const int len = I < I1 ? (__ldg(rp + 3 * I + 1) - __ldg(rp + 3 * I)) / 3 : 0;
      const int m = __reduce_max_sync(0xffffffffu, len);
      if ((threadIdx.x & 31) == 0) off[s + 1] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      off[0] = 0;
      for (int s = 0; s < nslice; ++s) off[s + 1] += off[s];
    }
    __syncthreads();
  }
  // component c's planes of slice s, and the columns with component 0
  __device__ __forceinline__ void fill(int s, int c, int I, int I1, const int32_t* __restrict__ rp,
                                       const int32_t* __restrict__ bcols, const double* __restrict__ gvals) {
    const int m = off[s + 1] - off[s], lane = threadIdx.x & 31;
    const int32_t b0 = I < I1 ? __ldg(rp + 3 * I) : 0, bc = I < I1 ? __ldg(rp + 3 * I + c) : 0;
    const int nbk = I < I1 ? (__ldg(rp + 3 * I + 1) - b0) / 3 : 0;
    for (int k = 0; k < m; ++k) {
      const bool in = k < nbk;
      const size_t e = 32 * (size_t)(off[s] + k);
      if (c == 0) cols[e + lane] = in ? __ldg(bcols + b0 / 9 + k) : (I < I1 ? I : 0);
#pragma unroll
      for (int b = 0; b < 3; ++b)
        vals[e * 9 + (3 * c + b) * 32 + lane] = in ? (float)__ldg(gvals + bc + 3 * k + b) : 0.f;
    }
  }
};

// One scalar row of a block slice (c: its first block column, v: the first
// value plane of its component), in the order of k_cgf_spmv_b3s.
template <bool SHARED>
__device__ __forceinline__ float res_row_dot3(const int32_t* c, const float* v, int m, const float* z) {
  constexpr int kChunk = 3;
  float acc = 0.f;
  for (int kb = 0; kb < m; kb += kChunk) {
    int32_t j[kChunk];
    float x[3 * kChunk], zz[3 * kChunk];
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int e = kb + u < m ? kb + u : 0;
      j[u] = 3 * (SHARED ? c[32 * e] : __ldg(c + 32 * e));
#pragma unroll
      for (int b = 0; b < 3; ++b) x[3 * u + b] = SHARED ? v[288 * e + 32 * b] : __ldg(v + 288 * (int64_t)e + 32 * b);
    }
#pragma unroll
    for (int u = 0; u < kChunk; ++u)
#pragma unroll
      for (int b = 0; b < 3; ++b) zz[3 * u + b] = z[j[u] + b];
#pragma unroll
    for (int u = 0; u < kChunk; ++u)
      if (kb + u < m)
#pragma unroll
        for (int b = 0; b < 3; ++b) acc = fmaf(x[3 * u + b], zz[3 * u + b], acc);
  }
  return acc;
}

// The FP32 inner CG of the mixed solver, up to `iters` iterations: the
// arithmetic of k_cgf_spmv_sl / k_cgf_spmv_b3s (w = A z, p = z + beta p,
// q = w + beta q) and k_cgf_update row by row.  B3: a warp takes one
// component of 32 block rows, and rows_pb counts block rows.
struct CgfResident {
  int n, rows_pb, iters, steps;
  const int32_t *rp, *cols;              // CSR; B3: the block columns
  const double* vals;
  const int32_t *soff, *scols;           // sliced copy, or null
  const float* svals;
  const float* dinv;
  const uint8_t* skip;
  float *x, *r, *z, *p, *q;
  ulonglong2* slots;
  int* err;
  CgState* st;
};

template <int K, bool B3, bool CL, bool TEST = false>
__global__ void __launch_bounds__(kResThreads, 1) k_cgf_resident(const ResArgs<TEST, CgfResident> a) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ ResCtl ctl;
  __shared__ int32_t soff_sh[K * kResThreads / 32 + 1];
  if (((volatile CgState*)a.st)->done) return;
  if constexpr (TEST)
    if ((int)blockIdx.x == a.waits.stall) return;
  static_assert(!(CL && TEST), "the cluster's barrier has no bound: no block may stay away");
  const int nb = gridDim.x, lane = threadIdx.x & 31;
  __shared__ ulonglong2 cluster_slots[CL ? 4 * kResCluster * kResWarps : 1];
  if constexpr (CL) cluster_sync();   // every block runs before one writes into another
  Grid<CL, TEST> grid;
  grid.slots = CL ? cluster_slots : a.slots;
  grid.sh = reinterpret_cast<double*>(dyn);
  grid.err = a.err;
  if constexpr (TEST) grid.spins = a.waits.spins;
  std::conditional_t<B3, ResMatrix3, ResMatrix<float>> mat;
  mat.off = soff_sh;
  mat.vals = reinterpret_cast<float*>(grid.sh + (2 * kResThreads > 2 * nb ? 2 * kResThreads : 2 * nb));
  mat.cols = reinterpret_cast<int32_t*>(mat.vals + (B3 ? 288 : 32) * (size_t)a.steps);
  mat.steps = a.steps;
  constexpr int C = B3 ? 3 : 1;
  const int rows = a.n / C;              // rows, or block rows
  const int r0 = blockIdx.x * a.rows_pb, r1 = min(rows, r0 + a.rows_pb);
  mat.offsets(a.rows_pb / 32, r0, r1, a.rp);
  const int units = C * a.rows_pb / 32;  // warps' worth of rows

  // unit of slot k: (slice, component) and the lane's row or block row
  auto unit = [&](int k) { return k * (kResThreads / 32) + (int)(threadIdx.x >> 5); };
  float r[K], d[K], x[K], p[K], q[K], z[K];
  unsigned counted = 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int u = unit(k), s = u / C, c = u - C * s, I = r0 + 32 * s + lane, row = C * I + c;
    r[k] = d[k] = x[k] = p[k] = q[k] = z[k] = 0.f;
    if (u < units) {
      if (mat.resident(s)) {
        if constexpr (B3) mat.fill(s, c, I, r1, a.rp, a.cols, a.vals);
        else mat.fill(s, row, r1, a.rp, a.cols, a.vals);
      }
      if (I < r1) {
        r[k] = a.r[row];
        d[k] = __ldg(a.dinv + row);
        x[k] = a.x[row];
        z[k] = a.z[row];
        p[k] = a.p[row];
        q[k] = a.q[row];
        if (!(a.skip && a.skip[row])) counted |= 1u << k;
      }
    }
  }
  __syncthreads();
  double rz = a.st->rz, rz_prev = 0.0;
  float beta = (float)a.st->beta;
  const double tol2 = a.st->tol2;
  const int max_iter = a.st->max_iter, iter0 = a.st->iter;
  int epq = kNoExponent, erz = sum_exponent(rz), err = sum_exponent(a.st->rr);   // of the sums' last values
  int it = 0;
  for (;;) {
    float pq[1] = {0.f};
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int u = unit(k), s = u / C, c = u - C * s, I = r0 + 32 * s + lane;
      if (u < units) {
        const int m = mat.off[s + 1] - mat.off[s];
        float w;
        if (mat.resident(s) || m == 0) {   // 0: past the matrix's last slice
          const int32_t* mc = mat.cols + 32 * (size_t)mat.off[s] + lane;
          if constexpr (B3) w = res_row_dot3<true>(mc, mat.vals + 288 * (size_t)mat.off[s] + 96 * c + lane, m, a.z);
          else w = res_row_dot<32, true>(mc, mat.vals + 32 * mat.off[s] + lane, m, a.z);
        } else {
          const int64_t at = (int64_t)kSlice * __ldg(a.soff + (r0 >> 5) + s);
          if constexpr (B3) w = res_row_dot3<false>(a.scols + at + lane, a.svals + 9 * at + 96 * c + lane, m, a.z);
          else w = res_row_dot<kSlice, false>(a.scols + at + lane, a.svals + at + lane, m, a.z);
        }
        if (I < r1) {
          p[k] = beta != 0.f ? fmaf(beta, p[k], z[k]) : z[k];
          q[k] = beta != 0.f ? fmaf(beta, q[k], w) : w;
          pq[0] = fmaf(p[k], q[k], pq[0]);
        }
      }
    }
    if (!grid.template sum<1, false>(pq, {epq}, ctl.total, ctl.slow, [&](int, double t) {
          const bool ok = t > 0.0 && isfinite(t);
          ctl.alpha = ok ? quotient(rz, t) : 0.0;
          ctl.status = ok ? AFEM_OK : AFEM_ERR_BREAKDOWN;
          ctl.done = !ok;
        }))
      return;
    epq = sum_exponent(ctl.total[0]);
    if (ctl.done) break;
    const float alpha = (float)ctl.alpha;
    float rs[2] = {0.f, 0.f};
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int u = unit(k), s = u / C, c = u - C * s, I = r0 + 32 * s + lane;
      if (u < units && I < r1) {
        x[k] = fmaf(alpha, p[k], x[k]);
        r[k] = fmaf(-alpha, q[k], r[k]);
        z[k] = d[k] * r[k];
        a.z[C * I + c] = z[k];
        rs[0] = fmaf(r[k], z[k], rs[0]);
        if (counted >> k & 1) rs[1] = fmaf(r[k], r[k], rs[1]);
      }
    }
    ++it;
    if (!grid.template sum<2, true>(rs, {erz, err}, ctl.total, ctl.slow, [&](int j, double t) {
          if (j == 0) {
            ctl.beta = quotient(t, rz);
            return;
          }
          ctl.done = !isfinite(t) || t <= tol2 || iter0 + it >= max_iter;
          ctl.status = isfinite(t) ? AFEM_OK : AFEM_ERR_BREAKDOWN;
        }))
      return;
    rz_prev = rz;
    rz = ctl.total[0];
    erz = sum_exponent(rz);
    err = sum_exponent(ctl.total[1]);
    beta = (float)ctl.beta;
    if (ctl.done || it == a.iters) break;
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int u = unit(k), s = u / C, c = u - C * s, I = r0 + 32 * s + lane, row = C * I + c;
    if (u < units && I < r1) {
      a.x[row] = x[k];
      a.r[row] = r[k];
      a.p[row] = p[k];
      a.q[row] = q[k];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (it > 0) {
      a.st->beta = ctl.beta;
      a.st->pad0 = rz_prev;
      a.st->rz = rz;
      a.st->rr = ctl.total[1];
    }
    a.st->iter = iter0 + it;
    a.st->status = ctl.status;
    a.st->done = ctl.done;
  }
}

// ---------------------------------------------------------------------------
// Host side.

// The split of `rows` rows of C components over the blocks.  At least 128
// scalar rows a block (one warp for each of an SM's four partitions): below
// that an exchange costs more than the rows.
struct ResPlan {
  unsigned grid = 0;
  int rows_pb = 0, K = 0, steps = 0;
  bool cluster = false;  // one cluster of blocks
  // dynamic shared memory: the cluster form's slots are static
  size_t smem() const { return kResSmem - (cluster ? sizeof(ulonglong2) * 4 * kResCluster * kResWarps : 0); }
  bool fits = false;     // every slice is likely to fit the shared memory (exactly: k_res_unfit)
  bool take = false;     // this form rather than the launches per iteration
};

// Where the line lies: one block an SM has the loads in flight for what the
// shared memory leaves over of a matrix up to about 80 MB (L2-resident), and
// registers for 6 rows a thread.  A solve, three launches an iteration against
// this form: 2D triangles 256^2 19.2 -> 8.6 ms, 600^2 98.5 -> 41.8; tetrahedra
// 57^3 8.8 -> 4.0, 75^3 17.7 -> 9.7; hexahedra 69^3 (34 MB left over)
// 11.2 -> 7.1; elasticity 40^3 (77 MB left over) 50.8 -> 29.1, mixed
// 35.1 -> 14.7.  Above, with 8 rows a thread: tetrahedra 84^3 23.7 -> 20.2, but
// renumbered at random 28.1 -> 34.2; hexahedra 84^3 17.9 -> 20.4.
// A matrix whose rows gather at random lives on what the L1 keeps of the
// gathered vector, and here shared memory takes most of the L1: with
// kResScatterEntries and more of them the launches win (random numbering,
// launches -> this form: triangles 600^2, 2.5 M entries, 105 -> 73 ms;
// hexahedra 50^3, 3.6 M, mixed 5.1 -> 5.2; 66^3, 8.1 M, 11.2 -> 12.0).
constexpr int64_t kResScatterEntries = 3300000;
constexpr int64_t kResStreamBytes = 80ll << 20;

constexpr int kResClusterUnits = 384;
constexpr int64_t kResClusterBytes = 1200 << 10;

inline ResPlan res_plan(afem_context ctx, int rows, int C, int64_t nnz, size_t step_bytes) {
  ResPlan p;
  auto split = [&](int64_t blocks) {
    const int64_t pb = (rows + blocks - 1) / blocks;
    p.rows_pb = (int)((pb + 31) / 32 * 32);
    p.grid = (unsigned)((rows + p.rows_pb - 1) / p.rows_pb);
    p.K = (int)(((int64_t)C * p.rows_pb + kResThreads - 1) / kResThreads);
  };
  // One cluster up to 384 rows a block and two thirds of its shared memory.  Eight blocks hold fewer rows at once
  // than the grid of 128 a block, but meet sooner (Grid): whole solves in FP64 1.36 -> 1.09 ms at 45^2 triangles,
  // 0.60 -> 0.54 at 13^3 tetrahedra, 2.10 -> 1.84 at 8^3 with three unknowns a node (1.0 MB of matrix); but, with
  // the sums still going by way of the blocks', 2.35 -> 2.37 at 9^3 (1.4 MB), and with 512 rows a block 0.67 -> 0.69
  // at 15^3, 2.53 -> 3.07 at 10^3 with three.
  int64_t blocks = 1;
  while (blocks < kResCluster && blocks * 64 < (int64_t)rows * C) blocks *= 2;
  split(blocks);
  p.cluster = (int64_t)C * p.rows_pb <= kResClusterUnits &&
              nnz / (C * C) * (int64_t)(step_bytes / 32) <= kResClusterBytes;
  if (p.cluster) p.grid = (unsigned)blocks;
  else split(std::min<int64_t>(std::min(ctx->sm_count, kResGrid), ((int64_t)rows * C + 127) / 128));
  p.steps = (int)((p.smem() - sizeof(double) * res_scratch_doubles(p.grid)) / step_bytes);
  // rows of a slice differ in length and the last block may be short: one step in ten for the padding
  p.take = p.K <= kResMaxRows &&
           (int64_t)(nnz / (C * C) * (step_bytes / 32)) - (int64_t)p.grid * (int64_t)kResSmem <= kResStreamBytes;
  p.fits = (double)nnz / (C * C) <= 0.9 * 32.0 * p.steps * p.grid;
  return p;
}

// Whether the slices of a block's rows (C scalar rows each) are more than `steps` long together, in any block: a block
// of the solve a block here, a warp a slice.  res_plan's `fits` expects slices of about equal rows; a node with far more
// neighbours than the others makes its slice as long as its row.  The mixed solver reads the answer with its first
// residual and makes the sliced copy then: walked in the CSR row, entry by entry with the values' conversions, a row of
// 5000 entries among 140^2 cost 190 ms a solve, from the copy 107 (launches per iteration 157 to 166).
static __global__ void __launch_bounds__(kResThreads) k_res_unfit(int rows, int rows_pb, int C, int steps,
                                                                  const int32_t* __restrict__ rp, int* unfit) {
  __shared__ int total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  const int r0 = blockIdx.x * rows_pb, r1 = min(rows, r0 + rows_pb);
  for (int s = threadIdx.x >> 5; 32 * s < r1 - r0; s += kResWarps) {
    const int I = r0 + 32 * s + (threadIdx.x & 31);
    const int len = I < r1 ? (__ldg(rp + C * I + 1) - __ldg(rp + C * I)) / C : 0;
    const int m = __reduce_max_sync(0xffffffffu, len);
    if ((threadIdx.x & 31) == 0) atomicAdd(&total, m);
  }
  __syncthreads();
  if (threadIdx.x == 0 && total > steps) *unfit = 1;
}

// Samples slices of 32 rows: counts[0] entries seen, counts[1] those more than
// 64 columns from the same entry of the row before.
static __global__ void k_scatter_sample(int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ cols,
                                        int32_t* counts) {
  const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x / 32);
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int64_t row = (int64_t)w * (n / 32) / warps * 32 + lane;
  const int32_t b = row < n ? __ldg(rp + row) : 0, e = row < n ? __ldg(rp + row + 1) : 0;
  const int m = __reduce_min_sync(0xffffffffu, e - b);
  int far = 0;
  for (int k = 0; k < m; ++k) {
    const int32_t c = __ldg(cols + b + k), before = __shfl_up_sync(0xffffffffu, c, 1);
    far += __popc(__ballot_sync(0xffffffffu, lane > 0 && abs(c - before) > 64));
  }
  if (lane == 0 && m > 0) {
    atomicAdd(counts, 31 * m);
    atomicAdd(counts + 1, far);
  }
}

// Whether the gathers of the rows are mostly scattered (one synchronising read).
inline afem_status res_scattered(afem_context ctx, int n, const int32_t* rp, const int32_t* cols, int32_t* counts,
                                 bool* scattered) {
  struct Two {
    int32_t seen, far;
  } c{};
  AFEM_CUDA(cudaMemsetAsync(counts, 0, sizeof(Two), ctx->stream));
  AFEM_TRY(launch(ctx, k_scatter_sample, 64, 256, 0, n, rp, cols, counts));
  AFEM_TRY(read_scalar(ctx, reinterpret_cast<const Two*>(counts), &c));
  *scattered = 2 * (int64_t)c.far > c.seen;
  return AFEM_OK;
}

inline size_t res_slots_bytes(const ResPlan& p) { return align256(sizeof(ulonglong2) * 2 * kSlotBuffers * kSlotStride * p.grid); }

// Iterations of one launch, for some 10 ms of work by the largest of the
// exchanges, the entries and the rows.
inline int res_launch_iters(int n, int64_t nnz) {
  return (int)std::max<int64_t>(64, 4000000000ll / (nnz + 20ll * n + 2000000ll));
}

template <class Args>
afem_status launch_resident(afem_context ctx, void (*k)(const Args), const ResPlan& p, const Args& a) {
  AFEM_CUDA(cudaMemsetAsync(a.slots, 0, res_slots_bytes(p), ctx->stream));
  AFEM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem()));
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(p.grid);
  lc.blockDim = dim3(kResThreads);
  lc.dynamicSmemBytes = p.smem();
  lc.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  if (p.cluster) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {p.grid, 1, 1};
  } else {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
  }
  lc.attrs = attr;
  lc.numAttrs = 1;
  AFEM_CUDA(cudaLaunchKernelEx(&lc, k, a));
  ++ctx->launches;
  return AFEM_OK;
}

template <class F>
afem_status dispatch_rows(int K, F&& f) {
  switch (K) {
    case 1: return f(std::integral_constant<int, 1>{});
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    case 4: return f(std::integral_constant<int, 4>{});
    default: return f(std::integral_constant<int, kResMaxRows>{});
  }
}

// Launch until the state says done; *hs is the final state.  A wait that ran
// out leaves the slots' owner with AFEM_ERR_TIMEOUT.
template <class Launch>
afem_status run_resident(afem_context ctx, CgState* st, int* err, CgState* hs, Launch&& go) {
  struct Both {
    CgState s;
    int err;
  };
  for (;;) {
    AFEM_TRY(go());
    auto* h = reinterpret_cast<Both*>(ctx->pinned);
    AFEM_CUDA(cudaMemcpyAsync(&h->s, st, sizeof(CgState), cudaMemcpyDeviceToHost, ctx->stream));
    AFEM_CUDA(cudaMemcpyAsync(&h->err, err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    AFEM_CUDA(cudaStreamSynchronize(ctx->stream));
    if (h->err) return fail((afem_status)h->err, "CG: a grid exchange ran out of time (status %d)", h->err);
    *hs = h->s;
    if (hs->done) return AFEM_OK;
  }
}

}  // namespace afem
