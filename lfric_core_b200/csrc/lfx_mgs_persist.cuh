// One Gram-Schmidt step of GMRES as one persistent launch (included by
// lfx_solver.cu): modified Gram-Schmidt of w against iv basis vectors, the
// norm, and the next basis vector. Same operations, orders and reductions as a
// launch per inner product, so the same bits.
#pragma once

#include "lfx_cg_persist.cuh"

namespace lfx {

constexpr int kMgsMaxVec = 64;
// chunks of w a block keeps in shared memory (of RCHUNK values)
constexpr size_t kMgsSmemMax = 224 * 1024;
template <class T>
constexpr int kMgsCap = (int)(kMgsSmemMax / (RCHUNK * sizeof(T)));

constexpr int kMgsAhead = 2;

template <class T>
struct MgsArgs {
  int64_t n;
  int nch, iv;
  const T* v[kMgsMaxVec];
  T* w;
  T* vn;        // next basis vector (nullable)
  double *h, *nh;  // column iv of H: h[0 .. iv), h[iv] = ||w||; nh = -h
  double *inv_hn, *sig;
  int* applies;
  double* partials;  // 2 nch
  GridBar bar;
  const int* skip;
};

// the RPER values of a lane of one chunk (m-th at p + m RT); FULL: the chunk has
// all its values, else those past the end are zero
template <class T, bool FULL, bool ONCE>
__device__ __forceinline__ void mgs_load(T (&v)[RPER], const T* p, int left) {
#pragma unroll
  for (int m = 0; m < RPER; ++m)
    v[m] = FULL || m < left ? (ONCE ? __ldcs(p + m * RT) : __ldcg(p + m * RT)) : T(0);
}

// Bound: a step of iv vectors has to bring each in once (40 MB at C96 x 30
// FP64, 6.2 us at 6.5 TB/s); w -= h_j v_j needs v_j again after its inner
// product. A launch per product (w -= h_{j-1} v_{j-1}; <v_j, w>) moves 160 MB, 25.6
// us. Here w stays with its block, 14 of its 17 chunks at that size in shared
// memory and the others in L2, and a pass reads two vectors: v_{j-1} (second
// touch, in the order opposite to the first, evict-first, all from L2: 40.8 MB a
// pass come from DRAM) and v_j. A warp holds the next chunk's values in registers
// while it works on one, also across the barrier, and warps do not meet between
// chunks: the chunk sums are added up after the pass. 15.8 us a pass: 27 % of the
// warps' time at barriers (a grid barrier and the sum of 2 457 chunk partials a
// pass), 27 % waiting for loads, the rest issue. The FP64 GMRES(10) solve at C96
// x 30: 6134 -> 4887 us; C48 x 30: 2192 -> 1825. Measured and not kept: 1024
// threads with 64 registers and no values ahead 5345 us; chunks 4 or 8 ahead into
// L2 instead of 2, no difference.
template <class T>
__global__ void __launch_bounds__(kCgThreads, 1) mgs_persist(const MgsArgs<T> A) {
  extern __shared__ __align__(16) unsigned char mgs_smem[];
  constexpr int kMaxSlots = 32;  // chunk sums held at a time
  __shared__ double wsum[kMaxSlots][RT / 32];
  __shared__ double sm[kCgSubs * (RT / 32)], tot[2];
  __shared__ int ok;
  if (*((volatile const int*)A.skip)) return;
  if (grid_failed(A.bar)) return;
  T* ws = reinterpret_cast<T*>(mgs_smem);
  const int sub = threadIdx.x / RT, tid = threadIdx.x % RT, lane = threadIdx.x & 31;
  const int warp = tid >> 5;
  // the block's chunks are blockIdx.x + gridDim.x i; sub-group `sub` takes i =
  // sub, sub + kCgSubs, ...
  const int nblk = (int)blockIdx.x < A.nch ? (A.nch - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  const int cnt = nblk > sub ? (nblk - 1 - sub) / kCgSubs + 1 : 0;
  auto slot = [&](int ph, int q) { return sub + kCgSubs * ((ph & 1) ? cnt - 1 - q : q); };
  auto first = [&](int i) { return (int64_t)(blockIdx.x + gridDim.x * i) * RCHUNK + tid; };
  // values of this lane in the chunk that starts (for this lane) at b
  auto values = [&](int64_t b) { return (int)max((int64_t)0, min((int64_t)RPER, (A.n - b + RT - 1) / RT)); };
  unsigned target = 0;
  double nh = 0.0;
  T pn[RPER], xn[RPER];  // the next chunk's values of v_{ph - 1} and v_ph
  auto fetch = [&](int ph, int q) {
    const int64_t b = first(slot(ph, q));
    if (b - tid + RCHUNK <= A.n) {
      if (ph > 0) mgs_load<T, true, true>(pn, A.v[ph - 1] + b, RPER);
      if (ph < A.iv) mgs_load<T, true, false>(xn, A.v[ph] + b, RPER);
    } else {
      const int left = values(b);
      if (ph > 0) mgs_load<T, false, true>(pn, A.v[ph - 1] + b, left);
      if (ph < A.iv) mgs_load<T, false, false>(xn, A.v[ph] + b, left);
    }
  };
  // chunks of the vectors' first touch go out to L2 kMgsAhead ahead, also into
  // the next pass (the second touch finds its chunk there)
  auto ahead = [&](int ph, int q) {
    if (tid != 0) return;
    if (q >= cnt) {
      q -= cnt;
      if (++ph > A.iv || q >= cnt) return;
    }
    if (ph >= A.iv) return;
    const int64_t e = first(slot(ph, q)) - tid;
    const unsigned bytes = (unsigned)(min((int64_t)RCHUNK, A.n - e) * sizeof(T)) & ~15u;
    if (bytes)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(A.v[ph] + e), "r"(bytes)
                   : "memory");
  };
  if (cnt) fetch(0, 0);
  for (int q = 1; q < kMgsAhead && q < cnt; ++q) ahead(0, q);
  for (int ph = 0; ph <= A.iv; ++ph) {
    double* part = A.partials + (size_t)(ph & 1) * A.nch;
    const T c = (T)nh;
    for (int q0 = 0; q0 < cnt; q0 += kMaxSlots / kCgSubs) {
      const int q1 = min(cnt, q0 + kMaxSlots / kCgSubs);
      for (int q = q0; q < q1; ++q) {
        const int i = slot(ph, q);
        const int64_t b = first(i);
        const bool own = i < kMgsCap<T>, full = b - tid + RCHUNK <= A.n;
        const int left = full ? RPER : values(b);
        T* wl = ws + (size_t)i * RCHUNK + tid;
        T* wg = A.w + b;
        T p[RPER], x[RPER], w[RPER];
#pragma unroll
        for (int m = 0; m < RPER; ++m) {
          p[m] = pn[m];
          x[m] = xn[m];
        }
        if (ph > 0 && own) {
#pragma unroll
          for (int m = 0; m < RPER; ++m) w[m] = wl[m * RT];
        } else if (full) {
          mgs_load<T, true, false>(w, wg, RPER);
        } else {
          mgs_load<T, false, false>(w, wg, left);
        }
        ahead(ph, q + kMgsAhead);
        if (q + 1 < cnt)
          fetch(ph, q + 1);
        else if (ph < A.iv)
          fetch(ph + 1, 0);
        if (ph > 0) {
#pragma unroll
          for (int m = 0; m < RPER; ++m) w[m] = fmaT(c, p[m], w[m]);
        }
        if (own) {
#pragma unroll
          for (int m = 0; m < RPER; ++m) wl[m * RT] = w[m];
        } else if (ph > 0) {
#pragma unroll
          for (int m = 0; m < RPER; ++m)
            if (m < left) __stcg(wg + m * RT, w[m]);
        }
        double acc = 0.0;
        if (ph == A.iv) {
#pragma unroll
          for (int m = 0; m < RPER; ++m) x[m] = w[m];
        }
        if (full) {
#pragma unroll
          for (int m = 0; m < RPER; ++m) acc = fma((double)x[m], (double)w[m], acc);
        } else {
#pragma unroll
          for (int m = 0; m < RPER; ++m)
            if (m < left) acc = fma((double)x[m], (double)w[m], acc);
        }
        acc = warp_butterfly(acc);
        if (lane == 0) wsum[sub + kCgSubs * (q - q0)][warp] = acc;
      }
      // the sub-group's chunk sums, the warps' left to right
      asm volatile("bar.sync %0, %1;" ::"r"(1 + sub), "n"(RT) : "memory");
      if (tid < q1 - q0) {
        const double* s = wsum[sub + kCgSubs * tid];
        double t = s[0];
#pragma unroll
        for (int k = 1; k < RT / 32; ++k) t = t + s[k];
        __stcg(part + blockIdx.x + (size_t)gridDim.x * slot(ph, q0 + tid), t);
      }
      if (q1 < cnt) asm volatile("bar.sync %0, %1;" ::"r"(1 + sub), "n"(RT) : "memory");
    }
    if (!cg_barrier<false>(A.bar, target, &ok)) return;
    cg_total<1>(part, A.nch, sm, tot);
    const double t = tot[0];
    if (ph < A.iv) {
      nh = -t;
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.h[ph] = t;
        A.nh[ph] = nh;
      }
    } else {
      const double hn = sqrt(t), inv = 1.0 / hn;
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.h[ph] = hn;
        *A.inv_hn = inv;
        *A.sig = inv;
        *A.applies += 1;
      }
      if (A.vn) {
        for (int q = 0; q < cnt; ++q) {
          const int i = sub + kCgSubs * q;
          const int64_t b = first(i);
          const bool own = i < kMgsCap<T>;
          const int left = values(b);
          const T* wl = own ? ws + (size_t)i * RCHUNK + tid : A.w + b;
#pragma unroll
          for (int m = 0; m < RPER; ++m)
            if (m < left) A.vn[b + m * RT] = (T)inv * wl[m * RT];
        }
      }
    }
  }
  cg_leave(A.bar);
}

}  // namespace lfx
