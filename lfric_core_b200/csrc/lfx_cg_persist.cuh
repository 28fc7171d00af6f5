// Conjugate gradients with a diagonal preconditioner as one persistent launch
// (included by lfx_solver.cu). Same operations, term orders and reductions as
// the launch per phase, so the same bits.
//
// A small solve is all latency: an iteration of five launches inside a CUDA
// graph takes 23.7 us at C8 x 6 (2 702 dofs) and 31.8 us at C24 x 20 (72 618
// dofs, the matrix in L2), of which the bytes would take under 1 and 6 us.
// Here the blocks stay resident, keep p, r, x and the diagonal of their chunks
// in shared memory, and the records and matrix rows of as many of their dof
// columns as fit beside them; they meet at a barrier where a launch ended
// (four an iteration). Whole solves, FP64, B200: C8 x 6 (67 iterations) 1390-1590 ->
// 598 us, C24 x 20 (192) 6100 -> 3141 us, C37 x 23 (263) 12.4 -> 6.9 ms. What is
// left is latency: 15 k cycles of 31 k at C24 x 20 are the gather (two passes of
// columns a warp, the second's matrix from L2), a grid barrier takes 2 to 3 k
// (0.6 to 1 k the cluster's), the two reductions with their division and root
// 3.4 and 2 k. 768 threads (80 registers, one cell at a time): 3463 us. In a
// form that read the vectors and the matrix from L2 in each phase: 5236 us.
#pragma once

#include "lfx_internal.cuh"

namespace lfx {

constexpr int kCgThreads = 512;
constexpr int kCgSubs = kCgThreads / RT;  // groups of RT threads, one 2048-value chunk each
// blocks of the cluster that carries the smallest solves (one column a warp):
// its barrier is in hardware
constexpr int kCgCluster = 16;
constexpr size_t kCgSmemMax = 224 * 1024;
// iterations of one launch (the next one carries on from the device state)
constexpr int kCgItersPerLaunch = 2000;

// barrier of a launch whose blocks are all resident
struct GridBar {
  unsigned* words;  // {arrivals, blocks gone}, zero between launches
  int* err;         // the context's error flag
  unsigned long long limit_ns;  // longest wait
  int poll;         // the clock and the flag are looked at every poll + 1 polls
};
inline GridBar grid_bar(const lfx_ctx* ctx) {
  // (a look costs more than a poll; a limit below a barrier's own time looks at once)
  return GridBar{ctx->d_ticket + 1, ctx->d_err, ctx->wait_ns, ctx->wait_ns < 1000000ull ? 0 : 255};
}

template <class T>
struct CgArgs {
  // gather layout of the operator and its matrix (lfx_lma_layout, lfx_op)
  int nent, nl, blk, gp_stride;
  size_t cell_stride;
  const int4* ent_pack;
  const int* grp_pack;
  const T* M;
  int64_t n;
  int nch;
  T *x, *r, *p, *z;
  const T* dg;
  double* partials;  // 3 nch
  GridBar bar;
  int iters;
  const T* b;
  // shared memory: the vectors of the block's chunks, then as many of its dof
  // columns (of maxg groups each) as fit
  int smem, maxg;
  int lw;  // lanes a column takes in the apply: 1 << lw
};

// one dof column in shared memory: per group its record and the matrix rows of
// up to two (cell, df) blocks
template <class T, int N>
__host__ __device__ constexpr size_t cg_group_bytes(int nl) {
  return 48 + ((2 * (size_t)N * nl * sizeof(T) + 15) / 16) * 16;
}
template <class T>
__host__ __device__ constexpr size_t cg_chunk_bytes() {
  return 4 * (size_t)RCHUNK * sizeof(T);  // p, r, x, diagonal
}

__device__ __forceinline__ unsigned long long cg_clock() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A launch that comes after a wait ran out (the host has not looked yet) leaves
// at once: the barrier's words are not zero. The whole block decides alike.
__device__ __forceinline__ bool grid_error(const GridBar& B) {
  return *((volatile const int*)B.err) != 0;
}
__device__ __forceinline__ bool grid_failed(const GridBar& B) {
  return __syncthreads_or(grid_error(B)) != 0;
}

// All blocks of the grid (every one resident: a cooperative launch, or one
// cluster). The grid form counts arrivals up; a wait past the limit sets
// LFX_TIMEOUT and every block leaves.
template <bool CLUSTER>
__device__ __forceinline__ bool cg_barrier(const GridBar& B, unsigned& target, int* ok) {
  if constexpr (CLUSTER) {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                     : "memory");
    return true;
  } else {
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(B.words) : "memory");
      *ok = 1;
      unsigned long long t0 = 0;
      for (int spin = 0;; ++spin) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(B.words) : "memory");
        if ((int)(v - target) >= 0) break;
        if ((spin & B.poll) == B.poll) {
          const unsigned long long t = cg_clock();
          if (!t0) t0 = t;
          if (grid_error(B) || t - t0 >= B.limit_ns) {
            atomicExch(B.err, (int)LFX_TIMEOUT);
            *ok = 0;
            break;
          }
        }
      }
    }
    __syncthreads();
    return *ok != 0;
  }
}

// the last block to leave makes the barrier ready for the next launch
__device__ __forceinline__ void cg_leave(const GridBar& B) {
  if (threadIdx.x == 0 && atomicAdd(B.words + 1, 1u) == gridDim.x - 1) {
    B.words[0] = 0u;
    B.words[1] = 0u;
  }
}

// One group's record {cell, records, map_from row} as the gather layout packs
// it (see the LMA apply: records at most two, df and vertical offset each), and
// its operands of one output row per lane. b0: the first record's x values; the
// second record's are those of the lane below where it sits one level above the
// first, and come from e where there is no such lane (edge).
template <class T, int N, bool EDGE>
struct CgGroup {
  T b0[N], e[EDGE ? N : 1];
  int cell, d0, d1, k0, k1;
  bool v0, v1, edge;
  template <bool CACHED>
  __device__ __forceinline__ void load(const CgArgs<T>& A, const T* p, const int* rec, int l,
                                       int lane) {
    const int4* gp = reinterpret_cast<const int4*>(rec);
    const int4 h0 = CACHED ? gp[0] : __ldg(gp);
    const int4 h1 = CACHED ? gp[1] : __ldg(gp + 1);
    int mf[N];
    mf[0] = h0.z; mf[1] = h0.w;
    mf[2] = h1.x; mf[3] = h1.y; mf[4] = h1.z; mf[5] = h1.w;
    if constexpr (N > 6) {
      const int4 h2 = CACHED ? gp[2] : __ldg(gp + 2);
      mf[6] = h2.x; mf[7] = h2.y;
    }
    const uint32_t pk = (uint32_t)h0.y;
    cell = h0.x;
    d0 = (pk >> 2) & 63u;
    d1 = (pk >> 11) & 63u;
    const int o0 = (pk >> 8) & 7u, o1 = (pk >> 17) & 7u, nrec = pk & 3u;
    k0 = l - o0;
    k1 = l - o1;
    v0 = (unsigned)k0 < (unsigned)A.nl;
    v1 = nrec > 1 && (unsigned)k1 < (unsigned)A.nl;
    edge = v1 && (o1 != o0 + 1 || lane == 0);
    const T* p0 = p + k0;
#pragma unroll
    for (int j = 0; j < N; ++j) b0[j] = v0 ? __ldcg(p0 + mf[j]) : T(0);
    if constexpr (EDGE) {
      const T* p1 = p + k1;
#pragma unroll
      for (int j = 0; j < N; ++j) e[j] = edge ? __ldcg(p1 + mf[j]) : T(0);
    }
  }
  // the terms in the order of the LMA apply (group_acc)
  __device__ __forceinline__ T add(const CgArgs<T>& A, const T* M0, const T* M1, T acc) const {
    M0 += v0 ? k0 : 0;
    M1 += v1 ? k1 : 0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
      T b1 = __shfl_up_sync(0xffffffffu, b0[j], 1);
      if (EDGE) b1 = edge ? e[j] : b1;
      if (v0) acc = fmaT(*M0, b0[j], acc);
      if (v1) acc = fmaT(*M1, b1, acc);
      M0 += A.nl;
      M1 += A.nl;
    }
    return acc;
  }
  __device__ __forceinline__ void none() {
    v0 = v1 = edge = false;
    cell = d0 = d1 = k0 = k1 = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) b0[j] = T(0);
#pragma unroll
    for (int j = 0; j < (EDGE ? N : 1); ++j) e[j] = T(0);
  }
};

// Column of slot s of this block, -1 past the end
__device__ __forceinline__ int cg_column(int nent, int s) {
  const int e = blockIdx.x + gridDim.x * s;
  return e < nent ? e : -1;
}

// the block's first ncache columns into shared memory
template <class T, int N>
__device__ __forceinline__ void cg_cache(const CgArgs<T>& A, unsigned char* cache, int ncache) {
  const int lane = threadIdx.x & 31;
  const size_t gb = cg_group_bytes<T, N>(A.nl);
  for (int s = threadIdx.x >> 5; s < ncache; s += kCgThreads / 32) {
    const int e = cg_column(A.nent, s);
    if (e < 0) break;
    const int4 ep = __ldg(A.ent_pack + e);
    for (int g = ep.z; g < ep.w; ++g) {
      unsigned char* dst = cache + ((size_t)s * A.maxg + (g - ep.z)) * gb;
      const int* rec = A.grp_pack + (size_t)g * A.gp_stride;
      if (lane < N + 2) reinterpret_cast<int*>(dst)[lane] = __ldg(rec + lane);
      const uint32_t pk = (uint32_t)__ldg(rec + 1);
      T* m = reinterpret_cast<T*>(dst + 48);
      const T* src = A.M + (size_t)__ldg(rec) * A.cell_stride;
      const T *s0 = src + (size_t)((pk >> 2) & 63u) * A.blk, *s1 = src + (size_t)((pk >> 11) & 63u) * A.blk;
      for (int i = lane; i < N * A.nl; i += 32) {
        m[i] = __ldg(s0 + i);
        if ((pk & 3u) > 1) m[N * A.nl + i] = __ldg(s1 + i);
      }
    }
  }
}

// A.z = A p: a lane takes a level of a dof column, a warp 32 >> lw columns of at
// most 1 << lw levels (lw = 5: one column of any height). Of a cached column the
// record and the matrix are in shared memory and a few cells' x values are
// loaded at once; of another one the matrix comes through L2.
template <class T, int N, bool EDGE>
__device__ __forceinline__ void cg_apply(const CgArgs<T>& A, const T* p, const unsigned char* cache,
                                         int ncache) {
  const int lane = threadIdx.x & 31;
  const int per = 32 >> A.lw, own = lane & ((1 << A.lw) - 1);
  const size_t gb = cg_group_bytes<T, N>(A.nl);
  constexpr int G = EDGE ? 1 : sizeof(T) == 4 ? 4 : 2;
  for (int s0 = (threadIdx.x >> 5) * per;; s0 += kCgThreads / 32 * per) {
    const int s = s0 + (lane >> A.lw);
    const int e = cg_column(A.nent, s);
    if (__all_sync(0xffffffffu, e < 0)) break;
    const int4 ep = e >= 0 ? __ldg(A.ent_pack + e) : make_int4(0, 0, 0, 0);
    const int ng = ep.w - ep.z;
    // the warp's columns are all cached or none is (ncache is a multiple of per)
    const bool cached = s0 < ncache;
    const int height = A.lw < 5 ? 1 : ep.y;
    for (int l0 = 0; l0 < height; l0 += 32) {
      const int l = l0 + own;
      T acc = T(0);
      if (cached) {
        const unsigned char* col = cache + (size_t)s * A.maxg * gb;
        for (int g0 = 0; __any_sync(0xffffffffu, g0 < ng); g0 += G) {
          CgGroup<T, N, EDGE> q[G];
#pragma unroll
          for (int u = 0; u < G; ++u) {
            if (g0 + u < ng)
              q[u].template load<true>(A, p, reinterpret_cast<const int*>(col + (g0 + u) * gb), l,
                                      own);
            else
              q[u].none();
          }
#pragma unroll
          for (int u = 0; u < G; ++u) {
            const T* m = reinterpret_cast<const T*>(col + (g0 + u < ng ? g0 + u : 0) * gb + 48);
            acc = q[u].add(A, m, m + N * A.nl, acc);
          }
        }
      } else {
        constexpr int GU = EDGE ? 1 : 2;
        for (int g0 = 0; __any_sync(0xffffffffu, g0 < ng); g0 += GU) {
          CgGroup<T, N, EDGE> q[GU];
#pragma unroll
          for (int u = 0; u < GU; ++u) {
            if (g0 + u < ng)
              q[u].template load<false>(A, p, A.grp_pack + (size_t)(ep.z + g0 + u) * A.gp_stride, l,
                                        own);
            else
              q[u].none();
          }
#pragma unroll
          for (int u = 0; u < GU; ++u) {
            const T* Mc = A.M + (size_t)q[u].cell * A.cell_stride;
            acc = q[u].add(A, Mc + (size_t)q[u].d0 * A.blk, Mc + (size_t)q[u].d1 * A.blk, acc);
          }
        }
      }
      if (l < ep.y) __stcg(A.z + ep.x + l, acc);
    }
  }
}

// Sum over the RT threads of a sub-group in the order of block_sum, by named
// barrier; valid in the sub-group's thread 0
__device__ __forceinline__ double cg_sub_sum(double acc, double* sm) {
  acc = warp_butterfly(acc);
  const int sub = threadIdx.x / RT, w = (threadIdx.x >> 5) % (RT / 32);
  if ((threadIdx.x & 31) == 0) sm[sub * (RT / 32) + w] = acc;
  asm volatile("bar.sync %0, %1;" ::"r"(1 + sub), "n"(RT) : "memory");
  double t = 0.0;
  if (threadIdx.x % RT == 0) {
    t = sm[sub * (RT / 32)];
#pragma unroll
    for (int i = 1; i < RT / 32; ++i) t = t + sm[sub * (RT / 32) + i];
  }
  return t;
}

// two such sums at once (sm: two arrays of the kernel's)
__device__ __forceinline__ void cg_sub_sum2(double& a, double& b, double* sm, double* sm2) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    a = a + __shfl_xor_sync(0xffffffffu, a, off);
    b = b + __shfl_xor_sync(0xffffffffu, b, off);
  }
  const int sub = threadIdx.x / RT, w = (threadIdx.x >> 5) % (RT / 32);
  if ((threadIdx.x & 31) == 0) {
    sm[sub * (RT / 32) + w] = a;
    sm2[sub * (RT / 32) + w] = b;
  }
  asm volatile("bar.sync %0, %1;" ::"r"(1 + sub), "n"(RT) : "memory");
  if (threadIdx.x % RT == 0) {
    a = sm[sub * (RT / 32)];
    b = sm2[sub * (RT / 32)];
#pragma unroll
    for (int i = 1; i < RT / 32; ++i) {
      a = a + sm[sub * (RT / 32) + i];
      b = b + sm2[sub * (RT / 32) + i];
    }
  }
}

// Total of the chunk partials, in chunk_kernel's order, by every block: sum s
// by sub-group s (NS <= kCgSubs sums), then to all threads through tot
template <int NS>
__device__ __forceinline__ void cg_total(const double* partials, int nch, double* sm, double* tot) {
  const int sub = threadIdx.x / RT;
  if (sub < NS) {
    double a = 0.0;
    for (int i = threadIdx.x % RT; i < nch; i += RT) a = a + __ldcg(partials + (size_t)sub * nch + i);
    a = cg_sub_sum(a, sm);
    if (threadIdx.x % RT == 0) tot[sub] = a;
  }
  __syncthreads();
}

// first: the solve starts here, from `init`, with r = b - A x; otherwise it goes
// on from the device state. S receives the state.
template <class T, int N, bool CLUSTER, bool EDGE, class State>
__global__ void __launch_bounds__(kCgThreads, 1) cg_persist(CgArgs<T> A, State* S, State init,
                                                            int first) {
  extern __shared__ __align__(16) unsigned char cg_smem[];
  __shared__ double sm[kCgSubs * (RT / 32)], sm2[kCgSubs * (RT / 32)], tot[2];
  __shared__ int ok;
  State c = first ? init : *S;  // every block keeps the scalars, computed alike
  if (c.done) return;
  if (grid_failed(A.bar)) return;
  const int sub = threadIdx.x / RT, tid = threadIdx.x % RT;
  const int ch = blockIdx.x + gridDim.x * sub;  // at most one chunk a sub-group
  const bool mine = ch < A.nch;
  const int64_t base = (int64_t)ch * RCHUNK + tid;
  // element m of this thread at [m * RT + tid]
  T* ps = reinterpret_cast<T*>(cg_smem) + (size_t)sub * 4 * RCHUNK;
  T *rs = ps + RCHUNK, *xs = rs + RCHUNK, *ds = xs + RCHUNK;
  const int left = mine ? (int)min((int64_t)RPER, (A.n - base + RT - 1) / RT) : 0;
  for (int m = 0; m < left; ++m) {
    const int64_t i = base + (int64_t)m * RT;
    if (!first) {
      ps[m * RT + tid] = A.p[i];
      rs[m * RT + tid] = A.r[i];
    }
    xs[m * RT + tid] = A.x[i];
    ds[m * RT + tid] = A.dg[i];
  }
  const int nsub = ((int)blockIdx.x < A.nch) + ((int)(blockIdx.x + gridDim.x) < A.nch);
  unsigned char* cache = cg_smem + nsub * cg_chunk_bytes<T>();
  const int per = 32 >> A.lw;
  const int ncache = (int)((A.smem - nsub * cg_chunk_bytes<T>()) /
                           (A.maxg * cg_group_bytes<T, N>(A.nl))) / per * per;
  cg_cache<T, N>(A, cache, ncache);
  __syncthreads();
  double* part_pq = A.partials;
  double* part_rr = A.partials + A.nch;  // <r, r>, then <r, z>
  unsigned target = 0;
  T zv[RPER];
  if (first) {
    cg_apply<T, N, EDGE>(A, A.x, cache, ncache);
    if (!cg_barrier<CLUSTER>(A.bar, target, &ok)) return;
    if (mine) {
      double a0 = 0.0, a1 = 0.0;
#pragma unroll
      for (int m = 0; m < RPER; ++m) {
        if (m < left) {
          const int64_t i = base + (int64_t)m * RT;
          const T ri = A.b[i] - __ldcg(A.z + i);
          const T zi = ri / ds[m * RT + tid];
          rs[m * RT + tid] = ri;
          ps[m * RT + tid] = zi;
          __stcg(A.p + i, zi);
          a0 = fma((double)ri, (double)ri, a0);
          a1 = fma((double)ri, (double)zi, a1);
        }
      }
      cg_sub_sum2(a0, a1, sm, sm2);
      if (tid == 0) {
        __stcg(part_rr + ch, a0);
        __stcg(part_rr + A.nch + ch, a1);
      }
    }
    if (!cg_barrier<CLUSTER>(A.bar, target, &ok)) return;
    cg_total<2>(part_rr, A.nch, sm, tot);
    c.applies = 1;
    c.r_nrm_0 = sqrt(tot[0]);
    c.rz = tot[1];
    if (c.r_nrm_0 < 2.220446049250313e-16) {  // :531
      c.done = 1;
      c.converged = 1;
      c.r_nrm = c.r_nrm_0;
    }
  }
  for (int it = 0; it < A.iters && !c.done; ++it) {
    cg_apply<T, N, EDGE>(A, A.p, cache, ncache);
    if (!cg_barrier<CLUSTER>(A.bar, target, &ok)) return;
    if (mine) {
#pragma unroll
      for (int m = 0; m < RPER; ++m) zv[m] = m < left ? __ldcg(A.z + base + m * RT) : T(0);
      double acc = 0.0;
#pragma unroll
      for (int m = 0; m < RPER; ++m)
        if (m < left) acc = fma((double)ps[m * RT + tid], (double)zv[m], acc);
      acc = cg_sub_sum(acc, sm);
      if (tid == 0) __stcg(part_pq + ch, acc);
    }
    if (!cg_barrier<CLUSTER>(A.bar, target, &ok)) return;
    cg_total<1>(part_pq, A.nch, sm, tot);
    c.applies += 1;
    const double alpha = c.rz / tot[0], neg_alpha = -alpha;
    if (mine) {
      double a0 = 0.0, a1 = 0.0;
#pragma unroll
      for (int m = 0; m < RPER; ++m) {
        if (m < left) {
          const int o = m * RT + tid;
          xs[o] = fmaT((T)alpha, ps[o], xs[o]);
          const T ri = fmaT((T)neg_alpha, zv[m], rs[o]);
          rs[o] = ri;
          a0 = fma((double)ri, (double)ri, a0);
          const T zi = ri / ds[o];
          zv[m] = zi;
          a1 = fma((double)ri, (double)zi, a1);
        }
      }
      cg_sub_sum2(a0, a1, sm, sm2);
      if (tid == 0) {
        __stcg(part_rr + ch, a0);
        __stcg(part_rr + A.nch + ch, a1);
      }
    }
    if (!cg_barrier<CLUSTER>(A.bar, target, &ok)) return;
    cg_total<2>(part_rr, A.nch, sm, tot);
    c.iter += 1;
    const double beta = tot[1] / c.rz;
    c.rz = tot[1];
    c.r_nrm = sqrt(tot[0]);
    if (mine) {
#pragma unroll
      for (int m = 0; m < RPER; ++m) {
        if (m < left) {
          const int o = m * RT + tid;
          ps[o] = fmaT((T)beta, ps[o], zv[m]);
          __stcg(A.p + base + m * RT, ps[o]);
        }
      }
    }
    if (c.monitor) {
      if (c.r_nrm / c.r_nrm_0 <= c.r_tol || c.r_nrm <= c.a_tol) {  // :563
        c.done = 1;
        c.converged = 1;
      } else if (isnan(c.r_nrm)) {
        c.done = 1;
        c.status = LFX_NAN_DETECTED;
      }
    }
    if (c.iter >= c.max_iter) c.done = 1;
    if (c.done) break;
    if (!cg_barrier<CLUSTER>(A.bar, target, &ok)) return;
  }
  for (int m = 0; m < left; ++m) {
    A.x[base + m * RT] = xs[m * RT + tid];
    A.r[base + m * RT] = rs[m * RT + tid];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *S = c;
  if (!CLUSTER) cg_leave(A.bar);
}

}  // namespace lfx
