// Batched, continuously admitted mixed-precision solves of many independent
// SPD systems (the W0 mass+diffusion and W2 Helmholtz operators are both SPD,
// with SPD Jacobi / column-tridiagonal preconditioners), run by ONE persistent
// kernel per CUDA graph replay.
//
// Algorithm per slot: preconditioned CG whose recurrences, operator apply and
// preconditioner run in FP32, with reliable updates: the steps accumulate in
// an FP32 correction; when the FP32 recursive residual has fallen by a factor
// kDelta since the last true residual (or reaches the tolerance), the
// correction is added to the FP64 solution and the true residual b - A x is
// recomputed with the FP64 operator and replaces it. A slot converges only on
// that FP64 true residual, ||b - A x|| / ||b - A x0||.
//
// One launch (cooperative: every block resident, so the grid-wide phase
// barriers cannot wait on a block that never runs) loops over `iters`
// super-iterations. Each super-iteration is a fixed sequence of phases, every
// phase covering all admitted slots through host-built work lists and ending
// at a grid barrier whose spin is bounded in time (a run-out sets an error
// flag, and every block leaves at its next barrier):
//   A   z = A32 p: the cell scatter of the reference's colour loop
//       (matrix_vector_kernel_mod.F90:107-140) over each slot's packed FP32
//       upper triangles, one phase per colour and per L2 group of slots (the
//       slots of one group keep p and the partial sums of z in L2 across
//       their colours); the last writer of every dof adds p_i z_i to its cell
//       column's share of <p, z>
//   F   alpha = rz / <p, z> per slot, the column shares summed in order
//   U   xc += alpha p, r -= alpha z, ||r||^2 (and, for a Jacobi slot, <r, r/d>
//       and beta); a slot whose residual fell by kDelta, reached its
//       tolerance or its iteration limit asks for a true residual
//   R   (only when some slot asked, or was just admitted) x += xc; the FP64
//       residual b - A64 x by the same cell scatter on the FP64 packed
//       triangles; r = r64, ||r64||, convergence
//   C   (slots with a column preconditioner) Thomas sweeps of the columns,
//       then z = r / d on the other rows with <r, z> and beta
//   P   p = z + beta p
// Work items: apply items of up to `cells_per_item` cell columns of one
// colour of one slot, one warp each (a column's segments in order);
// 4096-value chunk items (slot, one chunk or four), one block each, for the vector
// phases; 64-column items for the sweeps. Per-slot sums are reduced in an
// order fixed by the slot alone (per cell column, per 4096-value chunk, then
// in index order), so a slot's result is bit-identical whatever else is in
// the batch and whatever launch shape the autotuner picks.
//
// Memory: a slot's Krylov state (r64 FP64; r, p, z, xc FP32; its partial
// sums) is allocated at admission from the device's stream-ordered memory
// pool, and admission is refused while the device's free memory would drop
// under the batch's reserve. The operators, preconditioners and b, x belong
// to the caller and stay alive until the slot is retired.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <map>
#include <vector>

#include "lfx_internal.cuh"

using namespace lfx;

namespace {

enum { PH_EMPTY = 0, PH_INIT = 1, PH_RUN = 2, PH_DONE = 3 };

constexpr double kDelta = 1e-3;  // reliable update when ||r|| drops by this factor
constexpr int kBT = 256;         // threads per block of the persistent kernel
constexpr int kBW = kBT / 32;    // warps per block
constexpr int kMaxBps = 3;       // blocks per SM the kernel is built for (launch bounds)
constexpr int kBSub = 2;         // a chunk item: kBSub chunks of RCHUNK values (4096)
constexpr int kChGroup = 4;       // chunks a chunk item covers when there are many
constexpr int kMaxIters = 64;    // super-iterations per launch, at most
constexpr int kMaxSeg = 4;       // warps (segments of <= 31 levels) per cell column, at most
constexpr int kMaxColours = 8;   // cell colours of a slot, at most
constexpr int kBRows = 160;      // rows per preconditioner column, at most
// column sweeps: a warp's 32 columns move in chunks of kSwCh rows through a
// tile of kSwLd-float rows, beside the warp's table of its columns
constexpr int kSwCh = 8;                      // rows per chunk
constexpr int kSwLd = 33;                     // tile row stride (floats)
struct SweepCol {                             // a warp's columns, per lane
  const int* ind[32];
  const float* r[32];
  float* z[32];
  int f[32], nrow[32];
};
// per warp: the tile, the column table, then two buffers of the factors of a
// chunk (two arrays of kSwCh x 32 each)
constexpr size_t kSweepTileBytes = sizeof(float) * kSwCh * kSwLd;
constexpr size_t kSweepFacBytes = sizeof(float) * 2 * 2 * kSwCh * 32;
constexpr size_t kSweepWarpBytes = kSweepTileBytes + sizeof(SweepCol) + kSweepFacBytes;
constexpr size_t kSweepBytes = kBW * kSweepWarpBytes;

inline int64_t bchunks(int64_t n) {
  return (n + (int64_t)kBSub * RCHUNK - 1) / ((int64_t)kBSub * RCHUNK);
}

struct BSlot {
  // cell scatter: packed upper triangles [q][p][k] in the colour-loop order
  // (block stride sblk elements) and the per-cell descriptors {map row,
  // flags, partners} in the same order
  const float* S32;
  const double* S64;
  const int* cdesc;
  // the FP32 triangles level-major: [q][k][4 npv] (npv float4 per level)
  const float4* L32;
  int32_t sblk32, sblk64, cdints, nl;
  int32_t nseg, segL, nch, ncell;
  int32_t npv, cma, ncol, nrow;
  int32_t canon, pad1;  // canon: every cell has the space's reference pair structure
  int64_t n;
  double* part;  // [0, 2 nch): chunk sums; [2 nch, 2 nch + ncell): <p, z> per cell column
  // preconditioner: FP32 Jacobi diagonal (zero on the column rows of a
  // column preconditioner) and the Thomas factors [row][column]
  const float* diag;
  const float *fa, *finv, *fc;
  const int *first, *ind;
  // vectors: x (FP64, the caller's) moves only at true residuals; between
  // them the FP32 xc accumulates the steps
  const double* b;
  double* x;
  double* r64;
  float *r, *p, *z, *xc;
};

struct BState {
  int phase, flag, iter, status;
  int max_iter, fresh, resid, pad;
  double tol, r0, rlast, rnorm, rz, alpha, beta, true_rel;
};

// device-resident launch parameters (the graph's kernel takes their address,
// so lists can be rebuilt and reallocated between replays)
struct BParams {
  const int4* items32;  // FP32 apply items {slot, q0, columns, 0}
  const int* off32;     // [ncolour * ngr32 + 1]: items of group g, colour c from off32[g ncolour + c]
  const int4* items64;  // FP64 residual items {slot, q0, columns, 0}
  const int* off64;
  const int2* chunks;   // {slot, group of chgrp chunks}
  const int2* cols;     // {slot, column}
  const int* slotlist;  // the slots the lists cover
  const BSlot* slots;
  BState* st;
  unsigned* tickets;
  int* need;            // [kMaxIters]: a slot takes a true residual in super-iteration it
  unsigned* bar;        // grid barrier {count, generation}
  unsigned* wq;         // [2] FP32 apply work counters, alternate phases
  int* err;             // LFX_TIMEOUT when a wait ran out
  int ngr32, ngr64, nchunk, ncolitem;
  int iters, max_slots, any_cma, ncolour;
  int nslot, chgrp;
  unsigned long long timeout_ns;
};

struct BShared {
  int last;
  double red[kBT / 32];
  double red2[kChGroup][2][kBT / 32];
  int ok;
};

__device__ __forceinline__ bool ph_run(int ph) { return ph == PH_RUN; }

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned atom_add_acqrel(unsigned* p, unsigned v) {
  unsigned old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

// (each phase below is a separate, non-inlined function: the kernel's loop
// then keeps nothing of one phase live across the others, and no phase
// spills registers)
//
// Grid-wide barrier of a cooperative launch. Thread 0 of each block reads the
// generation, arrives, and the last to arrive resets the count and releases
// the next generation; the others spin on it for at most timeout_ns (and stop
// when another block has reported an error). Returns false when the block must
// leave the kernel. (Pauses of 100 ns between polls and fences beside the
// acquire and release cost 2 % of a small batch.)
__device__ bool grid_sync(const BParams& P, BShared& sh) {
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned gen = ld_acquire(P.bar + 1);
    const unsigned arrived = atom_add_acqrel(P.bar, 1u);
    if (arrived == gridDim.x - 1) {
      P.bar[0] = 0u;
      st_release(P.bar + 1, gen + 1u);
    } else {
      unsigned long long t0 = 0;
      for (int spin = 0; ld_acquire(P.bar + 1) == gen; ++spin) {
        if ((spin & 15) != 15) continue;
        if (*(volatile int*)P.err) {
          ok = 0;
          break;
        }
        const unsigned long long t = gtimer();
        if (!t0) t0 = t;
        if (t - t0 > P.timeout_ns) {
          atomicExch(P.err, (int)LFX_TIMEOUT);
          ok = 0;
          break;
        }
      }
    }
    if (*(volatile int*)P.err) ok = 0;
    sh.ok = ok;
  }
  __syncthreads();
  return sh.ok != 0;
}

// block sum in a fixed order (lane butterfly, then warps left to right);
// result valid in thread 0
__device__ __forceinline__ double bsum(double acc, double* red) {
  acc = warp_butterfly(acc);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = acc;
  __syncthreads();
  double tot = 0.0;
  if (threadIdx.x == 0) {
    tot = red[0];
#pragma unroll
    for (int i = 1; i < kBW; ++i) tot = tot + red[i];
  }
  __syncthreads();
  return tot;
}

// a slot's state as one thread sees it in L2 (other blocks write it)
__device__ __forceinline__ void copy_state_in(BState* d, const BState* s) {
  const int* a = reinterpret_cast<const int*>(s);
  int* b = reinterpret_cast<int*>(d);
#pragma unroll
  for (int i = 0; i < (int)(sizeof(BState) / 4); ++i) b[i] = __ldcg(a + i);
}
__device__ __forceinline__ void copy_state_out(BState* d, const BState& s) {
  const int* a = reinterpret_cast<const int*>(&s);
  int* b = reinterpret_cast<int*>(d);
#pragma unroll
  for (int i = 0; i < (int)(sizeof(BState) / 4); ++i) __stcg(b + i, a[i]);
}

template <int N>
__host__ __device__ constexpr int pidx(int i, int j) {
  return i <= j ? i * N - i * (i - 1) / 2 + (j - i) : j * N - j * (j - 1) / 2 + (i - j);
}

// row and column (row <= column) of packed upper-triangle entry p
template <int N>
__host__ __device__ constexpr int prow(int p) {
  int i = 0;
  while (p >= N - i) {
    p -= N - i;
    ++i;
  }
  return i;
}
template <int N>
__host__ __device__ constexpr int pcol(int p) {
  int i = 0;
  while (p >= N - i) {
    p -= N - i;
    ++i;
  }
  return i + p;
}

// One warp's share of the cell scatter: segment sg (L <= 31 output levels)
// of the cell column at colour-loop position q. Lane l (1 <= l <= L) holds
// level k = sg L + l - 1 and writes the dofs of that level (and the bottom
// dof of a pair, whose upper-record terms come from the lane below); lane 0
// holds the level below the segment only to supply those terms. A dof gets
// its terms in the reference's colour order: the first cell on its column
// starts from zero, later ones from the stored sum, and in the residual form
// the last writes b - sum. With DOT the lane returns the sum of p_i y_i over
// the dofs it finished (the last writer of each dof).
template <class T, int NDF, bool RESID, bool DOT, bool CANON>
__device__ __forceinline__ double scatter_unit(const T* __restrict__ Mq, const int* __restrict__ dsc,
                                               int nl, int L, int sg, int lane,
                                               const T* x, T* y, const double* __restrict__ b) {
  int mf[NDF];
#pragma unroll
  for (int j = 0; j < NDF; ++j) mf[j] = __ldg(dsc + j);
  const uint32_t flags = (uint32_t)__ldg(dsc + NDF), part = (uint32_t)__ldg(dsc + NDF + 1);
  const int k = sg * L + lane - 1;
  const bool own = lane >= 1 && lane <= L;
  const bool v = k >= 0 && k < nl && lane <= L;
  const T* Mc = Mq + (v ? k : 0);
  constexpr int NP = NDF * (NDF + 1) / 2;
  T m[NP], xv[NDF], yo[NDF];
  // the matrix is read once per apply (streaming loads); x and the partial
  // sums of y are written during the launch, so they are read through L2
#pragma unroll
  for (int p = 0; p < NP; ++p) m[p] = v ? __ldcs(Mc + p * nl) : T(0);
#pragma unroll
  for (int j = 0; j < NDF; ++j) xv[j] = v ? __ldcg(x + mf[j] + k) : T(0);
#pragma unroll
  for (int df = 0; df < NDF; ++df) {
    const bool lower = is_lower<NDF, CANON>(flags, df), upper = is_upper<NDF, CANON>(flags, df);
    const bool opens = (flags >> df) & 1u;
    const bool live = own && (lower ? k <= nl : v);
    yo[df] = (!upper && !opens && live) ? __ldcg(y + mf[df] + k) : T(0);
  }
  double dot = 0.0;
#define MV(i, j) m[pidx<NDF>(i, j)]
#pragma unroll
  for (int df = 0; df < NDF; ++df) {
    if (is_upper<NDF, CANON>(flags, df)) continue;  // upper record: summed with its lower one
    const bool last = (flags >> (24 + df)) & 1u;
    if (is_lower<NDF, CANON>(flags, df)) {
      const int bsel = partner<NDF, CANON>(part, df);
#pragma unroll
      for (int bb = df + 1; bb < NDF; ++bb) {
        if (bb != bsel) continue;
        T acc = yo[df];
#pragma unroll
        for (int j = 0; j < NDF; ++j) {
          const T mb = __shfl_up_sync(0xffffffffu, MV(bb, j), 1);
          const T xb = __shfl_up_sync(0xffffffffu, xv[j], 1);
          if (v) acc = fmaT(MV(df, j), xv[j], acc);
          if (own && k >= 1 && k <= nl) acc = fmaT(mb, xb, acc);
        }
        if (own && k <= nl) {
          const int row = mf[df] + k;
          if (RESID && last)
            __stcg(y + row, (T)(b[row] - (double)acc));
          else
            __stcg(y + row, acc);
          if (DOT && last) {
            const T pr = k < nl ? xv[df] : __ldcg(x + row);
            dot = fma((double)pr, (double)acc, dot);
          }
        }
      }
    } else {
      T acc = yo[df];
#pragma unroll
      for (int j = 0; j < NDF; ++j) acc = fmaT(MV(df, j), xv[j], acc);
      if (own && v) {
        const int row = mf[df] + k;
        if (RESID && last)
          __stcg(y + row, (T)(b[row] - (double)acc));
        else
          __stcg(y + row, acc);
        if (DOT && last) dot = fma((double)xv[df], (double)acc, dot);
      }
    }
  }
#undef MV
  return dot;
}
// one form per pair structure, each its own function (the apply phase keeps
// one register allocation for both)
template <class T, int NDF, bool FP64, bool CANON>
__device__ __noinline__ double scatter_unit_c(const T* __restrict__ Mq, const int* __restrict__ dsc,
                                              int nl, int L, int sg, int lane, const T* x, T* y,
                                              const double* __restrict__ b) {
  return scatter_unit<T, NDF, FP64, !FP64, CANON>(Mq, dsc, nl, L, sg, lane, x, y, b);
}

// The apply items [i0, i1) of one (group, colour) phase, one warp per item
// (no block-wide barrier: each warp walks its item's cell columns, and each
// column's segments, in order). FP32 (the form apply_phase32_ring restates on
// the level-major copy): z = A32 p for running slots, each column's share of
// <p, z> (lanes over the column's segments in order, then the lane
// butterfly) stored at its colour-loop position. FP64 (the form the kernel
// runs): r64 = b - A64 x for slots taking a true residual. An item's packed
// matrices are one
// contiguous run, which lane 0 asks the L2 to fetch in bulk
// (cp.async.bulk.prefetch) before the warp's first loads.
template <int NDF, bool FP64>
__device__ __noinline__ void apply_phase(const BParams& P, const int4* __restrict__ items, int i0,
                                         int i1) {
  using T = typename std::conditional<FP64, double, float>::type;
  const int lane = threadIdx.x & 31;
  const int gw = blockIdx.x * kBW + (threadIdx.x >> 5), nw = gridDim.x * kBW;
  for (int u = i0 + gw; u < i1; u += nw) {
    const int4 it = __ldg(items + u);
    const int s = it.x;
    const int ph = __ldcg(&P.st[s].phase), fl = __ldcg(&P.st[s].flag);
    if (FP64 ? !(ph == PH_INIT || (ph == PH_RUN && fl)) : !ph_run(ph)) continue;
    const BSlot* D = P.slots + s;
    const T* M = FP64 ? (const T*)D->S64 : (const T*)D->S32;
    const int sblk = FP64 ? D->sblk64 : D->sblk32;
    const int* cdesc = D->cdesc;
    const int cdints = D->cdints, nl = D->nl, nseg = D->nseg, L = D->segL;
    const T* x = FP64 ? (const T*)D->x : (const T*)D->p;
    T* y = FP64 ? (T*)D->r64 : (T*)D->z;
    const double* bb = D->b;
    const int q0 = it.y, nq = it.z;
    if (lane == 0) {
      const T* run = M + (size_t)q0 * sblk;
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(run),
                   "r"((unsigned)((size_t)nq * sblk * sizeof(T)))
                   : "memory");
    }
    double* part = FP64 ? nullptr : D->part + 2 * (int64_t)D->nch;
    for (int c = 0; c < nq; ++c) {
      const int q = q0 + c;
      double dot = 0.0;
      for (int sg = 0; sg < nseg; ++sg)
        dot += D->canon ? scatter_unit_c<T, NDF, FP64, true>(M + (size_t)q * sblk,
                                                             cdesc + (size_t)q * cdints, nl, L, sg,
                                                             lane, x, y, bb)
                        : scatter_unit_c<T, NDF, FP64, false>(M + (size_t)q * sblk,
                                                              cdesc + (size_t)q * cdints, nl, L,
                                                              sg, lane, x, y, bb);
      if (!FP64) {
        const double w = warp_butterfly(dot);
        if (lane == 0) __stcg(part + q, w);
      }
    }
  }
}

// ---- The FP32 apply with each warp's matrix stream on the bulk-copy
// engine. A warp walks its items' units (cell column, segment) in order; a
// unit's levels are one contiguous run of the level-major copy, which lane 0
// moves into the warp's ring in shared memory with one cp.async.bulk
// completing on the stage's mbarrier, kRing units ahead, so the bytes in
// flight cost no registers. The lanes gather x and the partial sums of y
// through L2 before they wait for the unit's matrix, then read their level's
// entries from the ring. Each lane forms the eight (six) row sums of its own
// cell; a dof on a vertical pair (bottom of level k, top of level k - 1)
// takes the row sum of the lane below with one shuffle, so the FP32 sums are
// grouped per cell (the FP64 form keeps the reference's term order; the FP64
// true residuals fix the accuracy of the solve). A wait is
// bounded by the batch's wait limit: on a time-out the warp records
// LFX_TIMEOUT, waits (bounded again) for the copies it still has in flight,
// and returns; the kernel leaves at its next grid barrier.
constexpr int kRing = 2;  // ring stages per warp

template <int NDF>
struct Ring {
  static constexpr int NP = NDF * (NDF + 1) / 2, NPV = (NP + 3) / 4;
  static constexpr int LEVEL = NPV * 16;           // bytes of one level
  static constexpr int STAGE = 32 * LEVEL;         // a segment: at most 32 levels
  static constexpr int WARP = kRing * STAGE;
};

// dynamic shared memory: the rings (or the sweeps' staging, which the
// phases never hold at once), then kRing mbarriers per warp past both
__host__ __device__ constexpr size_t ring_bar_offset(int ndf) {
  return ((ndf == 8 ? (size_t)kBW * Ring<8>::WARP : (size_t)kBW * Ring<6>::WARP) > kSweepBytes
              ? (ndf == 8 ? (size_t)kBW * Ring<8>::WARP : (size_t)kBW * Ring<6>::WARP)
              : kSweepBytes) +
         15 & ~(size_t)15;
}
__host__ __device__ constexpr size_t dyn_bytes(int ndf) {
  return ring_bar_offset(ndf) + (size_t)kBW * kRing * 8;
}

__device__ __forceinline__ unsigned su32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ bool ring_try(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(su32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// waits for the phase of the given parity for at most limit ns
__device__ __forceinline__ bool ring_wait(uint64_t* bar, unsigned parity,
                                          unsigned long long limit) {
  if (ring_try(bar, parity)) return true;
  const unsigned long long t0 = gtimer();
  while (!ring_try(bar, parity))
    if (gtimer() - t0 > limit) return false;
  return true;
}
__device__ __forceinline__ void ring_issue(void* dst, const void* src, unsigned bytes,
                                           uint64_t* bar) {
  // the stage was last read through the generic proxy
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(bar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          su32(dst)),
      "l"(src), "r"(bytes), "r"(su32(bar))
      : "memory");
}

// row sums of a cell from its packed triangle, entry by entry with the
// entry's (row, column) fixed at compile time: entry (a, b), a <= b, adds to
// row a (times x_b) and, mirrored, to row b
template <int NDF, int P>
__device__ __forceinline__ void row_entry(float e, const float (&xv)[NDF], float (&rs)[NDF]) {
  if constexpr (P < NDF * (NDF + 1) / 2) {
    constexpr int a = prow<NDF>(P), b = pcol<NDF>(P);
    rs[a] = fmaf(e, xv[b], rs[a]);
    if constexpr (a != b) rs[b] = fmaf(e, xv[a], rs[b]);
  }
}
template <int NDF, int PV>
__device__ __forceinline__ void row_sums(const float4* Ms, bool v, const float (&xv)[NDF],
                                         float (&rs)[NDF]) {
  if constexpr (PV < Ring<NDF>::NPV) {
    const float4 t = v ? Ms[PV] : make_float4(0.f, 0.f, 0.f, 0.f);
    row_entry<NDF, 4 * PV>(t.x, xv, rs);
    row_entry<NDF, 4 * PV + 1>(t.y, xv, rs);
    row_entry<NDF, 4 * PV + 2>(t.z, xv, rs);
    row_entry<NDF, 4 * PV + 3>(t.w, xv, rs);
    row_sums<NDF, PV + 1>(Ms, v, xv, rs);
  }
}

// one apply item (nq cell columns from q0 of slot record D) through the
// warp's ring; false when a ring wait ran out (recorded and drained)
template <int NDF, bool CANON>
__device__ __forceinline__ bool ring_item(const BParams& P, const BSlot& D, int q0, int nq,
                                          unsigned char* ring, uint64_t* bars, unsigned& seq,
                                          int lane) {
  using R = Ring<NDF>;
  constexpr int NPV = R::NPV;
  const float4* M4 = D.L32;
  const int* cdesc = D.cdesc;
  const int cdints = D.cdints, nl = D.nl, nseg = D.nseg, L = D.segL;
  const float* x = D.p;
  float* y = D.z;
  double* part = D.part + 2 * (int64_t)D.nch;
  const int nunit = nq * nseg;
  // unit j: column j / nseg, segment j % nseg; its levels kf..kl land at
  // ring slot (level - (sg L - 1)), so lane l finds level sg L + l - 1
  auto issue = [&](int j) {
    const int c = j / nseg, sg = j % nseg;
    const int kf = max(sg * L - 1, 0), kl = min(sg * L + L - 1, nl - 1);
    const unsigned st = (seq + (unsigned)j) % kRing;
    ring_issue(ring + st * R::STAGE + (kf - (sg * L - 1)) * R::LEVEL,
               M4 + ((size_t)(q0 + c) * nl + kf) * NPV, (unsigned)(kl - kf + 1) * R::LEVEL,
               bars + st);
  };
  if (lane == 0)
    for (int j = 0; j < kRing && j < nunit; ++j) issue(j);
  int mf[NDF];
  uint32_t flags = 0, prt = 0;
  double dot = 0.0;
  bool ok = true;
  int jf = 0;  // the unit whose wait ran out
  for (int j = 0; j < nunit; ++j) {
    const int c = j / nseg, sg = j % nseg;
    if (sg == 0) {
      const int* dsc = cdesc + (size_t)(q0 + c) * cdints;
#pragma unroll
      for (int jj = 0; jj < NDF; ++jj) mf[jj] = __ldg(dsc + jj);
      flags = (uint32_t)__ldg(dsc + NDF);
      prt = (uint32_t)__ldg(dsc + NDF + 1);
    }
    const int k = sg * L + lane - 1;
    const bool own = lane >= 1 && lane <= L;
    const bool v = k >= 0 && k < nl && lane <= L;
    float xv[NDF], yo[NDF];
#pragma unroll
    for (int jj = 0; jj < NDF; ++jj) xv[jj] = v ? __ldcg(x + mf[jj] + k) : 0.f;
#pragma unroll
    for (int df = 0; df < NDF; ++df) {
      const bool lower = is_lower<NDF, CANON>(flags, df), upper = is_upper<NDF, CANON>(flags, df);
      const bool opens = (flags >> df) & 1u;
      const bool live = own && (lower ? k <= nl : v);
      yo[df] = (!upper && !opens && live) ? __ldcg(y + mf[df] + k) : 0.f;
    }
    const unsigned g = seq + (unsigned)j, st = g % kRing;
    if (!ring_wait(bars + st, (g / kRing) & 1u, P.timeout_ns)) {
      ok = false;
      jf = j;
      break;
    }
    // row sums of this lane's cell, four packed entries at a time: entry
    // (a, b), a <= b, adds to row a (times x_b) and, mirrored, to row b
    float rs[NDF];
#pragma unroll
    for (int df = 0; df < NDF; ++df) rs[df] = 0.f;
    row_sums<NDF, 0>(reinterpret_cast<const float4*>(ring + st * R::STAGE) + lane * NPV, v, xv, rs);
    // every lane has read the stage: it takes unit j + kRing
    __syncwarp();
    if (lane == 0 && j + kRing < nunit) issue(j + kRing);
#pragma unroll
    for (int df = 0; df < NDF; ++df) {
      if (is_upper<NDF, CANON>(flags, df)) continue;  // upper record: summed with its lower one
      const bool last = (flags >> (24 + df)) & 1u;
      if (is_lower<NDF, CANON>(flags, df)) {
        const int bsel = partner<NDF, CANON>(prt, df);
#pragma unroll
        for (int bb = df + 1; bb < NDF; ++bb) {
          if (bb != bsel) continue;
          const float below = __shfl_up_sync(0xffffffffu, rs[bb], 1);
          float acc = yo[df] + rs[df];
          if (own && k >= 1 && k <= nl) acc = acc + below;
          if (own && k <= nl) {
            const int row = mf[df] + k;
            __stcg(y + row, acc);
            if (last) {
              const float pr = k < nl ? xv[df] : __ldcg(x + row);
              dot = fma((double)pr, (double)acc, dot);
            }
          }
        }
      } else {
        const float acc = yo[df] + rs[df];
        if (own && v) {
          __stcg(y + mf[df] + k, acc);
          if (last) dot = fma((double)xv[df], (double)acc, dot);
        }
      }
    }
    if (sg == nseg - 1) {
      const double w = warp_butterfly(dot);
      if (lane == 0) __stcg(part + q0 + c, w);
      dot = 0.0;
    }
  }
  if (!ok) {
    // record the time-out, then wait (bounded: the batch's wait limit, at
    // least 2 s, since a copy in flight lands within microseconds unless
    // the memory system has stopped) for this warp's copies still in
    // flight before the kernel leaves
    if (lane == 0) {
      atomicExch(P.err, (int)LFX_TIMEOUT);
      const unsigned long long drain = P.timeout_ns > 2000000000ull ? P.timeout_ns : 2000000000ull;
      // units jf .. jf + kRing - 1 were issued and not consumed
      for (int j = jf; j < nunit && j < jf + kRing; ++j) {
        const unsigned g = seq + (unsigned)j;
        ring_wait(bars + g % kRing, (g / kRing) & 1u, drain);
      }
    }
    __syncwarp();
    return false;
  }
  seq += (unsigned)nunit;
  return true;
}

template <int NDF>
__device__ __noinline__ unsigned apply_phase32_ring(const BParams& P, const int4* __restrict__ items,
                                                    int i0, int i1, unsigned char* ring,
                                                    uint64_t* bars, unsigned seq, unsigned* ctr) {
  const int lane = threadIdx.x & 31;
  // warps take items by the phase's counter (lane 0), the next one asked for
  // while the current item runs
  unsigned nxt = 0;
  if (lane == 0) nxt = atomicAdd(ctr, 1u);
  nxt = __shfl_sync(0xffffffffu, nxt, 0);
  for (;;) {
    const int u = i0 + (int)nxt;
    if (u >= i1) break;
    if (lane == 0) nxt = atomicAdd(ctr, 1u);
    const int4 it = __ldg(items + u);
    const int s = it.x;
    if (!ph_run(__ldcg(&P.st[s].phase))) {  // warp-uniform
      nxt = __shfl_sync(0xffffffffu, nxt, 0);
      continue;
    }
    const BSlot& D = P.slots[s];
    const bool ok = D.canon ? ring_item<NDF, true>(P, D, it.y, it.z, ring, bars, seq, lane)
                            : ring_item<NDF, false>(P, D, it.y, it.z, ring, bars, seq, lane);
    if (!ok) return seq;
    nxt = __shfl_sync(0xffffffffu, nxt, 0);
  }
  return seq;
}

constexpr int kItemCols = 8;  // cell columns per apply item, at most

// alpha = rz / <p, z> for every running slot: one block per slot sums the
// slot's per-column shares in a fixed order
__device__ __noinline__ void alpha_phase(const BParams& P, BShared& sh) {
  for (int k = blockIdx.x; k < P.nslot; k += gridDim.x) {
    const int s = __ldg(P.slotlist + k);
    if (!ph_run(__ldcg(&P.st[s].phase))) continue;  // block-uniform
    const BSlot* D = P.slots + s;
    const double* part = D->part + 2 * (int64_t)D->nch;
    const int nc = D->ncell;
    double a = 0.0;
    // (eight loads in flight: one at a time took 11 of an iteration's 290 us)
#pragma unroll 8
    for (int i = threadIdx.x; i < nc; i += kBT) a = a + __ldcg(part + i);
    const double pz = bsum(a, sh.red);
    if (threadIdx.x == 0) {
      BState S;
      copy_state_in(&S, P.st + s);
      S.alpha = S.rz / pz;
      S.fresh = 0;
      copy_state_out(P.st + s, S);
    }
  }
}

// ---- Vector phases. An item is (slot, chunks of kBSub * RCHUNK = 4096
// values: one, or kChGroup of them). The block takes an item; each thread takes four consecutive
// values per step (16-byte accesses, masked at the vector's end), with the
// loads of two steps in flight before any store. The slot record is read
// where it lies (read-only during a launch: broadcast loads); the state
// words the elementwise work needs are read through L2 (written by other
// blocks in earlier phases). A slot's item is skipped or taken by the whole
// block alike: its state changes in this phase only in fin, which runs after
// every item of the slot. Sums: FP64 per thread, then the block sum in a
// fixed order (lanes by butterfly, warps left to right) into the chunk's
// partial; the last block to finish a slot's chunks (ticket) sums the
// partials in chunk order and runs fin(record, state, totals).
// The chunk is small so that a few slots fill the grid: twelve uneven W0 slots
// (3.6 M rows) took 143 ms with 16384 values (220 items for 444 blocks), 139 with
// 8192, 138 with 4096; six W2 ones 7.8, 7.6, 7.4; sixty W0 ones 469, 452, 458.
// Where that gives every block of the largest grid 4 kChGroup chunks or more, an item
// takes kChGroup of them (each with its own partial, so the bits stay), with one
// block sum and one ticket an item: 256 uneven W0 slots (63 M rows, 15 424 chunks)
// took 3388 us an iteration with a chunk an item, 3291 so.
// Indices are 32 bits wide (a field has less than 2^31 values) and a phase without
// sums takes a group's chunks as one run: with 64-bit indices the group's counters
// spilled in the first phase (52 bytes; 4 now). 64 W2 slots (275 M rows) to 1e-10:
// 238.4 -> 235.3 ms, 16 (69 M) 67.0 -> 66.1, 6 (38 M) 42.6 -> 42.1; 256 W0 slots
// (59 M) 664 -> 663, 12 (2.5 M) 62.0 -> 61.3. With chunks of 16384 values and no
// groups those took 232.6, 66.0, 42.3, 658 and 69.5: the largest batches pay 1 % for
// what the few slots gain. (Sums of a group's chunks kept in shared memory and
// added up side by side: 241.5 ms for the 64.)
constexpr int kVStep = kBT * 4;                   // values per block step
constexpr int kVSteps = kBSub * RCHUNK / kVStep;  // steps per chunk (4)
static_assert(kVSteps % 2 == 0, "two steps per pass");

struct VState {
  int phase, fresh;
  float alpha, beta;
};

// four consecutive values from i (zeros past n); RO: read-only during the
// launch (non-coherent cache), else read through L2
template <bool RO>
__device__ __forceinline__ float4 vld(const float* a, unsigned i, unsigned n) {
  if (i + 3 < n)
    return RO ? __ldg(reinterpret_cast<const float4*>(a + i))
              : __ldcg(reinterpret_cast<const float4*>(a + i));
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (i < n) v.x = RO ? __ldg(a + i) : __ldcg(a + i);
  if (i + 1 < n) v.y = RO ? __ldg(a + i + 1) : __ldcg(a + i + 1);
  if (i + 2 < n) v.z = RO ? __ldg(a + i + 2) : __ldcg(a + i + 2);
  return v;
}
__device__ __forceinline__ void vst(float* a, unsigned i, unsigned n, float4 v) {
  if (i + 3 < n) {
    __stcg(reinterpret_cast<float4*>(a + i), v);
    return;
  }
  if (i < n) __stcg(a + i, v.x);
  if (i + 1 < n) __stcg(a + i + 1, v.y);
  if (i + 2 < n) __stcg(a + i + 2, v.z);
}
struct D4 {
  double v[4];
};
struct DF4 {
  D4 d;
  float4 f;
};
template <bool RO>
__device__ __forceinline__ D4 vldd(const double* a, unsigned i, unsigned n) {
  D4 r;
  if (i + 3 < n) {
    const double2 lo = RO ? __ldg(reinterpret_cast<const double2*>(a + i))
                          : __ldcg(reinterpret_cast<const double2*>(a + i));
    const double2 hi = RO ? __ldg(reinterpret_cast<const double2*>(a + i + 2))
                          : __ldcg(reinterpret_cast<const double2*>(a + i + 2));
    r.v[0] = lo.x; r.v[1] = lo.y; r.v[2] = hi.x; r.v[3] = hi.y;
    return r;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) r.v[c] = i + c < n ? (RO ? __ldg(a + i + c) : __ldcg(a + i + c)) : 0.0;
  return r;
}
__device__ __forceinline__ void vstd(double* a, unsigned i, unsigned n, const D4& r) {
  if (i + 3 < n) {
    __stcg(reinterpret_cast<double2*>(a + i), make_double2(r.v[0], r.v[1]));
    __stcg(reinterpret_cast<double2*>(a + i + 2), make_double2(r.v[2], r.v[3]));
    return;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
    if (i + c < n) __stcg(a + i + c, r.v[c]);
}
__device__ __forceinline__ void f4a(float4 v, float* o) {
  o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
__device__ __forceinline__ float4 a4f(const float* o) { return make_float4(o[0], o[1], o[2], o[3]); }

// ld(record, i, n) loads the four values at i; op(record, state, i, n,
// values, acc) computes and stores them (components past n left alone)
template <int NR, class Pred, class Ld, class Op, class Fin>
__device__ __noinline__ void vec_phase(const BParams& P, BShared& sh, Pred pred, Ld ld, Op op, Fin fin) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int u = blockIdx.x; u < P.nchunk; u += gridDim.x) {
    const int2 item = __ldg(P.chunks + u);
    const int s = item.x;
    const BState* Sg = P.st + s;
    if (!pred(__ldcg(&Sg->phase), __ldcg(&Sg->flag))) continue;  // block-uniform
    const BSlot& D = P.slots[s];
    VState V;
    V.phase = __ldcg(&Sg->phase);
    V.fresh = __ldcg(&Sg->fresh);
    V.alpha = (float)__ldcg(&Sg->alpha);
    V.beta = (float)__ldcg(&Sg->beta);
    const unsigned n = (unsigned)D.n;  // (below 2^31: 64-bit indices spill in the first phase)
    const int ch0 = item.y * P.chgrp, nk = min(P.chgrp, D.nch - ch0);
    const int reps = NR > 0 ? nk : 1, steps = NR > 0 ? kVSteps : nk * kVSteps;
    for (int k = 0; k < reps; ++k) {
      double acc[NR > 0 ? NR : 1];
#pragma unroll
      for (int r = 0; r < (NR > 0 ? NR : 1); ++r) acc[r] = 0.0;
      const unsigned c0 = (unsigned)(ch0 + k) * (kBSub * RCHUNK);
      for (int stp = 0; stp < steps; stp += 2) {
        if (c0 + stp * kVStep >= n) break;  // block-uniform
        const unsigned i0 = c0 + stp * kVStep + 4 * threadIdx.x, i1 = i0 + kVStep;
        const auto a = ld(D, i0, n);
        const auto b = ld(D, i1, n);
        if (i0 < n) op(D, V, i0, n, a, acc);
        if (i1 < n) op(D, V, i1, n, b, acc);
      }
      if constexpr (NR > 0) {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const double t = warp_butterfly(acc[r]);
          if (lane == 0) sh.red2[k][r][w] = t;
        }
      }
    }
    if constexpr (NR > 0) {
      const int nch = D.nch;
      double* part = D.part;
      __syncthreads();
      if (w == 0) {
        if (lane < nk * NR) {
          const int k = lane / NR, r = lane % NR;
          double t = sh.red2[k][r][0];
#pragma unroll
          for (int q = 1; q < kBW; ++q) t = t + sh.red2[k][r][q];
          __stcg(part + (int64_t)r * nch + ch0 + k, t);
          __threadfence();
        }
        __syncwarp();
        if (lane == 0) {
          __threadfence();
          sh.last = atomicAdd(&P.tickets[s], (unsigned)nk) == (unsigned)(nch - nk);
        }
      }
      __syncthreads();
      if (sh.last) {
        __threadfence();
        double a[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          a[r] = 0.0;
          for (int i = threadIdx.x; i < nch; i += kBT) a[r] = a[r] + __ldcg(part + (int64_t)r * nch + i);
          const double t = warp_butterfly(a[r]);
          if (lane == 0) sh.red2[0][r][w] = t;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
          double tot[NR];
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            tot[r] = sh.red2[0][r][0];
#pragma unroll
            for (int q = 1; q < kBW; ++q) tot[r] = tot[r] + sh.red2[0][r][q];
          }
          BState S;
          copy_state_in(&S, P.st + s);
          fin(D, S, tot);
          copy_state_out(P.st + s, S);
          P.tickets[s] = 0u;
        }
        __syncthreads();
      }
    }
  }
}

// Column sweeps, one warp per 32 consecutive list columns (one column a
// lane, any slots), no block barrier: rows move in chunks of kSwCh through a
// per-warp tile in shared memory (a column's rows are read and written as
// one coalesced run, kSwCh lanes a column), the factors come straight from
// [row][column] (coalesced across the lanes of one slot). The forward sweep
// leaves its values in z (FP32), the backward sweep reads them back; the
// arithmetic of thomas_sweep (FP64 carries, FP32 rows between the sweeps).
// 4-byte asynchronous copy of a read-only factor (zeros when !on)
__device__ __forceinline__ void sweep_fac_copy(float* dst, const float* src, bool on) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(su32(dst)), "l"(src),
               "r"(on ? 4 : 0)
               : "memory");
}

__device__ __noinline__ void sweep_phase_w(const BParams& P, unsigned char* wsm) {
  float (*tile)[kSwLd] = reinterpret_cast<float (*)[kSwLd]>(wsm);
  SweepCol& sc = *reinterpret_cast<SweepCol*>(wsm + kSweepTileBytes);
  float* facb = reinterpret_cast<float*>(wsm + kSweepTileBytes + sizeof(SweepCol));
  const int lane = threadIdx.x & 31;
  const int gw = blockIdx.x * kBW + (threadIdx.x >> 5), nw = gridDim.x * kBW;
  // a valid address for the copies that read nothing
  const float* dummy = reinterpret_cast<const float*>(P.cols);
  for (int u0 = gw * 32; u0 < P.ncolitem; u0 += nw * 32) {
    // this lane's column
    const int u = u0 + lane;
    int nrow = 0, nc = 1, c = 0;
    const float *fa = dummy, *finv = dummy, *fc = dummy;
    __syncwarp();
    sc.nrow[lane] = 0;
    if (u < P.ncolitem) {
      const int2 w = __ldg(P.cols + u);
      if (ph_run(__ldcg(&P.st[w.x].phase))) {
        const BSlot& D = P.slots[w.x];
        nrow = D.nrow;
        nc = D.ncol;
        c = w.y;
        fa = D.fa;
        finv = D.finv;
        fc = D.fc;
        sc.ind[lane] = D.ind;
        sc.r[lane] = D.r;
        sc.z[lane] = D.z;
        sc.f[lane] = __ldg(D.first + w.y);
        sc.nrow[lane] = nrow;
      }
    }
    int maxrow = nrow;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) maxrow = max(maxrow, __shfl_xor_sync(0xffffffffu, maxrow, o));
    __syncwarp();
    if (maxrow == 0) continue;
    // staging: lane = (column offset, row in the chunk); 32 / kSwCh columns
    // an instruction. The next chunk's rows (into registers, through L2:
    // other phases write r) and factors (into the other factor buffer, by
    // 4-byte cp.async: read-only) are in flight while a chunk is swept.
    constexpr int CPI = 32 / kSwCh, NG = 32 / CPI;
    const int hr = lane % kSwCh, hc = lane / kSwCh;
    auto fac = [&](int buf, int kind, int q) -> float* {
      return facb + ((buf * 2 + kind) * kSwCh + q) * 32 + lane;
    };
    auto gather = [&](const float* const* base, int i0, float (&v)[NG]) {
      const int i = i0 + hr;
#pragma unroll
      for (int m = 0; m < NG; ++m) {
        const int j = hc + CPI * m;
        v[m] = i < sc.nrow[j] ? __ldcg(base[j] + sc.f[j] + __ldg(sc.ind[j] + i)) : 0.f;
      }
    };
    auto stage = [&](int i0, const float (&v)[NG]) {
      const int i = i0 + hr;
#pragma unroll
      for (int m = 0; m < NG; ++m) {
        const int j = hc + CPI * m;
        if (i < sc.nrow[j]) tile[hr][j] = v[m];
      }
    };
    auto store = [&](int i0) {
      const int i = i0 + hr;
      for (int j = hc; j < 32; j += CPI)
        if (i < sc.nrow[j]) __stcg(sc.z[j] + sc.f[j] + __ldg(sc.ind[j] + i), tile[hr][j]);
    };
    float pv[NG];
    // forward: d_i = finv_i (r_i - fa_i d_{i-1}), left in z
    auto fwd_fac = [&](int i0, int buf) {
#pragma unroll
      for (int q = 0; q < kSwCh; ++q) {
        const int ii = i0 + q;
        const bool on = ii < nrow;
        sweep_fac_copy(fac(buf, 0, q), on ? finv + (size_t)ii * nc + c : dummy, on);
        sweep_fac_copy(fac(buf, 1, q), on ? fa + (size_t)ii * nc + c : dummy, on);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double d = 0.0;
    gather(sc.r, 0, pv);
    fwd_fac(0, 0);
    int buf = 0;
    for (int i0 = 0; i0 < maxrow; i0 += kSwCh, buf ^= 1) {
      stage(i0, pv);
      if (i0 + kSwCh < maxrow) {
        gather(sc.r, i0 + kSwCh, pv);
        fwd_fac(i0 + kSwCh, buf ^ 1);
      } else {
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
#pragma unroll
      for (int q = 0; q < kSwCh; ++q) {
        const int ii = i0 + q;
        if (ii < nrow) {
          const double iv = (double)*fac(buf, 0, q), av = (double)*fac(buf, 1, q);
          const double xv = (double)tile[q][lane];
          d = (ii == 0) ? iv * xv : iv * fma(-av, d, xv);
          tile[q][lane] = (float)d;
        }
      }
      __syncwarp();
      store(i0);
      __syncwarp();
    }
    // backward: z_i = d_i - fc_i z_{i+1}, rows nrow - 2 .. 0, chunks from the top
    auto bwd_fac = [&](int i0, int b2) {
#pragma unroll
      for (int q = 0; q < kSwCh; ++q) {
        const int ii = i0 + q;
        const bool on = ii < nrow - 1;
        sweep_fac_copy(fac(b2, 0, q), on ? fc + (size_t)ii * nc + c : dummy, on);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int top = ((maxrow - 1) / kSwCh) * kSwCh;
    gather(sc.z, top, pv);
    bwd_fac(top, buf);
    for (int i0 = top; i0 >= 0; i0 -= kSwCh, buf ^= 1) {
      stage(i0, pv);
      if (i0 - kSwCh >= 0) {
        gather(sc.z, i0 - kSwCh, pv);
        bwd_fac(i0 - kSwCh, buf ^ 1);
      } else {
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
#pragma unroll
      for (int q = kSwCh - 1; q >= 0; --q) {
        const int ii = i0 + q;
        if (ii == nrow - 1) {
          d = (double)tile[q][lane];
        } else if (ii < nrow - 1) {
          d = fma(-(double)*fac(buf, 0, q), d, (double)tile[q][lane]);
          tile[q][lane] = (float)d;
        }
      }
      __syncwarp();
      store(i0);
      __syncwarp();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
  }
}

template <class T> struct W5 { T a, b, c, d, e; };

// The persistent kernel: `iters` super-iterations of every admitted slot.
template <int NDF, bool CMA>
__global__ void __launch_bounds__(kBT, kMaxBps) batch_kernel(const BParams* __restrict__ PP) {
  // the apply rings, or the column sweeps' tiles, then the ring mbarriers
  // (dyn_bytes(NDF))
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  unsigned char* ring = dyn_smem + (size_t)(threadIdx.x >> 5) * Ring<NDF>::WARP;
  uint64_t* bars = reinterpret_cast<uint64_t*>(dyn_smem + ring_bar_offset(NDF)) +
                   (threadIdx.x >> 5) * kRing;
  if ((threadIdx.x & 31) == 0) {
    for (int i = 0; i < kRing; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(bars + i)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  unsigned seq = 0;  // ring units this warp has issued (and consumed)
  int aph = 0;       // FP32 apply phases run so far in this launch
  __shared__ BShared sh;
  __shared__ BParams sp;
  {
    const int* src = reinterpret_cast<const int*>(PP);
    int* dst = reinterpret_cast<int*>(&sp);
    for (int i = threadIdx.x; i < (int)(sizeof(BParams) / 4); i += kBT) dst[i] = src[i];
  }
  __syncthreads();
  const BParams& P = sp;
  // slots admitted since the last launch take their first residual in
  // super-iteration 0; later flags are raised by the iterations themselves
  if (blockIdx.x == 0 && threadIdx.x < 32) {
    int any = 0;
    for (int s = threadIdx.x; s < P.max_slots; s += 32) any |= (__ldcg(&P.st[s].phase) == PH_INIT);
    any = __any_sync(0xffffffffu, any);
    if (threadIdx.x == 0) {
      P.need[0] = any;
      for (int i = 1; i < P.iters; ++i) P.need[i] = 0;
    }
  }
  if (!grid_sync(P, sh)) return;

  for (int it = 0; it < P.iters; ++it) {
    // ---- A: z = A32 p, alpha
    for (int g = 0; g < P.ngr32; ++g)
      for (int c = 0; c < P.ncolour; ++c) {
        const int o = g * P.ncolour + c;
        // this apply phase takes counter aph & 1; the next one's is cleared
        // now (its last user finished before the last barrier)
        if (blockIdx.x == 0 && threadIdx.x == 0) P.wq[(aph + 1) & 1] = 0u;
        seq = apply_phase32_ring<NDF>(P, P.items32, __ldg(P.off32 + o), __ldg(P.off32 + o + 1),
                                      ring, bars, seq, P.wq + (aph & 1));
        ++aph;
        if (!grid_sync(P, sh)) return;
      }
    alpha_phase(P, sh);
    if (!grid_sync(P, sh)) return;
    // ---- U: xc += alpha p, r -= alpha z, ||r||^2 (+ <r, r/d>, beta for Jacobi slots)
    int* need = P.need + it;
    vec_phase<2>(
        P, sh, [](int ph, int) { return ph_run(ph); },
        [](const BSlot& D, unsigned i, unsigned n) {
          return W5<float4>{vld<false>(D.xc, i, n), vld<false>(D.p, i, n), vld<false>(D.r, i, n),
                            vld<false>(D.z, i, n),
                            D.cma ? make_float4(1.f, 1.f, 1.f, 1.f) : vld<true>(D.diag, i, n)};
        },
        [](const BSlot& D, const VState& S, unsigned i, unsigned n, const W5<float4>& v, double* a) {
          float xc[4], p[4], r[4], z[4], d[4];
          f4a(v.a, xc); f4a(v.b, p); f4a(v.c, r); f4a(v.d, z); f4a(v.e, d);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            xc[c] = fmaf(S.alpha, p[c], xc[c]);
            r[c] = fmaf(-S.alpha, z[c], r[c]);
            if (i + c < n) {
              a[0] = fma((double)r[c], (double)r[c], a[0]);
              if (!D.cma) a[1] = fma((double)r[c], (double)(r[c] / d[c]), a[1]);
            }
          }
          vst(D.xc, i, n, a4f(xc));
          vst(D.r, i, n, a4f(r));
        },
        [need](const BSlot& D, BState& S, const double* t) {
          S.iter += 1;
          S.rnorm = sqrt(t[0]);
          if (S.rnorm <= kDelta * S.rlast || S.rnorm <= S.tol * S.r0 || S.iter >= S.max_iter ||
              !(S.rnorm == S.rnorm)) {
            S.flag = 1;
            *need = 1;
          } else if (!D.cma) {
            S.beta = t[1] / S.rz;
            S.rz = t[1];
          }
        });
    if (!grid_sync(P, sh)) return;
    // ---- R: reliable update and FP64 true residual
    if (__ldcg(need)) {
      auto resid = [](int ph, int fl) { return ph == PH_INIT || (ph == PH_RUN && fl); };
      vec_phase<0>(
          P, sh, resid,
          [](const BSlot& D, unsigned i, unsigned n) {
            return DF4{vldd<false>(D.x, i, n), vld<false>(D.xc, i, n)};
          },
          [](const BSlot& D, const VState& S, unsigned i, unsigned n, const DF4& v, double*) {
            if (S.phase != PH_INIT) {
              float xc[4];
              f4a(v.f, xc);
              D4 x = v.d;
#pragma unroll
              for (int c = 0; c < 4; ++c) x.v[c] = x.v[c] + (double)xc[c];
              vstd(D.x, i, n, x);
            }
            vst(D.xc, i, n, make_float4(0.f, 0.f, 0.f, 0.f));
          },
          [](const BSlot&, BState&, const double*) {});
      if (!grid_sync(P, sh)) return;
      for (int g = 0; g < P.ngr64; ++g)
        for (int c = 0; c < P.ncolour; ++c) {
          const int o = g * P.ncolour + c;
          apply_phase<NDF, true>(P, P.items64, __ldg(P.off64 + o), __ldg(P.off64 + o + 1));
          if (!grid_sync(P, sh)) return;
        }
      vec_phase<2>(
          P, sh, resid,
          [](const BSlot& D, unsigned i, unsigned n) {
            return DF4{vldd<false>(D.r64, i, n), vld<true>(D.diag, i, n)};
          },
          [](const BSlot& D, const VState&, unsigned i, unsigned n, const DF4& v, double* a) {
            float d[4], r[4];
            f4a(v.f, d);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              r[c] = (float)v.d.v[c];
              if (i + c < n) {
                a[0] = fma(v.d.v[c], v.d.v[c], a[0]);
                if (!D.cma) a[1] = fma((double)r[c], (double)(r[c] / d[c]), a[1]);
              }
            }
            vst(D.r, i, n, a4f(r));
          },
          [](const BSlot& D, BState& S, const double* t) {
            const double nr = sqrt(t[0]);
            S.resid += 1;
            if (S.phase == PH_INIT) {
              S.r0 = nr;
              S.rlast = nr;
              S.true_rel = nr > 0.0 ? 1.0 : 0.0;
              if (nr < DBL_EPSILON) {
                S.phase = PH_DONE;
                S.true_rel = 0.0;
                return;
              }
              S.phase = PH_RUN;
              S.flag = 0;
              if (!D.cma) S.rz = t[1];
              return;
            }
            S.flag = 0;
            S.rlast = nr;
            S.true_rel = nr / S.r0;
            if (S.true_rel <= S.tol) {
              S.phase = PH_DONE;
            } else if (!(nr == nr)) {
              S.phase = PH_DONE;
              S.status = LFX_NAN_DETECTED;
            } else if (S.iter >= S.max_iter) {
              S.phase = PH_DONE;
              S.status = LFX_NOT_CONVERGED;
            } else if (!D.cma) {
              S.beta = t[1] / S.rz;
              S.rz = t[1];
            }
          });
      if (!grid_sync(P, sh)) return;
    }
    // ---- C: column sweeps, then the Jacobi rows with <r, z> and beta
    if (CMA && P.any_cma) {
      sweep_phase_w(P, dyn_smem + (size_t)(threadIdx.x >> 5) * kSweepWarpBytes);
      if (!grid_sync(P, sh)) return;
      vec_phase<1>(
          P, sh, [](int ph, int) { return ph_run(ph); },
          [](const BSlot& D, unsigned i, unsigned n) {
            if (!D.cma) return V3<float4>{};
            return V3<float4>{vld<false>(D.r, i, n), vld<true>(D.diag, i, n), vld<false>(D.z, i, n)};
          },
          [](const BSlot& D, const VState&, unsigned i, unsigned n, const V3<float4>& v, double* a) {
            if (!D.cma) return;
            // rows with a non-zero diagonal are Jacobi rows; the column rows
            // (written by the sweeps) carry a zero in the Jacobi diagonal
            float r[4], d[4], z[4];
            f4a(v.a, r); f4a(v.b, d); f4a(v.c, z);
            bool jac = false;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              if (d[c] != 0.0f) {
                z[c] = r[c] / d[c];
                jac = true;
              }
              if (i + c < n) a[0] = fma((double)r[c], (double)z[c], a[0]);
            }
            if (jac) vst(D.z, i, n, a4f(z));
          },
          [](const BSlot& D, BState& S, const double* t) {
            if (!D.cma) return;
            S.beta = S.fresh ? 0.0 : t[0] / S.rz;
            S.rz = t[0];
          });
      if (!grid_sync(P, sh)) return;
    }
    // ---- P: p = z + beta p (p = z for a slot that just started)
    vec_phase<0>(
        P, sh, [](int ph, int) { return ph_run(ph); },
        [](const BSlot& D, unsigned i, unsigned n) {
          return V3<float4>{vld<false>(D.p, i, n), D.cma ? vld<false>(D.z, i, n) : vld<false>(D.r, i, n),
                            D.cma ? make_float4(1.f, 1.f, 1.f, 1.f) : vld<true>(D.diag, i, n)};
        },
        [](const BSlot& D, const VState& S, unsigned i, unsigned n, const V3<float4>& v, double*) {
          float p[4], zr[4], d[4];
          f4a(v.a, p); f4a(v.b, zr); f4a(v.c, d);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float zi = D.cma ? zr[c] : zr[c] / d[c];
            p[c] = S.fresh ? zi : fmaf(S.beta, p[c], zi);
          }
          vst(D.p, i, n, a4f(p));
        },
        [](const BSlot&, BState&, const double*) {});
    if (!grid_sync(P, sh)) return;
  }
}

template <int NDF, bool CMA>
const void* kernel_ptr() {
  return reinterpret_cast<const void*>(&batch_kernel<NDF, CMA>);
}

}  // namespace

// host-side record of one slot
struct SlotHost {
  bool used = false;
  void* mem = nullptr;
  size_t mem_bytes = 0;
  lfx_vec* x = nullptr;
  int64_t tag = 0;
  int64_t n = 0;
  int nch = 0, nl = 0, ncol = 0;
  bool cma = false;
  std::vector<int32_t> cstart;  // colour starts in the colour-loop order
  int last_phase = PH_EMPTY;
};

// The work lists are expanded on the device from runs the host lays out: a
// run is one slot's range [a, e) (cell columns of one colour, chunks, or
// preconditioner columns) and the list index its entries start at, so a
// rebuild uploads a few hundred runs instead of the lists themselves.
struct ListRun {
  int s, a, e, off;
};

struct lfx_batch {
  lfx_ctx* ctx = nullptr;
  int ndf = 8, max_slots = 0, iters = 8;
  int64_t reserve = 0;
  // free device memory (plus the pool's unused bytes) as last queried,
  // less what admissions took since and plus what retirements gave back;
  // -1: query again (each step starts a new reading)
  int64_t avail = -1;
  BSlot* d_slots = nullptr;
  std::vector<BSlot> h_slots;
  BState* d_state = nullptr;
  BState* h_state = nullptr;  // pinned
  unsigned* d_tickets = nullptr;
  int* d_need = nullptr;
  unsigned* d_bar = nullptr;
  ListRun* d_runs = nullptr;
  size_t cap_runs = 0;
  int* d_err = nullptr;
  int* h_err = nullptr;  // pinned
  BParams* d_params = nullptr;
  BParams h_params{};
  // work lists (device, grown on demand)
  int4 *d_items32 = nullptr, *d_items64 = nullptr;
  int *d_off32 = nullptr, *d_off64 = nullptr;
  int2 *d_chunks = nullptr, *d_cols = nullptr;
  int* d_slotlist = nullptr;
  size_t cap_items32 = 0, cap_items64 = 0, cap_off32 = 0, cap_off64 = 0, cap_chunks = 0,
         cap_cols = 0, cap_slotlist = 0;
  std::vector<SlotHost> slots;
  bool dirty = true;
  int nactive = 0;
  // launch shape (autotuned) and its graphs
  int cells_per_item = 2, blocks_per_sm = 2, max_bps = 2;
  int64_t group_bytes = 64 << 20;
  float tuned_us = 0.f;
  std::map<int, cudaGraphExec_t> graphs;  // by blocks per SM
  bool cooperative = true;
  int64_t replays = 0;
  double timeout_s = 2.0;
};

namespace {

template <class T>
int grow(lfx_ctx* ctx, T** p, size_t* cap, size_t need) {
  if (need <= *cap && *p) return LFX_OK;
  size_t c = std::max<size_t>(need, *cap * 2);
  if (c < 64) c = 64;
  if (*p) LFX_CK(ctx, cudaFreeAsync(*p, ctx->stream));
  *p = nullptr;
  LFX_CK(ctx, cudaMallocAsync((void**)p, c * sizeof(T), ctx->stream));
  *cap = c;
  return LFX_OK;
}

template <class T>
int upload(lfx_ctx* ctx, T* dst, const std::vector<T>& src) {
  if (src.empty()) return LFX_OK;
  LFX_CK(ctx, cudaMemcpyAsync(dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice,
                              ctx->stream));
  return LFX_OK;
}


const void* pick_kernel(int ndf, bool cma) {
  if (ndf == 8) return cma ? kernel_ptr<8, true>() : kernel_ptr<8, false>();
  return cma ? kernel_ptr<6, true>() : kernel_ptr<6, false>();
}

// apply items {slot, first column, columns <= cb, 0} of each run
__global__ void expand_items(const ListRun* __restrict__ runs, int nrun, int cb,
                             int4* __restrict__ items) {
  for (int r = blockIdx.x; r < nrun; r += gridDim.x) {
    const ListRun R = runs[r];
    const int n = (R.e - R.a + cb - 1) / cb;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int q = R.a + i * cb;
      items[R.off + i] = make_int4(R.s, q, min(cb, R.e - q), 0);
    }
  }
}
// pairs {slot, k} for k in each run's range
__global__ void expand_pairs(const ListRun* __restrict__ runs, int nrun, int2* __restrict__ out) {
  for (int r = blockIdx.x; r < nrun; r += gridDim.x) {
    const ListRun R = runs[r];
    for (int i = threadIdx.x; i < R.e - R.a; i += blockDim.x) out[R.off + i] = make_int2(R.s, R.a + i);
  }
}

// apply item runs of one precision: slots greedily grouped so that a group's
// vectors (bytes_per_dof per dof) stay within group_bytes; per group and
// colour the slots' runs of cells_per_item cell columns. Returns the number
// of items; off receives each (group, colour)'s first item
int64_t build_apply_runs(const lfx_batch* B, const std::vector<int>& act, int ncolour,
                         int bytes_per_dof, std::vector<ListRun>& runs, std::vector<int>& off) {
  runs.clear();
  off.clear();
  std::vector<std::vector<int>> groups;
  int64_t acc = 0;
  for (int s : act) {
    const int64_t b = (int64_t)bytes_per_dof * B->slots[s].n;
    if (groups.empty() || (acc + b > B->group_bytes && !groups.back().empty())) {
      groups.emplace_back();
      acc = 0;
    }
    groups.back().push_back(s);
    acc += b;
  }
  const int cb = B->cells_per_item;
  int64_t n = 0;
  for (auto& g : groups)
    for (int c = 0; c < ncolour; ++c) {
      off.push_back((int)n);
      for (int s : g) {
        const SlotHost& H = B->slots[s];
        if (c + 1 >= (int)H.cstart.size()) continue;
        const int a = H.cstart[c], e = H.cstart[c + 1];
        if (e <= a) continue;
        runs.push_back(ListRun{s, a, e, (int)n});
        n += (e - a + cb - 1) / cb;
      }
    }
  off.push_back((int)n);
  return n;
}

int rebuild(lfx_batch* B) {
  lfx_ctx* ctx = B->ctx;
  std::vector<int> act;
  bool any_cma = false;
  for (int s = 0; s < B->max_slots; ++s) {
    const SlotHost& H = B->slots[s];
    if (H.used && H.last_phase != PH_DONE) {
      act.push_back(s);
      any_cma |= H.cma;
    }
  }
  B->nactive = (int)act.size();
  // colour phases: as many as the slot with the most colours has
  int ncolour = 1;
  for (int s : act) ncolour = std::max(ncolour, (int)B->slots[s].cstart.size() - 1);
  std::vector<ListRun> r32, r64, rch, rcol;
  std::vector<int> off32, off64;
  const int64_t n32 = build_apply_runs(B, act, ncolour, 8, r32, off32);
  const int64_t n64 = build_apply_runs(B, act, ncolour, 16, r64, off64);
  int64_t nch = 0, ncol = 0;
  for (int s : act) nch += B->slots[s].nch;
  // (vec_phase says why)
  const int chgrp = nch >= (int64_t)kChGroup * 4 * kMaxBps * ctx->num_sms ? kChGroup : 1;
  nch = 0;
  for (int s : act) {
    const SlotHost& H = B->slots[s];
    rch.push_back(ListRun{s, 0, (H.nch + chgrp - 1) / chgrp, (int)nch});
    nch += (H.nch + chgrp - 1) / chgrp;
    if (H.cma && H.ncol > 0) {
      rcol.push_back(ListRun{s, 0, H.ncol, (int)ncol});
      ncol += H.ncol;
    }
  }
  // one upload of all runs: apply32, apply64, chunks, columns
  std::vector<ListRun> runs;
  runs.reserve(r32.size() + r64.size() + rch.size() + rcol.size());
  runs.insert(runs.end(), r32.begin(), r32.end());
  runs.insert(runs.end(), r64.begin(), r64.end());
  runs.insert(runs.end(), rch.begin(), rch.end());
  runs.insert(runs.end(), rcol.begin(), rcol.end());
  int rc = grow(ctx, &B->d_items32, &B->cap_items32, (size_t)n32);
  if (!rc) rc = grow(ctx, &B->d_items64, &B->cap_items64, (size_t)n64);
  if (!rc) rc = grow(ctx, &B->d_off32, &B->cap_off32, off32.size());
  if (!rc) rc = grow(ctx, &B->d_off64, &B->cap_off64, off64.size());
  if (!rc) rc = grow(ctx, &B->d_chunks, &B->cap_chunks, (size_t)nch);
  if (!rc) rc = grow(ctx, &B->d_cols, &B->cap_cols, (size_t)ncol);
  if (!rc) rc = grow(ctx, &B->d_runs, &B->cap_runs, runs.size());
  if (rc) return rc;
  rc = upload(ctx, B->d_off32, off32);
  if (!rc) rc = upload(ctx, B->d_off64, off64);
  if (!rc) rc = upload(ctx, B->d_runs, runs);
  if (rc) return rc;
  {
    const ListRun* d = B->d_runs;
    const int g = ctx->num_sms * 4;
    int nl = 0;
    if (!r32.empty()) {
      expand_items<<<g, 256, 0, ctx->stream>>>(d, (int)r32.size(), B->cells_per_item, B->d_items32);
      ++nl;
    }
    d += r32.size();
    if (!r64.empty()) {
      expand_items<<<g, 256, 0, ctx->stream>>>(d, (int)r64.size(), B->cells_per_item, B->d_items64);
      ++nl;
    }
    d += r64.size();
    if (!rch.empty()) {
      expand_pairs<<<g, 256, 0, ctx->stream>>>(d, (int)rch.size(), B->d_chunks);
      ++nl;
    }
    d += rch.size();
    if (!rcol.empty()) {
      expand_pairs<<<g, 256, 0, ctx->stream>>>(d, (int)rcol.size(), B->d_cols);
      ++nl;
    }
    ctx->launches += nl;
    LFX_CK(ctx, cudaGetLastError());
  }
  rc = grow(ctx, &B->d_slotlist, &B->cap_slotlist, act.size());
  if (!rc) rc = upload(ctx, B->d_slotlist, act);
  if (rc) return rc;
  BParams& P = B->h_params;
  P.items32 = B->d_items32;
  P.off32 = B->d_off32;
  P.items64 = B->d_items64;
  P.off64 = B->d_off64;
  P.chunks = B->d_chunks;
  P.cols = B->d_cols;
  P.slotlist = B->d_slotlist;
  P.nslot = (int)act.size();
  P.slots = B->d_slots;
  P.st = B->d_state;
  P.tickets = B->d_tickets;
  P.need = B->d_need;
  P.bar = B->d_bar;
  P.wq = B->d_bar + 2;
  P.err = B->d_err;
  P.ngr32 = (int)(off32.size() - 1) / ncolour;
  P.ngr64 = (int)(off64.size() - 1) / ncolour;
  P.ncolour = ncolour;
  P.nchunk = (int)nch;
  P.chgrp = chgrp;
  P.ncolitem = (int)ncol;
  P.iters = B->iters;
  P.max_slots = B->max_slots;
  P.any_cma = any_cma ? 1 : 0;
  P.timeout_ns = (unsigned long long)(B->timeout_s * 1e9);
  LFX_CK(ctx, cudaMemcpyAsync(B->d_params, &P, sizeof(BParams), cudaMemcpyHostToDevice,
                              ctx->stream));
  B->dirty = false;
  return LFX_OK;
}

// the graph of one launch shape: reset the barrier, then the persistent
// kernel (cooperative where the graph takes it)
int graph_for(lfx_batch* B, int bps, cudaGraphExec_t* out) {
  auto f = B->graphs.find(bps);
  if (f != B->graphs.end()) {
    *out = f->second;
    return LFX_OK;
  }
  lfx_ctx* ctx = B->ctx;
  const void* k = pick_kernel(B->ndf, B->ndf == 6);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ctx->num_sms * bps));
  cfg.blockDim = dim3(kBT);
  cfg.dynamicSmemBytes = dyn_bytes(B->ndf);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  void* args[] = {(void*)&B->d_params};
  for (int attempt = 0; attempt < 2; ++attempt) {
    cfg.attrs = B->cooperative ? at : nullptr;
    cfg.numAttrs = B->cooperative ? 1 : 0;
    cudaGraph_t g = nullptr;
    LFX_CK(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    cudaError_t e1 = cudaMemsetAsync(B->d_bar, 0, 4 * sizeof(unsigned), ctx->stream);
    cudaError_t e2 = cudaLaunchKernelExC(&cfg, k, args);
    cudaError_t e3 = cudaStreamEndCapture(ctx->stream, &g);
    cudaGraphExec_t ex = nullptr;
    cudaError_t e4 = cudaErrorUnknown;
    if (e1 == cudaSuccess && e2 == cudaSuccess && e3 == cudaSuccess && g)
      e4 = cudaGraphInstantiate(&ex, g, 0);
    if (g) cudaGraphDestroy(g);
    if (e4 == cudaSuccess) {
      B->graphs[bps] = ex;
      *out = ex;
      return LFX_OK;
    }
    cudaGetLastError();
    if (!B->cooperative) {
      cudaError_t e = e1 != cudaSuccess ? e1 : e2 != cudaSuccess ? e2 : e3 != cudaSuccess ? e3 : e4;
      return cuda_fail(ctx, e, "batch graph capture");
    }
    // graphs that do not take a cooperative kernel: the grid is sized to
    // what the device holds at once, and every barrier wait is bounded
    B->cooperative = false;
  }
  return fail(ctx, LFX_CUDA_ERROR, "batch graph capture");
}

int replay(lfx_batch* B) {
  lfx_ctx* ctx = B->ctx;
  cudaGraphExec_t g = nullptr;
  int rc = graph_for(B, B->blocks_per_sm, &g);
  if (rc) return rc;
  LFX_CK(ctx, cudaGraphLaunch(g, ctx->stream));
  ctx->launches += 1;
  B->replays += 1;
  return LFX_OK;
}

// reads the slot states and the error flag back (synchronises)
int read_back(lfx_batch* B) {
  lfx_ctx* ctx = B->ctx;
  LFX_CK(ctx, cudaMemcpyAsync(B->h_state, B->d_state, sizeof(BState) * B->max_slots,
                              cudaMemcpyDeviceToHost, ctx->stream));
  LFX_CK(ctx, cudaMemcpyAsync(B->h_err, B->d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  LFX_CK(ctx, cudaStreamSynchronize(ctx->stream));
  if (*B->h_err) {
    const int e = *B->h_err;
    *B->h_err = 0;
    cudaMemsetAsync(B->d_err, 0, sizeof(int), ctx->stream);
    cudaStreamSynchronize(ctx->stream);
    return fail(ctx, e, "batch: a grid barrier wait ran out (the batch state is undefined)");
  }
  for (int s = 0; s < B->max_slots; ++s) {
    SlotHost& H = B->slots[s];
    if (!H.used) continue;
    H.last_phase = B->h_state[s].phase;
  }
  return LFX_OK;
}

// device memory the batch may still take: free memory plus what the
// stream-ordered pool holds unused
int64_t available_bytes(lfx_ctx* ctx) {
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  int64_t avail = (int64_t)fr;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, ctx->device) == cudaSuccess) {
    uint64_t res = 0, used = 0;
    if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &res) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess &&
        res > used)
      avail += (int64_t)(res - used);
  }
  cudaGetLastError();
  return avail;
}

// device bytes a slot of this operator takes at admission
int64_t slot_bytes(int64_t n, int64_t nch, int64_t ncell) {
  const int64_t v = ((8 * n + 255) / 256 + 4 * ((4 * n + 255) / 256)) * 256;
  return v + ((2 * nch + ncell) * 8 + 255) / 256 * 256;
}

}  // namespace

extern "C" {

int lfx_batch_create(lfx_ctx* ctx, int32_t ndf, int32_t max_slots, int64_t reserve_bytes,
                     int32_t iters_per_launch, lfx_batch** out) {
  if (!ctx || !out || (ndf != 6 && ndf != 8) || max_slots < 1 || reserve_bytes < 0 ||
      iters_per_launch < 1 || iters_per_launch > kMaxIters)
    return LFX_INVALID_ARGUMENT;
  *out = nullptr;
  lfx_batch* B = new lfx_batch();
  B->ctx = ctx;
  B->ndf = ndf;
  B->max_slots = max_slots;
  B->iters = iters_per_launch;
  B->reserve = reserve_bytes;
  B->slots.resize(max_slots);
  B->h_slots.assign(max_slots, BSlot{});
  int rc = dmalloc(ctx, (void**)&B->d_slots, sizeof(BSlot) * max_slots);
  if (!rc) rc = dmalloc(ctx, (void**)&B->d_state, sizeof(BState) * max_slots);
  if (!rc) rc = dmalloc(ctx, (void**)&B->d_tickets, sizeof(unsigned) * max_slots);
  if (!rc) rc = dmalloc(ctx, (void**)&B->d_need, sizeof(int) * kMaxIters);
  if (!rc) rc = dmalloc(ctx, (void**)&B->d_bar, sizeof(unsigned) * 4);
  if (!rc) rc = dmalloc(ctx, (void**)&B->d_err, sizeof(int));
  if (!rc) rc = dmalloc(ctx, (void**)&B->d_params, sizeof(BParams));
  if (!rc && cudaMallocHost((void**)&B->h_state, sizeof(BState) * max_slots) != cudaSuccess)
    rc = LFX_OUT_OF_MEMORY;
  if (!rc && cudaMallocHost((void**)&B->h_err, sizeof(int)) != cudaSuccess) rc = LFX_OUT_OF_MEMORY;
  if (!rc) {
    memset(B->h_state, 0, sizeof(BState) * max_slots);
    *B->h_err = 0;
    cudaMemsetAsync(B->d_slots, 0, sizeof(BSlot) * max_slots, ctx->stream);
    cudaMemsetAsync(B->d_state, 0, sizeof(BState) * max_slots, ctx->stream);
    cudaMemsetAsync(B->d_tickets, 0, sizeof(unsigned) * max_slots, ctx->stream);
    cudaMemsetAsync(B->d_need, 0, sizeof(int) * kMaxIters, ctx->stream);
    cudaMemsetAsync(B->d_bar, 0, sizeof(unsigned) * 4, ctx->stream);
    cudaMemsetAsync(B->d_err, 0, sizeof(int), ctx->stream);
    // memory returned by retired slots stays in the pool for the next ones
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, ctx->device) == cudaSuccess) {
      uint64_t thr = UINT64_MAX;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
    // the kernel holds at most kMaxBps blocks per SM (launch bounds); fewer
    // if the device says so
    int per_sm = 0;
    for (int cma = 0; cma < 2; ++cma)
      cudaFuncSetAttribute(pick_kernel(ndf, cma != 0), cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)dyn_bytes(ndf));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pick_kernel(ndf, ndf == 6), kBT,
                                                  dyn_bytes(ndf));
    B->max_bps = std::max(1, std::min(per_sm, kMaxBps));
    B->blocks_per_sm = B->max_bps;
    B->group_bytes = ctx->l2_bytes / 2;
    if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) rc = LFX_CUDA_ERROR;
    cudaGetLastError();
  }
  if (!rc) rc = rebuild(B);
  if (!rc) {
    cudaGraphExec_t g;
    rc = graph_for(B, B->blocks_per_sm, &g);
  }
  if (rc) {
    lfx_batch_destroy(B);
    return rc;
  }
  *out = B;
  return LFX_OK;
}

int lfx_batch_destroy(lfx_batch* B) {
  if (!B) return LFX_OK;
  lfx_ctx* ctx = B->ctx;
  cudaStreamSynchronize(ctx->stream);
  for (auto& kv : B->graphs) cudaGraphExecDestroy(kv.second);
  for (auto& H : B->slots)
    if (H.mem) cudaFreeAsync(H.mem, ctx->stream);
  for (void* p : {(void*)B->d_items32, (void*)B->d_items64, (void*)B->d_off32, (void*)B->d_off64,
                  (void*)B->d_chunks, (void*)B->d_cols, (void*)B->d_slotlist, (void*)B->d_runs})
    if (p) cudaFreeAsync(p, ctx->stream);
  cudaStreamSynchronize(ctx->stream);
  dfree(ctx, B->d_slots, sizeof(BSlot) * B->max_slots);
  dfree(ctx, B->d_state, sizeof(BState) * B->max_slots);
  dfree(ctx, B->d_tickets, sizeof(unsigned) * B->max_slots);
  dfree(ctx, B->d_need, sizeof(int) * kMaxIters);
  dfree(ctx, B->d_bar, sizeof(unsigned) * 4);
  dfree(ctx, B->d_err, sizeof(int));
  dfree(ctx, B->d_params, sizeof(BParams));
  if (B->h_state) cudaFreeHost(B->h_state);
  if (B->h_err) cudaFreeHost(B->h_err);
  cudaGetLastError();
  delete B;
  return LFX_OK;
}

int lfx_batch_admit(lfx_batch* B, lfx_op* op64, lfx_op* op32, lfx_prec* prec32, const lfx_vec* b,
                    lfx_vec* x, double tol, int32_t max_iter, int64_t tag, int32_t* slot_out) {
  if (!B || !op64 || !op32 || !prec32 || !b || !x || !slot_out || !(tol > 0.0) || max_iter < 1)
    return LFX_INVALID_ARGUMENT;
  lfx_ctx* ctx = B->ctx;
  *slot_out = -1;
  const lfx_lma_layout* L = op64->lay;
  if (op32->lay != L || op64->precision != LFX_R64 || op32->precision != LFX_R32)
    return fail(ctx, LFX_TYPE_MISMATCH, "batch needs FP64 and FP32 copies of one operator");
  if (L->ndf_from != B->ndf || L->ndf_to != B->ndf || !L->cs_ok || !op32->smat || !op64->smat)
    return fail(ctx, LFX_NOT_SUPPORTED,
                "batch needs a symmetric operator on one dofmap of the batch's cell size "
                "(the packed cell scatter)");
  const int nl = L->nlayers;
  // segments of at most 31 rows: lane 0 of a segment holds the row below it
  const int nseg = (nl + 1 + 30) / 31;
  if (nseg > kMaxSeg)
    return fail(ctx, LFX_NOT_SUPPORTED, "batch: at most 123 levels per column");
  const bool cma = prec32->kind == PREC_CMA;
  if (prec32->precision != LFX_R32 || (prec32->kind != PREC_DIAG && !cma) || !prec32->rdiag ||
      prec32->rdiag_n != L->undf_to || (cma && !prec32->jacobi_zeroed))
    return fail(ctx, LFX_NOT_SUPPORTED,
                "batch needs an FP32 Jacobi or column preconditioner with a diagonal");
  if (cma && (B->ndf != 6 || prec32->nrow > kBRows))
    return fail(ctx, LFX_NOT_SUPPORTED,
                "batch column preconditioner: 6-dof cells, at most 160 rows per column");
  if (b->precision != LFX_R64 || x->precision != LFX_R64 || b->undf[0] != L->undf_to ||
      x->undf[0] != L->undf_to)
    return fail(ctx, LFX_TYPE_MISMATCH, "b and x must be FP64 vectors of the operator's space");
  int s = -1;
  for (int i = 0; i < B->max_slots; ++i)
    if (!B->slots[i].used) {
      s = i;
      break;
    }
  if (s < 0) return fail(ctx, LFX_OUT_OF_MEMORY, "no free batch slot");
  const int64_t n = L->undf_to;
  const int64_t nch = bchunks(n);
  if (L->colour_start.size() < 2 || (int)L->colour_start.size() - 1 > kMaxColours)
    return fail(ctx, LFX_NOT_SUPPORTED, "batch: at most 8 cell colours");
  // admission by free device memory: the slot's state, its share of the
  // work lists, and the batch's reserve must fit
  const int64_t need = slot_bytes(n, nch, L->ncell_2d) + (int64_t)(op32->lmat ? 0 : op_level_major_bytes(op32));
  const int64_t lists = 16 * (2 * ((int64_t)L->ncell_2d / 32 + 8) + nch) + 8 * (cma ? prec32->ncell_2d : 0);
  if (B->avail < 0) B->avail = available_bytes(ctx);
  if (B->avail - need - 2 * lists < B->reserve)
    return fail(ctx, LFX_OUT_OF_MEMORY, "batch: not enough free device memory for the solve");
  {
    const int rcl = op_level_major(op32);
    if (rcl) return rcl;
  }
  SlotHost& H = B->slots[s];
  H = SlotHost();
  void* mem = nullptr;
  cudaError_t e = cudaMallocAsync(&mem, (size_t)need, ctx->stream);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(ctx, LFX_OUT_OF_MEMORY, "batch: slot state allocation failed");
  }
  H.used = true;
  H.mem = mem;
  H.mem_bytes = (size_t)need;
  H.x = x;
  H.tag = tag;
  H.n = n;
  H.nch = (int)nch;
  H.nl = nl;
  H.cma = cma;
  H.ncol = cma ? prec32->ncell_2d : 0;
  H.cstart = L->colour_start;
  H.last_phase = PH_INIT;
  BSlot D{};
  D.S32 = (const float*)op32->smat;
  D.S64 = (const double*)op64->smat;
  D.L32 = (const float4*)op32->lmat;
  D.npv = op32->lnpv;
  D.canon = layout_canon(L, B->ndf) ? 1 : 0;
  D.cdesc = L->cs_desc;
  D.sblk32 = op32->sblk;
  D.sblk64 = op64->sblk;
  D.cdints = L->cs_ints;
  D.nl = nl;
  D.nseg = nseg;
  D.segL = (nl + 1 + nseg - 1) / nseg;
  D.nch = (int)nch;
  D.ncell = L->ncell_2d;
  D.cma = cma ? 1 : 0;
  D.n = n;
  char* m = (char*)mem;
  D.r64 = (double*)m;
  m += (8 * n + 255) / 256 * 256;
  float* f[4];
  for (int i = 0; i < 4; ++i) {
    f[i] = (float*)m;
    m += (4 * n + 255) / 256 * 256;
  }
  D.r = f[0];
  D.p = f[1];
  D.z = f[2];
  D.xc = f[3];
  D.part = (double*)m;
  D.diag = (const float*)prec32->rdiag;
  if (cma) {
    D.fa = (const float*)prec32->fa;
    D.finv = (const float*)prec32->finv;
    D.fc = (const float*)prec32->fc;
    D.first = prec32->first_dof;
    D.ind = prec32->indirection;
    D.ncol = prec32->ncell_2d;
    D.nrow = prec32->nrow;
  }
  D.b = (const double*)b->data[0];
  D.x = (double*)x->data[0];
  B->h_slots[s] = D;
  BState S{};
  S.phase = PH_INIT;
  S.fresh = 1;
  S.tol = tol;
  S.max_iter = max_iter;
  B->h_state[s] = S;
  int rc = LFX_OK;
  // xc starts at zero (the first true residual leaves x as given)
  e = cudaMemsetAsync(D.xc, 0, 4 * n, ctx->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(B->d_slots + s, &B->h_slots[s], sizeof(BSlot), cudaMemcpyHostToDevice,
                        ctx->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(B->d_state + s, &B->h_state[s], sizeof(BState), cudaMemcpyHostToDevice,
                        ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(B->d_tickets + s, 0, sizeof(unsigned), ctx->stream);
  if (e != cudaSuccess) rc = cuda_fail(ctx, e, "batch admission");
  if (rc) {
    cudaFreeAsync(mem, ctx->stream);
    H = SlotHost();
    return rc;
  }
  B->dirty = true;
  B->avail -= need + 2 * lists;
  *slot_out = s;
  return LFX_OK;
}

// Runs one replay (iters super-iterations) for every admitted slot, then
// reads the slot states. *ndone receives the number of slots that are done
// (converged or failed) and not yet retired.
int lfx_batch_step(lfx_batch* B, int32_t* ndone) {
  if (!B) return LFX_INVALID_ARGUMENT;
  int rc = LFX_OK;
  // The work lists are rebuilt when slots were admitted (or the launch shape
  // changed), and when fewer than two thirds of the slots they cover still
  // run: every phase skips the items of a slot that is done or retired (its
  // state on the device says so before its memory is freed), so a slot
  // that finishes costs no rebuild.
  B->avail = -1;  // admissions after this step read free memory again
  int running = 0;
  for (int s = 0; s < B->max_slots; ++s)
    if (B->slots[s].used && B->slots[s].last_phase != PH_DONE) ++running;
  if (B->dirty || 3 * running < 2 * B->nactive) rc = rebuild(B);
  if (rc) return rc;
  if (running > 0) {
    rc = replay(B);
    if (!rc) rc = read_back(B);
    if (rc) return rc;
  }
  int nd = 0;
  for (int s = 0; s < B->max_slots; ++s)
    if (B->slots[s].used && B->slots[s].last_phase == PH_DONE) ++nd;
  if (ndone) *ndone = nd;
  return LFX_OK;
}

// Slot state: 0 empty, 1 starting, 2 iterating, 3 done.
int lfx_batch_slot_info(const lfx_batch* B, int32_t slot, int32_t* phase, int64_t* tag,
                        lfx_solve_info* info) {
  if (!B || slot < 0 || slot >= B->max_slots) return LFX_INVALID_ARGUMENT;
  const BState& S = B->h_state[slot];
  if (phase) *phase = B->slots[slot].used ? S.phase : PH_EMPTY;
  if (tag) *tag = B->slots[slot].tag;
  if (info) {
    memset(info, 0, sizeof *info);
    info->iterations = S.iter;
    info->converged = S.phase == PH_DONE && S.status == 0;
    info->initial_norm = S.r0;
    info->final_norm = S.rlast;
    info->final_rel = S.true_rel;
    info->applies = S.iter + S.resid;
    info->status = S.status;
    info->outer_iterations = S.resid;
    info->inner_iterations = S.iter;
  }
  return LFX_OK;
}

// Frees a done (or any) slot for new admissions; its state returns to the
// device's memory pool.
int lfx_batch_retire(lfx_batch* B, int32_t slot) {
  if (!B || slot < 0 || slot >= B->max_slots) return LFX_INVALID_ARGUMENT;
  lfx_ctx* ctx = B->ctx;
  SlotHost& H = B->slots[slot];
  if (!H.used) return LFX_OK;
  B->h_state[slot] = BState{};
  LFX_CK(ctx, cudaMemcpyAsync(B->d_state + slot, &B->h_state[slot], sizeof(BState),
                              cudaMemcpyHostToDevice, ctx->stream));
  if (H.mem) LFX_CK(ctx, cudaFreeAsync(H.mem, ctx->stream));
  if (B->avail >= 0) B->avail += (int64_t)H.mem_bytes;
  H = SlotHost();
  return LFX_OK;
}

int lfx_batch_get_tuning(const lfx_batch* B, lfx_batch_tuning* t) {
  if (!B || !t) return LFX_INVALID_ARGUMENT;
  t->cells_per_item = B->cells_per_item;
  t->blocks_per_sm = B->blocks_per_sm;
  t->grid = B->ctx->num_sms * B->blocks_per_sm;
  t->group_bytes = B->group_bytes;
  t->us_per_iteration = B->tuned_us;
  t->cooperative = B->cooperative ? 1 : 0;
  t->replays = B->replays;
  return LFX_OK;
}

int lfx_batch_set_tuning(lfx_batch* B, int32_t cells_per_item, int32_t blocks_per_sm,
                         int64_t group_bytes) {
  if (!B) return LFX_INVALID_ARGUMENT;
  if (cells_per_item < 1 || cells_per_item > kItemCols ||
      blocks_per_sm < 1 || blocks_per_sm > B->max_bps || group_bytes < 1)
    return fail(B->ctx, LFX_INVALID_ARGUMENT, "batch tuning out of range");
  B->cells_per_item = cells_per_item;
  B->blocks_per_sm = blocks_per_sm;
  B->group_bytes = group_bytes;
  B->dirty = true;
  return LFX_OK;
}

// Batch autotuner: times one replay of `iters` super-iterations per
// candidate launch shape on the admitted slots (the replays advance the
// solves; results do not depend on the shape) and keeps the fastest:
// blocks per SM, then cell columns per apply item, then the L2 group size.
int lfx_batch_autotune(lfx_batch* B, int32_t iters, lfx_batch_tuning* out) {
  if (!B || iters < 1 || iters > kMaxIters) return LFX_INVALID_ARGUMENT;
  lfx_ctx* ctx = B->ctx;
  const int keep_iters = B->iters;
  cudaEvent_t e0, e1;
  LFX_CK(ctx, cudaEventCreate(&e0));
  LFX_CK(ctx, cudaEventCreate(&e1));
  int rc = LFX_OK;
  auto trial = [&](float* us) -> int {
    int r = rebuild(B);
    if (r) return r;
    if (B->nactive == 0) {
      *us = 0.f;
      return LFX_OK;
    }
    cudaGraphExec_t g = nullptr;
    r = graph_for(B, B->blocks_per_sm, &g);  // captured before the timed replay
    if (r) return r;
    LFX_CK(ctx, cudaEventRecord(e0, ctx->stream));
    r = replay(B);
    if (r) return r;
    LFX_CK(ctx, cudaEventRecord(e1, ctx->stream));
    r = read_back(B);
    if (r) return r;
    float ms = 0.f;
    LFX_CK(ctx, cudaEventElapsedTime(&ms, e0, e1));
    *us = 1e3f * ms / iters;
    return LFX_OK;
  };
  B->iters = iters;
  float t = 0.f, best = 0.f;
  // one warm-up replay (first residuals of new slots)
  rc = trial(&t);
  int bb = B->blocks_per_sm, bc = B->cells_per_item;
  int64_t bg = B->group_bytes;
  const int64_t l2 = ctx->l2_bytes;
  for (int stage = 0; stage < 3 && !rc; ++stage) {
    std::vector<int64_t> cand;
    if (stage == 0)
      for (int v = 1; v <= B->max_bps; ++v) cand.push_back(v);
    if (stage == 1) cand = {1, 2, 4, 8};
    if (stage == 2) cand = {l2 / 4, l2 / 2, l2, int64_t(1) << 40};
    best = 0.f;
    for (int64_t c : cand) {
      B->blocks_per_sm = stage == 0 ? (int)c : bb;
      B->cells_per_item = stage == 1 ? (int)c : bc;
      B->group_bytes = stage == 2 ? c : bg;
      B->dirty = true;
      rc = trial(&t);
      if (rc) break;
      // a trial with no running slot measured nothing: it cannot win
      if (t > 0.f && (best == 0.f || t < best)) {
        best = t;
        if (stage == 0) bb = (int)c;
        if (stage == 1) bc = (int)c;
        if (stage == 2) bg = c;
      }
    }
  }
  B->blocks_per_sm = bb;
  B->cells_per_item = bc;
  B->group_bytes = bg;
  B->tuned_us = best;
  B->iters = keep_iters;
  B->dirty = true;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (!rc && out) rc = lfx_batch_get_tuning(B, out);
  return rc;
}

// Upper bound on one grid-barrier wait (seconds) before the kernel gives up
// with LFX_TIMEOUT.
int lfx_batch_set_wait_limit(lfx_batch* B, double seconds) {
  if (!B || !(seconds > 0.0)) return LFX_INVALID_ARGUMENT;
  B->timeout_s = seconds;
  B->dirty = true;
  return LFX_OK;
}

}  // extern "C"
