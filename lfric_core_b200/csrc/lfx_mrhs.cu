// Many right-hand sides of one LMA operator at once.
//
// Vectors of nrhs (16, 32 or 64) right-hand sides are stored dof-major,
// [undf][nrhs]. The operator must have the lowest-order nodal (W0) structure:
// ndf = 8, dofs 0..3 on the bottom and 4..7 on the top vertices, top = bottom
// + 1, so every dof lies on a vertex column of nlayers + 1 dofs. A row then
// couples to the levels l - 1, l, l + 1 of the vertex columns that share a
// cell with its own: at creation the local matrices are summed (in FP64) into
// these column stencils, 27 coefficients a row where four cells meet instead
// of the 64 of a cell level, and the apply gathers (mrhs_apply_k). No two
// threads add to one row, so there are no atomics, no colours, no barriers,
// and every sum has a fixed order.
//
// The vertex columns are ordered patch by patch (patches of cells grown
// breadth-first over shared vertices, a column in the patch that holds most
// of its cells), so that the columns of one thread block are neighbours and
// share the rows they read in L1.
//
// The solve wraps an FP32 preconditioned CG over all right-hand sides (each
// with its own step lengths; Jacobi preconditioner) in FP64 iterative
// refinement: the residual b - A x and the solution stay FP64 (RHS-major, the
// plain FP64 operator applies them), each inner solve reduces its residual by
// the inner tolerance, and a right-hand side converges on its true FP64
// residual ||b - A x|| / ||b - A x0||.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <queue>
#include <unordered_map>
#include <vector>

#include "lfx_internal.cuh"

using namespace lfx;

namespace {

constexpr int kMaxPC = 12;  // colours inside one patch (so cells around a vertex), at most
constexpr int kMaxSlot = 3 * kMaxPC + 1;  // vertex columns one column couples to, at most
constexpr int kDefaultPatch = 16;

// Column stencils. Slot t of a column names one vertex column it couples to
// (the column itself is its last slot); a slot holds, for every group of four
// rows, the coefficients {d = 0: level l - 1, d = 1: l, d = 2: l + 1} x
// {4 rows} contiguously in FP32, zero past the column's top and for levels
// that do not exist. FP32 for either kind: BF16 coefficients took the apply
// from 154 to 156 us (C48 x 30, 64 right-hand sides), and rounding a summed
// row to 8 bits moves its row sum by more than the cells' roundings did
// together, which cost block CG a third more iterations.
struct StencilArgs {
  const int* base;  // [ncol] first dof of each vertex column
  const int* off;   // [ncol + 1] first slot of each column
  const int* nbr;   // [nslot] first dof of the slot's vertex column
  float* coef;      // [nslot][g4][3][4]
  int ncol, h, g4;  // columns, rows of a column, groups of four rows
};

// the cells around each column: {cell, local vertex, slots of the cell's four
// vertices (a byte each), 0}
template <class TM>
__global__ void mrhs_assemble(StencilArgs A, const int* __restrict__ coff,
                              const int4* __restrict__ ccell, const TM* __restrict__ M, int nl,
                              int blk) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)A.ncol * A.h) return;
  const int v = (int)(i / A.h), l = (int)(i % A.h);
  const int s0 = A.off[v], ns = A.off[v + 1] - s0;
  double a[kMaxSlot][3];
  for (int t = 0; t < ns; ++t) a[t][0] = a[t][1] = a[t][2] = 0.0;
  for (int e = coff[v]; e < coff[v + 1]; ++e) {
    const int4 ce = ccell[e];
    // row l is the bottom vertex of cell level l and the top one of l - 1
    for (int top = 0; top < 2; ++top) {
      const int k = l - top;
      if (k < 0 || k >= nl) continue;
      const TM* Mr = M + ((int64_t)ce.x * 8 + ce.y + 4 * top) * (int64_t)blk + k;
      for (int j = 0; j < 4; ++j) {
        const int t = (ce.z >> (8 * j)) & 255;
        a[t][1 - top] += (double)Mr[(int64_t)j * nl];
        a[t][2 - top] += (double)Mr[(int64_t)(j + 4) * nl];
      }
    }
  }
  float* c = A.coef + (l & 3);
  for (int t = 0; t < ns; ++t)
    for (int d = 0; d < 3; ++d)
      c[(((int64_t)(s0 + t) * A.g4 + (l >> 2)) * 3 + d) * 4] = (float)a[t][d];
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

// ------------------------------------------------ dof-major vector kernels
// A thread handles four consecutive right-hand sides of a row (16-byte
// accesses): NR / 4 threads per row, RPB = 1024 / NR rows per block pass.

template <int NR>
struct MvShape {
  static constexpr int TPR = NR / 4;      // threads per row
  static constexpr int RPB = 256 / TPR;   // rows per block pass
};

__device__ __forceinline__ void l2_prefetch(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// The block's sums over its rows of sum r of every right-hand side, to
// partials[(r * NR + column) * blocks + block] (256 threads; acc[j] belongs to
// column 4 (threadIdx.x % TPR) + j). mv_fin adds the blocks up, in order.
template <int NR>
__device__ __forceinline__ void mv_block_sums(double (&acc)[4], double* partials, int r) {
  constexpr int TPR = MvShape<NR>::TPR;
  __shared__ double sm[8][NR];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll
    for (int o = 16; o >= TPR; o >>= 1) acc[j] = acc[j] + __shfl_xor_sync(0xffffffffu, acc[j], o);
    if (lane < TPR) sm[w][4 * lane + j] = acc[j];
  }
  __syncthreads();
  if (threadIdx.x < NR) {
    double s = sm[0][threadIdx.x];
#pragma unroll
    for (int q = 1; q < 8; ++q) s = s + sm[q][threadIdx.x];
    const size_t G = (size_t)gridDim.x * gridDim.y;
    partials[((size_t)r * NR + threadIdx.x) * G + (size_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
  }
  __syncthreads();
}

// Y = A X; with DOT also the block's share of <x, y> of every right-hand side.
// NR / 4 lanes (a group) take one vertex column, four right-hand sides a lane,
// and LB rows at a time: LB + 2 rows of each coupled column are loaded once
// (16 bytes a lane) and used for up to three rows of the result in registers.
//
// Bound: bytes in flight. Its 266 MB (x, y, coefficients; C48 x 30, 64
// right-hand sides) would take 41 us at 6.5 TB/s, the 27 FMAs a row and
// right-hand side 20 us on the FP32 cores; it takes 138 us (8 rows a pass; 157
// with 4 rows, where the two overlapping levels weigh more), from 250 us for
// products cell by cell on the tensor cores (mma.sync m16n8k8, TF32; BF16 300
// us) with sums through shared memory, seven colour barriers per block of
// levels and 1.7 cell levels computed per cell. Without the prefetches 154 us;
// coefficients through a cp.async ring and rows a step ahead in registers 165
// us (184 registers, one block an SM).
constexpr int LB = 8;      // rows held at once
constexpr int kAhead = 2;  // groups of LB rows a column's own rows are prefetched ahead

template <int RB, bool DOT>
__global__ void __launch_bounds__(256) mrhs_apply_k(StencilArgs A, const float* __restrict__ X,
                                                    float* __restrict__ Y,
                                                    double* __restrict__ partials) {
  constexpr int NR = 16 * RB, LPG = NR / 4, GPB = 256 / LPG;
  const int grp = threadIdx.x / LPG, c4 = threadIdx.x % LPG;
  const int v = blockIdx.x * GPB + grp;
  double dt[4] = {0.0, 0.0, 0.0, 0.0};
  if (v < A.ncol) {
    const int h = A.h, s0 = __ldg(A.off + v), s1 = __ldg(A.off + v + 1) - 1;
    const int nb = (h + LB - 1) / LB;
    const int b0 = (int)((int64_t)nb * blockIdx.y / gridDim.y);
    const int b1 = (int)((int64_t)nb * (blockIdx.y + 1) / gridDim.y);
    const int vb = __ldg(A.base + v);
    const float* Xc = X + 4 * c4;
    // the column's own rows go out to L2 ahead (every column of the grid does
    // the same, so a neighbour's rows are there too when they are read)
    auto ahead = [&](int l, int nr) {
      if (c4 == 0 && l < h)
        l2_prefetch(X + (int64_t)(vb + l) * NR, (unsigned)(min(nr, h - l) * NR * 4));
    };
    if (c4 == 0)
      l2_prefetch(A.coef + (int64_t)s0 * A.g4 * 12, (unsigned)((s1 + 1 - s0) * A.g4 * 48));
    ahead(b0 * LB, kAhead * LB);
    for (int rb = b0; rb < b1; ++rb) {
      const int l0 = rb * LB;
      if (rb + kAhead < nb) ahead(l0 + kAhead * LB, LB);
      float4 acc[LB];
#pragma unroll
      for (int r = 0; r < LB; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 xv[LB + 2];
      auto slot = [&](int t, int ub) {
#pragma unroll
        for (int q = 0; q < LB + 2; ++q) {
          const int l = l0 + q - 1;
          xv[q] = (unsigned)l < (unsigned)h
                      ? __ldg(reinterpret_cast<const float4*>(Xc + (int64_t)(ub + l) * NR))
                      : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int g = 0; g < LB / 4; ++g) {
          // (a group of rows past the column's top has no coefficients)
          if (g > 0 && l0 + 4 * g >= h) break;
          const int64_t ci = ((int64_t)t * A.g4 + (l0 >> 2) + g) * 3;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const float4 aq = __ldg(reinterpret_cast<const float4*>(A.coef) + ci + d);
            const float a[4] = {aq.x, aq.y, aq.z, aq.w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              float4& o = acc[4 * g + r];
              const float4 x = xv[4 * g + r + d];
              o.x = fmaf(a[r], x.x, o.x);
              o.y = fmaf(a[r], x.y, o.y);
              o.z = fmaf(a[r], x.z, o.z);
              o.w = fmaf(a[r], x.w, o.w);
            }
          }
        }
      };
#pragma unroll 2
      for (int t = s0; t < s1; ++t) slot(t, __ldg(A.nbr + t));
      slot(s1, vb);  // the column itself: its rows stay in xv
#pragma unroll
      for (int r = 0; r < LB; ++r) {
        if (l0 + r >= h) break;
        st4(Y + (int64_t)(vb + l0 + r) * NR + 4 * c4, acc[r]);
        if (DOT) {
          const float4 x = xv[r + 1];
          dt[0] = fma((double)x.x, (double)acc[r].x, dt[0]);
          dt[1] = fma((double)x.y, (double)acc[r].y, dt[1]);
          dt[2] = fma((double)x.z, (double)acc[r].z, dt[2]);
          dt[3] = fma((double)x.w, (double)acc[r].w, dt[3]);
        }
      }
    }
  }
  if (DOT) mv_block_sums<NR>(dt, partials, 0);
}

struct MvState {
  double rz[64], alpha[64], beta[64], r0[64], rn[64];
  int active[64], iters[64];
  int nactive;
};

#define LFX_MV_ROWS(NR)                                                      \
  const int c4 = threadIdx.x % MvShape<NR>::TPR;                             \
  _Pragma("unroll 2") for (int64_t row = (int64_t)blockIdx.x * MvShape<NR>::RPB +                \
                     threadIdx.x / MvShape<NR>::TPR;                         \
       row < n; row += (int64_t)gridDim.x * MvShape<NR>::RPB)

// The scalars of one right-hand side (a block each) from the G block sums of
// the kernel before: mode 0 after mv_init (r0, rz, active), 1 after the apply
// (alpha = rz / <p, q>), 2 after mv_residual (||r||, beta, rz and the inner
// convergence test ||r|| <= tol ||r0||). A launch of its own: a tail in the
// last block of those kernels took longer, its one block reading the sums of
// every right-hand side.
template <int NR>
__global__ void __launch_bounds__(128) mv_fin(int mode, int G, const double* __restrict__ partials,
                                              const int* act_out, double tol, MvState* S) {
  __shared__ double sm[2][4];
  const int c = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nred = mode == 1 ? 1 : 2;
  for (int r = 0; r < nred; ++r) {
    const double* p = partials + ((size_t)r * NR + c) * G;
    double s = 0.0;
    for (int b = threadIdx.x; b < G; b += 128) s = s + p[b];
    s = warp_butterfly(s);
    if (lane == 0) sm[r][w] = s;
  }
  __syncthreads();
  if (threadIdx.x) return;
  const double t0 = ((sm[0][0] + sm[0][1]) + sm[0][2]) + sm[0][3];
  const double t1 = nred == 2 ? ((sm[1][0] + sm[1][1]) + sm[1][2]) + sm[1][3] : 0.0;
  if (mode == 0) {
    const double r0 = sqrt(t0);
    S->r0[c] = r0;
    S->rn[c] = r0;
    S->rz[c] = t1;
    S->alpha[c] = 0.0;
    S->beta[c] = 0.0;
    const int on = act_out[c] && r0 > 0.0 && t1 > 0.0;
    S->active[c] = on;
    if (on) atomicAdd(&S->nactive, 1);
  } else if (mode == 1) {
    S->alpha[c] = (S->active[c] && t0 != 0.0) ? S->rz[c] / t0 : 0.0;
  } else if (S->active[c]) {
    const double rn = sqrt(t0);
    S->rn[c] = rn;
    S->beta[c] = t1 / S->rz[c];
    S->rz[c] = t1;
    S->iters[c] += 1;
    if (!(rn > tol * S->r0[c]) || !(t1 > 0.0)) {
      S->active[c] = 0;
      atomicSub(&S->nactive, 1);
    }
  } else {
    S->beta[c] = 0.0;
  }
}

// x = 0, p = z = D^-1 r; sums <r, r>, <r, z> per right-hand side
template <int NR>
__global__ void __launch_bounds__(256) mv_init(int64_t n, const float* __restrict__ dinv,
                                               const float* __restrict__ r, float* __restrict__ p,
                                               float* __restrict__ x, double* partials) {
  double acc[2][4] = {};
  LFX_MV_ROWS(NR) {
    const size_t i = (size_t)row * NR + 4 * c4;
    const float4 rv = ld4(r + i);
    const float d = dinv[row];
    const float4 zv = make_float4(rv.x * d, rv.y * d, rv.z * d, rv.w * d);
    st4(p + i, zv);
    st4(x + i, make_float4(0.f, 0.f, 0.f, 0.f));
    const float ra[4] = {rv.x, rv.y, rv.z, rv.w}, za[4] = {zv.x, zv.y, zv.z, zv.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[0][j] = fma((double)ra[j], (double)ra[j], acc[0][j]);
      acc[1][j] = fma((double)ra[j], (double)za[j], acc[1][j]);
    }
  }
  mv_block_sums<NR>(acc[0], partials, 0);
  mv_block_sums<NR>(acc[1], partials, 1);
}

// r -= alpha q; sums <r, r>, <r, D^-1 r>
template <int NR>
__global__ void __launch_bounds__(256) mv_residual(int64_t n, const float* __restrict__ dinv,
                                                   const float* __restrict__ q,
                                                   float* __restrict__ r, const MvState* S,
                                                   double* partials) {
  float a[4];
  {
    const int c0 = 4 * (threadIdx.x % MvShape<NR>::TPR);
#pragma unroll
    for (int j = 0; j < 4; ++j) a[j] = (float)S->alpha[c0 + j];
  }
  double acc[2][4] = {};
  LFX_MV_ROWS(NR) {
    const size_t i = (size_t)row * NR + 4 * c4;
    const float4 qv = ld4(q + i), rv = ld4(r + i);
    const float d = dinv[row];
    const float rn[4] = {fmaf(-a[0], qv.x, rv.x), fmaf(-a[1], qv.y, rv.y),
                         fmaf(-a[2], qv.z, rv.z), fmaf(-a[3], qv.w, rv.w)};
    st4(r + i, make_float4(rn[0], rn[1], rn[2], rn[3]));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[0][j] = fma((double)rn[j], (double)rn[j], acc[0][j]);
      acc[1][j] = fma((double)rn[j], (double)(rn[j] * d), acc[1][j]);
    }
  }
  mv_block_sums<NR>(acc[0], partials, 0);
  mv_block_sums<NR>(acc[1], partials, 1);
}

// x += alpha p, p = D^-1 r + beta p (p is read once for both)
template <int NR>
__global__ void __launch_bounds__(256) mv_direction(int64_t n, const float* __restrict__ dinv,
                                                    const float* __restrict__ r,
                                                    float* __restrict__ p, float* __restrict__ x,
                                                    const MvState* S) {
  float a[4], b[4];
  {
    const int c0 = 4 * (threadIdx.x % MvShape<NR>::TPR);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] = (float)S->alpha[c0 + j];
      b[j] = (float)S->beta[c0 + j];
    }
  }
  LFX_MV_ROWS(NR) {
    const size_t i = (size_t)row * NR + 4 * c4;
    const float4 rv = ld4(r + i), pv = ld4(p + i), xv = ld4(x + i);
    const float d = dinv[row];
    st4(x + i, make_float4(fmaf(a[0], pv.x, xv.x), fmaf(a[1], pv.y, xv.y), fmaf(a[2], pv.z, xv.z),
                           fmaf(a[3], pv.w, xv.w)));
    st4(p + i, make_float4(fmaf(b[0], pv.x, rv.x * d), fmaf(b[1], pv.y, rv.y * d),
                           fmaf(b[2], pv.z, rv.z * d), fmaf(b[3], pv.w, rv.w * d)));
  }
}
#undef LFX_MV_ROWS

// r[row][col] = (float) R[col * ld + row] (RHS-major FP64 to dof-major FP32)
template <int NR>
__global__ void mv_from_rhs_major(int64_t n, const double* __restrict__ R, int64_t ld,
                                  float* __restrict__ r) {
  constexpr int TW = NR < 32 ? NR : 32;
  __shared__ float tile[TW][33];
  const int64_t row0 = (int64_t)blockIdx.x * 32;
  const int col0 = blockIdx.y * TW;
  for (int j = threadIdx.y; j < TW; j += blockDim.y) {
    const int64_t row = row0 + threadIdx.x;
    if (row < n) tile[j][threadIdx.x] = (float)R[(size_t)(col0 + j) * ld + row];
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int64_t row = row0 + j;
    if (row < n && threadIdx.x < TW) r[(size_t)row * NR + col0 + threadIdx.x] = tile[threadIdx.x][j];
  }
}

// X[col * ld + row] += x[row][col]
template <int NR>
__global__ void mv_add_to_rhs_major(int64_t n, const float* __restrict__ x, double* __restrict__ X,
                                    int64_t ld) {
  constexpr int TW = NR < 32 ? NR : 32;
  __shared__ float tile[TW][33];
  const int64_t row0 = (int64_t)blockIdx.x * 32;
  const int col0 = blockIdx.y * TW;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int64_t row = row0 + j;
    if (row < n && threadIdx.x < TW) tile[threadIdx.x][j] = x[(size_t)row * NR + col0 + threadIdx.x];
  }
  __syncthreads();
  for (int j = threadIdx.y; j < TW; j += blockDim.y) {
    const int64_t row = row0 + threadIdx.x;
    if (row < n) X[(size_t)(col0 + j) * ld + row] += (double)tile[j][threadIdx.x];
  }
}

__global__ void k_dinv(int64_t n, const double* __restrict__ d, float* __restrict__ dinv) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dinv[i] = (float)(1.0 / d[i]);
}

// ------------------------------------------------ block CG
// Breakdown-free block preconditioned CG on all 64 right-hand sides at once
// (the block Krylov method of the reference's block_gcr_solve family,
// sci_iterative_solver_mod.f90:1461-1628, in its CG form):
//   Z = D^-1 R, P = orth(Z)
//   loop: Q = A P; alpha = (P^T Q)^-1 P^T R; X += P alpha; R -= Q alpha;
//         beta = -(P^T Q)^-1 Q^T D^-1 R; P = orth(D^-1 R + P beta)
// orth(W) = W T with T from a pivoted Cholesky factorisation of W^T W that
// stops at pivots below kBcgDrop times the largest one: directions the block
// no longer spans (right-hand sides that have converged, or become
// dependent) are dropped, so the method does not break down. The products
// with the tall n x 64 blocks run as 32-row chunks staged in shared memory,
// each thread holding a 4 x 4 (Gram) or 2 x 4 (update) register tile; the
// Gram sums are FP32 within a chunk, FP64 across chunks and blocks, in a
// fixed order; the 64 x 64 algebra runs in FP64 in one block.
constexpr int kBS = 64;          // right-hand sides of a block solve
constexpr int kBcgRows = 32;     // rows per staged chunk
// W is FP32 and its Gram sums carry relative errors near 1e-6 of the largest
// entry, so directions whose pivot falls below 1e-5 of the largest are noise
// and are dropped (the kept part of W then has a condition number under
// about 300, and W T is orthonormal to a few parts in a thousand)
constexpr double kBcgDrop = 1e-5;

struct BcgSmall {
  double C[2 * kBS * kBS];  // [v][i][j]: v = 0 P^T Q, v = 1 P^T R (gram of P with Q, R)
  double E[kBS * kBS];      // Q^T D^-1 R
  double G[kBS * kBS];      // W^T W
  double L1[kBS * kBS];     // inverse of the Cholesky factor of the active block of P^T Q
  double r0[kBS], rn[kBS];
  float coef[kBS * kBS];    // alpha, beta or T [k][j] for the next row update
  int active[kBS];          // right-hand sides the solve works on
  int rank, done, iters, fail;
};

// ---- The same Gram on the 5th-generation tensor cores (tcgen05).
// D (64 x 64 NV) = U^T [V_0 .. V_NV-1] accumulates in tensor memory (TMEM,
// FP32): A = U^T (64 x K) and B = V^T (64 NV x K) are both K-major in shared
// memory (kind::tf32 takes K-major operands only), in the canonical
// no-swizzle layout: core matrices of 8 MN-rows x 16 bytes (4 K values),
// MN-rows 16 bytes apart, MN groups of 8 rows 128 bytes apart (stride byte
// offset), K groups of 4 values MN/8 x 128 bytes apart (leading byte offset).
// Each FP32 value is split into TF32 parts hi + lo and a product taken as
// hi hi + hi lo + lo hi (three kind::tf32 MMAs of M = 64, K = 8 per K step),
// which keeps about FP32 accuracy. Two 32-row stages: the block stages the
// next chunk while the tensor core works on the last one; one elected thread
// issues the MMAs and commits them to the stage's mbarrier. Every mbarrier
// wait is bounded; a wait that runs out sets st->fail = 2 and the block
// stops issuing work (the final wait is bounded too before TMEM is freed).
constexpr int kTcRows = 32;
constexpr int kTcThreads = 128;
constexpr unsigned long long kTcWaitNs = 2000000000ull;  // 2 s

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// shared-memory matrix descriptor: start, leading (K group) and stride (MN
// group) byte offsets, version 1, no swizzle
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// instruction descriptor: FP32 accumulate, A and B TF32, both K-major, M = 64
template <int N>
__host__ __device__ constexpr uint32_t idesc_tf32_k() {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(64 >> 4) << 24);
}
__device__ __forceinline__ void tc_mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                       uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}
__device__ __forceinline__ unsigned long long tc_clock() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// wait for the mbarrier phase of the given parity, for at most kTcWaitNs
__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity) {
  const unsigned long long t0 = tc_clock();
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
    if (tc_clock() - t0 > kTcWaitNs) return false;
  }
}
__device__ __forceinline__ float tf32_round(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
// stage rows row0 .. row0 + 31 (the K dimension) of an n x MN block made of
// 64-column row-major sources (columns 0..63 from s0, 64.. from s1) as the
// K-major operand (MN x 32), TF32 hi and lo parts; rows past n are zero. A
// thread takes four consecutive rows of one column: the warp's loads of a row
// are coalesced and its 16-byte stores fill 512 contiguous bytes.
__device__ __forceinline__ void tc_stage(unsigned char* hi, unsigned char* lo, int MN,
                                         const float* s0, const float* s1, int64_t row0,
                                         int64_t n, const float* __restrict__ scale) {
  for (int e = threadIdx.x; e < (kTcRows / 4) * MN; e += kTcThreads) {
    const int m = e % MN, kq = e / MN;
    const float* src = m < kBS ? s0 + m : s1 + (m - kBS);
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t k = row0 + 4 * kq + q;
      v[q] = 0.f;
      if (k < n) {
        v[q] = __ldg(src + (size_t)k * kBS);
        if (scale) v[q] *= __ldg(scale + k);
      }
    }
    const float4 h = make_float4(tf32_round(v[0]), tf32_round(v[1]), tf32_round(v[2]), tf32_round(v[3]));
    const float4 l = make_float4(tf32_round(v[0] - h.x), tf32_round(v[1] - h.y),
                                 tf32_round(v[2] - h.z), tf32_round(v[3] - h.w));
    const size_t off = ((size_t)kq * (MN / 8) + m / 8) * 128 + (size_t)(m % 8) * 16;
    *reinterpret_cast<float4*>(hi + off) = h;
    *reinterpret_cast<float4*>(lo + off) = l;
  }
}

template <int NV>
__global__ void __launch_bounds__(kTcThreads) bcg_gram_tc(int64_t n, const float* __restrict__ U,
                                                         const float* __restrict__ V0,
                                                         const float* __restrict__ V1,
                                                         const float* __restrict__ vscale,
                                                         double* __restrict__ partials,
                                                         BcgSmall* st) {
  constexpr int N = kBS * NV, LBA = kBS / 8 * 128, LBB = N / 8 * 128;
  constexpr int ABYTES = kTcRows * kBS * 4, BBYTES = kTcRows * N * 4;
  constexpr int STAGE = 2 * ABYTES + 2 * BBYTES;
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  __shared__ __align__(8) uint64_t mbar[2];
  __shared__ uint32_t tmem_base;
  __shared__ int s_abort;
  if (st->done) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"((uint32_t)N)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[0])) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar[1])) : "memory");
    s_abort = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;
  constexpr uint32_t IDESC = idesc_tf32_k<N>();
  int j = 0;  // chunks of this block so far
  for (int64_t c = blockIdx.x; c * kTcRows < n; c += gridDim.x, ++j) {
    const int sidx = j & 1;
    unsigned char* base = tc_smem + (size_t)sidx * STAGE;
    if (j >= 2) {
      // the MMAs that last read this stage have completed
      if (threadIdx.x == 0 && !tc_wait(smem_u32(&mbar[sidx]), (uint32_t)((j / 2 - 1) & 1))) {
        s_abort = 1;
        st->fail = 2;
      }
      __syncthreads();
      if (s_abort) break;
    }
    tc_stage(base, base + ABYTES, kBS, U, U, c * kTcRows, n, nullptr);
    tc_stage(base + 2 * ABYTES, base + 2 * ABYTES + BBYTES, N, V0, NV > 1 ? V1 : V0,
             c * kTcRows, n, vscale);
    // generic-proxy writes of the operands become visible to the tensor core
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t a_hi = smem_u32(base), a_lo = a_hi + ABYTES;
      const uint32_t b_hi = a_hi + 2 * ABYTES, b_lo = b_hi + BBYTES;
#pragma unroll
      for (int kg = 0; kg < kTcRows / 8; ++kg) {
        // K step kg: K groups 2 kg and 2 kg + 1
        const uint64_t ah = umma_desc(a_hi + 2 * kg * LBA, LBA, 128);
        const uint64_t al = umma_desc(a_lo + 2 * kg * LBA, LBA, 128);
        const uint64_t bh = umma_desc(b_hi + 2 * kg * LBB, LBB, 128);
        const uint64_t bl = umma_desc(b_lo + 2 * kg * LBB, LBB, 128);
        tc_mma(tmem, ah, bh, IDESC, (j > 0 || kg > 0) ? 1u : 0u);
        tc_mma(tmem, ah, bl, IDESC, 1u);
        tc_mma(tmem, al, bh, IDESC, 1u);
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&mbar[sidx]))
                   : "memory");
    }
  }
  // the last commit covers every MMA of the block
  if (j > 0 && threadIdx.x == 0 &&
      !tc_wait(smem_u32(&mbar[(j - 1) & 1]), (uint32_t)(((j - 1) / 2) & 1))) {
    s_abort = 1;
    st->fail = 2;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  double* out = partials + (size_t)blockIdx.x * NV * kBS * kBS;
  // M = 64: row m sits in TMEM lane (m % 16) + 32 (m / 16); warp w reads
  // lanes 32 w .. 32 w + 31, whose first 16 hold rows 16 w .. 16 w + 15
#pragma unroll
  for (int c0 = 0; c0 < N; c0 += 32) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
        "%11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, "
        "%28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)c0));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (lane < 16) {
      const int m = 16 * warp + lane;
#pragma unroll
      for (int q = 0; q < 32; ++q) {
        const int jj = c0 + q, v = jj / kBS, jc = jj % kBS;
        out[((size_t)v * kBS + m) * kBS + jc] =
            (j > 0 && !s_abort) ? (double)__uint_as_float(r[q]) : 0.0;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"((uint32_t)N)
                 : "memory");
}

template <int NV>
constexpr size_t tc_gram_smem() {
  return 2 * (2 * (size_t)kTcRows * kBS * 4 + 2 * (size_t)kTcRows * kBS * NV * 4);
}

// out[e] = sum over the blocks, in block order, of partials[b][e]
// A block takes 32 entries, warp w the w-th eighth of the partials; the eight
// sums are added left to right. (One thread an entry, 16 blocks in all for a
// Gram, took 28 us of 296 x 32 KB.)
__global__ void __launch_bounds__(256) bcg_reduce(int nb, int ne,
                                                  const double* __restrict__ partials,
                                                  double* __restrict__ out, const BcgSmall* st) {
  __shared__ double sm[8][32];
  if (st->done) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + lane;
  const int b0 = nb * w / 8, b1 = nb * (w + 1) / 8;
  double s = 0.0;
#pragma unroll 8
  for (int b = b0; b < b1; ++b)
    if (e < ne) s = s + __ldg(partials + (size_t)b * ne + e);
  sm[w][lane] = s;
  __syncthreads();
  if (w == 0 && e < ne) {
#pragma unroll
    for (int q = 1; q < 8; ++q) s = s + sm[q][lane];
    out[e] = s;
  }
}

// ---- The same products with the tall blocks streamed. A block takes the
// 32-row chunks c = blockIdx.x + i gridDim.x of its operands (each chunk of
// an n x 64 row-major FP32 block is one contiguous 8 KB run) through a ring
// of S stages in shared memory: thread 0 moves a chunk's operands with
// cp.async.bulk copies completing on the stage's mbarrier, S - 1 chunks
// ahead of the compute, so the bytes in flight cost no registers. Every wait
// is bounded (kTcWaitNs); the block decides together (__syncthreads_and)
// and, on a time-out, sets st->fail = 2, waits (bounded) for the copies it
// issued and stops. Sums: FP32 within a chunk, FP64 across chunks and blocks, in a fixed order.
constexpr int kChunkBytes = kBcgRows * kBS * 4;  // one operand's chunk
template <int NA, int S>
struct ChunkRing {
  static constexpr int STAGE = NA * kChunkBytes;
  static constexpr size_t BYTES = (size_t)S * STAGE + (size_t)S * 8;
};
__device__ __forceinline__ bool chunk_try(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool chunk_wait(uint64_t* bar, unsigned parity) {
  if (chunk_try(bar, parity)) return true;
  const unsigned long long t0 = tc_clock();
  while (!chunk_try(bar, parity))
    if (tc_clock() - t0 > kTcWaitNs) return false;
  return true;
}
// thread 0: chunk c of the NA operands into stage buffer dst, on bar
template <int NA>
__device__ __forceinline__ void chunk_issue(const float* const (&src)[NA], int64_t c, int64_t n,
                                            unsigned char* dst, uint64_t* bar) {
  const int64_t row0 = c * kBcgRows;
  const int rows = (int)(n - row0 < (int64_t)kBcgRows ? n - row0 : (int64_t)kBcgRows);
  const unsigned bytes = (unsigned)rows * kBS * 4;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes * NA)
               : "memory");
#pragma unroll
  for (int a = 0; a < NA; ++a)
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst + a * kChunkBytes)),
        "l"(src[a] + (size_t)row0 * kBS), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
// the ring's set-up and its bounded drain after a time-out (chunks from..to-1:
// the one whose wait ran out and those issued after it)
template <int S>
__device__ __forceinline__ void chunk_ring_init(uint64_t* bar) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < S; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar + i)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
}
template <int S>
__device__ __forceinline__ void chunk_ring_drain(uint64_t* bar, int from, int to) {
  if (threadIdx.x == 0)
    for (int i = from; i < to; ++i) chunk_wait(bar + i % S, (unsigned)((i / S) & 1));
}

template <int NV>
__global__ void __launch_bounds__(256, 2) bcg_gram_s(int64_t n, const float* __restrict__ U,
                                                  const float* __restrict__ V0,
                                                  const float* __restrict__ V1,
                                                  const float* __restrict__ vscale,
                                                  double* __restrict__ partials, BcgSmall* st) {
  constexpr int NA = 1 + NV, S = 4;
  using RG = ChunkRing<NA, S>;
  extern __shared__ __align__(16) unsigned char ring_smem[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(ring_smem + S * RG::STAGE);
  if (st->done) return;
  const float* src[NA];
  src[0] = U;
  src[1] = V0;
  if (NV > 1) src[NA - 1] = V1;
  const int64_t nchunk = (n + kBcgRows - 1) / kBcgRows;
  const int nmine = blockIdx.x < nchunk ? (int)((nchunk - 1 - blockIdx.x) / gridDim.x + 1) : 0;
  chunk_ring_init<S>(bar);
  if (threadIdx.x == 0)
    for (int i = 0; i < S && i < nmine; ++i)
      chunk_issue<NA>(src, blockIdx.x + (int64_t)i * gridDim.x, n, ring_smem + i * RG::STAGE, bar + i);
  const int i0 = 4 * (threadIdx.x / 16), j0 = 4 * (threadIdx.x % 16);
  double acc[NV][4][4];
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[v][a][b] = 0.0;
  bool failed = false;
  for (int i = 0; i < nmine; ++i) {
    const int stg = i % S;
    const bool ok = chunk_wait(bar + stg, (unsigned)((i / S) & 1));
    if (!__syncthreads_and(ok)) {
      if (threadIdx.x == 0) st->fail = 2;
      chunk_ring_drain<S>(bar, i, nmine < i + S ? nmine : i + S);
      failed = true;
      break;
    }
    const int64_t c = blockIdx.x + (int64_t)i * gridDim.x, row0 = c * kBcgRows;
    const int rows = (int)(n - row0 < (int64_t)kBcgRows ? n - row0 : (int64_t)kBcgRows);
    const float (*Us)[kBS] = reinterpret_cast<const float (*)[kBS]>(ring_smem + stg * RG::STAGE);
    float a[NV][4][4];
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) a[v][x][y] = 0.f;
    // the row scales of this chunk: one load a lane, then shuffles (the
    // two-operand form measured faster this way; the one-operand form keeps
    // a load per row)
    const int lane = threadIdx.x & 31;
    const float sc_lane = (NV == 2 && vscale && lane < rows) ? __ldg(vscale + row0 + lane) : 1.f;
    for (int r = 0; r < rows; ++r) {
      const float4 u = *reinterpret_cast<const float4*>(&Us[r][i0]);
      const float uu[4] = {u.x, u.y, u.z, u.w};
      const float sc = !vscale ? 1.f
                       : NV == 2 ? __shfl_sync(0xffffffffu, sc_lane, r)
                                 : __ldg(vscale + row0 + r);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const float (*Vs)[kBS] =
            reinterpret_cast<const float (*)[kBS]>(ring_smem + stg * RG::STAGE + (1 + v) * kChunkBytes);
        float4 w = *reinterpret_cast<const float4*>(&Vs[r][j0]);
        if (vscale) {
          w.x *= sc; w.y *= sc; w.z *= sc; w.w *= sc;
        }
        const float ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) a[v][x][y] = fmaf(uu[x], ww[y], a[v][x][y]);
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) acc[v][x][y] += (double)a[v][x][y];
    __syncthreads();  // the stage is read: it takes chunk i + S
    if (threadIdx.x == 0 && i + S < nmine)
      chunk_issue<NA>(src, blockIdx.x + (int64_t)(i + S) * gridDim.x, n, ring_smem + stg * RG::STAGE,
                      bar + stg);
  }
  double* out = partials + (size_t)blockIdx.x * NV * kBS * kBS;
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y)
        out[((size_t)v * kBS + i0 + x) * kBS + j0 + y] = failed ? 0.0 : acc[v][x][y];
}

// Y (+)= B C streamed: mode 0 (P, Q, X, R): X += P C, R -= Q C and the column
// sums of R^2; mode 1 (P, R): W = D^-1 R + P C; mode 2 (W): P = W C
template <int MODE>
struct UpdOps {
  static constexpr int NA = MODE == 0 ? 4 : MODE == 1 ? 2 : 1;
  static constexpr int S = MODE == 0 ? 3 : 4;
};
template <int MODE>
__global__ void __launch_bounds__(256) bcg_update_s(int64_t n, const float* __restrict__ A0,
                                                    const float* __restrict__ A1, float* Y0,
                                                    float* Y1, const float* __restrict__ dinv,
                                                    const BcgSmall* st, int skip_p,
                                                    double* __restrict__ partials) {
  constexpr int NA = UpdOps<MODE>::NA, S = UpdOps<MODE>::S;
  using RG = ChunkRing<NA, S>;
  extern __shared__ __align__(16) unsigned char ring_smem[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(ring_smem + S * RG::STAGE);
  __shared__ __align__(16) float Cs[kBS][kBS];
  if (st->done) return;
  for (int e = threadIdx.x; e < kBS * kBS; e += blockDim.x) Cs[e / kBS][e % kBS] = st->coef[e];
  // streamed operands: mode 0 P, Q, X, R; mode 1 P, R; mode 2 W
  const float* src[NA];
  src[0] = A0;
  if (MODE == 0) {
    src[1] = A1;
    src[2] = Y0;
    src[3] = Y1;
  } else if (MODE == 1) {
    src[1] = A1;
  }
  const int64_t nchunk = (n + kBcgRows - 1) / kBcgRows;
  const int nmine = blockIdx.x < nchunk ? (int)((nchunk - 1 - blockIdx.x) / gridDim.x + 1) : 0;
  chunk_ring_init<S>(bar);
  if (threadIdx.x == 0)
    for (int i = 0; i < S && i < nmine; ++i)
      chunk_issue<NA>(src, blockIdx.x + (int64_t)i * gridDim.x, n, ring_smem + i * RG::STAGE, bar + i);
  // thread: column c of the output for the 8 rows 8 rg .. 8 rg + 7 of each
  // chunk, with column c of the coefficients in registers; the operand rows
  // are read four values at a time, every lane of a warp at the same address
  // (one shared-memory wavefront). Each output is one fmaf chain over
  // k = 0..63, as before the tiling changed.
  const int c = 32 * ((threadIdx.x >> 5) & 1) + (threadIdx.x & 31), rg = threadIdx.x >> 6;
  float cr[kBS];
  __syncthreads();  // Cs is written
#pragma unroll
  for (int k = 0; k < kBS; ++k) cr[k] = Cs[k][c];
  // the squared-residual sums of row pairs 4 rg + i, in the order of the
  // earlier two-rows-a-thread form (row 2q, then 2q + 1, chunk by chunk)
  double nrm[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = 0; i < nmine; ++i) {
    const int stg = i % S;
    const bool ok = chunk_wait(bar + stg, (unsigned)((i / S) & 1));
    if (!__syncthreads_and(ok)) {
      if (threadIdx.x == 0) const_cast<BcgSmall*>(st)->fail = 2;
      chunk_ring_drain<S>(bar, i, nmine < i + S ? nmine : i + S);
      break;
    }
    const int64_t ch = blockIdx.x + (int64_t)i * gridDim.x, row0 = ch * kBcgRows;
    const int rows = (int)(n - row0 < (int64_t)kBcgRows ? n - row0 : (int64_t)kBcgRows);
    const unsigned char* stage = ring_smem + stg * RG::STAGE;
    const float (*As0)[kBS] = reinterpret_cast<const float (*)[kBS]>(stage);
    const float (*As1)[kBS] = reinterpret_cast<const float (*)[kBS]>(stage + kChunkBytes);
    if (MODE == 1 && rows == kBcgRows) {
      // a full chunk: the thread's 8 rows with their fmaf chains
      // interleaved (independent chains, each still over k = 0..63 in
      // order; measured faster for this mode only)
      const int rb = 8 * rg;
      float d[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) d[q] = 0.f;
      if (!skip_p) {
#pragma unroll
        for (int k = 0; k < kBS; k += 4) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 a0 = *reinterpret_cast<const float4*>(&As0[rb + q][k]);
            d[q] = fmaf(a0.x, cr[k], d[q]);
            d[q] = fmaf(a0.y, cr[k + 1], d[q]);
            d[q] = fmaf(a0.z, cr[k + 2], d[q]);
            d[q] = fmaf(a0.w, cr[k + 3], d[q]);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int r = rb + q;
        const float rv = As1[r][c];
        const float dv = __ldg(dinv + row0 + r);
        Y0[(size_t)(row0 + r) * kBS + c] = fmaf(rv, dv, d[q]);
      }
    } else
#pragma unroll 1
    for (int i8 = 0; i8 < 8; ++i8) {
      const int r = 8 * rg + i8;
      if (r >= rows) break;
      const size_t o = (size_t)(row0 + r) * kBS + c;
      float d0 = 0.f, d1 = 0.f;
      if (!skip_p) {
#pragma unroll
        for (int k = 0; k < kBS; k += 4) {
          const float4 a0 = *reinterpret_cast<const float4*>(&As0[r][k]);
          d0 = fmaf(a0.x, cr[k], d0);
          d0 = fmaf(a0.y, cr[k + 1], d0);
          d0 = fmaf(a0.z, cr[k + 2], d0);
          d0 = fmaf(a0.w, cr[k + 3], d0);
          if (MODE == 0) {
            const float4 a1 = *reinterpret_cast<const float4*>(&As1[r][k]);
            d1 = fmaf(a1.x, cr[k], d1);
            d1 = fmaf(a1.y, cr[k + 1], d1);
            d1 = fmaf(a1.z, cr[k + 2], d1);
            d1 = fmaf(a1.w, cr[k + 3], d1);
          }
        }
      }
      if (MODE == 0) {
        const float x = reinterpret_cast<const float*>(stage + 2 * kChunkBytes)[r * kBS + c];
        const float rv = reinterpret_cast<const float*>(stage + 3 * kChunkBytes)[r * kBS + c];
        Y0[o] = x + d0;
        const float rn = rv - d1;
        Y1[o] = rn;
        const double rd = (double)rn;
        switch (i8 >> 1) {
          case 0: nrm[0] = fma(rd, rd, nrm[0]); break;
          case 1: nrm[1] = fma(rd, rd, nrm[1]); break;
          case 2: nrm[2] = fma(rd, rd, nrm[2]); break;
          default: nrm[3] = fma(rd, rd, nrm[3]); break;
        }
      } else if (MODE == 1) {
        const float rv = As1[r][c];
        const float dv = __ldg(dinv + row0 + r);
        Y0[o] = fmaf(rv, dv, d0);
      } else {
        Y0[o] = d0;
      }
    }
    __syncthreads();  // the stage is read: it takes chunk i + S
    if (threadIdx.x == 0 && i + S < nmine)
      chunk_issue<NA>(src, blockIdx.x + (int64_t)(i + S) * gridDim.x, n, ring_smem + stg * RG::STAGE,
                      bar + stg);
  }
  if (MODE == 0) {
    // column sums of R^2 in a fixed order, in the ring's memory (every
    // chunk has been consumed)
    __syncthreads();
    double (*red)[kBS] = reinterpret_cast<double (*)[kBS]>(ring_smem);
#pragma unroll
    for (int j = 0; j < 4; ++j) red[4 * rg + j][c] = nrm[j];
    __syncthreads();
    if (threadIdx.x < kBS) {
      double s = 0.0;
      for (int q = 0; q < 16; ++q) s = s + red[q][threadIdx.x];
      partials[(size_t)blockIdx.x * kBS + threadIdx.x] = s;
    }
  }
}

// column norms ||R_j|| of the initial residual (r0) and, for the columns not
// active, R_j = 0 so the block leaves them alone
__global__ void __launch_bounds__(256) bcg_mask(int64_t n, float* R, const int* act) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n * kBS;
       e += (int64_t)gridDim.x * blockDim.x)
    if (!act[e % kBS]) R[e] = 0.f;
}

// The 64 x 64 algebra of one step, in FP64, one block of 256 threads.
// mode 0 (alpha): L = chol(active r x r block of P^T Q); L1 = L^-1 (kept for
//   mode 1); alpha = L1^T (L1 P^T R)
// mode 1 (beta): rn = sqrt(column sums) (convergence: done when every active
//   right-hand side has rn <= tol r0); beta = -L1^T (L1 Q^T D^-1 R)
// mode 2 (orth): pivoted Cholesky of W^T W -> rank and T (P = W T)
// mode 3 (norms of the initial residual into r0)
//
// Both factorisations run as one elimination of [G | I] in registers: 256
// threads hold 4 x 4 entries of each half (rows tr + 16 a, columns tc + 16 b of
// thread 16 tr + tc), and a step subtracts multiples of the pivot's row, passed
// round through shared memory, from the rows not yet eliminated; their column of
// the pivot is that row by symmetry. The left half ends as D L^T and the right
// one, its rows scaled by 1 / sqrt(d), as L^-1, with no substitution after it.
// One barrier a step, with pivoting too: every warp keeps the diagonal, which
// the pivot's row updates. A form
// that factorised in shared memory, entry by entry, and then substituted took 88
// us (mode 0), 25 us (mode 1) and 129 us (mode 2); this one 31, 15 and 42: the
// chain of a step (row, division, products, barrier) is 0.4 to 0.6 us.
//
// The kernel's whole shared state is one dynamic buffer laid out here (no
// static shared variables beside it): three 64 x 65 FP64 matrices, the pivot's
// row (two buffers), the pivots, then the step of each row.
constexpr size_t kBcgMatBytes = sizeof(double) * kBS * (kBS + 1);
constexpr size_t kBcgSmallSmem =
    3 * kBcgMatBytes + sizeof(double) * (4 * kBS + kBS) + sizeof(int) * kBS;

// this thread's entries of [G | I] (I: the first r rows)
struct BcgElim {
  double A[4][4], B[4][4];
  int tr, tc;
  __device__ __forceinline__ void load(const double* G, int r) {
    tr = threadIdx.x >> 4;
    tc = threadIdx.x & 15;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int i = tr + 16 * a, j = tc + 16 * b;
        A[a][b] = G[i * kBS + j];
        B[a][b] = i == j && i < r ? 1.0 : 0.0;
      }
  }
  // row p into R[0 .. 64) and R[64 .. 128)
  __device__ __forceinline__ void put(int p, double* R) const {
#pragma unroll
    for (int a = 0; a < 4; ++a)
      if (tr + 16 * a == p) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          R[tc + 16 * b] = A[a][b];
          R[kBS + tc + 16 * b] = B[a][b];
        }
      }
  }
  // the rows of `rest` lose their multiple of row R: row groups A0 .. 3, of the
  // left half the columns of the same groups and of the right one those of
  // groups 0 .. B1
  template <int A0, int B1>
  __device__ __forceinline__ void sub(const double* R, double inv, unsigned long long rest) {
    double ra[4], rb[4];
#pragma unroll
    for (int b = A0; b < 4; ++b) ra[b] = R[tc + 16 * b];
#pragma unroll
    for (int b = 0; b <= B1; ++b) rb[b] = R[kBS + tc + 16 * b];
    rest >>= tr;
#pragma unroll
    for (int a = A0; a < 4; ++a) {
      const double m = (rest >> (16 * a)) & 1ull ? -(R[tr + 16 * a] * inv) : 0.0;
      if (m == 0.0) continue;
#pragma unroll
      for (int b = A0; b < 4; ++b) A[a][b] = fma(m, ra[b], A[a][b]);
#pragma unroll
      for (int b = 0; b <= B1; ++b) B[a][b] = fma(m, rb[b], B[a][b]);
    }
  }
  // steps 16 KA .. of the unpivoted elimination; false when a pivot is not positive
  template <int KA>
  __device__ __forceinline__ bool steps(int r, unsigned long long upto, double* row, double* piv) {
    for (int k = 16 * KA; k < min(r, 16 * KA + 16); ++k) {
      double* R = row + (k & 1) * 2 * kBS;
      if (tr == k - 16 * KA) {
#pragma unroll
        for (int b = KA; b < 4; ++b) R[tc + 16 * b] = A[KA][b];
#pragma unroll
        for (int b = 0; b <= KA; ++b) R[kBS + tc + 16 * b] = B[KA][b];
      }
      __syncthreads();
      const double d = R[k];
      if (!(d > 0.0)) return false;  // every thread reads the same d
      if (threadIdx.x == 0) piv[k] = d;
      sub<KA, KA>(R, 1.0 / d, k == 63 ? 0ull : upto & (~0ull << (k + 1)));
    }
    return true;
  }
};

// Out = op(A) B for 64 x 64 operands, op(A) = A or A^T; each thread the 4 x 4
// entries (tr + 16 x, tc + 16 y), so that the 16 threads of a row read 16
// neighbouring columns of B; k in increasing order
template <bool TRANS>
__device__ __forceinline__ void small_mm(const double (*A)[kBS + 1], const double (*B)[kBS + 1],
                                         double (*Out)[kBS + 1], double scale) {
  const int tr = threadIdx.x / 16, tc = threadIdx.x % 16;
  double acc[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) acc[x][y] = 0.0;
#pragma unroll 4
  for (int k = 0; k < kBS; ++k) {
    double a[4], bv[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) a[x] = TRANS ? A[k][tr + 16 * x] : A[tr + 16 * x][k];
#pragma unroll
    for (int y = 0; y < 4; ++y) bv[y] = B[k][tc + 16 * y];
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) acc[x][y] = fma(a[x], bv[y], acc[x][y]);
  }
  __syncthreads();  // Out may alias B
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) Out[tr + 16 * x][tc + 16 * y] = scale * acc[x][y];
  __syncthreads();
}

__global__ void __launch_bounds__(256) bcg_small(int mode, BcgSmall* st, double tol) {
  extern __shared__ __align__(16) unsigned char bcg_dyn[];
  double (*M)[kBS + 1] = reinterpret_cast<double (*)[kBS + 1]>(bcg_dyn);
  double (*Bm)[kBS + 1] = reinterpret_cast<double (*)[kBS + 1]>(bcg_dyn + kBcgMatBytes);
  double (*Y)[kBS + 1] = reinterpret_cast<double (*)[kBS + 1]>(bcg_dyn + 2 * kBcgMatBytes);
  double* row = reinterpret_cast<double*>(bcg_dyn + 3 * kBcgMatBytes);  // [2][2 kBS]
  double* piv = row + 4 * kBS;
  int* pos = reinterpret_cast<int*>(piv + kBS);
  const int t = threadIdx.x;
  if (st->done) return;
  if (mode == 3) {
    // the column sums of R^2 were reduced into rn
    if (t < kBS) {
      st->r0[t] = sqrt(st->rn[t]);
      st->rn[t] = st->r0[t];
    }
    return;
  }
  if (mode == 0 || mode == 1) {
    const int r = st->rank;
    if (mode == 0) {
      // elimination of the r x r active block of P^T Q
      BcgElim e;
      e.load(st->C, r);
      const unsigned long long upto = r == 64 ? ~0ull : (1ull << r) - 1ull;
      const bool stop = !(e.steps<0>(r, upto, row, piv) && e.steps<1>(r, upto, row, piv) &&
                          e.steps<2>(r, upto, row, piv) && e.steps<3>(r, upto, row, piv));
      if (stop) {
        if (t == 0) { st->fail = 1; st->done = 1; }
        return;
      }
      __syncthreads();
      // L1 = L^-1, kept for mode 1; rows and columns past r are zero
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int i = e.tr + 16 * a;
        const double sc = i < r ? 1.0 / sqrt(piv[i]) : 0.0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const double v = i < r ? e.B[a][b] * sc : 0.0;
          Bm[i][e.tc + 16 * b] = v;
          st->L1[i * kBS + e.tc + 16 * b] = v;
        }
      }
      // right-hand sides: P^T R; rows past r do not take part
      for (int q = t; q < kBS * kBS; q += blockDim.x)
        M[q / kBS][q % kBS] = q / kBS < r ? st->C[kBS * kBS + q] : 0.0;
    } else {
      int over = 0;
      if (t < kBS) {
        const double rn = sqrt(st->rn[t]);
        st->rn[t] = rn;
        over = st->active[t] && rn > tol * st->r0[t];
      }
      const int go_on = __syncthreads_or(over);
      if (t == 0) {
        st->iters += 1;
        if (!go_on) st->done = 1;
      }
      if (!go_on) return;
      for (int q = t; q < kBS * kBS; q += blockDim.x) {
        Bm[q / kBS][q % kBS] = st->L1[q];
        M[q / kBS][q % kBS] = q / kBS < r ? st->E[q] : 0.0;
      }
    }
    __syncthreads();
    // Y = L1 B, then the coefficients L1^T Y (negated for beta)
    small_mm<false>(Bm, M, Y, 1.0);
    small_mm<true>(Bm, Y, Y, mode == 0 ? 1.0 : -1.0);
    for (int q = t; q < kBS * kBS; q += blockDim.x) st->coef[q] = (float)Y[q / kBS][q % kBS];
    return;
  }
  // mode 2: pivoted elimination of G = W^T W, stopping at pivots below kBcgDrop
  // times the first. Nothing is swapped: `rest` are the rows left and pos[i] the
  // step that took row i. The pivot is the largest diagonal entry left to 14
  // bits (the first of those that agree): its leading bits and its row make one
  // 32-bit key for the warp's maximum. A row whose entry is not positive is none.
  BcgElim e;
  e.load(st->G, kBS);
  const int lane = t & 31;
  double dg[2] = {st->G[lane * (kBS + 1)], st->G[(lane + 32) * (kBS + 1)]};
  unsigned long long rest = ~0ull;
  int r = 0;
  double dmax = 0.0;
  for (int k = 0; k < kBS; ++k) {
    unsigned key = 0u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = lane + 32 * h;
      if (((rest >> i) & 1ull) && dg[h] > 0.0)
        key = max(key, ((unsigned)__double2hiint(dg[h]) & ~63u) | (unsigned)(63 - i));
    }
    key = __reduce_max_sync(0xffffffffu, key);
    if (key < 64u) break;  // (the same in every thread, as below)
    const int p = 63 - (int)(key & 63u);
    const double d = __shfl_sync(0xffffffffu, p < 32 ? dg[0] : dg[1], p & 31);
    if (k == 0) dmax = d;
    if (!(d > kBcgDrop * dmax)) break;
    double* R = row + (k & 1) * 2 * kBS;
    e.put(p, R);
    if (t == 0) {
      piv[k] = d;
      pos[p] = k;
    }
    rest &= ~(1ull << p);
    r = k + 1;
    const double inv = 1.0 / d;
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double x = R[lane + 32 * h];
      dg[h] = fma(-(x * inv), x, dg[h]);
    }
    e.sub<0, 3>(R, inv, rest);
  }
  for (int q = t; q < kBS * kBS; q += blockDim.x) st->coef[q] = 0.f;
  __syncthreads();
  // T(c, j) = L^-1(j, c), the step of a row naming its column of T
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int i = e.tr + 16 * a;
    if ((rest >> i) & 1ull) continue;
    const int j = pos[i];
    const double sc = 1.0 / sqrt(piv[j]);
#pragma unroll
    for (int b = 0; b < 4; ++b) st->coef[(e.tc + 16 * b) * kBS + j] = (float)(e.B[a][b] * sc);
  }
  if (t == 0) {
    st->rank = r;
    if (r == 0) st->done = 1;
  }
}

}  // namespace

struct lfx_mrhs {
  lfx_ctx* ctx = nullptr;
  int32_t nrhs = 64, nl = 0, ncell_2d = 0;
  int64_t undf = 0;
  int32_t npatch = 0, own_max = 0, max_colours = 0;
  int64_t nent = 0;
  StencilArgs st{};     // column stencils (device arrays owned here)
  size_t base_b = 0, off_b = 0, nbr_b = 0, coef_b = 0;
  // solve work space, allocated by the first solve
  float *x32 = nullptr, *r32 = nullptr, *p32 = nullptr, *q32 = nullptr, *dinv = nullptr;
  double* R64 = nullptr;
  double* nrm = nullptr;      // [nrhs] device
  double* h_nrm = nullptr;    // [nrhs] pinned
  int* d_act = nullptr;       // [nrhs]
  MvState* S = nullptr;
  MvState* h_S = nullptr;     // pinned
  double* partials = nullptr;  // block sums, npart doubles
  int grid = 0;
  int64_t npart = 0;
  // block CG: W, the small algebra state and the Gram partials
  float* w32 = nullptr;
  BcgSmall* bcg = nullptr;
  BcgSmall* h_bcg = nullptr;  // pinned
  double* bpart = nullptr;
  int bgrid = 0;
  int gram_tc = 0;  // block CG Gram products on the tcgen05 tensor cores (1) or the FP32 cores (0)
};

namespace {

// blocks of the apply: patches of columns, and the groups of LB rows split
// over blockIdx.y where the columns alone do not give about four waves
dim3 apply_grid(const lfx_mrhs* m) {
  const int gpb = 1024 / m->nrhs;
  const int gx = (m->st.ncol + gpb - 1) / gpb, nb = (m->nl + 1 + LB - 1) / LB;
  const int want = (12 * m->ctx->num_sms + gx - 1) / gx;
  return dim3((unsigned)gx, (unsigned)std::max(1, std::min(nb, want)));
}

template <int RB>
void launch_t(lfx_mrhs* m, const float* x, float* y, double* part) {
  const dim3 g = apply_grid(m);
  if (part)
    mrhs_apply_k<RB, true><<<g, 256, 0, m->ctx->stream>>>(m->st, x, y, part);
  else
    mrhs_apply_k<RB, false><<<g, 256, 0, m->ctx->stream>>>(m->st, x, y, nullptr);
}

// y = A x; with part the block sums of <x, y> too (one per block of apply_grid)
int mrhs_launch(lfx_mrhs* m, const float* x, float* y, double* part = nullptr) {
  lfx_ctx* ctx = m->ctx;
  switch (m->nrhs) {
    case 16: launch_t<1>(m, x, y, part); break;
    case 32: launch_t<2>(m, x, y, part); break;
    default: launch_t<4>(m, x, y, part); break;
  }
  ctx->launches++;
  LFX_CK(ctx, cudaGetLastError());
  return LFX_OK;
}

void mrhs_free(lfx_mrhs* m) {
  lfx_ctx* ctx = m->ctx;
  dfree(ctx, (void*)m->st.base, m->base_b);
  dfree(ctx, (void*)m->st.off, m->off_b);
  dfree(ctx, (void*)m->st.nbr, m->nbr_b);
  dfree(ctx, m->st.coef, m->coef_b);
  const size_t v32 = (size_t)m->undf * m->nrhs * 4;
  dfree(ctx, m->x32, v32);
  dfree(ctx, m->r32, v32);
  dfree(ctx, m->p32, v32);
  dfree(ctx, m->q32, v32);
  dfree(ctx, m->dinv, (size_t)m->undf * 4);
  dfree(ctx, m->R64, (size_t)m->undf * m->nrhs * 8);
  dfree(ctx, m->nrm, sizeof(double) * 64);
  dfree(ctx, m->d_act, sizeof(int) * 64);
  dfree(ctx, m->S, sizeof(MvState));
  dfree(ctx, m->partials, sizeof(double) * m->npart);
  if (m->h_nrm) cudaFreeHost(m->h_nrm);
  if (m->h_S) cudaFreeHost(m->h_S);
  dfree(ctx, m->w32, v32);
  dfree(ctx, m->bcg, sizeof(BcgSmall));
  dfree(ctx, m->bpart, sizeof(double) * 2 * kBS * kBS * m->bgrid);
  if (m->h_bcg) cudaFreeHost(m->h_bcg);
}

}  // namespace

int lfx_mrhs_create(const lfx_op* op, int32_t kind, int32_t nrhs, int32_t cells_per_patch,
                    lfx_mrhs** out) {
  if (!op || !out) return LFX_INVALID_ARGUMENT;
  *out = nullptr;
  lfx_ctx* ctx = op->ctx;
  const lfx_lma_layout* L = op->lay;
  if (kind != LFX_MRHS_TF32 && kind != LFX_MRHS_BF16)
    return fail(ctx, LFX_INVALID_ARGUMENT, "kind must be LFX_MRHS_TF32 or LFX_MRHS_BF16");
  if (nrhs != 16 && nrhs != 32 && nrhs != 64)
    return fail(ctx, LFX_INVALID_ARGUMENT, "nrhs must be 16, 32 or 64");
  if (cells_per_patch < 0 || cells_per_patch > 256)
    return fail(ctx, LFX_INVALID_ARGUMENT, "cells_per_patch must be in [0, 256]");
  const int P = cells_per_patch ? cells_per_patch : kDefaultPatch;
  if (L->ndf_to != 8 || L->ndf_from != 8 || L->undf_to != L->undf_from)
    return fail(ctx, LFX_NOT_SUPPORTED, "multi-RHS apply needs a square ndf = 8 (W0) operator");
  const int nc = L->ncell_2d, nl = L->nlayers;
  std::vector<int32_t> mt((size_t)nc * 8), mf((size_t)nc * 8);
  LFX_CK(ctx, cudaMemcpy(mt.data(), L->map_to, mt.size() * 4, cudaMemcpyDeviceToHost));
  LFX_CK(ctx, cudaMemcpy(mf.data(), L->map_from, mf.size() * 4, cudaMemcpyDeviceToHost));
  if (mt != mf) return fail(ctx, LFX_NOT_SUPPORTED, "multi-RHS apply needs map_to == map_from");
  // vertex columns
  std::unordered_map<int32_t, int32_t> vid;
  std::vector<int32_t> vbase;
  std::vector<int32_t> cv((size_t)nc * 4);
  for (int c = 0; c < nc; ++c)
    for (int v = 0; v < 4; ++v) {
      const int32_t b = mt[(size_t)c * 8 + v];
      if (mt[(size_t)c * 8 + 4 + v] != b + 1)
        return fail(ctx, LFX_NOT_SUPPORTED,
                    "multi-RHS apply needs W0 dofs: top vertex dof = bottom dof + 1");
      if (b < 0 || (int64_t)b + nl >= L->undf_to)
        return fail(ctx, LFX_INVALID_ARGUMENT, "dofmap entry out of range");
      auto it = vid.find(b);
      int id;
      if (it == vid.end()) {
        id = (int)vbase.size();
        vid.emplace(b, id);
        vbase.push_back(b);
      } else {
        id = it->second;
      }
      cv[(size_t)c * 4 + v] = id;
    }
  const int nv = (int)vbase.size();
  if ((int64_t)nv * (nl + 1) != L->undf_to)
    return fail(ctx, LFX_NOT_SUPPORTED, "multi-RHS apply needs every dof on a vertex column");
  std::vector<int32_t> voff(nv + 1, 0), vcells;
  for (int c = 0; c < nc; ++c)
    for (int v = 0; v < 4; ++v) voff[cv[(size_t)c * 4 + v] + 1]++;
  for (int i = 0; i < nv; ++i) voff[i + 1] += voff[i];
  vcells.resize(voff[nv]);
  {
    std::vector<int32_t> fill(voff.begin(), voff.end() - 1);
    for (int c = 0; c < nc; ++c)
      for (int v = 0; v < 4; ++v) vcells[fill[cv[(size_t)c * 4 + v]]++] = c;
  }
  // compact patches: breadth-first over cells sharing a vertex (their colours, which
  // the gather does without, are what lfx_mrhs_info reports)
  std::vector<int32_t> patch(nc, -1);
  int npatch = 0;
  {
    std::vector<int32_t> queue;
    for (int s = 0; s < nc; ++s) {
      if (patch[s] >= 0) continue;
      queue.clear();
      queue.push_back(s);
      patch[s] = npatch;
      int taken = 1;
      for (size_t h = 0; h < queue.size() && taken < P; ++h) {
        const int c = queue[h];
        for (int v = 0; v < 4 && taken < P; ++v) {
          const int id = cv[(size_t)c * 4 + v];
          for (int k = voff[id]; k < voff[id + 1] && taken < P; ++k) {
            const int n2 = vcells[k];
            if (patch[n2] < 0) {
              patch[n2] = npatch;
              queue.push_back(n2);
              ++taken;
            }
          }
        }
      }
      ++npatch;
    }
  }
  // owner of a vertex column: the patch holding most of its cells (ties: the
  // patch of its lowest cell)
  std::vector<int32_t> owner(nv);
  for (int i = 0; i < nv; ++i) {
    int best = -1, bestn = 0;
    for (int k = voff[i]; k < voff[i + 1]; ++k) {
      const int pk = patch[vcells[k]];
      int n = 0;
      for (int k2 = voff[i]; k2 < voff[i + 1]; ++k2) n += patch[vcells[k2]] == pk;
      if (n > bestn || (n == bestn && pk < best)) {
        best = pk;
        bestn = n;
      }
    }
    owner[i] = best;
  }
  std::vector<std::vector<int32_t>> pown(npatch);
  for (int i = 0; i < nv; ++i) pown[owner[i]].push_back(i);
  std::vector<int> h_own;  // vertex columns patch by patch
  int64_t nent = 0;
  int own_max = 0, max_col = 0;
  std::vector<int32_t> slot_of(nv, -1);
  for (int p = 0; p < npatch; ++p) {
    const auto& ov = pown[p];
    if (ov.size() > 254) return fail(ctx, LFX_NOT_SUPPORTED, "patch owns too many vertex columns");
    for (size_t s = 0; s < ov.size(); ++s) slot_of[ov[s]] = (int)s;
    std::vector<int32_t> need;
    for (int id : ov)
      for (int k = voff[id]; k < voff[id + 1]; ++k) need.push_back(vcells[k]);
    std::sort(need.begin(), need.end());
    need.erase(std::unique(need.begin(), need.end()), need.end());
    // greedy colours: cells sharing an owned vertex differ
    std::vector<uint32_t> used(ov.size(), 0u);
    int ncol = 0;
    for (size_t i = 0; i < need.size(); ++i) {
      uint32_t forbid = 0u;
      for (int v = 0; v < 4; ++v) {
        const int s = slot_of[cv[(size_t)need[i] * 4 + v]];
        if (s >= 0) forbid |= used[s];
      }
      int col = 0;
      while (forbid & (1u << col)) ++col;
      if (col >= kMaxPC) return fail(ctx, LFX_NOT_SUPPORTED, "patch needs too many colours");
      ncol = std::max(ncol, col + 1);
      for (int v = 0; v < 4; ++v) {
        const int s = slot_of[cv[(size_t)need[i] * 4 + v]];
        if (s >= 0) used[s] |= 1u << col;
      }
    }
    nent += (int64_t)need.size();
    h_own.insert(h_own.end(), ov.begin(), ov.end());
    for (int id : ov) slot_of[id] = -1;
    own_max = std::max(own_max, (int)ov.size());
    max_col = std::max(max_col, ncol);
  }

  auto* m = new lfx_mrhs();
  m->ctx = ctx;
  m->nrhs = nrhs;
  m->nl = nl;
  m->ncell_2d = nc;
  m->undf = L->undf_to;
  m->npatch = npatch;
  m->own_max = own_max;
  m->max_colours = max_col;
  m->nent = nent;
  int rc = LFX_OK;
  // the columns each column couples to: those sharing a cell, in the order they
  // are met, then the column itself; and the cells around it
  std::vector<int> h_base, h_off{0}, h_nbr, h_coff{0};
  std::vector<int4> h_ccell;
  h_nbr.reserve((size_t)nv * 9);
  h_ccell.reserve(vcells.size());
  int32_t near[kMaxSlot];
  for (int id : h_own) {
    int nn = 0;
    const size_t e0 = h_ccell.size();
    for (int k = voff[id]; k < voff[id + 1]; ++k) {
      const int c = vcells[k];
      // (a cell that holds the column at two of its vertices is listed once
      // for each)
      int seen = 0;
      for (int k2 = voff[id]; k2 < k; ++k2) seen += vcells[k2] == c;
      unsigned slots = 0u;
      int mine = -1;
      for (int v = 0; v < 4; ++v) {
        const int32_t u = cv[(size_t)c * 4 + v];
        int t = 255;  // the column itself: its slot is known at the end
        if (u != id) {
          for (t = 0; t < nn && near[t] != u; ++t) {
          }
          if (t == kMaxSlot - 1) {
            rc = fail(ctx, LFX_NOT_SUPPORTED, "a vertex column has too many neighbours");
            t = 0;
          } else if (t == nn) {
            near[nn++] = u;
          }
        } else if (seen-- == 0) {
          mine = v;
        }
        slots |= (unsigned)t << (8 * v);
      }
      h_ccell.push_back(make_int4(c, mine, (int)slots, 0));
    }
    for (size_t e = e0; e < h_ccell.size(); ++e)
      for (int v = 0; v < 4; ++v)
        if ((((unsigned)h_ccell[e].z >> (8 * v)) & 255u) == 255u)
          h_ccell[e].z = (int)(((unsigned)h_ccell[e].z & ~(255u << (8 * v))) | ((unsigned)nn << (8 * v)));
    h_base.push_back(vbase[id]);
    for (int t = 0; t < nn; ++t) h_nbr.push_back(vbase[near[t]]);
    h_nbr.push_back(vbase[id]);
    h_off.push_back((int)h_nbr.size());
    h_coff.push_back((int)h_ccell.size());
  }
  auto up = [&](void** dst, size_t* held, const void* src, size_t bytes) {
    if (rc) return;
    rc = dmalloc(ctx, dst, bytes);
    if (!rc) *held = bytes;
    if (!rc && cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice) != cudaSuccess)
      rc = fail(ctx, LFX_CUDA_ERROR, "upload of the patch tables failed");
  };
  StencilArgs& st = m->st;
  st.ncol = (int)h_base.size();
  st.h = nl + 1;
  st.g4 = (nl + 1 + 3) / 4;
  int *coff = nullptr, *ccell = nullptr;
  size_t coff_b = 0, ccell_b = 0;
  up((void**)&st.base, &m->base_b, h_base.data(), h_base.size() * sizeof(int));
  up((void**)&st.off, &m->off_b, h_off.data(), h_off.size() * sizeof(int));
  up((void**)&st.nbr, &m->nbr_b, h_nbr.data(), h_nbr.size() * sizeof(int));
  up((void**)&coff, &coff_b, h_coff.data(), h_coff.size() * sizeof(int));
  up((void**)&ccell, &ccell_b, h_ccell.data(), h_ccell.size() * sizeof(int4));
  const size_t cbytes = h_nbr.size() * st.g4 * 12 * sizeof(float);
  if (!rc) rc = dmalloc(ctx, (void**)&st.coef, cbytes);
  if (!rc) {
    m->coef_b = cbytes;
    cudaMemsetAsync(st.coef, 0, cbytes, ctx->stream);
    const int blocks = (int)(((int64_t)st.ncol * st.h + 127) / 128);
    const int4* cc = reinterpret_cast<const int4*>(ccell);
    if (op->precision == LFX_R64)
      mrhs_assemble<double><<<blocks, 128, 0, ctx->stream>>>(st, coff, cc, (const double*)op->mat, nl, op->blk);
    else
      mrhs_assemble<float><<<blocks, 128, 0, ctx->stream>>>(st, coff, cc, (const float*)op->mat, nl, op->blk);
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(ctx->stream) != cudaSuccess)
      rc = fail(ctx, LFX_CUDA_ERROR, "stencil assembly failed");
  }
  dfree(ctx, coff, coff_b);
  dfree(ctx, ccell, ccell_b);
  if (rc) {
    mrhs_free(m);
    delete m;
    return rc;
  }
  *out = m;
  return LFX_OK;
}

int lfx_mrhs_destroy(lfx_mrhs* m) {
  if (!m) return LFX_OK;
  mrhs_free(m);
  delete m;
  return LFX_OK;
}

int lfx_mrhs_info(const lfx_mrhs* m, int32_t* npatch, int64_t* cell_entries, int32_t* max_owned,
                  int32_t* max_colours, int64_t* matrix_bytes) {
  if (!m) return LFX_INVALID_ARGUMENT;
  if (npatch) *npatch = m->npatch;
  if (cell_entries) *cell_entries = m->nent * m->nl;
  if (max_owned) *max_owned = m->own_max;
  if (max_colours) *max_colours = m->max_colours;
  if (matrix_bytes) *matrix_bytes = (int64_t)m->coef_b;
  return LFX_OK;
}

// The kernels read and write 16 bytes a lane. With 16 right-hand sides x may
// start on any multiple of 8 bytes: such an x is copied first.
int lfx_mrhs_apply(lfx_mrhs* m, const float* x, float* y) {
  if (!m || !x || !y || x == y) return LFX_INVALID_ARGUMENT;
  if (((uintptr_t)y & 15) || ((uintptr_t)x & (m->nrhs == 16 ? 7 : 15)))
    return fail(m->ctx, LFX_INVALID_ARGUMENT, "x and y must be 16-byte aligned");
  if (((uintptr_t)x & 15) == 0) return mrhs_launch(m, x, y);
  lfx_ctx* ctx = m->ctx;
  const size_t bytes = (size_t)m->undf * m->nrhs * sizeof(float);
  float* t = nullptr;
  LFX_CK(ctx, cudaMallocAsync((void**)&t, bytes, ctx->stream));
  int rc = cudaMemcpyAsync(t, x, bytes, cudaMemcpyDeviceToDevice, ctx->stream) == cudaSuccess
               ? mrhs_launch(m, t, y)
               : fail(ctx, LFX_CUDA_ERROR, "copy of x failed");
  cudaFreeAsync(t, ctx->stream);
  return rc;
}

int lfx_mrhs_time_apply(lfx_mrhs* m, const float* x, float* y, int32_t reps, float* us) {
  if (!m || !x || !y || x == y || reps < 1 || !us) return LFX_INVALID_ARGUMENT;
  lfx_ctx* ctx = m->ctx;
  int rc = lfx_mrhs_apply(m, x, y);  // warm
  if (rc) return rc;
  cudaEvent_t e0, e1;
  LFX_CK(ctx, cudaEventCreate(&e0));
  LFX_CK(ctx, cudaEventCreate(&e1));
  cudaEventRecord(e0, ctx->stream);
  for (int r = 0; r < reps && !rc; ++r) rc = lfx_mrhs_apply(m, x, y);
  cudaEventRecord(e1, ctx->stream);
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess && !rc)
    rc = fail(ctx, LFX_CUDA_ERROR, "multi-RHS apply timing failed");
  float ms = 0.f;
  if (!rc) cudaEventElapsedTime(&ms, e0, e1);
  *us = 1e3f * ms / reps;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return rc;
}

// The apply has one launch shape: reps applies are timed and its rows per
// pass reported.
int lfx_mrhs_autotune(lfx_mrhs* m, int32_t reps, int32_t* lb, float* us) {
  if (!m || reps < 1) return LFX_INVALID_ARGUMENT;
  lfx_ctx* ctx = m->ctx;
  const size_t bytes = (size_t)m->undf * m->nrhs * sizeof(float);
  float *x = nullptr, *y = nullptr, t = 0.f;
  int rc = dmalloc(ctx, (void**)&x, bytes);
  if (!rc) rc = dmalloc(ctx, (void**)&y, bytes);
  if (!rc && cudaMemsetAsync(x, 0, bytes, ctx->stream) != cudaSuccess)
    rc = fail(ctx, LFX_CUDA_ERROR, "multi-RHS apply timing failed");
  if (!rc) rc = lfx_mrhs_time_apply(m, x, y, reps, &t);
  dfree(ctx, x, bytes);
  dfree(ctx, y, bytes);
  if (rc) return rc;
  if (lb) *lb = LB;
  if (us) *us = t;
  return LFX_OK;
}

namespace {

int ensure_work(lfx_mrhs* m) {
  if (m->x32) return LFX_OK;
  lfx_ctx* ctx = m->ctx;
  const size_t v32 = (size_t)m->undf * m->nrhs * 4;
  m->grid = ctx->num_sms * 4;
  int rc = dmalloc(ctx, (void**)&m->x32, v32);
  if (!rc) rc = dmalloc(ctx, (void**)&m->r32, v32);
  if (!rc) rc = dmalloc(ctx, (void**)&m->p32, v32);
  if (!rc) rc = dmalloc(ctx, (void**)&m->q32, v32);
  if (!rc) rc = dmalloc(ctx, (void**)&m->dinv, (size_t)m->undf * 4);
  if (!rc) rc = dmalloc(ctx, (void**)&m->R64, (size_t)m->undf * m->nrhs * 8);
  if (!rc) rc = dmalloc(ctx, (void**)&m->nrm, sizeof(double) * 64);
  if (!rc) rc = dmalloc(ctx, (void**)&m->d_act, sizeof(int) * 64);
  if (!rc) rc = dmalloc(ctx, (void**)&m->S, sizeof(MvState));
  {
    // two sums a block of the vector kernels, one a block of the apply
    const dim3 g = apply_grid(m);
    m->npart = (int64_t)m->nrhs * std::max((int64_t)2 * m->grid, (int64_t)g.x * g.y);
  }
  if (!rc) rc = dmalloc(ctx, (void**)&m->partials, sizeof(double) * m->npart);
  if (!rc && cudaMallocHost(&m->h_nrm, sizeof(double) * 64) != cudaSuccess)
    rc = fail(ctx, LFX_OUT_OF_MEMORY, "pinned allocation failed");
  if (!rc && cudaMallocHost(&m->h_S, sizeof(MvState)) != cudaSuccess)
    rc = fail(ctx, LFX_OUT_OF_MEMORY, "pinned allocation failed");
  if (!rc) LFX_CK(ctx, cudaMemsetAsync(m->S, 0, sizeof(MvState), ctx->stream));
  return rc;
}

// R = B - A64 X per right-hand side, and ||R|| into m->h_nrm
int outer_residual(lfx_mrhs* m, lfx_op* op64, const double* b, double* x, int64_t ld) {
  lfx_ctx* ctx = m->ctx;
  const int64_t n = m->undf;
  for (int r = 0; r < m->nrhs; ++r) {
    int rc = op_apply_impl(op64, x + (size_t)r * ld, m->R64 + (size_t)r * n, b + (size_t)r * ld,
                           nullptr);
    if (rc) return rc;
    const double* R = m->R64 + (size_t)r * n;
    double* out = m->nrm + r;
    rc = launch_chunks<1>(
        ctx, n, [=] __device__(int64_t i) { return V1<double>{R[i]}; },
        [=] __device__(int64_t, const V1<double>& v, double* acc) {
          acc[0] = fma(v.a, v.a, acc[0]);
        },
        [=] __device__(const double* tot) { *out = sqrt(tot[0]); });
    if (rc) return rc;
  }
  LFX_CK(ctx, cudaMemcpyAsync(m->h_nrm, m->nrm, sizeof(double) * m->nrhs, cudaMemcpyDeviceToHost,
                              ctx->stream));
  LFX_CK(ctx, cudaStreamSynchronize(ctx->stream));
  return LFX_OK;
}

template <int NR>
int inner_solve(lfx_mrhs* m, const int* act, double tol, int max_inner, int* inner_its) {
  lfx_ctx* ctx = m->ctx;
  const int64_t n = m->undf;
  const int G = m->grid;
  const dim3 tb(32, 8), tg((unsigned)((n + 31) / 32), NR < 32 ? 1 : NR / 32);
  mv_from_rhs_major<NR><<<tg, tb, 0, ctx->stream>>>(n, m->R64, n, m->r32);
  LFX_CK(ctx, cudaMemcpyAsync(m->d_act, act, sizeof(int) * NR, cudaMemcpyHostToDevice, ctx->stream));
  LFX_CK(ctx, cudaMemsetAsync(&m->S->nactive, 0, sizeof(int), ctx->stream));
  mv_init<NR><<<G, 256, 0, ctx->stream>>>(n, m->dinv, m->r32, m->p32, m->x32, m->partials);
  mv_fin<NR><<<NR, 128, 0, ctx->stream>>>(0, G, m->partials, m->d_act, tol, m->S);
  ctx->launches += 3;
  LFX_CK(ctx, cudaGetLastError());
  const dim3 ga = apply_grid(m);
  int it = 0;
  constexpr int kCheck = 8;
  while (it < max_inner) {
    const int nb = std::min(kCheck, max_inner - it);
    for (int s = 0; s < nb; ++s) {
      int rc = mrhs_launch(m, m->p32, m->q32, m->partials);
      if (rc) return rc;
      mv_fin<NR><<<NR, 128, 0, ctx->stream>>>(1, (int)(ga.x * ga.y), m->partials, nullptr, tol, m->S);
      mv_residual<NR><<<G, 256, 0, ctx->stream>>>(n, m->dinv, m->q32, m->r32, m->S, m->partials);
      mv_fin<NR><<<NR, 128, 0, ctx->stream>>>(2, G, m->partials, nullptr, tol, m->S);
      mv_direction<NR><<<G, 256, 0, ctx->stream>>>(n, m->dinv, m->r32, m->p32, m->x32, m->S);
      ctx->launches += 4;
    }
    LFX_CK(ctx, cudaGetLastError());
    it += nb;
    LFX_CK(ctx, cudaMemcpyAsync(&m->h_S->nactive, &m->S->nactive, sizeof(int),
                                cudaMemcpyDeviceToHost, ctx->stream));
    LFX_CK(ctx, cudaStreamSynchronize(ctx->stream));
    if (m->h_S->nactive == 0) break;
  }
  *inner_its = it;
  return LFX_OK;
}

// partials of U^T [V0 (V1)] (rows of V scaled by vscale when given) on the
// tensor cores or the FP32 cores, then the fixed-order reduction into out
template <int NV>
int gram(lfx_mrhs* m, const float* U, const float* V0, const float* V1, const float* vscale,
         BcgSmall* st, double* out) {
  lfx_ctx* ctx = m->ctx;
  const int64_t n = m->undf;
  if (m->gram_tc) {
    LFX_CK(ctx, ctx->kernels.allow_smem((const void*)bcg_gram_tc<NV>, tc_gram_smem<NV>()));
    bcg_gram_tc<NV><<<m->bgrid, kTcThreads, tc_gram_smem<NV>(), ctx->stream>>>(n, U, V0, V1,
                                                                               vscale, m->bpart, st);
  } else {
    constexpr size_t smem = ChunkRing<1 + NV, 4>::BYTES;
    LFX_CK(ctx, ctx->kernels.allow_smem((const void*)bcg_gram_s<NV>, smem));
    bcg_gram_s<NV><<<m->bgrid, 256, smem, ctx->stream>>>(n, U, V0, V1, vscale, m->bpart, st);
  }
  const int ne = NV * kBS * kBS;
  bcg_reduce<<<(ne + 31) / 32, 256, 0, ctx->stream>>>(m->bgrid, ne, m->bpart, out, st);
  ctx->launches += 2;
  LFX_CK(ctx, cudaGetLastError());
  return LFX_OK;
}

int ensure_bcg(lfx_mrhs* m) {
  if (m->bcg) return LFX_OK;
  lfx_ctx* ctx = m->ctx;
  LFX_CK(ctx, ctx->kernels.allow_smem((const void*)bcg_small, kBcgSmallSmem));
  m->bgrid = ctx->num_sms * 2;
  int rc = dmalloc(ctx, (void**)&m->w32, (size_t)m->undf * m->nrhs * 4);
  if (!rc) rc = dmalloc(ctx, (void**)&m->bcg, sizeof(BcgSmall));
  if (!rc) rc = dmalloc(ctx, (void**)&m->bpart, sizeof(double) * 2 * kBS * kBS * m->bgrid);
  if (!rc && cudaMallocHost((void**)&m->h_bcg, sizeof(BcgSmall)) != cudaSuccess)
    rc = fail(ctx, LFX_OUT_OF_MEMORY, "pinned allocation failed");
  return rc;
}

// the streamed update kernel of a mode with its shared memory set: returns a
// callable taking the kernel's arguments
template <int MODE>
auto upd_launch(lfx_ctx* ctx, int G) {
  using RG = ChunkRing<UpdOps<MODE>::NA, UpdOps<MODE>::S>;
  ctx->kernels.allow_smem((const void*)bcg_update_s<MODE>, RG::BYTES);
  return [ctx, G](int64_t n, const float* A0, const float* A1, float* Y0, float* Y1,
                  const float* dinv, const BcgSmall* st, int skip_p, double* partials) {
    bcg_update_s<MODE><<<G, 256, RG::BYTES, ctx->stream>>>(n, A0, A1, Y0, Y1, dinv, st, skip_p,
                                                            partials);
  };
}

// One inner block-CG solve of A X = R (R from the outer residual, X = 0),
// each active right-hand side reduced by tol, at most max_inner iterations.
int bcg_inner(lfx_mrhs* m, const int* act, double tol, int max_inner, int* inner_its,
              int* failed) {
  lfx_ctx* ctx = m->ctx;
  const int64_t n = m->undf;
  const int G = m->bgrid;
  BcgSmall* st = m->bcg;
  const dim3 tb(32, 8), tg((unsigned)((n + 31) / 32), kBS / 32);
  mv_from_rhs_major<kBS><<<tg, tb, 0, ctx->stream>>>(n, m->R64, n, m->r32);
  LFX_CK(ctx, cudaMemsetAsync(st, 0, sizeof(BcgSmall), ctx->stream));
  LFX_CK(ctx, cudaMemcpyAsync(st->active, act, sizeof(int) * kBS, cudaMemcpyHostToDevice,
                              ctx->stream));
  LFX_CK(ctx, cudaMemsetAsync(m->x32, 0, (size_t)n * kBS * 4, ctx->stream));
  bcg_mask<<<ctx->num_sms * 8, 256, 0, ctx->stream>>>(n, m->r32, st->active);
  // r0: column norms of R (the update kernel's norm pass, products left out)
  upd_launch<0>(ctx, G)(n, m->p32, m->q32, m->x32, m->r32, m->dinv, st, 1,
                                            m->bpart);
  bcg_reduce<<<kBS / 32, 256, 0, ctx->stream>>>(G, kBS, m->bpart, st->rn, st);
  bcg_small<<<1, 256, kBcgSmallSmem, ctx->stream>>>(3, st, tol);
  // P = orth(D^-1 R)
  upd_launch<1>(ctx, G)(n, m->p32, m->r32, m->w32, nullptr, m->dinv, st, 1,
                                            nullptr);
  int rc = gram<1>(m, m->w32, m->w32, nullptr, nullptr, st, st->G);
  if (rc) return rc;
  bcg_small<<<1, 256, kBcgSmallSmem, ctx->stream>>>(2, st, tol);
  upd_launch<2>(ctx, G)(n, m->w32, nullptr, m->p32, nullptr, nullptr, st, 0,
                                            nullptr);
  ctx->launches += 10;
  LFX_CK(ctx, cudaGetLastError());
  // four iterations between the host's looks at the state (every kernel but the
  // apply idles once the solve is done)
  constexpr int kCheck = 4;
  for (int it = 1; it <= max_inner; ++it) {
    // Q = A P; alpha
    rc = mrhs_launch(m, m->p32, m->q32);
    if (!rc) rc = gram<2>(m, m->p32, m->q32, m->r32, nullptr, st, st->C);
    if (rc) return rc;
    bcg_small<<<1, 256, kBcgSmallSmem, ctx->stream>>>(0, st, tol);
    // X += P alpha, R -= Q alpha, ||R_j||
    upd_launch<0>(ctx, G)(n, m->p32, m->q32, m->x32, m->r32, m->dinv, st, 0,
                                              m->bpart);
    bcg_reduce<<<kBS / 32, 256, 0, ctx->stream>>>(G, kBS, m->bpart, st->rn, st);
    // beta (and convergence)
    rc = gram<1>(m, m->q32, m->r32, nullptr, m->dinv, st, st->E);
    if (rc) return rc;
    bcg_small<<<1, 256, kBcgSmallSmem, ctx->stream>>>(1, st, tol);
    // P = orth(D^-1 R + P beta)
    upd_launch<1>(ctx, G)(n, m->p32, m->r32, m->w32, nullptr, m->dinv, st, 0,
                                              nullptr);
    rc = gram<1>(m, m->w32, m->w32, nullptr, nullptr, st, st->G);
    if (rc) return rc;
    bcg_small<<<1, 256, kBcgSmallSmem, ctx->stream>>>(2, st, tol);
    upd_launch<2>(ctx, G)(n, m->w32, nullptr, m->p32, nullptr, nullptr, st,
                                              0, nullptr);
    ctx->launches += 13;
    LFX_CK(ctx, cudaGetLastError());
    if (it % kCheck && it < max_inner) continue;
    LFX_CK(ctx, cudaMemcpyAsync(&m->h_bcg->rank, &st->rank, 4 * sizeof(int),
                                cudaMemcpyDeviceToHost, ctx->stream));
    LFX_CK(ctx, cudaStreamSynchronize(ctx->stream));
    if (m->h_bcg->done) break;
  }
  *inner_its = m->h_bcg->iters;
  *failed = m->h_bcg->fail;
  return LFX_OK;
}

template <int NR>
int add_correction(lfx_mrhs* m, double* x, int64_t ld) {
  lfx_ctx* ctx = m->ctx;
  const int64_t n = m->undf;
  const dim3 tb(32, 8), tg((unsigned)((n + 31) / 32), NR < 32 ? 1 : NR / 32);
  mv_add_to_rhs_major<NR><<<tg, tb, 0, ctx->stream>>>(n, m->x32, x, ld);
  ctx->launches++;
  LFX_CK(ctx, cudaGetLastError());
  return LFX_OK;
}

}  // namespace

int lfx_mrhs_set_gram(lfx_mrhs* m, int32_t tensor) {
  if (!m || (tensor != 0 && tensor != 1)) return LFX_INVALID_ARGUMENT;
  m->gram_tc = tensor;
  return LFX_OK;
}

int lfx_mrhs_gram(lfx_mrhs* m, const float* U, const float* V0, const float* V1, int32_t nv,
                  int32_t tensor, double* out) {
  if (!m || !U || !V0 || !out || (nv != 1 && nv != 2) || (nv == 2 && !V1) ||
      (tensor != 0 && tensor != 1))
    return LFX_INVALID_ARGUMENT;
  lfx_ctx* ctx = m->ctx;
  if (m->nrhs != kBS) return fail(ctx, LFX_NOT_SUPPORTED, "Gram products of 64 columns only");
  int rc = ensure_work(m);
  if (!rc) rc = ensure_bcg(m);
  if (rc) return rc;
  LFX_CK(ctx, cudaMemsetAsync(m->bcg, 0, sizeof(BcgSmall), ctx->stream));
  const int keep = m->gram_tc;
  m->gram_tc = tensor;
  rc = nv == 1 ? gram<1>(m, U, V0, nullptr, nullptr, m->bcg, out)
               : gram<2>(m, U, V0, V1, nullptr, m->bcg, out);
  m->gram_tc = keep;
  if (rc) return rc;
  LFX_CK(ctx, cudaStreamSynchronize(ctx->stream));
  int h_fail = 0;
  LFX_CK(ctx, cudaMemcpy(&h_fail, &m->bcg->fail, sizeof(int), cudaMemcpyDeviceToHost));
  if (h_fail) return fail(ctx, LFX_TIMEOUT, "a tensor-core wait ran out");
  return LFX_OK;
}

int lfx_mrhs_solve(lfx_mrhs* m, lfx_op* op64, const lfx_vec* diag, const double* b, double* x,
                   int64_t ld, const lfx_mrhs_cfg* cfg, lfx_solve_info* info) {
  if (!m || !op64 || !diag || !b || !x || !cfg || !info) return LFX_INVALID_ARGUMENT;
  lfx_ctx* ctx = m->ctx;
  if (op64->precision != LFX_R64 || op64->lay->undf_to != m->undf || op64->lay->undf_from != m->undf)
    return fail(ctx, LFX_INVALID_ARGUMENT, "op64 must be the FP64 operator of the same space");
  if (diag->precision != LFX_R64 || diag->data.size() != 1 || diag->undf[0] != m->undf)
    return fail(ctx, LFX_INVALID_ARGUMENT, "diag must be one FP64 field of undf values");
  if (ld < m->undf) return fail(ctx, LFX_INVALID_ARGUMENT, "ld must be at least undf");
  if (!(cfg->r_tol > 0.0) || !(cfg->inner_tol > 0.0) || !(cfg->inner_tol < 1.0) ||
      cfg->max_outer < 1 || cfg->max_inner < 1 ||
      (cfg->method != LFX_MRHS_PER_RHS_CG && cfg->method != LFX_MRHS_BLOCK_CG))
    return fail(ctx, LFX_INVALID_ARGUMENT, "bad tolerances, iteration limits or method");
  const bool block = cfg->method == LFX_MRHS_BLOCK_CG;
  if (block && m->nrhs != kBS)
    return fail(ctx, LFX_NOT_SUPPORTED, "block CG runs 64 right-hand sides");
  int rc = ensure_work(m);
  if (!rc && block) rc = ensure_bcg(m);
  if (rc) return rc;
  std::vector<int> bcg_its(m->nrhs, 0);
  const int nr = m->nrhs;
  const int64_t n = m->undf;
  k_dinv<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(n, (const double*)diag->data[0],
                                                                m->dinv);
  LFX_CK(ctx, cudaGetLastError());
  LFX_CK(ctx, cudaMemsetAsync(m->S, 0, sizeof(MvState), ctx->stream));
  std::vector<double> r0(nr), rn(nr);
  std::vector<int> act(64, 0), outer_n(nr, 0);
  // With products accurate to FP32 an inner solve meets its tolerance on the
  // true residual as well, so that the last step of the refinement can end just
  // under r_tol (products rounded to TF32 fell short and took a step more). CG on
  // each right-hand side therefore goes to half the tolerance. Largest error of the
  // solution against FP64, N(0, 1) right-hand sides, inner_tol 1e-2, r_tol 1e-6, 1e-7,
  // .. 1e-11; whole tolerance / half / rounded products: C24 x 20 2.4e-5 1.6e-7 1.6e-7
  // 2.4e-9 2.4e-9 1.6e-11 / 3.0e-6 1.3e-6 1.1e-8 1.1e-8 9.3e-11 9.3e-11 / 2.0e-5 2.1e-7
  // 1.5e-7 2.9e-9 1.6e-9 2.2e-11; C48 x 30 5.5e-5 4.8e-7 4.8e-7 6.2e-9 6.2e-9 4.3e-11 /
  // 6.5e-6 2.7e-8 2.7e-8 2.7e-8 1.9e-10 1.9e-10 / 1.6e-6 1.6e-6 2.4e-8 2.4e-8 3.0e-10
  // 3.0e-10, in 3 to 6 steps, 3 to 5 and 4 to 7. Block CG, whose step ends with its
  // slowest right-hand side, keeps the whole tolerance: half of it gave C48 x 30 at
  // 1e-8 2.8e-7 for 1.1e-7, 410 iterations for 361.
  const double inner_tol = (block ? 1.0 : 0.5) * cfg->inner_tol;
  rc = outer_residual(m, op64, b, x, ld);
  if (rc) return rc;
  for (int r = 0; r < nr; ++r) r0[r] = rn[r] = m->h_nrm[r];
  int outer = 0, inner_total = 0;
  for (;;) {
    int nact = 0;
    for (int r = 0; r < nr; ++r) {
      const bool conv = r0[r] == 0.0 || rn[r] <= cfg->r_tol * r0[r];
      act[r] = !conv && std::isfinite(rn[r]);
      nact += act[r];
    }
    if (nact == 0 || outer >= cfg->max_outer) break;
    int its = 0, bfail = 0;
    if (block) {
      rc = bcg_inner(m, act.data(), inner_tol, cfg->max_inner, &its, &bfail);
      for (int r = 0; r < nr; ++r)
        if (act[r]) bcg_its[r] += its;
    } else {
      rc = nr == 16 ? inner_solve<16>(m, act.data(), inner_tol, cfg->max_inner, &its)
           : nr == 32 ? inner_solve<32>(m, act.data(), inner_tol, cfg->max_inner, &its)
                      : inner_solve<64>(m, act.data(), inner_tol, cfg->max_inner, &its);
    }
    if (!rc) rc = nr == 16 ? add_correction<16>(m, x, ld)
                  : nr == 32 ? add_correction<32>(m, x, ld)
                             : add_correction<64>(m, x, ld);
    if (rc) return rc;
    inner_total += its;
    for (int r = 0; r < nr; ++r) outer_n[r] += act[r];
    ++outer;
    rc = outer_residual(m, op64, b, x, ld);
    if (rc) return rc;
    for (int r = 0; r < nr; ++r) rn[r] = m->h_nrm[r];
  }
  LFX_CK(ctx, cudaMemcpyAsync(m->h_S, m->S, sizeof(MvState), cudaMemcpyDeviceToHost, ctx->stream));
  LFX_CK(ctx, cudaStreamSynchronize(ctx->stream));
  rc = lfx_ctx_check_device_error(ctx);
  for (int r = 0; r < nr; ++r) {
    lfx_solve_info& I = info[r];
    memset(&I, 0, sizeof I);
    I.initial_norm = r0[r];
    I.final_norm = rn[r];
    I.final_rel = r0[r] > 0.0 ? rn[r] / r0[r] : 0.0;
    I.converged = r0[r] == 0.0 || rn[r] <= cfg->r_tol * r0[r];
    I.outer_iterations = outer_n[r];
    I.inner_iterations = block ? bcg_its[r] : m->h_S->iters[r];
    I.iterations = I.inner_iterations;
    I.applies = inner_total;
    I.status = I.converged ? LFX_OK : (std::isfinite(rn[r]) ? LFX_NOT_CONVERGED : LFX_NAN_DETECTED);
  }
  return rc;
}
