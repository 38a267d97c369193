// solver.cu -- preconditioner and restarted GMRES, resident on the device.
//
//   block preconditioner   src/precond_fmm.c:147-263, 553-652: one dense block
//                          per level (depth-1) cube, 2*nPnls square, entries
//                          block[i*M+j] from panelIA0(pnlX=j, pnlY=i) which
//                          LAPACK reads column-major, plus the area diagonal;
//                          LU-factored once (dgetrf)
//   cached-LU apply        src/precond_fmm.c:861-953 (dgetrs per block)
//   diagonal apply         src/precond_fmm.c:664-728
//   GMRES                  src/gmres.c:153-373 (Templates GMRES, left
//                          preconditioned, modified Gram-Schmidt basis,
//                          Givens rotations, x0 = initial guess)
//
// B200 design: the block matrices are assembled by a kernel in FP64 (the
// exact panelIA0 cases) and replaced by their explicit inverses, so each
// preconditioner apply is one block-diagonal GEMV kernel streaming the
// inverses from HBM instead of ~3 launches per block; the inverses are formed
// by size class in thread-block clusters (cuSOLVER above the last class).  The
// Krylov vectors, the Hessenberg columns and the Givens rotations live on the
// device, with deterministic reductions; a status record crosses to the host
// once per step.
#include <cusolverDn.h>

#include <climits>
#include <cmath>
#include <vector>

#include <cooperative_groups.h>

#include "context.cuh"
#include "quad.cuh"

namespace fb {

struct PrecondDev {
  int mode = -1;
  DevArena arena;
  int nBlocks = 0;
  std::vector<int> hStart, hSize;
  std::vector<long long> hOff;
  int *d_start = nullptr, *d_size = nullptr;
  int2 *d_tiles = nullptr;   // (block, first row) tiles of the apply
  int *d_colSrc = nullptr;   // per block (offset 2*start): input component of each stored column
  int *d_rowDst = nullptr;   // output component of each stored row
  int nTiles = 0;
  long long *d_off = nullptr;
  double *d_inv = nullptr;
  float *d_invF = nullptr;   // mixed contexts: the inverses stored in FP32 (applied with FP64 sums)
  int maxM = 0;
  // GMRES workspace
  int restart = 0;
  double *d_V = nullptr, *d_r = nullptr, *d_av = nullptr, *d_w = nullptr;
  double *d_h = nullptr, *d_part = nullptr, *d_y = nullptr;
  double *d_G = nullptr;                    // Gram entries of the current cycle's basis (row k: j < k)
  double *d_H = nullptr, *d_sv = nullptr;   // Hessenberg (+ cs, sn columns) and rotated residual vector
  void *d_status = nullptr;                 // GmresStatus on the device
  void *h_status = nullptr;                 // pinned host copy (and two host-read norms)
  cudaEvent_t evStatus = nullptr;           // marks the status copy (the host spins on it)
  int partCap = 0;
};

void free_precond(Context &c) {
  if (c.pc) {
    c.pc->arena.release();
    if (c.pc->h_status) cudaFreeHost(c.pc->h_status);
    if (c.pc->evStatus) cudaEventDestroy(c.pc->evStatus);
    delete c.pc;
    c.pc = nullptr;
  }
}

// ---------------------------------------------------------------------------
// block assembly: A(j, i) = -K1(X=j,Y=i) etc. in column-major M x M
// (src/precond_fmm.c:147-263: panelIA0 over the cube's panel pairs).
// From the near field's own coefficients: every pair's one-point
// term A_X A_Y KER4(p_X - p_Y) at the one-point nodes p = v0/2 + v1/4 + v2/4 (0
// for X = Y), then, in pc_special_kernel, the exact-minus-one-point correction
// of the special pairs (shared vertex, edge, self) from the near field's table,
// so a block equals panelIA0's at -q=1 without its singularity tests per pair.
template <typename TO>
__global__ void pc_onepoint_kernel(int nBlocks, const int *__restrict__ bStart, const int *__restrict__ bSize,
                                   const long long *__restrict__ bOff, const double *__restrict__ vtx,
                                   const double *__restrict__ nrm, const double *__restrict__ area, double kappa,
                                   double eps, double s1, double s2, TO *A) {
  for (int b = blockIdx.y; b < nBlocks; b += gridDim.y) {   // (the grid's y extent is capped at 65535)
    const int hm = bSize[b], st = bStart[b], M = 2 * hm;
    const long long pairs = (long long)hm * hm;
    TO *Ab = A + bOff[b];
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < pairs;
         p += (long long)gridDim.x * blockDim.x) {
      const int i = (int)(p / hm), j = (int)(p % hm);  // i: pnlY (column), j: pnlX (row)
      const int Xi = st + j, Yi = st + i;
      double K[4] = {0.0, 0.0, 0.0, 0.0};
      if (Xi != Yi) {
        const double *vx = vtx + 9 * (size_t)Xi, *vy = vtx + 9 * (size_t)Yi;
        double r[3], nX[3], nY[3];
        for (int c = 0; c < 3; c++) {
          const double mx = vx[c] + 0.5 * ((vx[3 + c] - vx[c]) + 0.5 * (vx[6 + c] - vx[3 + c]));
          const double my = vy[c] + 0.5 * ((vy[3 + c] - vy[c]) + 0.5 * (vy[6 + c] - vy[3 + c]));
          r[c] = mx - my;
          nX[c] = nrm[3 * (size_t)Xi + c];
          nY[c] = nrm[3 * (size_t)Yi + c];
        }
        if (r[0] != 0.0 || r[1] != 0.0 || r[2] != 0.0) {
          double y[4];
          ker4_d(kappa, eps, r, nX, nY, y);
          const double w = area[Xi] * area[Yi];
          for (int k = 0; k < 4; k++) K[k] = w * y[k];
        }
      }
      const double d0 = (i == j) ? s1 * area[Yi] : 0.0;
      const double d1 = (i == j) ? s2 * area[Yi] : 0.0;
      Ab[(size_t)i * M + j] = (TO)(-K[1] + d0);
      Ab[(size_t)i * M + j + hm] = (TO)(-K[0]);
      Ab[(size_t)(i + hm) * M + j] = (TO)(-K[3]);
      Ab[(size_t)(i + hm) * M + j + hm] = (TO)(-K[2] + d1);
    }
  }
}

// the special pairs (X, Y) of a block: add their correction (each entry has one writer)
template <typename TO>
__global__ void pc_special_kernel(int nBlocks, const int *__restrict__ bStart, const int *__restrict__ bSize,
                                  const long long *__restrict__ bOff, const int *__restrict__ spOff,
                                  const int *__restrict__ spSrc, const double4 *__restrict__ spK, TO *A) {
  for (int b = blockIdx.y; b < nBlocks; b += gridDim.y) {
    const int hm = bSize[b], st = bStart[b], M = 2 * hm;
    TO *Ab = A + bOff[b];
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < hm; j += gridDim.x * blockDim.x) {
      const int Xi = st + j;
      for (int e = spOff[Xi]; e < spOff[Xi + 1]; e++) {
        const int Yi = spSrc[e];
        if (Yi < st || Yi >= st + hm) continue;
        const int i = Yi - st;
        const double4 d = spK[e];   // (K0, K1, K2, K3) exact minus one-point
        TO *a0 = Ab + (size_t)i * M + j, *a1 = Ab + (size_t)i * M + j + hm;
        TO *a2 = Ab + (size_t)(i + hm) * M + j, *a3 = Ab + (size_t)(i + hm) * M + j + hm;
        *a0 = (TO)((double)*a0 - d.y);
        *a1 = (TO)((double)*a1 - d.x);
        *a2 = (TO)((double)*a2 - d.w);
        *a3 = (TO)((double)*a3 - d.z);
      }
    }
  }
}

// the listed blocks of I := identity, and their column and row indices the identity
__global__ void identity_kernel(int nList, const int *__restrict__ list, const int *__restrict__ bStart,
                                const int *__restrict__ bSize, const long long *__restrict__ bOff, double *I,
                                int *colSrc, int *rowDst) {
  for (int li = blockIdx.y; li < nList; li += gridDim.y) {   // (y extent capped at 65535)
    const int b = list[li];
    const int M = 2 * bSize[b];
    const long long e = (long long)M * M;
    double *Ib = I + bOff[b];
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < e; p += (long long)gridDim.x * blockDim.x)
      Ib[p] = ((p / M) == (p % M)) ? 1.0 : 0.0;
    if (blockIdx.x == 0)
      for (int c = threadIdx.x; c < M; c += blockDim.x)
        colSrc[2LL * bStart[b] + c] = rowDst[2LL * bStart[b] + c] = c;
  }
}

// In-place inversion of the preconditioner blocks of up to 1,536 rows by
// blocked Gauss-Jordan elimination with partial pivoting, all blocks of a size
// class in one launch; a block is inverted by a cluster of CS thread blocks.
// Per panel of NB columns:
//   * every CTA of the cluster eliminates the panel in its shared memory (the
//     same data, so the same result), eight columns at a time with its rows in
//     registers (row i belongs to thread i mod NT), one barrier per pivot: the
//     warps' candidates (largest |a| among the rows not yet taken) carry their
//     rows along; each eight columns are then a rank-8 update of the panel's rest;
//   * each CTA takes its share of the other columns, dealt in tiles:
//     A(:, j) = A(:, j) without the pivot rows + Panel * A(pivot rows, j).
// Rows are never interchanged: perm[k] is the row that column k was eliminated
// with, stored column c multiplies input component colSrc[c] = perm[c], and
// stored row perm[k] is output component rowDst[perm[k]] = k.  info[b] = k + 1
// for the first column whose pivot is zero, not finite or without a finite
// reciprocal; perm stays a permutation of the rows whatever the values are.
//
// 2 M^3 operations; bound by latency: at two CTAs per SM the updates' loads
// from the block and from shared memory and the pivots' barriers each stall
// about as much (every panel reads and writes a whole block, at a quarter of the
// DRAM's peak rate).  So panels are as wide as shared memory allows.  A panel of 32 columns of a 575-row block on
// two CTAs: 46 us of pivots and in-panel updates, 26 gathering the pivot rows,
// 115 updating.  With interchanged rows, panels of 16 eliminated in shared
// memory with two barriers per pivot and the interchange list formed by one
// thread, the 1,108 blocks of a 204,800-panel star surface (mean 370 rows, 96
// above 768 and one of 1,672) took 74 ms in FP32; 28 now, as long as the one
// block of the next kernel takes.
constexpr int kInvSub = 8;   // columns eliminated in registers

template <typename TV>
struct InvShape;   // quads of rows and columns per thread in the update
template <>
struct InvShape<float> {
  static constexpr int QR = 2;
  typedef float4 V4;
};
template <>
struct InvShape<double> {
  static constexpr int QR = 1;
  typedef double4 V4;
};

template <typename TV, int NB, int QC>
__host__ __device__ constexpr size_t inv_smem_bytes(int maxM) {
  return sizeof(TV) * ((size_t)NB * ((maxM + 3) & ~3) + (size_t)NB * 64 * QC) + (size_t)maxM * (sizeof(int) + 1);
}

// the largest value of the warp and the lowest index among the lanes that hold it (v >= 0, or -1 for none; a NaN,
// its sign cleared, counts as larger than infinity)
__device__ __forceinline__ int warp_first_max(float v, int i) {
  const unsigned b = v < 0.f ? 0u : __float_as_uint(v) + 1u;
  const unsigned m = __reduce_max_sync(0xffffffffu, b);
  return __reduce_min_sync(0xffffffffu, b == m ? i : INT_MAX);
}
__device__ __forceinline__ int warp_first_max(double v, int i) {
  const unsigned hi = v < 0.0 ? 0u : (unsigned)__double2hiint(v) + 1u;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == mh ? (unsigned)__double2loint(v) : 0u;
  const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
  return __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? i : INT_MAX);
}

// d = 1/pivot (0 for a zero pivot): the elimination can go on with finite numbers
template <typename TV>
__device__ __forceinline__ bool usable_pivot(TV d) {
  return fabs(d) > (TV)0 && !isinf(d);
}

template <typename TV, int NB, int CS, int RPT, int QC, int NT>
__global__ void __launch_bounds__(NT, NT == 256 ? 2 : 1)
pc_invert_kernel(const int *__restrict__ list, const int *__restrict__ bStart, const int *__restrict__ bSize,
                 const long long *__restrict__ bOff, TV *inv, int *colSrc, int *rowDst, int *info) {
  typedef typename Vec2<TV>::t V2;
  typedef typename InvShape<TV>::V4 V4;
  constexpr int QR = InvShape<TV>::QR, TR = 64 * QR, TC = 64 * QC;
  constexpr int W = NT / 32;
  extern __shared__ double4 invSmem[];
  __shared__ TV cVal[2][W], cRow[2][W][kInvSub], sY[NB][kInvSub];
  __shared__ int cIdx[2][W];
  const int rank = (CS > 1) ? (int)(blockIdx.x % CS) : 0;
  const int b = list[blockIdx.x / CS];
  const int M = 2 * bSize[b], Mp = (M + 3) & ~3;
  TV *A = inv + bOff[b];
  TV *P = reinterpret_cast<TV *>(invSmem);       // the panel, [NB][Mp]
  TV *Yt = P + (size_t)NB * Mp;                  // the pivot rows of a column tile, [NB][TC]
  int *perm = reinterpret_cast<int *>(Yt + (size_t)NB * TC);   // [M]
  unsigned char *flag = reinterpret_cast<unsigned char *>(perm + M);   // [M]: a pivot row of this panel
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int grp = t / 256, tr = t % 16, tc = (t % 256) / 16;   // groups of 256 threads take the row tiles in turn
  unsigned used = 0;   // of this thread's rows
  int bad = 0;
  for (int k0 = 0; k0 < M; k0 += NB) {
    const int nb = min(NB, M - k0);
    if (CS > 1) {   // the owners' updates of these columns are complete and visible
      __threadfence();
      cooperative_groups::this_cluster().sync();
    } else {
      __syncthreads();
    }
    for (int i = t; i < M; i += NT) {
      flag[i] = 0;
      const TV *src = A + (size_t)k0 * M + i;
#pragma unroll 16
      for (int c = 0; c < nb; c++) P[c * Mp + i] = src[(size_t)c * M];
    }
    // (row i of P and of flag: written and read by thread i mod NT until the next barrier)
    for (int c0 = 0; c0 < nb; c0 += kInvSub) {
      const int sb = min(kInvSub, nb - c0);
      TV v[RPT][kInvSub];
      unsigned sub = 0;   // pivot rows of these columns
#pragma unroll
      for (int r = 0; r < RPT; r++) {
        const int i = t + r * NT;
#pragma unroll
        for (int c = 0; c < kInvSub; c++) v[r][c] = i < M && c < sb ? P[(c0 + c) * Mp + i] : (TV)0;
      }
#pragma unroll
      for (int kk = 0; kk < kInvSub; kk++) {
        if (kk >= sb) break;   // uniform
        TV best = (TV)-1;
        int bi = INT_MAX;
#pragma unroll
        for (int r = 0; r < RPT; r++) {
          const int i = t + r * NT;
          const TV a = fabs(v[r][kk]);
          if (i < M && !((used >> r) & 1u) && !(a <= best)) {   // a NaN is taken too: some row always is
            best = a;
            bi = i;
          }
        }
        const int wi = warp_first_max(best, bi), par = kk & 1;
        if (wi == INT_MAX) {   // no row left in this warp
          if (lane == 0) {
            cVal[par][warp] = (TV)-1;
            cIdx[par][warp] = INT_MAX;
          }
        } else if (bi == wi) {
          cVal[par][warp] = best;
          cIdx[par][warp] = wi;
#pragma unroll
          for (int r = 0; r < RPT; r++)
            if (t + r * NT == wi)
#pragma unroll
              for (int c = 0; c < kInvSub; c++) cRow[par][warp][c] = v[r][c];
        }
        __syncthreads();   // (two buffers: a step's writes cannot meet the previous step's reads)
        const int ci = lane < W ? cIdx[par][lane] : INT_MAX;
        const int pv = warp_first_max(lane < W ? cVal[par][lane] : (TV)-1, ci);
        const int pw = __ffs(__ballot_sync(0xffffffffu, ci == pv)) - 1;
        const TV piv = cRow[par][pw][kk];
        const TV d = piv != (TV)0 ? (TV)1 / piv : (TV)0;
        if (!usable_pivot(d)) bad = bad ? bad : k0 + c0 + kk + 1;
        if (t == 0) perm[k0 + c0 + kk] = pv;
        TV row[kInvSub];
#pragma unroll
        for (int c = 0; c < kInvSub; c++) row[c] = c == kk ? d : cRow[par][pw][c] * d;
#pragma unroll
        for (int r = 0; r < RPT; r++) {
          const TV f = v[r][kk];
          if (t + r * NT == pv) {
            used |= 1u << r;
            sub |= 1u << r;
            flag[pv] = 1;
#pragma unroll
            for (int c = 0; c < kInvSub; c++) v[r][c] = row[c];
          } else {
#pragma unroll
            for (int c = 0; c < kInvSub; c++) v[r][c] = c == kk ? -f * d : v[r][c] - f * row[c];
          }
        }
      }
#pragma unroll
      for (int r = 0; r < RPT; r++) {
        const int i = t + r * NT;
        if (i < M)
#pragma unroll
          for (int c = 0; c < kInvSub; c++)
            if (c < sb) P[(c0 + c) * Mp + i] = v[r][c];
      }
      if (nb > kInvSub) {   // the panel's other columns
        __syncthreads();    // perm, and the previous rows' columns, are written
        for (int e = t; e < nb * kInvSub; e += NT) {
          const int c = e / kInvSub, kk = e % kInvSub;
          sY[c][kk] = kk < sb && (c < c0 || c >= c0 + sb) ? P[c * Mp + perm[k0 + c0 + kk]] : (TV)0;
        }
        __syncthreads();
        for (int c = 0; c < nb; c++) {
          if (c >= c0 && c < c0 + sb) continue;
          TV y[kInvSub];
#pragma unroll
          for (int kk = 0; kk < kInvSub; kk++) y[kk] = sY[c][kk];
#pragma unroll
          for (int r = 0; r < RPT; r++) {
            const int i = t + r * NT;
            if (i < M) {
              TV s = (sub >> r) & 1u ? (TV)0 : P[c * Mp + i];
#pragma unroll
              for (int kk = 0; kk < kInvSub; kk++) s += v[r][kk] * y[kk];
              P[c * Mp + i] = s;
            }
          }
        }
      }
    }
    if (CS > 1) cooperative_groups::this_cluster().sync();   // every CTA has read the panel's columns
    else __syncthreads();
    if (rank == 0)
      for (int c = 0; c < nb; c++)
        for (int i = t; i < M; i += NT) A[(size_t)(k0 + c) * M + i] = P[c * Mp + i];
    for (int jt = TC * rank; jt < M; jt += TC * CS) {
      __syncthreads();   // the previous tile's reads of Yt are done
#pragma unroll 8
      for (int e = t; e < nb * TC; e += NT) {
        const int kk = e / TC, j = jt + e % TC;
        Yt[e] = j < M ? A[(size_t)j * M + perm[k0 + kk]] : (TV)0;
      }
      __syncthreads();
      // row tiles, the next one's values loaded while the current one is computed
      auto load_tile = [&](int it, TV (&v)[QC * 4][QR * 4]) {
#pragma unroll
        for (int q = 0; q < QR; q++) {
          const int i0 = it + 64 * q + 4 * tr;
          const bool in = i0 < M, hi = i0 + 2 < M;   // M is even: a row quad is full or holds two rows
#pragma unroll
          for (int c = 0; c < QC * 4; c++) {
            const int j = jt + 64 * (c / 4) + 4 * tc + c % 4;
            V2 a{(TV)0, (TV)0}, z{(TV)0, (TV)0};
            if (in && j < M) {
              const V2 *src = reinterpret_cast<const V2 *>(A + (size_t)j * M + i0);
              a = src[0];
              if (hi) z = src[1];
            }
            v[c][4 * q] = a.x;
            v[c][4 * q + 1] = a.y;
            v[c][4 * q + 2] = z.x;
            v[c][4 * q + 3] = z.y;
          }
        }
      };
      constexpr int kStep = TR * (NT / 256);
      TV nxt[QC * 4][QR * 4];
      if (TR * grp < M) load_tile(TR * grp, nxt);
      for (int it = TR * grp; it < M; it += kStep) {
        TV acc[QC * 4][QR * 4];
        int ir[QR];
#pragma unroll
        for (int q = 0; q < QR; q++) {
          const int i0 = it + 64 * q + 4 * tr;
          ir[q] = i0 < M ? i0 : -1;
#pragma unroll
          for (int r = 0; r < 4; r++) {
            const bool f = i0 + r < M && flag[i0 + r];   // a pivot row starts from zero
#pragma unroll
            for (int c = 0; c < QC * 4; c++) acc[c][4 * q + r] = f ? (TV)0 : nxt[c][4 * q + r];
          }
        }
        if (it + kStep < M) load_tile(it + kStep, nxt);
#pragma unroll 2
        for (int kk = 0; kk < nb; kk++) {
          V4 w[QR], y[QC];
#pragma unroll
          for (int q = 0; q < QR; q++) w[q] = *reinterpret_cast<const V4 *>(P + (size_t)kk * Mp + (ir[q] < 0 ? 0 : ir[q]));
#pragma unroll
          for (int q = 0; q < QC; q++) y[q] = *reinterpret_cast<const V4 *>(Yt + kk * TC + 64 * q + 4 * tc);
#pragma unroll
          for (int c = 0; c < QC * 4; c++) {
            const V4 &yq = y[c / 4];
            const TV yc = c % 4 == 0 ? yq.x : c % 4 == 1 ? yq.y : c % 4 == 2 ? yq.z : yq.w;
#pragma unroll
            for (int q = 0; q < QR; q++) {
              acc[c][4 * q] += w[q].x * yc;
              acc[c][4 * q + 1] += w[q].y * yc;
              acc[c][4 * q + 2] += w[q].z * yc;
              acc[c][4 * q + 3] += w[q].w * yc;
            }
          }
        }
#pragma unroll
        for (int c = 0; c < QC * 4; c++) {
          const int j = jt + 64 * (c / 4) + 4 * tc + c % 4;
          if (j >= M || (j >= k0 && j < k0 + nb)) continue;
#pragma unroll
          for (int q = 0; q < QR; q++)
            if (ir[q] >= 0) {
              V2 *dst = reinterpret_cast<V2 *>(A + (size_t)j * M + ir[q]);
              dst[0] = V2{acc[c][4 * q], acc[c][4 * q + 1]};
              if (ir[q] + 2 < M) dst[1] = V2{acc[c][4 * q + 2], acc[c][4 * q + 3]};
            }
        }
      }
    }
  }
  __syncthreads();
  if (rank == 0) {
    int *cs = colSrc + 2 * bStart[b], *rd = rowDst + 2 * bStart[b];
    for (int k = t; k < M; k += NT) {
      cs[k] = perm[k];
      rd[perm[k]] = k;
    }
    if (t == 0) info[b] = bad;
  }
}

// The same for larger blocks, whose panel's rows do not fit in registers: the
// panel eliminated in shared memory, with row interchanges.  Per panel of NB
// columns:
//   * every CTA of the cluster eliminates the panel in its shared memory (the
//     same data, so the same result; pivot = first largest |a| at or below
//     the diagonal, as idamax) and rank 0 writes it back;
//   * each CTA takes its share of the other columns (64-column tiles dealt
//     round-robin): the panel's row interchanges, the panel rows moved to a
//     scratch Y and zeroed, then A(:, j) += Panel * Y(:, j), the composite
//     elimination of the panel as a rank-NB update (4x4 outputs per thread);
//   * a cluster barrier before the next panel, whose columns some CTA owns.
// The column interchanges that end Gauss-Jordan are not carried out:
// colSrc[c] records which input component stored column c multiplies, and
// the apply kernels gather through it (rowDst is the identity).  info[b] = k+1
// for the first pivot k that is zero, not finite or without a finite reciprocal.
constexpr int kGjThreads = 256;

template <typename TV, int NB>
__host__ __device__ constexpr size_t gj_smem_bytes(int maxM) {
  return (size_t)NB * maxM * sizeof(TV) + 64 * NB * sizeof(TV) + (size_t)maxM * sizeof(int);
}

// resident blocks per SM the register allocation of pc_gj_invert_kernel<float>
// aims at (the FP64 kernel keeps one: at two it spills)
#ifndef FB_GJ_MIN_BLOCKS
#define FB_GJ_MIN_BLOCKS 2
#endif
template <typename TV, int NB, int CS>
__global__ void __launch_bounds__(kGjThreads, sizeof(TV) == 4 ? FB_GJ_MIN_BLOCKS : 1)
pc_gj_invert_kernel(const int *__restrict__ list, const int *__restrict__ bStart, const int *__restrict__ bSize,
                    const long long *__restrict__ bOff, const long long *__restrict__ yOff, TV *inv, TV *yAll,
                    int *colSrc, int *rowDst, int *info) {
  typedef typename Vec2<TV>::t V2;
  extern __shared__ double gjSmemD[];
  TV *gjSmem = reinterpret_cast<TV *>(gjSmemD);
  __shared__ TV wbest[kGjThreads / 32];
  __shared__ int wbi[kGjThreads / 32];
  __shared__ int sPos[2 * NB], sSrc[2 * NB], sCnt;
  __shared__ TV gBuf[64 * 2 * NB];   // one column tile's moved rows
  __shared__ TV sRk[NB], sOk[NB];
  const int rank = (CS > 1) ? (int)(blockIdx.x % CS) : 0;
  const int b = list[blockIdx.x / CS];
  const int M = 2 * bSize[b];
  TV *A = inv + bOff[b];
  TV *Y = yAll + yOff[b];
  TV *P = gjSmem;                          // panel, [NB][M]
  TV *Yt = gjSmem + (size_t)NB * M;        // Y tile, [64][NB]
  int *perm = (int *)(Yt + 64 * NB);           // [M]
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int bad = 0;
  for (int k0 = 0; k0 < M; k0 += NB) {
    const int nb = min(NB, M - k0);
    if (CS > 1) {   // the owners' updates of these columns are complete and visible
      __threadfence();
      cooperative_groups::this_cluster().sync();
    }
    for (int e = t; e < nb * M; e += kGjThreads) P[e] = A[(size_t)k0 * M + e];   // columns k0.. are contiguous
    __syncthreads();
    // Row i of the panel belongs to thread i mod kGjThreads throughout: each
    // step's write phase also finds the thread's candidate pivot of the next
    // column among its own rows, so a step needs two barriers.
    TV best = (TV)-1;
    int bi = INT_MAX;
    for (int i = t; i < M; i += kGjThreads) {
      if (i < k0) continue;
      const TV v = fabs(P[i]);
      if (!(v <= best)) { best = v; bi = i; }   // a NaN is taken too: some row always is
    }
    for (int kk = 0; kk < nb; kk++) {
      const int k = k0 + kk;
      const int wi = warp_first_max(best, bi);   // first largest within the warp
      if (wi == INT_MAX) {   // no row left in this warp
        if (lane == 0) { wbest[warp] = (TV)-1; wbi[warp] = INT_MAX; }
      } else if (bi == wi) {
        wbest[warp] = best;
        wbi[warp] = wi;
      }
      __syncthreads();
      const int pv = warp_first_max(lane < kGjThreads / 32 ? wbest[lane] : (TV)-1,
                                    lane < kGjThreads / 32 ? wbi[lane] : INT_MAX);
      if (t == 0) perm[k] = pv;
      // read phase: the pivot row (old row pv, scaled; sRk[kk] = 1/pivot) and
      // the old row k, which moves to row pv
      if (t < nb) {
        const TV piv = P[kk * M + pv];
        const TV d = (piv != (TV)0) ? (TV)1 / piv : (TV)0;
        sRk[t] = (t == kk) ? d : P[t * M + pv] * d;
        sOk[t] = P[t * M + k];
      }
      __syncthreads();
      // write phase, and the candidates for the next column
      const TV d = sRk[kk];
      if (!usable_pivot(d)) bad = bad ? bad : k + 1;
      best = (TV)-1;
      bi = INT_MAX;
      const bool more = kk + 1 < nb;
      for (int i = t; i < M; i += kGjThreads) {
        if (i == k) {
          for (int c = 0; c < nb; c++) P[c * M + k] = sRk[c];
          continue;   // the pivot row is no candidate
        }
        if (i == pv) {   // (only reached when pv != k) the old row k, eliminated
          const TV f = sOk[kk];
          for (int c = 0; c < nb; c++) P[c * M + i] = (c == kk) ? -f * d : sOk[c] - f * sRk[c];
        } else {
          const TV f = P[kk * M + i];
          for (int c = 0; c < nb; c++) P[c * M + i] = (c == kk) ? -f * d : P[c * M + i] - f * sRk[c];
        }
        if (more && i > k) {
          const TV v = fabs(P[(kk + 1) * M + i]);
          if (!(v <= best)) { best = v; bi = i; }
        }
      }
      // the next step's first barrier orders this write phase before its reads
    }
    __syncthreads();
    if (rank == 0)
      for (int e = t; e < nb * M; e += kGjThreads) A[(size_t)k0 * M + e] = P[e];
    // the panel's row interchanges as one gather: row r takes the value of row sSrc of the same column
    if (t == 0) {
      int cnt = 0;
      auto add = [&](int r) {
        for (int q = 0; q < cnt; q++)
          if (sPos[q] == r) return;
        sPos[cnt] = r;
        sSrc[cnt] = r;
        cnt++;
      };
      for (int kk = 0; kk < nb; kk++) {
        add(k0 + kk);
        add(perm[k0 + kk]);
      }
      for (int kk = 0; kk < nb; kk++) {   // replay the swaps on the source indices
        const int k = k0 + kk, pv = perm[k];
        int qa = 0, qb = 0;
        for (int q = 0; q < cnt; q++) {
          if (sPos[q] == k) qa = q;
          if (sPos[q] == pv) qb = q;
        }
        const int tmp = sSrc[qa];
        sSrc[qa] = sSrc[qb];
        sSrc[qb] = tmp;
      }
      sCnt = cnt;
    }
    __syncthreads();
    // this CTA's columns: gather the interchanged rows, rows k0.. to Y, zero
    // them; per 64-column tile all (column, moved row) reads are issued
    // together into gBuf, then, after a barrier, written back
    const int cnt = sCnt;
    for (int jt = 64 * rank; jt < M; jt += 64 * CS) {
      const int ne = 64 * cnt;
#pragma unroll 4
      for (int e = t; e < ne; e += kGjThreads) {
        const int jl = e / cnt, q = e - jl * cnt, j = jt + jl;
        if (j < M && (j < k0 || j >= k0 + nb)) gBuf[e] = A[(size_t)j * M + sSrc[q]];
      }
      __syncthreads();
      for (int e = t; e < ne; e += kGjThreads) {
        const int jl = e / cnt, q = e - jl * cnt, j = jt + jl;
        if (j < M && (j < k0 || j >= k0 + nb)) {
          const int r = sPos[q];
          TV *col = A + (size_t)j * M;
          if (r >= k0 && r < k0 + nb) {
            Y[(size_t)j * NB + (r - k0)] = gBuf[e];
            col[r] = (TV)0;
          } else {
            col[r] = gBuf[e];
          }
        }
      }
      __syncthreads();
    }
    // A(:, j) += P * Y(:, j) over this CTA's 64-column tiles; thread: 4 rows x 4 columns
    const int tr = t % 16, tc = t / 16;
    for (int jt = 64 * rank; jt < M; jt += 64 * CS) {
      for (int e = t; e < 64 * NB; e += kGjThreads) {
        const int jl = e / NB, kk = e % NB, j = jt + jl;
        const bool ok = j < M && (j < k0 || j >= k0 + nb) && kk < nb;
        Yt[e] = ok ? Y[(size_t)j * NB + kk] : (TV)0;
      }
      __syncthreads();
      // row tiles, the next tile's A values loaded while the current one is computed
      auto load_tile = [&](int it, TV (&v)[4][4]) {
        const int i0 = it + 4 * tr;
        const bool in = i0 < M, full = i0 + 4 <= M;   // M is even: a row quad is full or holds two rows
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const int j = jt + 4 * tc + c;
          if (in && j < M) {
            const V2 *src = reinterpret_cast<const V2 *>(A + (size_t)j * M + i0);
            const V2 lo = src[0], hi = full ? src[1] : V2{(TV)0, (TV)0};
            v[c][0] = lo.x; v[c][1] = lo.y; v[c][2] = hi.x; v[c][3] = hi.y;
          } else {
            v[c][0] = v[c][1] = v[c][2] = v[c][3] = (TV)0;
          }
        }
      };
      TV acc[4][4], nxt[4][4];
      load_tile(0, acc);
      for (int it = 0; it < M; it += 64) {
        const int i0 = it + 4 * tr;
        if (it + 64 < M) load_tile(it + 64, nxt);
        if (i0 < M) {
          const bool full = i0 + 4 <= M;
          for (int kk = 0; kk < nb; kk++) {
            const V2 *pw = reinterpret_cast<const V2 *>(P + (size_t)kk * M + i0);
            const V2 wlo = pw[0], whi = full ? pw[1] : V2{(TV)0, (TV)0};
            const TV w[4] = {wlo.x, wlo.y, whi.x, whi.y};
            TV y[4];
#pragma unroll
            for (int c = 0; c < 4; c++) y[c] = Yt[(4 * tc + c) * NB + kk];
#pragma unroll
            for (int c = 0; c < 4; c++)
#pragma unroll
              for (int r = 0; r < 4; r++) acc[c][r] += w[r] * y[c];
          }
#pragma unroll
          for (int c = 0; c < 4; c++) {
            const int j = jt + 4 * tc + c;
            if (j < M && (j < k0 || j >= k0 + nb)) {
              V2 *dst = reinterpret_cast<V2 *>(A + (size_t)j * M + i0);
              dst[0] = V2{acc[c][0], acc[c][1]};
              if (full) dst[1] = V2{acc[c][2], acc[c][3]};
            }
          }
        }
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
          for (int r = 0; r < 4; r++) acc[c][r] = nxt[c][r];
      }
      __syncthreads();
    }
  }
  // the pending column interchanges, as an index: stored column c multiplies input component colSrc[c]
  __syncthreads();
  if (rank == 0 && t == 0) {
    // sigma: final column j = stored column sigma[j], built by replaying the swaps in reverse
    int *cs = colSrc + 2 * bStart[b];
    for (int c = 0; c < M; c++) cs[c] = c;   // cs temporarily holds sigma
    for (int k = M - 1; k >= 0; k--) {
      const int pv = perm[k];
      if (pv != k) {
        const int a = cs[k];
        cs[k] = cs[pv];
        cs[pv] = a;
      }
    }
    // invert: colSrc[sigma[j]] = j
    for (int j = 0; j < M; j++) perm[cs[j]] = j;
    for (int c = 0; c < M; c++) cs[c] = perm[c];
    for (int c = 0; c < M; c++) rowDst[2 * bStart[b] + c] = c;
    info[b] = bad;
  }
  if (CS > 1) cooperative_groups::this_cluster().sync();   // no CTA leaves while others may still read
}

// x = blockdiag(inv) * b, block b gathers its pot/dpdn halves
// Block-diagonal apply with the explicit inverses, one thread block per tile
// of kPcRows rows of one diagonal block (tiles of large blocks spread over
// many SMs).  The block's inputs are gathered into shared memory (in chunks
// of kPcChunk columns); warp w sums the columns c = w mod kPcWarps, each lane
// kPcRpl consecutive rows (8- or 16-byte loads of the column-major inverse,
// eight columns in flight), and the warps' partial sums are added in a fixed
// order.  The reference's per-block solve order (x = [pot; dpdn]
// of the cube's panels) is src/precond_fmm.c:861-953.
#ifndef FB_PC_RPL
#define FB_PC_RPL 4
#endif
constexpr int kPcRpl = FB_PC_RPL;   // rows per lane (2 or 4)
constexpr int kPcRows = 32 * kPcRpl, kPcWarps = 8, kPcChunk = 2048;

// streams the block factorisations are spread over
#ifndef FB_PC_STREAMS
#define FB_PC_STREAMS 16
#endif

template <typename TI>
__global__ void __launch_bounds__(kPcWarps * 32)
pc_apply_kernel(int n, const int2 *__restrict__ tiles, const int *__restrict__ bStart, const int *__restrict__ bSize,
                const long long *__restrict__ bOff, const int *__restrict__ colSrc, const int *__restrict__ rowDst,
                const TI *__restrict__ inv, const double *__restrict__ rhs, double *x) {
  typedef typename Vec2<TI>::t V2;
  __shared__ double xs[kPcChunk];
  __shared__ double red[kPcWarps][kPcRows];
  const int2 tl = tiles[blockIdx.x];
  const int b = tl.x, r0 = tl.y;
  const int hm = bSize[b], st = bStart[b], M = 2 * hm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = r0 + kPcRpl * lane;   // M is even: rows r and r + 1 are both in or both out
  const TI *Ib = inv + bOff[b];
  const int *cs = colSrc + 2 * (size_t)st;
  double y0 = 0.0, y1 = 0.0, y2 = 0.0, y3 = 0.0;
  const bool q2 = kPcRpl == 4 && r + 2 < M;
  for (int k0 = 0; k0 < M; k0 += kPcChunk) {
    const int kn = min(kPcChunk, M - k0);
    __syncthreads();   // the previous chunk's reads are done
    for (int c = threadIdx.x; c < kn; c += blockDim.x) {
      const int g = cs[k0 + c];
      xs[c] = (g < hm) ? rhs[st + g] : rhs[n + st + g - hm];
    }
    __syncthreads();
    if (r < M) {
      const TI *col = Ib + (size_t)k0 * M + r;
      for (int c = warp; c < kn; c += 8 * kPcWarps) {
        V2 lo[8], hi[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
          if (c + u * kPcWarps < kn) {   // warp-uniform
            const V2 *src = reinterpret_cast<const V2 *>(col + (size_t)(c + u * kPcWarps) * M);
            lo[u] = src[0];
            if (kPcRpl == 4 && q2) hi[u] = src[1];
          }
#pragma unroll
        for (int u = 0; u < 8; u++)
          if (c + u * kPcWarps < kn) {
            const double xc = xs[c + u * kPcWarps];
            y0 += (double)lo[u].x * xc;
            y1 += (double)lo[u].y * xc;
            if (kPcRpl == 4 && q2) {
              y2 += (double)hi[u].x * xc;
              y3 += (double)hi[u].y * xc;
            }
          }
      }
    }
  }
  red[warp][kPcRpl * lane] = y0;
  red[warp][kPcRpl * lane + 1] = y1;
  if (kPcRpl == 4) {
    red[warp][kPcRpl * lane + 2] = y2;
    red[warp][kPcRpl * lane + 3] = y3;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kPcRows; i += blockDim.x) {
    const int rr = r0 + i;
    if (rr < M) {
      double t = red[0][i];
#pragma unroll
      for (int w = 1; w < kPcWarps; w++) t += red[w][i];
      const int g = rowDst[2 * (size_t)st + rr];
      if (g < hm) x[st + g] = t;
      else x[n + st + g - hm] = t;
    }
  }
}

// Transposed block-diagonal apply (adjoint solves): output c of a block is
// column c of its inverse dotted with the block's input.  Tiles of kPcRows
// outputs; the block's input is staged in shared memory in chunks, a warp takes
// four output columns at a time, each lane two consecutive rows per step.
template <typename TI>
__global__ void __launch_bounds__(kPcWarps * 32)
pc_apply_t_kernel(int n, const int2 *__restrict__ tiles, const int *__restrict__ bStart, const int *__restrict__ bSize,
                  const long long *__restrict__ bOff, const int *__restrict__ colSrc, const int *__restrict__ rowDst,
                  const TI *__restrict__ inv, const double *__restrict__ rhs, double *x) {
  typedef typename Vec2<TI>::t V2;
  __shared__ double xs[kPcChunk];
  const int2 tl = tiles[blockIdx.x];
  const int b = tl.x, c0 = tl.y;
  const int hm = bSize[b], st = bStart[b], M = 2 * hm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const TI *Ib = inv + bOff[b];
  constexpr int kCols = kPcRows / kPcWarps;   // output columns per warp
  double y[kCols];
#pragma unroll
  for (int q = 0; q < kCols; q++) y[q] = 0.0;
  for (int k0 = 0; k0 < M; k0 += kPcChunk) {
    const int kn = min(kPcChunk, M - k0);
    __syncthreads();
    for (int i = threadIdx.x; i < kn; i += blockDim.x) {
      const int g = rowDst[2 * (size_t)st + k0 + i];
      xs[i] = (g < hm) ? rhs[st + g] : rhs[n + st + g - hm];
    }
    __syncthreads();
    // four columns at a time: their loads overlap and share the staged input
#pragma unroll
    for (int q = 0; q < kCols; q += 4) {
      if (c0 + warp + q * kPcWarps >= M) break;   // warp-uniform
      const TI *col[4];
#pragma unroll
      for (int u = 0; u < 4; u++)   // (a column past the block: the last one again, dropped below)
        col[u] = Ib + (size_t)min(c0 + warp + (q + u) * kPcWarps, M - 1) * M + k0;
#pragma unroll 2
      for (int i = 2 * lane; i < kn; i += 64) {   // kn is even
        const double x0 = xs[i], x1 = xs[i + 1];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const V2 a = *reinterpret_cast<const V2 *>(col[u] + i);
          y[q + u] += (double)a.x * x0 + (double)a.y * x1;
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kCols; q++) {
    double v = y[q];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int c = c0 + warp + q * kPcWarps;
    if (lane == 0 && c < M) {
      const int g = colSrc[2 * (size_t)st + c];   // stored column c is output component g
      if (g < hm) x[st + g] = v;
      else x[n + st + g - hm] = v;
    }
  }
}

__global__ void pc_diag_kernel(int n, const double *__restrict__ area, double s1, double s2,
                               const double *__restrict__ b, double *x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  x[i] = b[i] / (s1 * area[i]);
  x[n + i] = b[n + i] / (s2 * area[i]);
}

// LU and explicit inverse of every block with cuSOLVER (blocks above the
// Gauss-Jordan kernel's size limit), spread over several streams so that
// independent blocks run side by side.  Inverts d_A into p.d_inv.
static bool factor_cusolver(Context &c, PrecondDev &p, const std::vector<int> &blocks) {
  cudaStream_t s = c.stream;
  if (blocks.empty()) return true;
  // copy the assembled blocks out of d_inv, which then starts as the identity
  std::vector<long long> aOff(p.nBlocks, -1);
  long long atot = 0;
  int maxM = 0;
  for (int b : blocks) {
    aOff[b] = atot;
    atot += 4LL * p.hSize[b] * p.hSize[b];
    maxM = std::max(maxM, 2 * p.hSize[b]);
  }
  double *d_A = nullptr;
  FB_CUDA(cudaMalloc((void **)&d_A, (size_t)atot * sizeof(double)));
  for (int b : blocks)
    FB_CUDA(cudaMemcpyAsync(d_A + aOff[b], p.d_inv + p.hOff[b], 4LL * p.hSize[b] * p.hSize[b] * sizeof(double),
                            cudaMemcpyDeviceToDevice, s));
  const int ns = std::min(FB_PC_STREAMS, std::max((int)blocks.size(), 1));
  std::vector<cusolverDnHandle_t> hs(ns, nullptr);
  std::vector<cudaStream_t> ss(ns, nullptr);
  std::vector<double *> works(ns, nullptr);
  std::vector<int *> pivs(ns, nullptr);
  int lwork = 0, *d_info = nullptr;
  int *d_list = nullptr;
  FB_CUDA(cudaMalloc((void **)&d_list, blocks.size() * sizeof(int)));
  FB_CUDA(cudaMemcpyAsync(d_list, blocks.data(), blocks.size() * sizeof(int), cudaMemcpyHostToDevice, s));
  dim3 grid(64, (unsigned)std::min<size_t>(blocks.size(), 65535));
  identity_kernel<<<grid, 256, 0, s>>>((int)blocks.size(), d_list, p.d_start, p.d_size, p.d_off, p.d_inv, p.d_colSrc,
                                  p.d_rowDst);
  cudaEvent_t evA = nullptr;
  bool ok = cudaEventCreateWithFlags(&evA, cudaEventDisableTiming) == cudaSuccess;
  ok = ok && cudaEventRecord(evA, s) == cudaSuccess;
  for (int k = 0; ok && k < ns; k++) {
    ok = cudaStreamCreateWithFlags(&ss[k], cudaStreamNonBlocking) == cudaSuccess &&
         cusolverDnCreate(&hs[k]) == CUSOLVER_STATUS_SUCCESS && cusolverDnSetStream(hs[k], ss[k]) == CUSOLVER_STATUS_SUCCESS &&
         cudaStreamWaitEvent(ss[k], evA, 0) == cudaSuccess;
  }
  if (ok && cusolverDnDgetrf_bufferSize(hs[0], maxM, maxM, d_A, maxM, &lwork) != CUSOLVER_STATUS_SUCCESS) ok = false;
  for (int k = 0; ok && k < ns; k++)
    ok = cudaMalloc((void **)&works[k], (size_t)std::max(lwork, 1) * sizeof(double)) == cudaSuccess &&
         cudaMalloc((void **)&pivs[k], (size_t)maxM * sizeof(int)) == cudaSuccess;
  ok = ok && cudaMalloc((void **)&d_info, (size_t)p.nBlocks * sizeof(int)) == cudaSuccess;
  ok = ok && cudaMemsetAsync(d_info, 0, (size_t)p.nBlocks * sizeof(int), s) == cudaSuccess;
  std::vector<int> order(blocks);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return p.hSize[a] > p.hSize[b]; });
  for (int q = 0; ok && q < (int)order.size(); q++) {
    const int b = order[q], k = q % ns;
    int M = 2 * p.hSize[b];
    if (M == 0) continue;
    double *Ab = d_A + aOff[b], *Ib = p.d_inv + p.hOff[b];
    if (cusolverDnDgetrf(hs[k], M, M, Ab, M, works[k], pivs[k], d_info + b) != CUSOLVER_STATUS_SUCCESS) ok = false;
    if (ok && cusolverDnDgetrs(hs[k], CUBLAS_OP_N, M, M, Ab, M, pivs[k], Ib, M, d_info + b) != CUSOLVER_STATUS_SUCCESS)
      ok = false;
  }
  for (int k = 0; k < ns; k++) {
    if (!ss[k]) continue;
    cudaEvent_t ev = nullptr;
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) == cudaSuccess) {
      cudaEventRecord(ev, ss[k]);
      cudaStreamWaitEvent(s, ev, 0);
      cudaEventDestroy(ev);
    } else {
      ok = false;
    }
  }
  std::vector<int> info(p.nBlocks, 0);
  if (ok) ok = cudaMemcpyAsync(info.data(), d_info, info.size() * sizeof(int), cudaMemcpyDeviceToHost, s) == cudaSuccess;
  if (ok) ok = cudaStreamSynchronize(s) == cudaSuccess;
  for (int k = 0; k < ns; k++) {
    if (ss[k]) cudaStreamSynchronize(ss[k]);
    if (hs[k]) cusolverDnDestroy(hs[k]);
    if (ss[k]) cudaStreamDestroy(ss[k]);
    cudaFree(works[k]);
    cudaFree(pivs[k]);
  }
  if (evA) cudaEventDestroy(evA);
  cudaFree(d_info);
  cudaFree(d_list);
  cudaFree(d_A);
  FB_CHECK(ok, "preconditioner factorisation failed: %s", cudaGetErrorString(cudaGetLastError()));
  for (int b = 0; b < p.nBlocks; b++)
    FB_CHECK(info[b] == 0, "dgetrf failed in preconditioner block %d (info=%d)", b, info[b]);
  return true;
}

// Blocks up to this many rows (and up to the size classes below) go to the
// Gauss-Jordan kernel; larger ones to cuSOLVER (several streams, FP64 only).
// Measured on the 204,800-panel star surface, sending everything to the
// kernel is fastest (cuSOLVER launches run slowly beside the kernel's
// resident blocks).
#ifndef FB_PC_GJ_MAXM
#define FB_PC_GJ_MAXM 11000
#endif
template <typename TV, int NB, int CS>
static bool launch_gj_t(int nList, int maxM, cudaStream_t st, const int *d_list, PrecondDev &p, const long long *d_yOff,
                        TV *inv, TV *d_y, int *d_info) {
  const size_t shm = gj_smem_bytes<TV, NB>(maxM);
  cudaFuncAttributes fa{};
  FB_CUDA(cudaFuncGetAttributes(&fa, pc_gj_invert_kernel<TV, NB, CS>));
  int dev = 0, optin = 0;
  FB_CUDA(cudaGetDevice(&dev));
  FB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  FB_CHECK(shm + fa.sharedSizeBytes <= (size_t)optin,
           "Gauss-Jordan class NB=%d: %d rows need %zu + %zu bytes of shared memory, above the %d available", NB,
           maxM, shm, (size_t)fa.sharedSizeBytes, optin);
  // (the same value every time: another thread's set-up may come between this and the launch)
  FB_CUDA(cudaFuncSetAttribute(pc_gj_invert_kernel<TV, NB, CS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               optin - (int)fa.sharedSizeBytes));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nList * CS));
  cfg.blockDim = dim3(kGjThreads);
  cfg.dynamicSmemBytes = shm;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  FB_CUDA(cudaLaunchKernelEx(&cfg, pc_gj_invert_kernel<TV, NB, CS>, d_list, (const int *)p.d_start,
                             (const int *)p.d_size, (const long long *)p.d_off, d_yOff, inv, d_y, p.d_colSrc,
                             p.d_rowDst, d_info));
  return true;
}

template <typename TV>
static bool launch_gj(int nb, int nList, int maxM, cudaStream_t st, const int *d_list, PrecondDev &p,
                      const long long *d_yOff, TV *inv, TV *d_y, int *d_info) {
  if constexpr (sizeof(TV) == 4) {
    if (nb == 16) return launch_gj_t<TV, 16, 8>(nList, maxM, st, d_list, p, d_yOff, inv, d_y, d_info);
    if (nb == 4) return launch_gj_t<TV, 4, 8>(nList, maxM, st, d_list, p, d_yOff, inv, d_y, d_info);
  }
  return launch_gj_t<TV, 8, 8>(nList, maxM, st, d_list, p, d_yOff, inv, d_y, d_info);
}

template <typename TV, int NB, int CS, int RPT, int QC, int NT>
static bool launch_inv_t(int nList, int maxM, cudaStream_t st, const int *d_list, PrecondDev &p, TV *inv,
                         int *d_info, bool share) {
  FB_CHECK(maxM <= RPT * NT, "inversion class of %d rows given %d", RPT * NT, maxM);
  const size_t shm = inv_smem_bytes<TV, NB, QC>(maxM);
  // (the same value every time: another thread's set-up may come between this and the launch)
  FB_CUDA(cudaFuncSetAttribute(pc_invert_kernel<TV, NB, CS, RPT, QC, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)inv_smem_bytes<TV, NB, QC>(RPT * NT)));
  FB_CUDA(cudaFuncSetAttribute(pc_invert_kernel<TV, NB, CS, RPT, QC, NT>,
                               cudaFuncAttributePreferredSharedMemoryCarveout,
                               share ? cudaSharedmemCarveoutMaxShared : cudaSharedmemCarveoutDefault));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nList * CS));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = shm;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  FB_CUDA(cudaLaunchKernelEx(&cfg, pc_invert_kernel<TV, NB, CS, RPT, QC, NT>, d_list, (const int *)p.d_start,
                             (const int *)p.d_size, (const long long *)p.d_off, inv, p.d_colSrc, p.d_rowDst,
                             d_info));
  return true;
}

// Size classes per precision.  Blocks of up to 1,536 rows go to
// pc_invert_kernel on one, two or four CTAs of 256 threads, two per SM, so that
// one's pivots hide behind the other's updates (FP64 above 768 rows: 512
// threads, one per SM); larger ones to pc_gj_invert_kernel; blocks above the
// last class go to cuSOLVER (FP64).  FP32, 422 blocks of 385 to 768 rows: 11.7
// ms on two CTAs, 14.6 on four, 21.9 on eight (each CTA repeats the pivots),
// 13.7 with 512 threads; 91 blocks of 769 to 1,226 rows, panels of 16: 15.0 ms
// on four, 21.7 on two, 18.1 on eight; panels of 32: 15.7 and more (one CTA per
// SM).  FP64, the same 91: 37.4 ms, 53 on eight; but eight where four a block
// would leave SMs idle (8 blocks of up to 1,192 rows: 18.2 ms on four, 11.7 on
// eight; 28 of up to 1,474: 33 and 22).
constexpr int kSms = 148;
static bool wide_clusters(int nList) { return nList * 4 <= kSms; }   // FP64 blocks of 769 to 1,536 rows
struct InvClass { int hi, nb, cs; };   // rows up to, panel width, CTAs per block
template <typename TV>
static const InvClass *inv_classes(int *count) {
  // FP64 stops at 3200 rows: above it cuSOLVER's factorisation of a single
  // large block (all SMs) beats the kernel's narrow panels (measured on a
  // 2.1M-panel surface: 7.9 s against 9.8 s for the whole inversion)
  static const InvClass d64[4] = {{384, 16, 1}, {768, 16, 2}, {1536, 16, 4}, {3200, 8, 8}};
  static const InvClass d32[6] = {{384, 32, 1}, {768, 32, 2}, {1536, 16, 4}, {3200, 16, 8}, {6000, 8, 8}, {11000, 4, 8}};
  *count = sizeof(TV) == 8 ? 4 : 6;
  return sizeof(TV) == 8 ? d64 : d32;
}

template <typename TV>
static bool launch_inversion(int ci, int nb, int nList, int maxM, cudaStream_t st, const int *d_list, PrecondDev &p,
                             const long long *d_yOff, TV *inv, TV *d_y, int *d_info, bool share) {
  constexpr bool f = sizeof(TV) == 4;
  if (ci == 0) return launch_inv_t<TV, f ? 32 : 16, 1, 2, 1, 256>(nList, maxM, st, d_list, p, inv, d_info, share);
  if (ci == 1) return launch_inv_t<TV, f ? 32 : 16, 2, 3, 1, 256>(nList, maxM, st, d_list, p, inv, d_info, share);
  if constexpr (!f) {
    if (ci == 2 && wide_clusters(nList)) return launch_inv_t<TV, 16, 8, 3, 1, 512>(nList, maxM, st, d_list, p, inv, d_info, share);
  }
  if (ci == 2) return launch_inv_t<TV, 16, 4, f ? 6 : 3, 1, f ? 256 : 512>(nList, maxM, st, d_list, p, inv, d_info, share);
  return launch_gj<TV>(nb, nList, maxM, st, d_list, p, d_yOff, inv, d_y, d_info);
}

template <typename TV>
static int gj_max_rows() {
  int n = 0;
  const InvClass *c = inv_classes<TV>(&n);
  return std::min(c[n - 1].hi, FB_PC_GJ_MAXM);
}

// about 20 us
__global__ void pause_kernel() {
  for (int i = 0; i < 20; i++) __nanosleep(1000);
}

// Gauss-Jordan inversion of every block of inv (assembled there), class by
// class; blocks above the kernels' size limit (FP64 only) go to cuSOLVER.
template <typename TV>
static bool factor_gauss_jordan(Context &c, PrecondDev &p, TV *inv) {
  cudaStream_t s = c.stream;
  const int cut = gj_max_rows<TV>();
  int ncls = 0;
  const InvClass *cls = inv_classes<TV>(&ncls);
  std::vector<int> big;
  for (int b = 0; b < p.nBlocks; b++)
    if (2 * p.hSize[b] > cut) big.push_back(b);
  FB_CHECK(big.empty() || sizeof(TV) == 8, "preconditioner block of %d rows above the FP32 limit %d", p.maxM, cut);
  std::vector<long long> yOff(p.nBlocks);
  long long ytot = 0;
  for (int b = 0; b < p.nBlocks; b++) {
    yOff[b] = ytot;
    if (2 * p.hSize[b] > cls[2].hi) ytot += 16LL * 2 * p.hSize[b];   // only pc_gj_invert_kernel uses it
  }
  long long *d_yOff = nullptr;
  TV *d_y = nullptr;
  int *d_info = nullptr;
  DevArena tmp;
  if (!tmp.upload(&d_yOff, yOff, s) || !tmp.alloc_n(&d_y, (size_t)std::max(ytot, 1LL)) ||
      !tmp.alloc_n(&d_info, (size_t)p.nBlocks))
    return false;
  FB_CUDA(cudaMemsetAsync(d_info, 0, (size_t)p.nBlocks * sizeof(int), s));
  struct Job {
    int ci, maxM = 0;
    std::vector<int> list;
    int *d_list = nullptr;
  };
  std::vector<Job> jobs;   // the classes with blocks, the largest blocks first
  for (int ci = ncls - 1; ci >= 0; ci--) {
    const int lo = ci ? cls[ci - 1].hi : 0, hi = std::min(cls[ci].hi, cut);
    Job j{ci};
    for (int b = 0; b < p.nBlocks; b++) {
      const int M = 2 * p.hSize[b];
      if (hi > lo && M > lo && M <= hi) {
        j.list.push_back(b);
        j.maxM = std::max(j.maxM, M);
      }
    }
    if (j.list.empty()) continue;
    std::stable_sort(j.list.begin(), j.list.end(), [&](int a, int b) { return p.hSize[a] > p.hSize[b]; });
    jobs.push_back(std::move(j));
  }
  bool ok = true;
  for (Job &j : jobs) ok = ok && tmp.upload(&j.d_list, j.list, s);
  // The classes run side by side, the largest blocks' clusters placed first, on the context's other streams (its own is
  // left to cuSOLVER when there are blocks for it): a class alone leaves SMs idle, when it has few blocks and at its
  // end.  FP64, 263 blocks of up to 996 rows: 23.4 ms in turn, 11.3 side by side; FP64, 55 of up to 1,100: 26.8 and
  // 16.4; FP32, three stars of 1,100 blocks: 61.8, 37.8 and 28.9 in turn, 30.0, 29.9 and 26.3.
  const bool fork = jobs.size() > 1 || !big.empty();
  cudaStream_t lane[3] = {c.farStream, c.sideStream, big.empty() ? s : c.sideStream};
  if (fork)
    ok = ok && cudaEventRecord(c.evFork, s) == cudaSuccess && cudaStreamWaitEvent(lane[0], c.evFork, 0) == cudaSuccess &&
         cudaStreamWaitEvent(lane[1], c.evFork, 0) == cudaSuccess;
  // Classes whose CTAs outnumber the SMs share them, which blocks of two kernels on an SM can only if its shared memory
  // need not be divided anew: all ask for the largest share then.  (The 263 blocks: 16.4 ms without, 11.3 with it.
  // But 8 FP32 blocks of up to 1,192 rows with the smaller L1 9.8 -> 10.4.)
  long long ctas = 0;
  for (const Job &j : jobs) ctas += (long long)j.list.size() * cls[j.ci].cs;
  const bool share = jobs.size() > 1 && ctas > kSms;
  for (size_t k = 0; ok && k < jobs.size(); k++) {
    const Job &j = jobs[k];
    cudaStream_t st = fork ? lane[std::min<size_t>(k, 2)] : s;
    // the next class starts after this one: its event comes before this launch, and a pause holds it back until this
    // one's clusters have their SMs (without it smaller blocks can take them first: FP64, 1,100 blocks in three classes
    // 13.5 ms without it, 10.6 with it; the first star 41 and 29.9)
    if (k > 0) {
      ok = ok && cudaStreamWaitEvent(st, c.evJoin, 0) == cudaSuccess;
      if (ok) pause_kernel<<<1, 1, 0, st>>>();
      c.launches += 1;
    }
    if (fork) ok = ok && cudaEventRecord(c.evJoin, st) == cudaSuccess;
    ok = ok && launch_inversion<TV>(j.ci, cls[j.ci].nb, (int)j.list.size(), j.maxM, st, j.d_list, p, d_yOff, inv, d_y,
                                    d_info, share);
    c.launches += 1;
    ok = ok && cudaGetLastError() == cudaSuccess;
  }
  // the large blocks meanwhile, through cuSOLVER on its own streams
  if (ok && !big.empty()) {
    if constexpr (sizeof(TV) == 8) ok = factor_cusolver(c, p, big);
  }
  for (int k = 0; fork && k < 2; k++)
    if (cudaEventRecord(c.evJoin, lane[k]) != cudaSuccess || cudaStreamWaitEvent(s, c.evJoin, 0) != cudaSuccess) ok = false;
  std::vector<int> info(p.nBlocks, 0);
  if (ok) ok = cudaMemcpyAsync(info.data(), d_info, info.size() * sizeof(int), cudaMemcpyDeviceToHost, s) == cudaSuccess;
  if (ok) ok = cudaStreamSynchronize(s) == cudaSuccess;
  tmp.release();
  FB_CHECK(ok, "preconditioner inversion failed: %s", cudaGetErrorString(cudaGetLastError()));
  for (int b = 0; b < p.nBlocks; b++)
    FB_CHECK(info[b] == 0, "zero or non-finite pivot in preconditioner block %d (step %d)", b, info[b]);
  return true;
}

static bool setup_blocks(Context &c) {
  PrecondDev &p = *c.pc;
  const Octree &t = c.pt.t;
  const int lev = t.depth - 1;
  FB_CHECK(lev >= 0, "block preconditioner needs depth >= 1");
  long long off = 0;
  for (int cc = t.levStart[lev]; cc < t.levStart[lev + 1]; cc++) {
    int hm = t.itemCount[cc];
    p.hStart.push_back(t.itemStart[cc]);
    p.hSize.push_back(hm);
    p.hOff.push_back(off);
    off += 4LL * hm * hm;
    p.maxM = std::max(p.maxM, 2 * hm);
  }
  p.nBlocks = (int)p.hSize.size();
  // apply tiles, the largest blocks' first (a tile's cost grows with its block's size)
  std::vector<int> order(p.nBlocks);
  for (int b = 0; b < p.nBlocks; b++) order[b] = b;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return p.hSize[a] > p.hSize[b]; });
  std::vector<int2> tiles;
  for (int b : order)
    for (int r0 = 0; r0 < 2 * p.hSize[b]; r0 += kPcRows) tiles.push_back(make_int2(b, r0));
  p.nTiles = (int)tiles.size();
  FB_CHECK(p.maxM <= 46340, "preconditioner block %d too large (increase -t)", p.maxM);
  cudaStream_t s = c.stream;
  StageTimer tm("precond_setup", s);
  if (!p.arena.upload(&p.d_start, p.hStart, s) || !p.arena.upload(&p.d_size, p.hSize, s) ||
      !p.arena.upload(&p.d_tiles, tiles, s) || !p.arena.upload(&p.d_off, p.hOff, s) ||
      !p.arena.alloc_n(&p.d_colSrc, 2 * (size_t)c.n) || !p.arena.alloc_n(&p.d_rowDst, 2 * (size_t)c.n))
    return false;
  // FP64 contexts invert in FP64; mixed contexts assemble and invert in FP32
  // (the preconditioner only steers GMRES; its inverse is stored in FP32)
  const double s1 = (1.0 + c.epsilon) / 2.0, s2 = (1.0 + 1.0 / c.epsilon) / 2.0;
  dim3 grid(64, std::min(p.nBlocks, 65535));
  bool ok;
  if (c.mixed) {
    FB_CHECK(p.maxM <= gj_max_rows<float>(), "preconditioner block of %d rows above the FP32 limit %d", p.maxM,
             gj_max_rows<float>());
    if (!p.arena.alloc_n(&p.d_invF, (size_t)off)) return false;
    pc_onepoint_kernel<float><<<grid, 128, 0, s>>>(p.nBlocks, p.d_start, p.d_size, p.d_off, c.d_vtx, c.d_nrm,
                                                   c.d_area, c.prm.kappa, c.epsilon, s1, s2, p.d_invF);
    pc_special_kernel<float><<<dim3(4, grid.y), 128, 0, s>>>(p.nBlocks, p.d_start, p.d_size, p.d_off, c.d_spOff,
                                                             c.d_spSrc, c.d_spK, p.d_invF);
    c.launches += 2;
    FB_CUDA(cudaGetLastError());
    tm.mark("assemble");
    ok = factor_gauss_jordan<float>(c, p, p.d_invF);
  } else {
    if (!p.arena.alloc_n(&p.d_inv, (size_t)off)) return false;
    pc_onepoint_kernel<double><<<grid, 128, 0, s>>>(p.nBlocks, p.d_start, p.d_size, p.d_off, c.d_vtx, c.d_nrm,
                                                    c.d_area, c.prm.kappa, c.epsilon, s1, s2, p.d_inv);
    pc_special_kernel<double><<<dim3(4, grid.y), 128, 0, s>>>(p.nBlocks, p.d_start, p.d_size, p.d_off, c.d_spOff,
                                                              c.d_spSrc, c.d_spK, p.d_inv);
    c.launches += 2;
    FB_CUDA(cudaGetLastError());
    tm.mark("assemble");
    ok = factor_gauss_jordan<double>(c, p, p.d_inv);
  }
  tm.mark("factor_invert");
  return ok;
}

bool precond_setup(Context &c, int mode) {
  free_precond(c);
  c.pc = new PrecondDev();
  c.pc->mode = mode;   // -1 identity and 3 diagonal need no setup
  if (mode != 2 || setup_blocks(c)) return true;
  free_precond(c);   // no half-built inverse for a later call
  return false;
}

bool precond_apply(Context &c, const double *b, double *x, bool adjoint) {
  FB_CHECK(c.pc != nullptr, "preconditioner not set up");
  PrecondDev &p = *c.pc;
  if (p.mode == 2 && adjoint) {
    if (p.d_invF)
      pc_apply_t_kernel<float><<<p.nTiles, kPcWarps * 32, 0, c.stream>>>(c.n, p.d_tiles, p.d_start, p.d_size,
                                                                             p.d_off, p.d_colSrc, p.d_rowDst, p.d_invF, b, x);
    else
      pc_apply_t_kernel<double><<<p.nTiles, kPcWarps * 32, 0, c.stream>>>(c.n, p.d_tiles, p.d_start, p.d_size,
                                                                              p.d_off, p.d_colSrc, p.d_rowDst, p.d_inv, b, x);
  } else if (p.mode == 2) {
    if (p.d_invF)
      pc_apply_kernel<float><<<p.nTiles, kPcWarps * 32, 0, c.stream>>>(c.n, p.d_tiles, p.d_start, p.d_size,
                                                                           p.d_off, p.d_colSrc, p.d_rowDst, p.d_invF, b, x);
    else
      pc_apply_kernel<double><<<p.nTiles, kPcWarps * 32, 0, c.stream>>>(c.n, p.d_tiles, p.d_start, p.d_size,
                                                                             p.d_off, p.d_colSrc, p.d_rowDst, p.d_inv, b, x);
  } else if (p.mode == 3) {
    pc_diag_kernel<<<ceil_div(c.n, 256), 256, 0, c.stream>>>(c.n, c.d_area, (1.0 + c.epsilon) / 2.0,
                                                            (1.0 + 1.0 / c.epsilon) / 2.0, b, x);
  } else {
    FB_CUDA(cudaMemcpyAsync(x, b, 2 * (size_t)c.n * sizeof(double), cudaMemcpyDeviceToDevice, c.stream));
    return true;
  }
  c.launches += 1;
  FB_CUDA(cudaGetLastError());
  return true;
}

// ---------------------------------------------------------------------------
// level-1 kernels with deterministic reductions
// ---------------------------------------------------------------------------
constexpr int kRedBlocks = 296;   // 2 x 148 SMs
constexpr int kRedThreads = 256;

// part[b] = sum over the block's grid-stride share of x.*y
__global__ void dot_partial_kernel(long long n, const double *__restrict__ x, const double *__restrict__ y,
                                   double *part) {
  __shared__ double red[kRedThreads];
  double s = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    s += x[i] * y[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if ((int)threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// out[0] = sum(part) (or sqrt of it), fixed order
__global__ void dot_final_kernel(int k, const double *__restrict__ part, double *out, int takeSqrt) {
  __shared__ double red[kRedThreads];
  double s = 0.0;
  for (int i = threadIdx.x; i < k; i += blockDim.x) s += part[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int m = blockDim.x / 2; m > 0; m >>= 1) {
    if ((int)threadIdx.x < m) red[threadIdx.x] += red[threadIdx.x + m];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = takeSqrt ? sqrt(red[0]) : red[0];
}

// y -= (*h) * x
__global__ void axpy_neg_dev_kernel(long long n, const double *__restrict__ h, const double *__restrict__ x, double *y) {
  const double a = -(*h);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] += a * x[i];
}

// v = w / (*h) when *h > 0, else v = w
__global__ void scale_copy_dev_kernel(long long n, const double *__restrict__ h, const double *__restrict__ w, double *v) {
  const double d = *h;
  const double s = (d > 0.0) ? 1.0 / d : 1.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    v[i] = (d > 0.0) ? w[i] * s : w[i];
}

__global__ void scale_copy_kernel(long long n, double s, const double *__restrict__ w, double *v) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    v[i] = w[i] * s;
}

// x += V y  (k columns of length n, column stride ldv)
__global__ void update_kernel(long long n, int k, const double *__restrict__ V, long long ldv,
                              const double *__restrict__ y, double *x) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double s = x[i];
    for (int j = 0; j < k; j++) s += y[j] * V[(size_t)j * ldv + i];
    x[i] = s;
  }
}

// Sum of kRedBlocks partials in a fixed order (the dot_final_kernel order),
// by every thread block alike; returns the total to all threads.
__device__ __forceinline__ double block_sum_partials(const double *__restrict__ part, double *red) {
  double s = 0.0;
  for (int i = threadIdx.x; i < kRedBlocks; i += blockDim.x) s += part[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int m = blockDim.x / 2; m > 0; m >>= 1) {
    if ((int)threadIdx.x < m) red[threadIdx.x] += red[threadIdx.x + m];
    __syncthreads();
  }
  const double t = red[0];
  __syncthreads();
  return t;
}

__device__ __forceinline__ void block_store_partial(double acc, double *red, double *partOut) {
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int m = blockDim.x / 2; m > 0; m >>= 1) {
    if ((int)threadIdx.x < m) red[threadIdx.x] += red[threadIdx.x + m];
    __syncthreads();
  }
  if (threadIdx.x == 0) partOut[blockIdx.x] = red[0];
}

// Modified Gram-Schmidt of one Arnoldi step (gmres.c's ddot + daxpy pairs) in
// two passes over the basis whatever its length.  MGS takes h_k = v_k.(w -
// sum_{j<k} h_j v_j); with the products c_k = v_k.w and the basis' own Gram
// entries L_kj = v_k.v_j (j < k; rounding-sized, kept for the cycle) that is the
// triangular solve (I + L) h = c, the one-reduction form of MGS of Swirydowicz,
// Langou, Ananthan, Yang and Thomas (Numer. Linear Algebra Appl. 28, 2021).
// gs_dots_kernel takes all products at once (and the newest column's Gram row),
// gs_update_kernel solves and subtracts, mgs_norm_scale_kernel normalises and
// takes the Givens step: three launches per step (four above kGsStage columns,
// where gs_solve_kernel solves).  One launch per column
// took 5.3 us each (20,000 panels: 529 us for the 19 steps of two solves); these
// take 4.6, 4.7 and 5.0 us (271 us).
constexpr int kGsCols = 8;   // columns per pass over w in gs_dots_kernel

// the sum of one product's partials, in a fixed order, in every lane
__device__ __forceinline__ double warp_sum_partials(const double *__restrict__ part, int lane) {
  double s = 0.0;
  for (int b = lane; b < kRedBlocks; b += 32) s += part[b];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// part[k][block] = partial of w.v_k (k < i), part[i + k][block] = partial of v_{i-1}.v_k (k < i - 1)
__global__ void __launch_bounds__(kRedThreads)
gs_dots_kernel(long long n, int i, const double *__restrict__ V, const double *__restrict__ w, double *part) {
  __shared__ double red[2 * kGsCols][kRedThreads / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double *last = V + (size_t)(i - 1) * n;
  for (int k0 = 0; k0 < i; k0 += kGsCols) {
    double c[kGsCols], g[kGsCols];
#pragma unroll
    for (int q = 0; q < kGsCols; q++) c[q] = g[q] = 0.0;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
      const double we = w[e], le = last[e];
#pragma unroll
      for (int q = 0; q < kGsCols; q++)
        if (k0 + q < i) {   // uniform
          const double v = V[(size_t)(k0 + q) * n + e];
          c[q] += we * v;
          g[q] += le * v;
        }
    }
    __syncthreads();   // the previous columns' sums are read
#pragma unroll
    for (int q = 0; q < kGsCols; q++) {
      for (int o = 16; o > 0; o >>= 1) {
        c[q] += __shfl_xor_sync(0xffffffffu, c[q], o);
        g[q] += __shfl_xor_sync(0xffffffffu, g[q], o);
      }
      if (lane == 0) {
        red[q][warp] = c[q];
        red[kGsCols + q][warp] = g[q];
      }
    }
    __syncthreads();
    if (threadIdx.x < 2 * kGsCols) {
      const int q = threadIdx.x % kGsCols, gram = threadIdx.x / kGsCols;
      if (k0 + q < i - gram) {
        double s = 0.0;
        for (int v = 0; v < kRedThreads / 32; v++) s += red[threadIdx.x][v];
        part[(size_t)(gram * i + k0 + q) * gridDim.x + blockIdx.x] = s;
      }
    }
  }
}

// every block: the sums of the partials in the same order, h from (I + L) h = c (block 0 stores h and the newest Gram
// row), its share of w -= V h and the partial of w.w.  SOLVE: up to kGsStage columns, whose Gram rows every block holds
// in gs_smem(i) bytes of dynamic shared memory; above, gs_solve_kernel has formed h and the Gram row.
constexpr int kGsStage = 64;
static size_t gs_smem(int i) { return i <= kGsStage ? sizeof(double) * i * (i + 1) : 0; }
template <bool SOLVE>
__global__ void __launch_bounds__(kRedThreads)
gs_update_kernel(long long n, int i, int ldg, const double *__restrict__ V, const double *__restrict__ part,
                 double *G, double *hOut, double *w, double *partOut) {
  extern __shared__ double gsSmem[];
  __shared__ double red[kRedThreads];
  const double *h = hOut;
  if constexpr (SOLVE) {
    double *c = gsSmem, *row = gsSmem + i, *L = row + i;   // [i], the newest Gram row, the others [i - 1][i] (row k: j < k)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int e = threadIdx.x; e < (i - 1) * i; e += blockDim.x) {
      const int k = e / i, j = e % i;
      if (j < k) L[e] = G[(size_t)k * ldg + j];
    }
    for (int q = warp; q < 2 * i - 1; q += kRedThreads / 32) {
      const double s = warp_sum_partials(part + (size_t)q * kRedBlocks, lane);
      if (lane == 0) (q < i ? c[q] : row[q - i]) = s;
    }
    __syncthreads();
    if (warp == 0)   // forward substitution, column by column
      for (int k = 0; k < i; k++) {
        const double hk = c[k];
        for (int j = k + 1 + lane; j < i; j += 32) c[j] -= hk * (j == i - 1 ? row[k] : L[j * i + k]);
        __syncwarp();
      }
    __syncthreads();
    if (blockIdx.x == 0)
      for (int k = threadIdx.x; k < i; k += blockDim.x) {
        hOut[k] = c[k];
        if (k < i - 1) G[(size_t)(i - 1) * ldg + k] = row[k];
      }
    h = c;
  }
  double acc = 0.0;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    double we = w[e];
#pragma unroll 8
    for (int k = 0; k < i; k++) we -= h[k] * V[(size_t)k * n + e];
    w[e] = we;
    acc += we * we;
  }
  block_store_partial(acc, red, partOut);
}

// h and the newest Gram row of a step with more than kGsStage columns, any number of them, by one block, 32 rows of
// (I + L) h = c at a time: a warp per row sums the columns solved before, then one warp solves the triangle of 32.
// Bound by the latency of i / 32 dependent rounds.  (1,568 panels, a step's mean time in a cycle of 200, 1,000 and
// 2,000 columns: 554, 2,505 and 4,874 us with a launch per column, 179, 1,316 and 5,530 with every block of the update
// solving for itself from global memory, 158, 486 and 1,015 so.)
constexpr int kGsRows = 32;
__global__ void __launch_bounds__(kGsRows * 32)
gs_solve_kernel(int i, int ldg, const double *__restrict__ part, double *G, double *h) {
  __shared__ double rest[kGsRows];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *row = G + (size_t)(i - 1) * ldg;
  for (int q = warp; q < 2 * i - 1; q += kGsRows) {
    const double s = warp_sum_partials(part + (size_t)q * kRedBlocks, lane);
    if (lane == 0) (q < i ? h[q] : row[q - i]) = s;
  }
  __syncthreads();
  for (int k0 = 0; k0 < i; k0 += kGsRows) {
    const int k = k0 + warp;
    if (k < i) {   // warp-uniform
      double s = 0.0;
#pragma unroll 4
      for (int j = lane; j < k0; j += 32) s += G[(size_t)k * ldg + j] * h[j];
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) rest[warp] = h[k] - s;
    }
    __syncthreads();
    if (warp == 0) {
      const int m = min(kGsRows, i - k0);
      const double *Lr = G + (size_t)(k0 + min(lane, m - 1)) * ldg + k0;   // this lane's row
      double x = lane < m ? rest[lane] : 0.0;
      for (int j = 0; j < m; j++) {
        const double hj = __shfl_sync(0xffffffffu, x, j);
        if (lane > j && lane < m) x -= Lr[j] * hj;
      }
      if (lane < m) h[k0 + lane] = x;
    }
    __syncthreads();
  }
}

static bool dot_dev(Context &c, long long n, const double *x, const double *y, double *out, bool sq) {
  PrecondDev &p = *c.pc;
  dot_partial_kernel<<<kRedBlocks, kRedThreads, 0, c.stream>>>(n, x, y, p.d_part);
  dot_final_kernel<<<1, kRedThreads, 0, c.stream>>>(kRedBlocks, p.d_part, out, sq ? 1 : 0);
  c.launches += 2;
  FB_CUDA(cudaGetLastError());
  return true;
}

// x . y to the host (fixed-order reduction); needs a preconditioner record
// for its scratch
bool dot_to_host(Context &c, long long n, const double *x, const double *y, double *out) {
  FB_CHECK(c.pc != nullptr, "dot_to_host without a preconditioner record");
  PrecondDev &p = *c.pc;
  if (!p.d_part && !p.arena.alloc_n(&p.d_part, 2 * (size_t)kRedBlocks + 2)) return false;
  if (!dot_dev(c, n, x, y, p.d_part + kRedBlocks, false)) return false;
  FB_CUDA(cudaMemcpyAsync(out, p.d_part + kRedBlocks, sizeof(double), cudaMemcpyDeviceToHost, c.stream));
  FB_CUDA(cudaStreamSynchronize(c.stream));
  return true;
}

// ---------------------------------------------------------------------------
// GMRES state on the device.  The Hessenberg matrix, the Givens rotations
// (cs, sn), the rotated residual vector s and the residual estimate live in
// device memory; one single-warp kernel per Arnoldi step applies the previous
// rotations to the new column, forms the next rotation (netlib drotg, the
// BLAS the reference calls at src/gmres.c:281-293), rotates s and decides
// whether the cycle ends.  The host reads back only the small GmresStatus
// record (pinned) after each step, to know whether to queue another one; the
// triangular solve and the x update of src/gmres.c:364-373 are kernels too.
// Every product and sum of the rotations is rounded separately (no fused
// multiply-add), as the reference's BLAS calls compute them.
// ---------------------------------------------------------------------------
struct GmresStatus {
  double resid;   // |s_i| / ||b|| after the last step, or the restart residual
  double rnorm;   // norm of the preconditioned residual at the cycle start
  int i;          // columns of the current cycle
  int iters;      // Arnoldi steps so far
  int state;      // 0 running, 1 converged, 2 cycle full (i == restart or iters == maxit), 3 zero/NaN residual
  int pad;
};

__device__ __forceinline__ void drot_d(double *x, double *y, double cc, double ss) {
  const double xv = *x, yv = *y;
  *x = __dadd_rn(__dmul_rn(cc, xv), __dmul_rn(ss, yv));
  *y = __dsub_rn(__dmul_rn(cc, yv), __dmul_rn(ss, xv));
}

__device__ void drotg_d(double *a, double *b, double *cc, double *ss) {
  const double aa = *a, bb = *b;
  const double roe = (fabs(aa) > fabs(bb)) ? aa : bb;
  const double scale = __dadd_rn(fabs(aa), fabs(bb));
  double r, z;
  if (scale == 0.0) {
    *cc = 1.0; *ss = 0.0; r = 0.0; z = 0.0;
  } else {
    const double ua = __ddiv_rn(aa, scale), ub = __ddiv_rn(bb, scale);
    r = __dmul_rn(scale, __dsqrt_rn(__dadd_rn(__dmul_rn(ua, ua), __dmul_rn(ub, ub))));
    if (roe < 0.0) r = -r;
    *cc = __ddiv_rn(aa, r);
    *ss = __ddiv_rn(bb, r);
    z = 1.0;
    if (fabs(aa) > fabs(bb)) z = *ss;
    if (fabs(bb) >= fabs(aa) && *cc != 0.0) z = __ddiv_rn(1.0, *cc);
  }
  *a = r;
  *b = z;
}

// Cycle start: rnorm = sqrt(sum of the dot partials of r.r); the restart
// residual test of src/gmres.c:225-232 / :352-356 (strict < tol at the very
// first test, <= at a restart); s = (rnorm, 0, ...).
__global__ void gmres_cycle_start_kernel(const double *__restrict__ part, int nPart, double bnrm2, double tol,
                                         int first, int restrt, double *sv, GmresStatus *st) {
  __shared__ double red[kRedThreads];
  double s = 0.0;
  for (int k = threadIdx.x; k < nPart; k += blockDim.x) s += part[k];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int m = blockDim.x / 2; m > 0; m >>= 1) {
    if ((int)threadIdx.x < m) red[threadIdx.x] += red[threadIdx.x + m];
    __syncthreads();
  }
  const double rn = sqrt(red[0]);
  for (int k = threadIdx.x; k < restrt + 2; k += blockDim.x) sv[k] = (k == 0) ? rn : 0.0;
  if (threadIdx.x == 0) {
    const double res = rn / bnrm2;
    st->rnorm = rn;
    st->resid = res;
    st->i = 0;
    if (first ? (res < tol) : (res <= tol)) st->state = 1;
    else if (!(rn > 0.0) || rn != rn) st->state = 3;
    else st->state = 0;
  }
}

// h_i = sqrt(w.w) from the partials; v_i = w / h_i (w itself when h_i is 0); then, in block 0, the Givens step
// of column i (1-based, as src/gmres.c): H(:, i-1) = h, previous rotations, the new rotation, s rotated, residual
// estimate.  A step queued after the cycle ended (state != 0) changes nothing in H and the status.
__global__ void __launch_bounds__(kRedThreads)
mgs_norm_scale_kernel(long long n, const double *__restrict__ partIn, const double *__restrict__ h,
                      const double *__restrict__ w, double *v, double *H, int ldh, int restrt, double *sv, int i,
                      int iters, int maxit, double bnrm2, double tol, GmresStatus *st) {
  __shared__ double red[kRedThreads];
  const double d = sqrt(block_sum_partials(partIn, red));
  const double sc = (d > 0.0) ? 1.0 / d : 1.0;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
    v[e] = (d > 0.0) ? w[e] * sc : w[e];
  if (blockIdx.x != 0 || threadIdx.x != 0 || st->state != 0) return;
  double *cs = H + (size_t)restrt * ldh, *sn = H + (size_t)(restrt + 1) * ldh;
  double *hc = H + (size_t)(i - 1) * ldh;
  double cur = h[0];   // the rotated column's running entry
  for (int k = 0; k < i - 1; k++) {
    double nxt = h[k + 1];
    drot_d(&cur, &nxt, cs[k], sn[k]);
    hc[k] = cur;
    cur = nxt;
  }
  double aa = cur, bb = d, cc, ss;
  drotg_d(&aa, &bb, &cc, &ss);
  cs[i - 1] = cc;
  sn[i - 1] = ss;
  double x = cur, y = d;
  drot_d(&x, &y, cc, ss);
  hc[i - 1] = x;
  hc[i] = y;
  x = sv[i - 1];
  y = sv[i];
  drot_d(&x, &y, cc, ss);
  sv[i - 1] = x;
  sv[i] = y;
  const double res = fabs(y) / bnrm2;
  st->resid = res;
  st->i = i;
  st->iters = iters;
  if (res <= tol) st->state = 1;
  else if (iters == maxit || i >= restrt) st->state = 2;
}

// y = H(0:k, 0:k)^-1 s (upper triangular, netlib dtrsv order), k = st->i
__global__ void gmres_trsv_kernel(const double *__restrict__ H, int ldh, const double *__restrict__ sv, double *y,
                                  const GmresStatus *st) {
  if (threadIdx.x != 0) return;
  const int k = st->i;
  for (int j = 0; j < k; j++) y[j] = sv[j];
  for (int j = k - 1; j >= 0; j--) {
    if (y[j] != 0.0) {
      y[j] = __ddiv_rn(y[j], H[(size_t)j * ldh + j]);
      const double t = y[j];
      for (int r = j - 1; r >= 0; r--) y[r] = __dsub_rn(y[r], __dmul_rn(t, H[(size_t)j * ldh + r]));
    }
  }
}

// x += V y over the first st->i columns
__global__ void gmres_update_kernel(long long n, const double *__restrict__ V, long long ldv,
                                    const double *__restrict__ y, const GmresStatus *st, double *x) {
  const int k = st->i;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double s = x[i];
    for (int j = 0; j < k; j++) s += y[j] * V[(size_t)j * ldv + i];
    x[i] = s;
  }
}

static bool gmres_log_enabled() {
  static const bool on = [] {
    const char *e = getenv("FABIPB_GMRES_LOG_RESID");
    return e != nullptr && atoi(e) > 0;
  }();
  return on;
}

// the status record to the host (pinned), after everything queued so far.
// The host spins on an event query rather than blocking in a stream
// synchronize: a thread put to sleep by a blocking wait can take milliseconds
// to be woken, once per Arnoldi step (measured: GMRES at 204,800 panels 10.7 to
// 57 ms from run to run when blocking, 10.7 to 12.9 when the host stays busy).
static bool read_status(Context &c, const GmresStatus *d_st, GmresStatus *h_st) {
  PrecondDev &p = *c.pc;
  if (!p.evStatus) FB_CUDA(cudaEventCreateWithFlags(&p.evStatus, cudaEventDisableTiming));
  FB_CUDA(cudaMemcpyAsync(h_st, d_st, sizeof(GmresStatus), cudaMemcpyDeviceToHost, c.stream));
  FB_CUDA(cudaEventRecord(p.evStatus, c.stream));
  cudaError_t e;
  while ((e = cudaEventQuery(p.evStatus)) == cudaErrorNotReady) {
  }
  FB_CUDA(e);
  return true;
}

// x := x + V y with y from the device triangular solve
static bool gmres_update_dev(Context &c, int ldh, const GmresStatus *d_st, double *x) {
  PrecondDev &p = *c.pc;
  const long long n2 = 2LL * c.n;
  gmres_trsv_kernel<<<1, 32, 0, c.stream>>>(p.d_H, ldh, p.d_sv, p.d_y, d_st);
  gmres_update_kernel<<<kRedBlocks * 4, 256, 0, c.stream>>>(n2, p.d_V, n2, p.d_y, d_st, x);
  c.launches += 2;
  FB_CUDA(cudaGetLastError());
  return true;
}

// Restarted, left-preconditioned GMRES of src/gmres.c:153-362 with every
// vector and the Hessenberg/Givens state on the device.  Residual measure:
// ||P^-1 (b - A x)|| / ||b||, estimated by |s_i| / ||b|| inside a cycle.
bool gmres_solve(Context &c, const double *b, double *x, int restrt, int maxit, double tol, int *iters, double *resid,
                 int *info, bool adjoint, int *steps) {
  FB_CHECK(c.pc != nullptr, "call fabipb_b200_precond_setup before solving (mode -1 for none)");
  FB_CHECK(restrt >= 1, "GMRES restart must be at least 1");
  PrecondDev &p = *c.pc;
  const long long n2 = 2LL * c.n;
  const int ldh = restrt + 1;
  cudaStream_t s = c.stream;
  if (p.restart != restrt || p.d_V == nullptr) {
    p.restart = restrt;
    if (!p.arena.alloc_n(&p.d_V, (size_t)n2 * (restrt + 1)) || !p.arena.alloc_n(&p.d_r, (size_t)n2) ||
        !p.arena.alloc_n(&p.d_av, (size_t)n2) || !p.arena.alloc_n(&p.d_w, (size_t)n2) ||
        !p.arena.alloc_n(&p.d_h, (size_t)ldh + 1) || !p.arena.alloc_n(&p.d_part, (2 * (size_t)restrt + 2) * kRedBlocks + 2) ||
        !p.arena.alloc_n(&p.d_G, (size_t)restrt * restrt) || !p.arena.alloc_n(&p.d_y, (size_t)restrt + 1) || !p.arena.alloc_n(&p.d_H, (size_t)ldh * (restrt + 2)) ||
        !p.arena.alloc_n(&p.d_sv, (size_t)restrt + 2) || !p.arena.alloc(&p.d_status, sizeof(GmresStatus)))
      return false;
    if (!p.h_status) FB_CUDA(cudaMallocHost(&p.h_status, 4 * sizeof(GmresStatus)));
  }
  GmresStatus *d_st = static_cast<GmresStatus *>(p.d_status);
  GmresStatus *h_st = static_cast<GmresStatus *>(p.h_status);
  const bool logResid = gmres_log_enabled();
  *info = 0;
  *iters = maxit;
  *resid = tol;
  // ||x0|| decides whether b - A x0 needs the operator; ||b|| scales the test
  double *norms = static_cast<double *>(p.h_status) + 2 * sizeof(GmresStatus) / sizeof(double);
  if (!dot_dev(c, n2, x, x, p.d_part + kRedBlocks, true)) return false;
  if (!dot_dev(c, n2, b, b, p.d_part + kRedBlocks + 1, true)) return false;
  FB_CUDA(cudaMemcpyAsync(norms, p.d_part + kRedBlocks, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
  FB_CUDA(cudaStreamSynchronize(s));   // once per solve
  const double xn = norms[0];
  double bnrm2 = norms[1];
  if (bnrm2 == 0.0) bnrm2 = 1.0;
  FB_CUDA(cudaMemcpyAsync(p.d_av, b, n2 * sizeof(double), cudaMemcpyDeviceToDevice, s));
  if (xn != 0.0) {
    if (!op_matvec(c, -1.0, x, 1.0, p.d_av, adjoint)) return false;
  }
  if (!precond_apply(c, p.d_av, p.d_r, adjoint)) return false;
  int it = 0;
  bool first = true;
  int stepsLocal = 0;
  if (!steps) steps = &stepsLocal;
  *steps = 0;
  for (;;) {
    // cycle start: rnorm, the restart residual test, v_0 = r / rnorm
    dot_partial_kernel<<<kRedBlocks, kRedThreads, 0, s>>>(n2, p.d_r, p.d_r, p.d_part);
    gmres_cycle_start_kernel<<<1, kRedThreads, 0, s>>>(p.d_part, kRedBlocks, bnrm2, tol, first ? 1 : 0, restrt,
                                                       p.d_sv, d_st);
    c.launches += 2;
    FB_CUDA(cudaGetLastError());
    if (!read_status(c, d_st, h_st)) return false;
    if (first && h_st->state == 1) return true;   // converged at x0: iters and resid keep their entry values
    *resid = h_st->resid;
    if (!first && logResid) printf("GMRES residual: iter=%d resid=%e\n", it, h_st->resid);
    if (h_st->state == 1) {
      *iters = it;
      return true;
    }
    if (first) {
      *iters = 0;
      first = false;
    } else if (it == maxit) {
      *iters = it;
      *info = 1;
      return true;
    }
    if (h_st->state == 3) {
      const double rn = h_st->rnorm;
      *resid = (rn != rn) ? rn : 0.0;
      *info = (rn != rn) ? 2 : 0;
      *iters = it;
      return true;
    }
    scale_copy_dev_kernel<<<kRedBlocks * 4, 256, 0, s>>>(n2, &d_st->rnorm, p.d_r, p.d_V);
    c.launches += 1;
    int i = 0;
    for (;;) {
      ++i;
      ++it;
      *steps = it;
      if (!op_matvec(c, 1.0, p.d_V + (size_t)(i - 1) * n2, 0.0, p.d_av, adjoint)) return false;
      if (!precond_apply(c, p.d_av, p.d_w, adjoint)) return false;
      // modified Gram-Schmidt of w against v_0 .. v_{i-1}, then the Givens step
      double *norm = p.d_part + 2 * (size_t)restrt * kRedBlocks;
      gs_dots_kernel<<<kRedBlocks, kRedThreads, 0, s>>>(n2, i, p.d_V, p.d_w, p.d_part);
      if (i > kGsStage) gs_solve_kernel<<<1, kGsRows * 32, 0, s>>>(i, restrt, p.d_part, p.d_G, p.d_h);
      auto update = i <= kGsStage ? gs_update_kernel<true> : gs_update_kernel<false>;
      update<<<kRedBlocks, kRedThreads, gs_smem(i), s>>>(n2, i, restrt, p.d_V, p.d_part, p.d_G, p.d_h, p.d_w, norm);
      mgs_norm_scale_kernel<<<kRedBlocks, kRedThreads, 0, s>>>(n2, norm, p.d_h, p.d_w, p.d_V + (size_t)i * n2, p.d_H,
                                                               ldh, restrt, p.d_sv, i, it, maxit, bnrm2, tol, d_st);
      c.launches += i > kGsStage ? 4 : 3;
      FB_CUDA(cudaGetLastError());
      if (!read_status(c, d_st, h_st)) return false;
      *resid = h_st->resid;
      if (logResid) printf("GMRES residual: iter=%d resid=%e\n", it, h_st->resid);
      if (h_st->state == 1) {
        *iters = it;
        return gmres_update_dev(c, ldh, d_st, x);
      }
      if (h_st->state != 0) break;
    }
    // end of a cycle: x += V y, r = P^-1 (b - A x)
    if (!gmres_update_dev(c, ldh, d_st, x)) return false;
    FB_CUDA(cudaMemcpyAsync(p.d_av, b, n2 * sizeof(double), cudaMemcpyDeviceToDevice, s));
    if (!op_matvec(c, -1.0, x, 1.0, p.d_av, adjoint)) return false;
    if (!precond_apply(c, p.d_av, p.d_r, adjoint)) return false;
    *iters = it;
  }
}

}  // namespace fb

namespace fb {

__global__ void add_kernel(long long n, const double *__restrict__ d, double *x) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    x[i] += d[i];
}

// Mixed-precision iterative refinement.  First the whole system A x = b is
// solved from the given x by GMRES with the context's own operator (the FP32
// P2P in a mixed context), to tolInner, or to 0.9 of the outer tolerance when
// tolInner is not looser than tol (the FP32 operator's error then rarely lifts
// the FP64 residual above tol); then, until ||P^-1 r|| / ||b|| <= tol (the
// reference GMRES measure, src/gmres.c:225-232), the residual r = b - A x is
// formed with the FP64 operator (in a mixed context the FP64 near-field P2P),
// the correction A d = r is solved by GMRES with the context's operator from
// d = 0, and x += d.  The outer residuals and updates are FP64 vectors.  A
// correction is solved to the relative tolerance tolInner, or only to half
// the reduction the outer test still needs when that is looser: the inner
// GMRES stops at ||P^-1 r_inner|| <= tolStep ||r||, so tolStep =
// 0.5 tol ||b|| / ||r|| leaves the next outer residual near tol / 2, and a
// residual just above tol costs a few inner iterations, not a full tolInner
// reduction far below tol.  When the first solve already meets tol in FP64
// terms, the whole refined solve costs one FP64 residual more than the plain
// solve.
bool refined_solve(Context &c, const double *b, double *x, int restart, int maxit, double tolInner, double tol,
                   int maxOuter, int *outer, int *iters, double *resid, int *info) {
  FB_CHECK(c.pc != nullptr, "call fabipb_b200_precond_setup before solving (mode -1 for none)");
  const long long n2 = 2LL * c.n;
  if (!c.d_refR && (!c.arena.alloc_n(&c.d_refR, (size_t)n2) || !c.arena.alloc_n(&c.d_refD, (size_t)n2) ||
                    !c.arena.alloc_n(&c.d_refZ, (size_t)n2)))
    return false;
  double bn = 0.0;
  if (!dot_to_host(c, n2, b, b, &bn)) return false;
  bn = sqrt(bn);
  if (bn == 0.0) bn = 1.0;
  *outer = 0;
  *iters = 0;
  *info = 0;
  {   // the first solve: the full system from x, on the context's operator
    int it = 0, inf = 0, st = 0;
    double res = 0.0;
    const double tolFirst = tolInner > tol ? tolInner : 0.9 * tol;
    if (!gmres_solve(c, b, x, restart, maxit, tolFirst, &it, &res, &inf, false, &st)) return false;
    *iters += st;
    ++(*outer);
  }
  for (;;) {
    FB_CUDA(cudaMemcpyAsync(c.d_refR, b, n2 * sizeof(double), cudaMemcpyDeviceToDevice, c.stream));
    if (!op_matvec(c, -1.0, x, 1.0, c.d_refR, false, true)) return false;
    if (!precond_apply(c, c.d_refR, c.d_refZ)) return false;
    double zn = 0.0;
    if (!dot_to_host(c, n2, c.d_refZ, c.d_refZ, &zn)) return false;
    *resid = sqrt(zn) / bn;
    if (*resid <= tol || !(*resid == *resid)) {
      if (!(*resid == *resid)) *info = 2;
      return true;
    }
    if (*outer >= maxOuter || *iters >= maxit) {
      *info = 1;
      return true;
    }
    ++(*outer);
    FB_CUDA(cudaMemsetAsync(c.d_refD, 0, n2 * sizeof(double), c.stream));
    int it = 0, inf = 0;
    double res = 0.0;
    double rn = 0.0;
    if (!dot_to_host(c, n2, c.d_refR, c.d_refR, &rn)) return false;
    rn = sqrt(rn);
    const double tolStep = rn > 0.0 ? fmax(tolInner, 0.5 * tol * bn / rn) : tolInner;
    int st = 0;
    if (!gmres_solve(c, c.d_refR, c.d_refD, restart, maxit - *iters, tolStep, &it, &res, &inf, false, &st))
      return false;
    *iters += st;
    add_kernel<<<kRedBlocks * 4, 256, 0, c.stream>>>(n2, c.d_refD, x);
    c.launches += 1;
    FB_CUDA(cudaGetLastError());
  }
}

}  // namespace fb
