// near.cu -- Galerkin near field on the device.
//
// The near field couples every panel X of a leaf with every panel Y of each
// leaf in its near list (src/fmm.c:554-593).  With the one-point rule (-q=1,
// the reference default) a disjoint pair is K = Ax*Ay*KER4(mX - mY)
// (src/numQuad.c:586-618 at q=1, src/gpu/gpu_nearfield_cuda.inc:1127-1137);
// pairs that share a vertex, an edge, or are the same panel use the Sauter
// rules instead (src/numQuad.c:401-571).
//
// B200 design:
//   * nothing per pair is stored.  Pairs of distinct near parts (leaves, or
//     runs of panels in a direct FP64 context) are tasks: a warp or a half-warp
//     evaluates each unordered panel pair once for both directions, one or two
//     targets per lane in registers and the other part in shared-memory tiles,
//     and leaves the sums in scratch slots.  A finishing kernel takes what is
//     left (each part with itself, parts of a few panels) and adds the slots in
//     a fixed order.  The work is FP32 (or FP64) arithmetic: two MUFU per pair
//     in FP32, own reciprocal root and exponential in FP64 (fastmath.cuh);
//   * positions are stored relative to their own part's centre, and a target
//     is moved into each source part's frame once per pair of parts, which keeps
//     FP32 differences of close panels accurate to ~1e-7 relative;
//   * the coincident pair is masked (r = 0 gives 0), and every pair with a
//     shared vertex carries an FP64 correction "exact Sauter value minus the
//     one-point value" in a CSR table built once on the device, applied in
//     FP64 by the finishing kernel.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <thread>
#include <unordered_map>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "context.cuh"
#include "fastmath.cuh"
#include "near_plan.hpp"
#include "quad.cuh"

namespace fb {

template <typename T>
struct Vec4;
template <>
struct Vec4<float> {
  typedef float4 t;
};
template <>
struct Vec4<double> {
  typedef double4 t;
};
// FP32: the single MUFU instructions (PTX rsqrt.approx / ex2.approx, flush
// to zero; relative error ~2^-22, far below the FP32 P2P tolerance).
__device__ __forceinline__ float rsqrt_t(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 2^x: e^{-kappa r} is taken at x = -kappa log2(e) r
__device__ __forceinline__ float expneg_t(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <typename T>
__global__ void near_targets_kernel(int n, const double *__restrict__ vtx, const double *__restrict__ nrm,
                                    const double *__restrict__ area, const int *__restrict__ leafOfPanel,
                                    const double *__restrict__ leafCtr, typename Vec4<T>::t *tgtP,
                                    typename Vec4<T>::t *tgtN) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double *v = vtx + 9 * (size_t)i;
  const double *c = leafCtr + 3 * (size_t)leafOfPanel[i];
  double m[3];
  for (int k = 0; k < 3; k++) {
    double a2 = v[3 + k] - v[k], a0 = v[6 + k] - v[3 + k];
    m[k] = v[k] + 0.5 * (a2 + 0.5 * a0);
  }
  typename Vec4<T>::t p, q;
  p.x = (T)(m[0] - c[0]); p.y = (T)(m[1] - c[1]); p.z = (T)(m[2] - c[2]); p.w = (T)area[i];
  q.x = (T)nrm[3 * (size_t)i]; q.y = (T)nrm[3 * (size_t)i + 1]; q.z = (T)nrm[3 * (size_t)i + 2]; q.w = (T)0;
  tgtP[i] = p;
  tgtN[i] = q;
}

// Record of panel i for the density sgm: {position, A*sigma_dpdn}, {normal, A*sigma_pot}.
template <typename T>
__device__ __forceinline__ void near_record(int i, int n, const typename Vec4<T>::t *__restrict__ tgtP,
                                            const typename Vec4<T>::t *__restrict__ tgtN,
                                            const double *__restrict__ area, const double *__restrict__ sgm,
                                            typename Vec4<T>::t &a, typename Vec4<T>::t &b) {
  a = tgtP[i];
  b = tgtN[i];
  const double A = area[i];
  a.w = (T)(A * sgm[n + i]);   // weight of the dpdn density
  b.w = (T)(A * sgm[i]);       // weight of the potential density
}

// the records of one apply, for the symmetric tasks, which read each many times
template <typename T>
__global__ void near_pack_kernel(int n, const typename Vec4<T>::t *__restrict__ tgtP,
                                 const typename Vec4<T>::t *__restrict__ tgtN, const double *__restrict__ area,
                                 const double *__restrict__ sgm, typename Vec4<T>::t *recA,
                                 typename Vec4<T>::t *recB) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  typename Vec4<T>::t a, b;
  near_record<T>(i, n, tgtP, tgtN, area, sgm, a, b);
  recA[i] = a;
  recB[i] = b;
}

constexpr int kNearWarps = 4;

// One disjoint pair, one-point rule: the four KER4 kernels (src/kernel.c:109-147)
// at d = target - source, times the source weights a.w = A*sigma_dpdn and
// b.w = A*sigma_pot (the 4 pi and the target area are applied once at the end).
// With g = 1/r, h = g^3, c = (kappa r + 1) e^{-kappa r}, the pair's terms are
//   F  = h (eps c - 1),   Fi = h (c/eps - 1),   H1 = h (c - 1),
//   y0 = g - g e,   y1 = (n_s.d) F,   y2 = (n_t.d) Fi,
//   y3 = (n_t.n_s) H1 - (n_t.d)(n_s.d) (3 g^2 H1 + kappa^2 h e).
//
// ADJ: the transposed pair block.  Swapping the roles of the two panels gives
// K0 and K3 unchanged, K1(s,t) = -(n_t.d) F and K2(s,t) = -(n_s.d) Fi, so
//   out_pot  += y3 * a.w - (n_t.d) F * b.w
//   out_dpdn += y0 * b.w - (n_s.d) Fi * a.w
// with a.w = A*lambda_dpdn and b.w = A*lambda_pot of the source panel.
struct NearConstD {
  double kappa, kexp, eps, ieps, kap2;
};
struct NearConstF {
  float kappa, kexp, eps, ieps, kap2;
};

struct NearPairD {
  double y0, y3, a1, a2, b1, b2;   // a1 = (n_s.d) F, a2 = (n_t.d) F, b1 = (n_s.d) Fi, b2 = (n_t.d) Fi
};
// SELF: the two sides may hold panels with the same one-point node (the target's own leaf; any two parts of a
// direct context, whose runs of panels cut leaves): 1/r of a coincident pair is 0.  (The test reads r2's high word,
// beside the FP64 pipe; an r2 below the normal numbers counts as 0.)
template <bool SELF>
__device__ __forceinline__ NearPairD near_terms(double dx, double dy, double dz, double tnx, double tny, double tnz,
                                                double snx, double sny, double snz, const NearConstD &K,
                                                const double *tab) {
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double g = SELF && __double2hiint(r2) < 0x00100000 ? 0.0 : rsqrt_pos(r2);
  const double r = r2 * g;
  const double e = exp_tab(K.kexp * r, tab);
  const double g2 = g * g, h = g2 * g, he = h * e, hc = he * (K.kappa * r + 1.0);
  const double H1 = hc - h, F = K.eps * hc - h, Fi = K.ieps * hc - h;
  const double ipX = tnx * dx + tny * dy + tnz * dz;
  const double ipY = snx * dx + sny * dy + snz * dz;
  const double ip0 = tnx * snx + tny * sny + tnz * snz;
  NearPairD p;
  p.y0 = g - g * e;
  p.y3 = ip0 * H1 - ipX * ipY * (3.0 * (g2 * H1) + K.kap2 * he);
  p.a1 = ipY * F;
  p.a2 = ipX * F;
  p.b1 = ipY * Fi;
  p.b2 = ipX * Fi;
  return p;
}

template <bool ADJ, bool SELF>
__device__ __forceinline__ void near_pair(const double4 a, const double4 b, double tx, double ty, double tz,
                                          const double4 tn, const NearConstD &K, const double *tab, double &acc0,
                                          double &acc1) {
  const NearPairD p = near_terms<SELF>(tx - a.x, ty - a.y, tz - a.z, tn.x, tn.y, tn.z, b.x, b.y, b.z, K, tab);
  if (ADJ) {
    acc0 += p.y3 * a.w - p.a2 * b.w;
    acc1 += p.y0 * b.w - p.b1 * a.w;
  } else {
    acc0 += p.y0 * a.w + p.a1 * b.w;
    acc1 += p.b2 * a.w + p.y3 * b.w;
  }
}

// The same in FP32 for two sources at once (packed f32x2: sm_100
// FFMA2/FMUL2/FADD2).  A source pair is four float4
//   A = (-x0 -x1 -y0 -y1), B = (-z0 -z1 wa0 wa1), C = (nx0 nx1 ny0 ny1), D = (nz0 nz1 wb0 wb1),
// so the packed operands come straight from the loads.  Signs are arranged so
// that no packed operand has to be negated but 1/r.  ADJ: wb is stored negated
// and acc1 is the negated sum:
//   acc0 += y3 wa + (n_t.d) F wb,  acc1 += y0 wb + (n_s.d) Fi wa.
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

struct NearPairF2 {
  float2 y0, y3, a1, a2, b1, b2;   // a1 = (n_s.d) F, a2 = (n_t.d) F, b1 = (n_s.d) Fi, b2 = (n_t.d) Fi
};
template <int G>
struct NearTargetsF2 {   // G targets, each value in both halves
  float2 x[G], y[G], z[G], nx[G], ny[G], nz[G];
};

// The terms of a source pair and G targets, operation by operation over the
// targets: a packed FMA with three register operands takes three to four
// cycles of register reads instead of two, and neighbours that share one are
// what the operand reuse of the scheduler can shorten.
// SELF (the target's own leaf, the only tile holding the coincident pair
// d = 0): 1/r is taken as 0 there, which zeroes every term.
template <bool SELF, int G>
__device__ __forceinline__ void near_terms2(const float4 A, const float4 B, const float4 C, const float4 D,
                                            const NearTargetsF2<G> &t, const NearConstF &K, NearPairF2 (&p)[G]) {
#define FB_EACH _Pragma("unroll") for (int k = 0; k < G; k++)
  const float2 nx = make_float2(C.x, C.y), ny = make_float2(C.z, C.w), nz = make_float2(D.x, D.y);
  float2 dx[G], dy[G], dz[G], r2[G], g[G], ng[G], e[G], c1[G], g2[G], nh[G], he[G], hc[G], H1[G], F[G], Fi[G];
  float2 ipX[G], ipY[G], ip0[G], w[G];
  FB_EACH dx[k] = __fadd2_rn(t.x[k], make_float2(A.x, A.y));
  FB_EACH dy[k] = __fadd2_rn(t.y[k], make_float2(A.z, A.w));
  FB_EACH dz[k] = __fadd2_rn(t.z[k], make_float2(B.x, B.y));
  FB_EACH r2[k] = __fmul2_rn(dx[k], dx[k]);
  FB_EACH r2[k] = __ffma2_rn(dy[k], dy[k], r2[k]);
  FB_EACH r2[k] = __ffma2_rn(dz[k], dz[k], r2[k]);
  FB_EACH {
    if (SELF) {
      g[k].x = r2[k].x > 0.f ? rsqrt_t(r2[k].x) : 0.f;
      g[k].y = r2[k].y > 0.f ? rsqrt_t(r2[k].y) : 0.f;
    } else {   // distinct leaves: distinct panel centroids, r > 0
      g[k].x = rsqrt_t(r2[k].x);
      g[k].y = rsqrt_t(r2[k].y);
    }
    ng[k] = make_float2(-g[k].x, -g[k].y);
  }
  FB_EACH r2[k] = __fmul2_rn(r2[k], g[k]);   // r
  FB_EACH {
    const float2 ea = __fmul2_rn(f2(K.kexp), r2[k]);
    e[k].x = expneg_t(ea.x);
    e[k].y = expneg_t(ea.y);
  }
  FB_EACH c1[k] = __ffma2_rn(f2(-K.kappa), r2[k], f2(-1.f));   // -(kappa r + 1)
  FB_EACH g2[k] = __fmul2_rn(g[k], g[k]);
  FB_EACH nh[k] = __fmul2_rn(g2[k], ng[k]);                    // -h
  FB_EACH he[k] = __fmul2_rn(nh[k], e[k]);                     // -h e
  FB_EACH hc[k] = __fmul2_rn(he[k], c1[k]);                    // h c
  FB_EACH H1[k] = __fadd2_rn(hc[k], nh[k]);
  FB_EACH F[k] = __ffma2_rn(f2(K.eps), hc[k], nh[k]);
  FB_EACH Fi[k] = __ffma2_rn(f2(K.ieps), hc[k], nh[k]);
  FB_EACH ipX[k] = __fmul2_rn(t.nx[k], dx[k]);                 // n_t.d
  FB_EACH ipX[k] = __ffma2_rn(t.ny[k], dy[k], ipX[k]);
  FB_EACH ipX[k] = __ffma2_rn(t.nz[k], dz[k], ipX[k]);
  FB_EACH ipY[k] = __fmul2_rn(nx, dx[k]);                      // n_s.d
  FB_EACH ipY[k] = __ffma2_rn(ny, dy[k], ipY[k]);
  FB_EACH ipY[k] = __ffma2_rn(nz, dz[k], ipY[k]);
  FB_EACH ip0[k] = __fmul2_rn(nx, t.nx[k]);                    // n_t.n_s
  FB_EACH ip0[k] = __ffma2_rn(ny, t.ny[k], ip0[k]);
  FB_EACH ip0[k] = __ffma2_rn(nz, t.nz[k], ip0[k]);
  FB_EACH w[k] = __ffma2_rn(f2(-3.f), __fmul2_rn(g2[k], H1[k]), __fmul2_rn(f2(K.kap2), he[k]));
  FB_EACH p[k].y0 = __ffma2_rn(ng[k], e[k], g[k]);
  FB_EACH p[k].y3 = __ffma2_rn(__fmul2_rn(ipX[k], ipY[k]), w[k], __fmul2_rn(ip0[k], H1[k]));
  FB_EACH p[k].a1 = __fmul2_rn(ipY[k], F[k]);
  FB_EACH p[k].a2 = __fmul2_rn(ipX[k], F[k]);
  FB_EACH p[k].b1 = __fmul2_rn(ipY[k], Fi[k]);
  FB_EACH p[k].b2 = __fmul2_rn(ipX[k], Fi[k]);
}

template <bool ADJ, bool SELF>
__device__ __forceinline__ void near_pair2(const float4 A, const float4 B, const float4 C, const float4 D,
                                           const NearTargetsF2<1> &t, const NearConstF &K, float2 &acc0,
                                           float2 &acc1) {
  NearPairF2 p[1];
  near_terms2<SELF, 1>(A, B, C, D, t, K, p);
  const float2 wa = make_float2(B.z, B.w), wb = make_float2(D.z, D.w);
  if (ADJ) {
    acc0 = __ffma2_rn(p[0].a2, wb, __ffma2_rn(p[0].y3, wa, acc0));
    acc1 = __ffma2_rn(p[0].b1, wa, __ffma2_rn(p[0].y0, wb, acc1));
  } else {
    acc0 = __ffma2_rn(p[0].a1, wb, __ffma2_rn(p[0].y0, wa, acc0));
    acc1 = __ffma2_rn(p[0].y3, wb, __ffma2_rn(p[0].b2, wa, acc1));
  }
}

// ---------------------------------------------------------------------------
// Symmetric near field.  The pair terms of K(X, Y) and K(Y, X) share r, 1/r,
// e^{-kappa r}, the normal products and F, Fi, y0, y3; with d = x_X - x_Y,
// swapping the panels negates d, so
//   K(Y,X): out_pot  += y0 wa_X - (n_X.d) F wb_X,
//           out_dpdn += y3 wb_X - (n_Y.d) Fi wa_X.
// So every unordered pair of distinct near leaves (R, T) is evaluated once
// for both directions, without atomics: the sums go to a scratch slot per
// (leaf, task), which the finishing kernel adds in a fixed order.
//
// A task is a leaf pair, or a chunk of R's panels against all of T, on W lanes
// (a warp, or a half-warp for pairs that pad badly into 32-panel groups).
// Every lane holds one or two target panels of R in registers; T passes in
// tiles of W sources through shared memory.  In step s, lane t takes the
// tile's sources t + s and t + s + W/2 (mod W) as one packed pair, so the
// lanes hold distinct sources; the sources' own sums travel with them, one
// lane down per step, and are added to by the same FMAs that form the terms.
//
// Bound by the FP32 FMA pipe: 44 packed operations (two cycles each) for the
// two directions of two pairs.  Two targets per lane halve the shared-memory
// reads and shuffles per pair, which beside 46 + 2 operations with one target
// per lane and gathered sums had left the pipe at 75%.
// Measured (whole products, before -> after): two-shell 2,096,704 panels 25.8
// -> 23.4 ms, its quarter transposed 9.45 -> 8.11 ms, star 204,800 panels 605 ->
// 553 us, sphere 20,480 panels 144 -> 80 us (there by the split into tasks).
// ---------------------------------------------------------------------------
// steps of a tile unrolled together, and resident blocks per SM that the
// register allocation aims at (two targets per lane: 4 at 128 registers)
#ifndef FB_NEAR_SYM_UNROLL
#define FB_NEAR_SYM_UNROLL 2
#endif
#ifndef FB_NEAR_SYM_MIN_BLOCKS
#define FB_NEAR_SYM_MIN_BLOCKS 4
#endif
constexpr int kSymUnroll = FB_NEAR_SYM_UNROLL;
constexpr int kSymWarps = 4;

// a task: leaves R (registers) and T (tiles), R's panels [r0, r1), and the
// first scratch slots of R's and T's sums
struct NearTask {
  int R, T, r0, r1, scrR, scrT;
};

// G * W targets of R from r0 against all of T.  first: the sums of T start here.
template <bool ADJ, int W, int G>
__device__ __forceinline__ void near_sym_group(float4 *Q, unsigned mask, int hl, int r0, int r1, int rb, int tb,
                                               int tc, float sx, float sy, float sz, bool first,
                                               const float4 *__restrict__ recA, const float4 *__restrict__ recB,
                                               const NearConstF &K, float2 *scrR, float2 *scrT) {
  NearTargetsF2<G> tg;
  float2 wat[G], wbt[G], nwat[G], nwbt[G], acc0[G], acc1[G];
#pragma unroll
  for (int k = 0; k < G; k++) {
    const int t = r0 + k * W + hl;
    // a lane past the end: far away, zero weights (its terms vanish, its sums are dropped)
    const float4 a = t < r1 ? recA[rb + t] : make_float4(1e4f, 1e4f, 1e4f, 0.f);
    const float4 b = t < r1 ? recB[rb + t] : make_float4(0.f, 0.f, 1.f, 0.f);
    tg.x[k] = f2(a.x + sx); tg.y[k] = f2(a.y + sy); tg.z[k] = f2(a.z + sz);
    tg.nx[k] = f2(b.x); tg.ny[k] = f2(b.y); tg.nz[k] = f2(b.z);
    wat[k] = f2(a.w); wbt[k] = f2(b.w); nwat[k] = f2(-a.w); nwbt[k] = f2(-b.w);
    acc0[k] = acc1[k] = f2(0.f);
  }
  // the tile's source hl, or a padding source far away with zero weights; loaded one tile ahead
  const float4 farA = make_float4(-1e4f, -1e4f, -1e4f, 0.f), farB = make_float4(0.f, 0.f, 1.f, 0.f);
  float4 na = hl < tc ? recA[tb + hl] : farA, nb = hl < tc ? recB[tb + hl] : farB;
  for (int j0 = 0; j0 < tc; j0 += W) {
    const int j = j0 + hl;
    const float4 sa = na, sb = nb;
    na = j + W < tc ? recA[tb + j + W] : farA;
    nb = j + W < tc ? recB[tb + j + W] : farB;
    const float2 prev = first || j >= tc ? f2(0.f) : scrT[j];
    // slot m holds source m first and source m + W/2 (mod W) second
    const float ox = __shfl_xor_sync(mask, sa.x, W / 2), oy = __shfl_xor_sync(mask, sa.y, W / 2);
    const float oz = __shfl_xor_sync(mask, sa.z, W / 2), ow = __shfl_xor_sync(mask, sa.w, W / 2);
    const float px = __shfl_xor_sync(mask, sb.x, W / 2), py = __shfl_xor_sync(mask, sb.y, W / 2);
    const float pz = __shfl_xor_sync(mask, sb.z, W / 2), pw = __shfl_xor_sync(mask, sb.w, W / 2);
    __syncwarp(mask);   // the previous tile's reads are done
    Q[hl] = make_float4(-sa.x, -ox, -sa.y, -oy);
    Q[W + hl] = make_float4(-sa.z, -oz, sa.w, ow);
    Q[2 * W + hl] = make_float4(sb.x, px, sb.y, py);
    Q[3 * W + hl] = ADJ ? make_float4(sb.z, pz, -sb.w, -pw) : make_float4(sb.z, pz, sb.w, pw);
    __syncwarp(mask);
    float2 o0 = f2(0.f), o1 = f2(0.f);   // the travelling sums (pot, dpdn) of this lane's two sources
#pragma unroll kSymUnroll
    for (int st = 0; st < W / 2; st++) {
      const int slot = (hl + st) & (W - 1);
      const float4 A = Q[slot], B = Q[W + slot], C = Q[2 * W + slot], D = Q[3 * W + slot];
      const float2 wa = make_float2(B.z, B.w), wb = make_float2(D.z, D.w);
      NearPairF2 p[G];
      near_terms2<false, G>(A, B, C, D, tg, K, p);
      if (ADJ) {   // wb negated, acc1 the negated sum
        FB_EACH acc0[k] = __ffma2_rn(p[k].y3, wa, acc0[k]);
        FB_EACH acc1[k] = __ffma2_rn(p[k].b1, wa, acc1[k]);
        FB_EACH acc0[k] = __ffma2_rn(p[k].a2, wb, acc0[k]);
        FB_EACH acc1[k] = __ffma2_rn(p[k].y0, wb, acc1[k]);
        FB_EACH {
          o0 = __ffma2_rn(p[k].a1, wbt[k], __ffma2_rn(p[k].y3, wat[k], o0));
          o1 = __ffma2_rn(p[k].b2, wat[k], __ffma2_rn(p[k].y0, wbt[k], o1));
        }
      } else {
        FB_EACH acc0[k] = __ffma2_rn(p[k].y0, wa, acc0[k]);
        FB_EACH acc1[k] = __ffma2_rn(p[k].b2, wa, acc1[k]);
        FB_EACH acc0[k] = __ffma2_rn(p[k].a1, wb, acc0[k]);
        FB_EACH acc1[k] = __ffma2_rn(p[k].y3, wb, acc1[k]);
        FB_EACH {
          o0 = __ffma2_rn(p[k].a2, nwbt[k], __ffma2_rn(p[k].y0, wat[k], o0));
          o1 = __ffma2_rn(p[k].b1, nwat[k], __ffma2_rn(p[k].y3, wbt[k], o1));
        }
      }
      const int up = (hl + 1) & (W - 1);
      o0.x = __shfl_sync(mask, o0.x, up, W);
      o0.y = __shfl_sync(mask, o0.y, up, W);
      o1.x = __shfl_sync(mask, o1.x, up, W);
      o1.y = __shfl_sync(mask, o1.y, up, W);
    }
    // after W/2 steps the second source's sums are home, the first's half a turn away
    const float s0 = o0.y + __shfl_xor_sync(mask, o0.x, W / 2), s1 = o1.y + __shfl_xor_sync(mask, o1.x, W / 2);
    if (j < tc) scrT[j] = make_float2(prev.x + s0, prev.y + s1);
  }
#pragma unroll
  for (int k = 0; k < G; k++) {
    const int t = r0 + k * W + hl;
    const float v1 = acc1[k].x + acc1[k].y;
    if (t < r1) scrR[t] = make_float2(acc0[k].x + acc0[k].y, ADJ ? -v1 : v1);
  }
}

template <bool ADJ, int W>
__device__ __forceinline__ void near_sym_task(const NearTask tk, float4 *Q, const int *__restrict__ leafStart,
                                              const int *__restrict__ leafCount, const double *__restrict__ leafCtr,
                                              const float4 *__restrict__ recA, const float4 *__restrict__ recB,
                                              const NearConstF &K, float2 *scr) {
  const int hl = threadIdx.x % W;
  const unsigned mask = W == 32 ? 0xffffffffu : 0xffffu << (threadIdx.x & 16);
  const int rb = leafStart[tk.R], tb = leafStart[tk.T], tc = leafCount[tk.T];
  const float sx = (float)(leafCtr[3 * tk.R] - leafCtr[3 * tk.T]);
  const float sy = (float)(leafCtr[3 * tk.R + 1] - leafCtr[3 * tk.T + 1]);
  const float sz = (float)(leafCtr[3 * tk.R + 2] - leafCtr[3 * tk.T + 2]);
  float2 *scrR = scr + tk.scrR, *scrT = scr + tk.scrT;
  int r0 = tk.r0;
  for (; r0 + W < tk.r1; r0 += 2 * W)
    near_sym_group<ADJ, W, 2>(Q, mask, hl, r0, tk.r1, rb, tb, tc, sx, sy, sz, r0 == tk.r0, recA, recB, K, scrR, scrT);
  if (r0 < tk.r1)
    near_sym_group<ADJ, W, 1>(Q, mask, hl, r0, tk.r1, rb, tb, tc, sx, sy, sz, r0 == tk.r0, recA, recB, K, scrR, scrT);
}

// one launch: the first blocks take the warp tasks, the rest the half-warp ones
template <bool ADJ>
__global__ void __launch_bounds__(kSymWarps * 32, FB_NEAR_SYM_MIN_BLOCKS)
near_sym_f2_kernel(int n32, int nTasks, const NearTask *__restrict__ tasks, const int *__restrict__ leafStart,
                   const int *__restrict__ leafCount, const double *__restrict__ leafCtr,
                   const float4 *__restrict__ recA, const float4 *__restrict__ recB, NearConstF K, float2 *scr) {
  __shared__ float4 sQ[kSymWarps * 32 * 4];
  const int blocks32 = (n32 + kSymWarps - 1) / kSymWarps;
  if ((int)blockIdx.x < blocks32) {
    const int warp = threadIdx.x >> 5, task = blockIdx.x * kSymWarps + warp;
    if (task < n32)   // warp-uniform
      near_sym_task<ADJ, 32>(tasks[task], sQ + warp * 128, leafStart, leafCount, leafCtr, recA, recB, K, scr);
  } else {
    const int half = threadIdx.x >> 4, task = n32 + ((int)blockIdx.x - blocks32) * 2 * kSymWarps + half;
    if (task < nTasks)   // uniform over the half-warp
      near_sym_task<ADJ, 16>(tasks[task], sQ + half * 64, leafStart, leafCount, leafCtr, recA, recB, K, scr);
  }
}

// The same symmetric scheme in FP64 scalar arithmetic: lane t takes source
// (t + s) mod W in step s of W.  Bound by the FP64 pipe: 58 operations for the
// two directions of a pair, 15 of them 1/r and the exponential.
// Measured (whole FP64 products, before -> after): star 204,800 panels 1.73 ->
// 1.34 ms, direct 12,797 panels 1.43 -> 0.44 ms (that one also by taking the
// direct operator's pairs in equal runs of panels, once for both directions).
// MEET: parts that may hold coincident panels (near_terms).
template <bool ADJ, bool MEET, int W, int G>
__device__ __forceinline__ void near_sym_group(double2 *Q, unsigned mask, int hl, int r0, int r1, int rb, int tb,
                                               int tc, double sx, double sy, double sz, bool first,
                                               const double4 *__restrict__ recA, const double4 *__restrict__ recB,
                                               const NearConstD &K, const double *tab, double2 *scrR, double2 *scrT) {
  double4 ta[G], tn[G];
  double acc0[G], acc1[G];
#pragma unroll
  for (int k = 0; k < G; k++) {
    const int t = r0 + k * W + hl;
    // a lane past the end: far away, zero weights
    ta[k] = t < r1 ? recA[rb + t] : make_double4(1e4, 1e4, 1e4, 0.0);
    tn[k] = t < r1 ? recB[rb + t] : make_double4(0.0, 0.0, 1.0, 0.0);
    ta[k].x += sx;
    ta[k].y += sy;
    ta[k].z += sz;
    acc0[k] = acc1[k] = 0.0;
  }
  for (int j0 = 0; j0 < tc; j0 += W) {
    const int j = j0 + hl;
    const double4 sa = j < tc ? recA[tb + j] : make_double4(-1e4, -1e4, -1e4, 0.0);
    const double4 sb = j < tc ? recB[tb + j] : make_double4(0.0, 0.0, 1.0, 0.0);
    const double2 prev = first || j >= tc ? make_double2(0.0, 0.0) : scrT[j];
    __syncwarp(mask);   // the previous tile's reads are done
    Q[hl] = make_double2(sa.x, sa.y);
    Q[W + hl] = make_double2(sa.z, sa.w);
    Q[2 * W + hl] = make_double2(sb.x, sb.y);
    Q[3 * W + hl] = make_double2(sb.z, sb.w);
    __syncwarp(mask);
    double o0 = 0.0, o1 = 0.0;   // the travelling sums of this lane's source
#pragma unroll 1
    for (int st = 0; st < W; st++) {
      const int slot = (hl + st) & (W - 1);
      const double2 A = Q[slot], B = Q[W + slot], C = Q[2 * W + slot], D = Q[3 * W + slot];
      const double wa = B.y, wb = D.y;
#pragma unroll
      for (int k = 0; k < G; k++) {
        const NearPairD p = near_terms<MEET>(ta[k].x - A.x, ta[k].y - A.y, ta[k].z - B.x, tn[k].x, tn[k].y, tn[k].z,
                                              C.x, C.y, D.x, K, tab);
        if (ADJ) {
          acc0[k] += p.y3 * wa - p.a2 * wb;
          acc1[k] += p.y0 * wb - p.b1 * wa;
          o0 += p.y3 * ta[k].w + p.a1 * tn[k].w;
          o1 += p.y0 * tn[k].w + p.b2 * ta[k].w;
        } else {
          acc0[k] += p.y0 * wa + p.a1 * wb;
          acc1[k] += p.b2 * wa + p.y3 * wb;
          o0 += p.y0 * ta[k].w - p.a2 * tn[k].w;
          o1 += p.y3 * tn[k].w - p.b1 * ta[k].w;
        }
      }
      const int up = (hl + 1) & (W - 1);
      o0 = __shfl_sync(mask, o0, up, W);
      o1 = __shfl_sync(mask, o1, up, W);
    }
    if (j < tc) scrT[j] = make_double2(prev.x + o0, prev.y + o1);   // after W steps the sums are home
  }
#pragma unroll
  for (int k = 0; k < G; k++) {
    const int t = r0 + k * W + hl;
    if (t < r1) scrR[t] = make_double2(acc0[k], acc1[k]);
  }
}

template <bool ADJ, bool MEET, int W>
__device__ __forceinline__ void near_sym_task(const NearTask tk, double2 *Q, const int *__restrict__ leafStart,
                                              const int *__restrict__ leafCount, const double *__restrict__ leafCtr,
                                              const double4 *__restrict__ recA, const double4 *__restrict__ recB,
                                              const NearConstD &K, const double *tab, double2 *scr) {
  const int hl = threadIdx.x % W;
  const unsigned mask = W == 32 ? 0xffffffffu : 0xffffu << (threadIdx.x & 16);
  const int rb = leafStart[tk.R], tb = leafStart[tk.T], tc = leafCount[tk.T];
  const double sx = leafCtr[3 * tk.R] - leafCtr[3 * tk.T];
  const double sy = leafCtr[3 * tk.R + 1] - leafCtr[3 * tk.T + 1];
  const double sz = leafCtr[3 * tk.R + 2] - leafCtr[3 * tk.T + 2];
  double2 *scrR = scr + tk.scrR, *scrT = scr + tk.scrT;
  int r0 = tk.r0;
  for (; r0 + W < tk.r1; r0 += 2 * W)
    near_sym_group<ADJ, MEET, W, 2>(Q, mask, hl, r0, tk.r1, rb, tb, tc, sx, sy, sz, r0 == tk.r0, recA, recB, K, tab, scrR,
                              scrT);
  if (r0 < tk.r1)
    near_sym_group<ADJ, MEET, W, 1>(Q, mask, hl, r0, tk.r1, rb, tb, tc, sx, sy, sz, r0 == tk.r0, recA, recB, K, tab, scrR,
                              scrT);
}

#ifndef FB_NEAR_SYM64_MIN_BLOCKS
#define FB_NEAR_SYM64_MIN_BLOCKS 4
#endif
template <bool ADJ, bool MEET>
__global__ void __launch_bounds__(kSymWarps * 32, FB_NEAR_SYM64_MIN_BLOCKS)
near_sym_kernel(int n32, int nTasks, const NearTask *__restrict__ tasks, const int *__restrict__ leafStart,
                const int *__restrict__ leafCount, const double *__restrict__ leafCtr,
                const double4 *__restrict__ recA, const double4 *__restrict__ recB, NearConstD K, double2 *scr) {
  __shared__ double2 sQ[kSymWarps * 32 * 4];
  __shared__ double tab[kExpTab];
  load_exp_tab(tab);
  __syncthreads();
  const int blocks32 = (n32 + kSymWarps - 1) / kSymWarps;
  if ((int)blockIdx.x < blocks32) {
    const int warp = threadIdx.x >> 5, task = blockIdx.x * kSymWarps + warp;
    if (task < n32)   // warp-uniform
      near_sym_task<ADJ, MEET, 32>(tasks[task], sQ + warp * 128, leafStart, leafCount, leafCtr, recA, recB, K, tab, scr);
  } else {
    const int half = threadIdx.x >> 4, task = n32 + ((int)blockIdx.x - blocks32) * 2 * kSymWarps + half;
    if (task < nTasks)   // uniform over the half-warp
      near_sym_task<ADJ, MEET, 16>(tasks[task], sQ + half * 64, leafStart, leafCount, leafCtr, recA, recB, K, tab, scr);
  }
}

// ---------------------------------------------------------------------------
// The finishing kernel: the pairs that the symmetric tasks leave out (each
// leaf with itself, pairs with a leaf of a few panels, every pair when there
// are no tasks), the tasks' scratch sums, and the special pairs in FP64.
//
// A block of four warps takes up to 32 target panels of one leaf (one target
// per lane; a short group of mt targets gives each target 32/mt lanes).  The
// warps share all three sums -- whole source leaves when there are several,
// else equal parts of the leaf's panels; every fourth scratch slot and special
// pair -- and the partial sums are added in a fixed order.  The kernel is a
// chain of dependent loads per target, which four warps shorten (one warp per
// group took 23.4 us for 20,480 panels, four take 12.5).
// ---------------------------------------------------------------------------
// this lane's share (every step-th slot from first) of the scratch sums of panel xo of the leaf
template <typename P, typename S>
__device__ __forceinline__ void near_gather(int g0, int g1, int first, int step, int xo,
                                            const int *__restrict__ slot, const P *__restrict__ scr, S &a0, S &a1) {
#pragma unroll 4
  for (int i = g0 + first; i < g1; i += step) {
    const P v = scr[(size_t)slot[i] + xo];
    a0 += v.x;
    a1 += v.y;
  }
}

// this lane's share of the FP64 special-pair corrections of target X
__device__ __forceinline__ void special_sums(int X, int n, int first, int step, const int *__restrict__ spOff,
                                             const int *__restrict__ spSrc, const double4 *__restrict__ spK,
                                             const double *__restrict__ sgm, double &e0, double &e1) {
  const int end = spOff[X + 1];
#pragma unroll 4
  for (int e = spOff[X] + first; e < end; e += step) {
    const int Y = spSrc[e];
    const double4 d = spK[e];
    const double sp = sgm[Y], sd = sgm[n + Y];
    e0 += d.x * sd + d.y * sp;
    e1 += d.z * sd + d.w * sp;
  }
}

// adds the warps' and lanes' partial sums; thread t < mt of the block returns with target t's
struct NearPartial {
  double s0, s1, e0, e1;
};
__device__ __forceinline__ NearPartial near_partials(NearPartial p, int mt, int k) {
  __shared__ NearPartial red[kNearWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  red[warp][lane] = p;
  __syncthreads();
  NearPartial t{0.0, 0.0, 0.0, 0.0};
  if ((int)threadIdx.x < mt)
    for (int w = 0; w < kNearWarps; w++)
      for (int i = 0; i < k; i++) {
        const NearPartial v = red[w][threadIdx.x * k + i];
        t.s0 += v.s0;
        t.s1 += v.s1;
        t.e0 += v.e0;
        t.e1 += v.e1;
      }
  return t;
}

// this warp's share of source leaf S: all of it when the leaves are dealt over the warps, else a quarter
__device__ __forceinline__ void near_share(int warp, bool byLeaf, int cnt, int &j0, int &j1) {
  j0 = 0;
  j1 = cnt;
  if (!byLeaf) {
    const int part = ((cnt + kNearWarps - 1) / kNearWarps + 1) & ~1;
    j0 = min(cnt, warp * part);
    j1 = min(cnt, j0 + part);
  }
}

__device__ __forceinline__ void near_store(int X, int n, const NearPartial t, const double *__restrict__ area,
                                           double coef, int accumulate, double *out) {
  const double AX = area[X] * kFourPiI;
  const double v0 = coef * (AX * t.s0 + t.e0), v1 = coef * (AX * t.s1 + t.e1);
  out[X] = accumulate ? out[X] + v0 : v0;   // each output has exactly one writer
  out[X + n] = accumulate ? out[X + n] + v1 : v1;
}

template <bool ADJ>
__global__ void __launch_bounds__(kNearWarps * 32)
near_apply_f2_kernel(const int2 *__restrict__ work, const int *__restrict__ leafStart,
                     const int *__restrict__ leafCount, const int *__restrict__ ordOff,
                     const int *__restrict__ ordSrc, const double *__restrict__ leafCtr,
                     const float4 *__restrict__ tgtP, const float4 *__restrict__ tgtN,
                     const int *__restrict__ spOff, const int *__restrict__ spSrc, const double4 *__restrict__ spK,
                     const double *__restrict__ sgm, const double *__restrict__ area, int n, NearConstF K,
                     double coef, int accumulate, double *out, const int *__restrict__ gatOff,
                     const int *__restrict__ gatSlot, const float2 *__restrict__ scr) {
  __shared__ float4 sP[kNearWarps][16][4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int2 wk = work[blockIdx.x];
  const int L = wk.x;
  const int base = leafStart[L], cnt = leafCount[L];
  const int g0 = 32 * wk.y;
  const int mt = min(32, cnt - g0);   // targets in this group
  const int k = 32 / mt;              // lanes per target
  const int t = lane / k, sub = lane - t * k;
  const bool valid = t < mt;
  const int X = base + g0 + (valid ? t : 0);
  const float4 tp = tgtP[X], tn = tgtN[X];
  NearTargetsF2<1> tg;
  tg.nx[0] = f2(tn.x); tg.ny[0] = f2(tn.y); tg.nz[0] = f2(tn.z);
  const double cx = leafCtr[3 * L], cy = leafCtr[3 * L + 1], cz = leafCtr[3 * L + 2];
  float2 acc0 = f2(0.f), acc1 = f2(0.f);
  float *pf = reinterpret_cast<float *>(&sP[warp][lane >> 1][0]) + (lane & 1);
  const int p1 = ordOff[L + 1], p0 = ordOff[L];
  const bool byLeaf = p1 - p0 >= kNearWarps;
  for (int p = p0 + (byLeaf ? warp : 0); p < p1; p += byLeaf ? kNearWarps : 1) {
    const int S = ordSrc[p], sb = leafStart[S];
    int jb, je;
    near_share(warp, byLeaf, leafCount[S], jb, je);
    tg.x[0] = f2(tp.x + (float)(cx - leafCtr[3 * S]));
    tg.y[0] = f2(tp.y + (float)(cy - leafCtr[3 * S + 1]));
    tg.z[0] = f2(tp.z + (float)(cz - leafCtr[3 * S + 2]));
    for (int j0 = jb; j0 < je; j0 += 32) {
      const int m = min(32, je - j0);
      float4 a = make_float4(1e4f, 1e4f, 1e4f, 0.f), b = make_float4(0.f, 0.f, 0.f, 0.f);
      if (lane < m) {
        near_record<float>(sb + j0 + lane, n, tgtP, tgtN, area, sgm, a, b);
      }
      pf[0] = -a.x; pf[2] = -a.y; pf[4] = -a.z; pf[6] = a.w;
      pf[8] = b.x; pf[10] = b.y; pf[12] = b.z; pf[14] = ADJ ? -b.w : b.w;
      __syncwarp();
      const int np = (m + 1) >> 1;
      if (S == L) {   // warp-uniform
#pragma unroll 4
        for (int q = sub; q < np; q += k)
          near_pair2<ADJ, true>(sP[warp][q][0], sP[warp][q][1], sP[warp][q][2], sP[warp][q][3], tg, K, acc0,
                                acc1);
      } else {
#pragma unroll 4
        for (int q = sub; q < np; q += k)
          near_pair2<ADJ, false>(sP[warp][q][0], sP[warp][q][1], sP[warp][q][2], sP[warp][q][3], tg, K, acc0,
                                 acc1);
      }
      __syncwarp();
    }
  }
  float s0 = acc0.x + acc0.y, s1 = ADJ ? -(acc1.x + acc1.y) : acc1.x + acc1.y;
  NearPartial p{0.0, 0.0, 0.0, 0.0};
  if (valid) {
    const int first = warp * k + sub, step = kNearWarps * k;
    if (gatOff) near_gather(gatOff[L], gatOff[L + 1], first, step, X - base, gatSlot, scr, s0, s1);
    special_sums(X, n, first, step, spOff, spSrc, spK, sgm, p.e0, p.e1);
  }
  p.s0 = (double)s0;
  p.s1 = (double)s1;
  p = near_partials(p, mt, k);
  if ((int)threadIdx.x < mt) near_store(base + g0 + threadIdx.x, n, p, area, coef, accumulate, out);
}

// MEET: any two parts may hold coincident panels (near_terms)
template <bool ADJ, bool MEET>
__global__ void __launch_bounds__(kNearWarps * 32)
near_apply_kernel(const int2 *__restrict__ work, const int *__restrict__ leafStart,
                  const int *__restrict__ leafCount, const int *__restrict__ ordOff,
                  const int *__restrict__ ordSrc, const double *__restrict__ leafCtr,
                  const double4 *__restrict__ tgtP, const double4 *__restrict__ tgtN,
                  const int *__restrict__ spOff, const int *__restrict__ spSrc, const double4 *__restrict__ spK,
                  const double *__restrict__ sgm, const double *__restrict__ area, int n, NearConstD K, double coef,
                  int accumulate, double *out, const int *__restrict__ gatOff, const int *__restrict__ gatSlot,
                  const double2 *__restrict__ scr) {
  __shared__ double4 sA[kNearWarps][32], sB[kNearWarps][32];
  __shared__ double tab[kExpTab];
  load_exp_tab(tab);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int2 wk = work[blockIdx.x];
  const int L = wk.x;
  const int base = leafStart[L], cnt = leafCount[L];
  const int g0 = 32 * wk.y;
  const int mt = min(32, cnt - g0);   // targets in this group
  const int k = 32 / mt;              // lanes per target
  const int t = lane / k, sub = lane - t * k;
  const bool valid = t < mt;
  const int X = base + g0 + (valid ? t : 0);
  const double4 tp = tgtP[X], tn = tgtN[X];
  const double cx = leafCtr[3 * L], cy = leafCtr[3 * L + 1], cz = leafCtr[3 * L + 2];
  NearPartial p{0.0, 0.0, 0.0, 0.0};
  const int p1 = ordOff[L + 1], p0 = ordOff[L];
  const bool byLeaf = p1 - p0 >= kNearWarps;
  for (int q = p0 + (byLeaf ? warp : 0); q < p1; q += byLeaf ? kNearWarps : 1) {
    const int S = ordSrc[q], sb = leafStart[S];
    int jb, je;
    near_share(warp, byLeaf, leafCount[S], jb, je);
    const double tx = tp.x + (cx - leafCtr[3 * S]), ty = tp.y + (cy - leafCtr[3 * S + 1]),
                 tz = tp.z + (cz - leafCtr[3 * S + 2]);
    for (int j0 = jb; j0 < je; j0 += 32) {
      const int m = min(32, je - j0);
      if (lane < m)
        near_record<double>(sb + j0 + lane, n, tgtP, tgtN, area, sgm, sA[warp][lane], sB[warp][lane]);
      __syncwarp();
      if (MEET || S == L) {   // warp-uniform
#pragma unroll 2
        for (int jj = sub; jj < m; jj += k)
          near_pair<ADJ, true>(sA[warp][jj], sB[warp][jj], tx, ty, tz, tn, K, tab, p.s0, p.s1);
      } else {
#pragma unroll 2
        for (int jj = sub; jj < m; jj += k)
          near_pair<ADJ, false>(sA[warp][jj], sB[warp][jj], tx, ty, tz, tn, K, tab, p.s0, p.s1);
      }
      __syncwarp();
    }
  }
  if (valid) {
    const int first = warp * k + sub, step = kNearWarps * k;
    if (gatOff) near_gather(gatOff[L], gatOff[L + 1], first, step, X - base, gatSlot, scr, p.s0, p.s1);
    special_sums(X, n, first, step, spOff, spSrc, spK, sgm, p.e0, p.e1);
  }
  p = near_partials(p, mt, k);
  if ((int)threadIdx.x < mt) near_store(base + g0 + threadIdx.x, n, p, area, coef, accumulate, out);
}

// FP64 correction for every special pair: exact panelIA0 minus the
// one-point value the P2P loop computes for the same pair.
__global__ void special_coeff_kernel(long long nSp, const int *__restrict__ spDst, const int *__restrict__ spSrc,
                                     const double *__restrict__ vtx, const double *__restrict__ nrm,
                                     const double *__restrict__ area, int q, double kappa, double eps,
                                     double4 *spK, int *caseOut) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nSp) return;
  int Xi = spDst[e], Yi = spSrc[e];
  PanelD X, Y;
  const double *vx = vtx + 9 * (size_t)Xi, *vy = vtx + 9 * (size_t)Yi;
  for (int k = 0; k < 3; k++) {
    for (int c = 0; c < 3; c++) { X.v[k][c] = vx[3 * k + c]; Y.v[k][c] = vy[3 * k + c]; }
  }
  for (int c = 0; c < 3; c++) {
    X.a[0][c] = X.v[2][c] - X.v[1][c]; X.a[1][c] = X.v[0][c] - X.v[2][c]; X.a[2][c] = X.v[1][c] - X.v[0][c];
    Y.a[0][c] = Y.v[2][c] - Y.v[1][c]; Y.a[1][c] = Y.v[0][c] - Y.v[2][c]; Y.a[2][c] = Y.v[1][c] - Y.v[0][c];
    X.n[c] = nrm[3 * (size_t)Xi + c];
    Y.n[c] = nrm[3 * (size_t)Yi + c];
  }
  X.area = area[Xi];
  Y.area = area[Yi];
  double K[4], M[4] = {0, 0, 0, 0};
  int cs = 0;
  panel_ia0_d(q, kappa, eps, X, Y, Xi == Yi, K, &cs);
  if (Xi != Yi) {
    double r[3];
    for (int c = 0; c < 3; c++) {
      double mx = X.v[0][c] + 0.5 * (X.a[2][c] + 0.5 * X.a[0][c]);
      double my = Y.v[0][c] + 0.5 * (Y.a[2][c] + 0.5 * Y.a[0][c]);
      r[c] = mx - my;
    }
    if (r[0] != 0.0 || r[1] != 0.0 || r[2] != 0.0) {
      double y[4];
      ker4_d(kappa, eps, r, X.n, Y.n, y);
      for (int i = 0; i < 4; i++) M[i] = X.area * Y.area * y[i];
    }
  }
  spK[e] = make_double4(K[0] - M[0], K[1] - M[1], K[2] - M[2], K[3] - M[3]);
  if (caseOut) caseOut[e] = cs;
}

// Near field at panel quadrature order q > 1 (src/fmm.c:554-593 with
// panelIA0 at order q, src/numQuad.c:629-697), FP64 in every context.
// Forward (target X, K = panelIA0(X, Y)):
//   out_pot[X] += K0 s_dpdn[Y] + K1 s_pot[Y],  out_dpdn[X] += K2 s_dpdn[Y] + K3 s_pot[Y].
// ADJ, the transposed operator (target Y, K = panelIA0(X, Y) of the forward
// pair; the near-leaf relation is symmetric):
//   out_pot[Y] += K1 l_pot[X] + K3 l_dpdn[X],  out_dpdn[Y] += K0 l_pot[X] + K2 l_dpdn[X].
//
// FP64-bound: q^4 kernel evaluations per disjoint pair.  One warp per target
// panel, its q^2 points in shared memory, the sources of all its near leaves
// dealt flat over the lanes (leaves hold fewer panels than a warp has lanes),
// so 2,048 panels are 2,048 warps; the touching pairs, a few per target, are
// left out of that loop and taken from the special-pair table, which holds
// their order-q value minus the one-point value.
// One thread per target, looping over every near pair with the singular rules
// in line, took 9.4 ms for the product of 2,048 panels at q = 2 (243 near
// panels each, 16 blocks on the chip); with this it takes 0.093 ms.
constexpr int kQuadWarps = 4;
constexpr int kQuadPoints = 100;   // q <= 10

struct NearSums {
  double k0, k1, k2, k3;
};

// w times the four kernels (times 4 pi) at d = x - y, added to s
__device__ __forceinline__ void near_quad_eval(double dx, double dy, double dz, double nx, double ny, double nz,
                                               double mx, double my, double mz, double ip0, double w, double kappa,
                                               double kexp, double eps, double ieps, double kap2, const double *tab,
                                               NearSums &s) {
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double g = rsqrt_pos(r2), r = r2 * g;
  const double e = exp_tab(kexp * r, tab);
  const double c = (kappa * r + 1.0) * e;
  const double g2 = g * g, h = g2 * g;
  const double ipX = nx * dx + ny * dy + nz * dz, ipY = mx * dx + my * dy + mz * dz;
  const double t1 = ipY * h, t2 = ipX * h, u = ipX * t1;
  const double dd = (ip0 * g - 3.0 * u) * g2;
  s.k0 += w * (g - g * e);
  s.k1 += w * (t1 * (eps * c - 1.0));
  s.k2 += w * (t2 * (c * ieps - 1.0));
  s.k3 += w * (dd * (c - 1.0) - kap2 * e * u);
}

template <bool ADJ>
__global__ void __launch_bounds__(kQuadWarps * 32)
near_quad_kernel(int n, int q, const int *__restrict__ leafOfPanel, const int *__restrict__ leafStart,
                 const int *__restrict__ leafCount, const int *__restrict__ nearOff, const int *__restrict__ nearSrc,
                 const double *__restrict__ vtx, const double *__restrict__ nrm, const double *__restrict__ area,
                 const int *__restrict__ spOff, const int *__restrict__ spSrc, const double4 *__restrict__ spK,
                 double kappa, double eps, const double *__restrict__ sgm, double coef, int accumulate,
                 double *out) {
  __shared__ double tab[kExpTab];
  __shared__ double4 pts[kQuadWarps][kQuadPoints];   // the target's points and their weights
  load_exp_tab(tab);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int T = blockIdx.x * kQuadWarps + warp;
  const bool live = T < n;
  const int Ts = live ? T : 0;
  const double *t = c_tLeg[q], *w = c_wLeg[q];
  const int qq = q * q;
  const double *vt = vtx + 9 * (size_t)Ts;
  for (int i = lane; i < qq; i += 32) {
    const int a = i / q, b = i - a * q;
    double p[3];
    for (int k = 0; k < 3; k++) p[k] = vt[k] + t[a] * ((vt[3 + k] - vt[k]) + t[b] * (vt[6 + k] - vt[3 + k]));
    pts[warp][i] = make_double4(p[0], p[1], p[2], t[a] * w[a] * w[b]);
  }
  __syncthreads();
  if (!live) return;
  const double tn[3] = {nrm[3 * (size_t)T], nrm[3 * (size_t)T + 1], nrm[3 * (size_t)T + 2]};
  const double kexp = -kappa * kExpScale, ieps = 1.0 / eps, kap2 = kappa * kappa;
  const int L = leafOfPanel[T];
  const int s0 = spOff[T], s1 = spOff[T + 1];
  double e0 = 0.0, e1 = 0.0;   // sums without the target's area
  for (int p0 = nearOff[L], p1 = nearOff[L + 1]; p0 < p1; p0 += 32) {
    // 32 near leaves: their first panels and the running number of panels
    const int S = p0 + lane < p1 ? nearSrc[p0 + lane] : -1;
    const int cnt = S < 0 ? 0 : leafCount[S];
    int end = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += v;
    }
    const int shift = (S < 0 ? 0 : leafStart[S]) - (end - cnt);   // flat index to panel index
    const int total = __shfl_sync(0xffffffffu, end, 31);
    for (int i0 = 0; i0 < total; i0 += 32) {
      const int i = i0 + lane;
      int j = 0;   // the leaf of flat index i: the number of leaves that end at or before it
      for (int o = 16; o > 0; o >>= 1) {
        const int v = __shfl_sync(0xffffffffu, end, j + o - 1);
        if (v <= i) j += o;
      }
      const int Y = i + __shfl_sync(0xffffffffu, shift, j);
      if (i >= total) continue;
      int lo = s0, hi = s1;   // a touching panel is taken from the table
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (spSrc[mid] < Y) lo = mid + 1;
        else hi = mid;
      }
      if (lo < s1 && spSrc[lo] == Y) continue;
      const double *v = vtx + 9 * (size_t)Y;
      double v0[3], a2[3], a0[3], sn[3];
      for (int k = 0; k < 3; k++) {
        v0[k] = v[k];
        a2[k] = v[3 + k] - v[k];
        a0[k] = v[6 + k] - v[3 + k];
        sn[k] = nrm[3 * (size_t)Y + k];
      }
      const double ip0 = tn[0] * sn[0] + tn[1] * sn[1] + tn[2] * sn[2];
      NearSums K{0.0, 0.0, 0.0, 0.0};
      for (int a = 0; a < q; a++)
        for (int b = 0; b < q; b++) {
          const double ws = t[a] * w[a] * w[b];
          const double px = v0[0] + t[a] * (a2[0] + t[b] * a0[0]), py = v0[1] + t[a] * (a2[1] + t[b] * a0[1]),
                       pz = v0[2] + t[a] * (a2[2] + t[b] * a0[2]);
          for (int k = 0; k < qq; k++) {
            const double4 P = pts[warp][k];
            if (ADJ)   // panelIA0(source, target)
              near_quad_eval(px - P.x, py - P.y, pz - P.z, sn[0], sn[1], sn[2], tn[0], tn[1], tn[2], ip0, ws * P.w,
                             kappa, kexp, eps, ieps, kap2, tab, K);
            else
              near_quad_eval(P.x - px, P.y - py, P.z - pz, tn[0], tn[1], tn[2], sn[0], sn[1], sn[2], ip0, ws * P.w,
                             kappa, kexp, eps, ieps, kap2, tab, K);
          }
        }
      const double wp = 4.0 * area[Y] * sgm[Y], wd = 4.0 * area[Y] * sgm[n + Y];
      if (ADJ) {
        e0 += K.k1 * wp + K.k3 * wd;
        e1 += K.k0 * wp + K.k2 * wd;
      } else {
        e0 += K.k0 * wd + K.k1 * wp;
        e1 += K.k2 * wd + K.k3 * wp;
      }
    }
  }
  e0 *= area[T] * kFourPiI;
  e1 *= area[T] * kFourPiI;
  // the touching pairs: the table's value (spK, or spKT arranged for the transposed sums) plus the
  // one-point value that it leaves out
  for (int e = s0 + lane; e < s1; e += 32) {
    const int Y = spSrc[e];
    const double4 d = spK[e];
    const double sp = sgm[Y], sd = sgm[n + Y];
    double y[4] = {0.0, 0.0, 0.0, 0.0};
    if (Y != T) {
      const double *v = vtx + 9 * (size_t)Y;
      double r[3];
      for (int k = 0; k < 3; k++) {
        const double mx = vt[k] + 0.5 * ((vt[3 + k] - vt[k]) + 0.5 * (vt[6 + k] - vt[3 + k]));
        const double my = v[k] + 0.5 * ((v[3 + k] - v[k]) + 0.5 * (v[6 + k] - v[3 + k]));
        r[k] = ADJ ? my - mx : mx - my;
      }
      if (r[0] != 0.0 || r[1] != 0.0 || r[2] != 0.0) {
        const double *m = nrm + 3 * (size_t)Y;
        if (ADJ) ker4_d(kappa, eps, r, m, tn, y);
        else ker4_d(kappa, eps, r, tn, m, y);
      }
    }
    const double ww = area[T] * area[Y];
    if (ADJ) {
      e0 += (d.x + ww * y[3]) * sd + (d.y + ww * y[1]) * sp;
      e1 += (d.z + ww * y[2]) * sd + (d.w + ww * y[0]) * sp;
    } else {
      e0 += (d.x + ww * y[0]) * sd + (d.y + ww * y[1]) * sp;
      e1 += (d.z + ww * y[2]) * sd + (d.w + ww * y[3]) * sp;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    e0 += __shfl_xor_sync(0xffffffffu, e0, o);
    e1 += __shfl_xor_sync(0xffffffffu, e1, o);
  }
  if (lane == 0) {   // each output has exactly one writer
    out[T] = accumulate ? out[T] + coef * e0 : coef * e0;
    out[T + n] = accumulate ? out[T + n] + coef * e1 : coef * e1;
  }
}

namespace {

struct VKey {
  uint64_t a, b, c;
  bool operator==(const VKey &o) const { return a == o.a && b == o.b && c == o.c; }
};
struct VKeyHash {
  size_t operator()(const VKey &k) const {
    uint64_t h = k.a * 0x9E3779B97F4A7C15ULL;
    h ^= k.b + 0x7F4A7C159E3779B9ULL + (h << 6) + (h >> 2);
    h ^= k.c + 0x94D049BB133111EBULL + (h << 6) + (h >> 2);
    return (size_t)h;
  }
};
inline uint64_t dbits(double v) {
  if (v == 0.0) v = 0.0;  // -0.0 and 0.0 compare equal in nrCommonVtx
  uint64_t u;
  memcpy(&u, &v, 8);
  return u;
}

}  // namespace

// ---------------------------------------------------------------------------
// Special-pair search on the device: the panels sharing a vertex with X (by
// exact coordinates, -0.0 = 0.0, as nrCommonVtx, src/numQuad.c:312), X itself,
// kept when their leaves are near, ascending, as CSR by X.  The 3N corners are
// sorted by a 64-bit hash of their coordinates; equal-hash runs are checked
// for exact equality (a collision sends the search to the host path, as does
// a panel with more than kSpCand candidates).
// ---------------------------------------------------------------------------
constexpr int kSpCand = 64;

__device__ __forceinline__ unsigned long long vtx_bits(double v) {
  return (unsigned long long)__double_as_longlong(v == 0.0 ? 0.0 : v);
}
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {   // splitmix64 finaliser
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

__global__ void corner_keys_kernel(int nc, const double *__restrict__ vtx, unsigned long long *keys, int *vals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nc) return;
  const double *x = vtx + 3 * (size_t)i;   // corner i = vertex i%3 of panel i/3
  keys[i] = mix64(vtx_bits(x[0]) + mix64(vtx_bits(x[1]) + mix64(vtx_bits(x[2]))));
  vals[i] = i;
}

__global__ void corner_runs_kernel(int nc, const unsigned long long *__restrict__ keys, const int *__restrict__ vals,
                                   const double *__restrict__ vtx, int *flag, int *err) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nc) return;
  int f = 1;
  if (p > 0 && keys[p] == keys[p - 1]) {
    f = 0;
    const double *a = vtx + 3 * (size_t)vals[p], *b = vtx + 3 * (size_t)vals[p - 1];
    for (int k = 0; k < 3; k++)
      if (vtx_bits(a[k]) != vtx_bits(b[k])) atomicExch(err, 1);   // hash collision
  }
  flag[p] = f;
}

// gid: inclusive scan of the run flags (group g = gid - 1)
__global__ void corner_groups_kernel(int nc, const int *__restrict__ flag, const int *__restrict__ gid,
                                     const int *__restrict__ vals, int *gStart, int *cornerGroup) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= nc) return;
  const int g = gid[p] - 1;
  if (flag[p]) gStart[g] = p;
  if (p == nc - 1) gStart[g + 1] = nc;
  cornerGroup[vals[p]] = g;
}

// WRITE = false: count per panel into cnt; true: write the sources at off[X]
template <bool WRITE>
__global__ void special_pairs_kernel(int n, const int *__restrict__ cornerGroup, const int *__restrict__ gStart,
                                     const int *__restrict__ vals, const int *__restrict__ leafOf,
                                     const int *__restrict__ nearOff, const int *__restrict__ nearSorted, int *cnt,
                                     const int *__restrict__ off, int *spSrc, int *spDst, int *err) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x;
  if (X >= n) return;
  int cand[kSpCand];
  int m = 0;
  cand[m++] = X;
  for (int k = 0; k < 3; k++) {
    const int g = cornerGroup[3 * X + k];
    for (int p = gStart[g]; p < gStart[g + 1]; p++) {
      if (m == kSpCand) {
        atomicExch(err, 2);
        if (!WRITE) cnt[X] = 0;
        return;
      }
      cand[m++] = vals[p] / 3;
    }
  }
  for (int i = 1; i < m; i++) {   // insertion sort of the few candidates
    const int v = cand[i];
    int j = i - 1;
    while (j >= 0 && cand[j] > v) {
      cand[j + 1] = cand[j];
      j--;
    }
    cand[j + 1] = v;
  }
  const int L = leafOf[X];
  const int *ns = nearSorted + nearOff[L];
  const int nn = nearOff[L + 1] - nearOff[L];
  int o = WRITE ? off[X] : 0, c = 0;
  for (int i = 0; i < m; i++) {
    if (i > 0 && cand[i] == cand[i - 1]) continue;
    const int Y = cand[i], LY = leafOf[Y];
    int lo = 0, hi = nn;   // LY in the sorted near list of L?
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (ns[mid] < LY) lo = mid + 1;
      else hi = mid;
    }
    if (lo < nn && ns[lo] == LY) {
      if (WRITE) {
        spSrc[o] = Y;
        spDst[o] = X;
        o++;
      }
      c++;
    }
  }
  if (!WRITE) cnt[X] = c;
}

// 1: tables built (c.d_spOff, c.d_spSrc, *d_spDst, c.nSpecial); 0: use the
// host search instead; -1: CUDA error (message set)
static int special_pairs_device(Context &c, const std::vector<int> &nearSortedFlat, int **d_spDst) {
  const int n = c.n, nc = 3 * n;
  cudaStream_t s = c.stream;
  DevArena tmp;
  ArenaScope scope{tmp};
  unsigned long long *keys = nullptr, *keysS = nullptr;
  int *vals = nullptr, *valsS = nullptr, *flag = nullptr, *gid = nullptr, *cornerGroup = nullptr, *gStart = nullptr;
  int *cnt = nullptr, *err = nullptr, *d_nearSorted = nullptr;
  if (!tmp.alloc_n(&keys, nc) || !tmp.alloc_n(&keysS, nc) || !tmp.alloc_n(&vals, nc) || !tmp.alloc_n(&valsS, nc) ||
      !tmp.alloc_n(&flag, nc) || !tmp.alloc_n(&gid, nc) || !tmp.alloc_n(&cornerGroup, nc) ||
      !tmp.alloc_n(&gStart, (size_t)nc + 1) || !tmp.alloc_n(&cnt, (size_t)n + 1) || !tmp.alloc_n(&err, 1) ||
      !tmp.upload(&d_nearSorted, nearSortedFlat, s))
    return -1;
  FB_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
  size_t tb1 = 0, tb2 = 0, tb3 = 0;
  FB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb1, keys, keysS, vals, valsS, nc, 0, 64, s));
  FB_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tb2, flag, gid, nc, s));
  FB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb3, cnt, cnt, n + 1, s));
  void *tbuf = nullptr;
  if (!tmp.alloc(&tbuf, std::max(tb1, std::max(tb2, tb3)))) return -1;
  const size_t tbytes = std::max(tb1, std::max(tb2, tb3));
  corner_keys_kernel<<<ceil_div(nc, 256), 256, 0, s>>>(nc, c.d_vtx, keys, vals);
  size_t tb = tbytes;
  FB_CUDA(cub::DeviceRadixSort::SortPairs(tbuf, tb, keys, keysS, vals, valsS, nc, 0, 64, s));
  corner_runs_kernel<<<ceil_div(nc, 256), 256, 0, s>>>(nc, keysS, valsS, c.d_vtx, flag, err);
  tb = tbytes;
  FB_CUDA(cub::DeviceScan::InclusiveSum(tbuf, tb, flag, gid, nc, s));
  corner_groups_kernel<<<ceil_div(nc, 256), 256, 0, s>>>(nc, flag, gid, valsS, gStart, cornerGroup);
  special_pairs_kernel<false><<<ceil_div(n, 128), 128, 0, s>>>(n, cornerGroup, gStart, valsS, c.d_leafOfPanel,
                                                               c.d_nearOff, d_nearSorted, cnt, nullptr, nullptr,
                                                               nullptr, err);
  FB_CUDA(cudaMemsetAsync(cnt + n, 0, sizeof(int), s));
  if (!c.arena.alloc_n(&c.d_spOff, (size_t)n + 1)) return -1;
  tb = tbytes;
  FB_CUDA(cub::DeviceScan::ExclusiveSum(tbuf, tb, cnt, c.d_spOff, n + 1, s));
  int hErr = 0, total = 0;
  FB_CUDA(cudaMemcpyAsync(&hErr, err, sizeof(int), cudaMemcpyDeviceToHost, s));
  FB_CUDA(cudaMemcpyAsync(&total, c.d_spOff + n, sizeof(int), cudaMemcpyDeviceToHost, s));
  FB_CUDA(cudaStreamSynchronize(s));
  FB_CUDA(cudaGetLastError());
  if (hErr) return 0;
  c.nSpecial = total;
  if (!c.arena.alloc_n(&c.d_spSrc, (size_t)std::max(total, 1)) || !c.arena.alloc_n(d_spDst, (size_t)std::max(total, 1)))
    return -1;
  special_pairs_kernel<true><<<ceil_div(n, 128), 128, 0, s>>>(n, cornerGroup, gStart, valsS, c.d_leafOfPanel,
                                                              c.d_nearOff, d_nearSorted, nullptr, c.d_spOff,
                                                              c.d_spSrc, *d_spDst, err);
  FB_CUDA(cudaGetLastError());
  FB_CUDA(cudaStreamSynchronize(s));   // the temporaries are freed on return
  return 1;
}

static bool special_pairs_host(Context &c, const std::vector<int> &nearSortedFlat, int **d_spDst);
static bool setup_near_targets(Context &c);
static bool setup_near_parts(Context &c);

bool setup_near(Context &c) {
  const PanelTree &pt = c.pt;
  cudaStream_t s = c.stream;
  // -q=1: the one-point P2P kernels plus the FP64 special-pair corrections;
  // -q>1: near_quad_kernel (panelIA0 at order q for every near pair).  The
  // special-pair table is built at order q either way (the preconditioners
  // assemble their blocks from it).
  if (c.prm.quad_order < 1 || c.prm.quad_order > 10) {
    set_error("panel quadrature order -q=%d outside 1..10", c.prm.quad_order);
    return false;
  }
  // the direct operator: every leaf is near every leaf
  if (c.dense) {
    PanelTree &w = c.pt;
    w.nearOff.assign(w.nLeaves + 1, 0);
    w.nearSrc.clear();
    w.nearDst.clear();
    for (int L = 0; L < w.nLeaves; L++) {
      w.nearOff[L] = (int)w.nearSrc.size();
      for (int S = 0; S < w.nLeaves; S++) { w.nearSrc.push_back(S); w.nearDst.push_back(L); }
    }
    w.nearOff[w.nLeaves] = (int)w.nearSrc.size();
    if (!c.arena.upload(&c.d_nearOff, w.nearOff, s) || !c.arena.upload(&c.d_nearSrc, w.nearSrc, s)) return false;
  }
  c.maxLeaf = 0;
  c.nearPanelPairs = 0;
  for (int L = 0; L < pt.nLeaves; L++) {
    int cnt = pt.leafCount[L];
    c.maxLeaf = std::max(c.maxLeaf, cnt);
    long long srcs = 0;
    for (int p = pt.nearOff[L]; p < pt.nearOff[L + 1]; p++) srcs += pt.leafCount[pt.nearSrc[p]];
    c.nearPanelPairs += srcs * cnt;
  }
  if (!setup_near_parts(c)) return false;

  StageTimer tm("near_setup", s);
  // special pairs: panels sharing a vertex (exact coordinates), restricted to
  // near leaf pairs, plus the panel itself -- on the device, or on the host
  // when the device search declines
  std::vector<int> nearSortedFlat(pt.nearSrc.size());
  for (int L = 0; L < pt.nLeaves; L++) {
    std::copy(pt.nearSrc.begin() + pt.nearOff[L], pt.nearSrc.begin() + pt.nearOff[L + 1],
              nearSortedFlat.begin() + pt.nearOff[L]);
    std::sort(nearSortedFlat.begin() + pt.nearOff[L], nearSortedFlat.begin() + pt.nearOff[L + 1]);
  }
  int *d_spDst = nullptr;
  // FABIPB_B200_HOST_SPECIAL=1 forces the host search (the tests compare the two)
  const int onDevice = getenv("FABIPB_B200_HOST_SPECIAL") ? 0 : special_pairs_device(c, nearSortedFlat, &d_spDst);
  if (onDevice < 0) return false;
  if (onDevice == 0 && !special_pairs_host(c, nearSortedFlat, &d_spDst)) return false;
  tm.mark("special_pairs");
  if (!c.arena.alloc_n(&c.d_spK, (size_t)std::max<long long>(c.nSpecial, 1))) return false;
  if (c.nSpecial > 0) {
    special_coeff_kernel<<<ceil_div(c.nSpecial, 128), 128, 0, s>>>(
        c.nSpecial, d_spDst, c.d_spSrc, c.d_vtx, c.d_nrm, c.d_area, c.prm.quad_order, c.prm.kappa,
        c.epsilon, c.d_spK, nullptr);
    FB_CUDA(cudaGetLastError());
  }
  tm.mark("special_coeff");
  return setup_near_targets(c);
}

// The host search (used when the device search declines): vertex ids from a
// hash map of exact coordinates, per panel its sharing panels, on host threads.
static bool special_pairs_host(Context &c, const std::vector<int> &nearSortedFlat, int **d_spDst) {
  const PanelTree &pt = c.pt;
  const int n = c.n;
  cudaStream_t s = c.stream;
  if (c.h_vtx.size() != 9 * (size_t)n) {   // the device tree keeps the tree-order panels on the device only
    c.h_vtx.resize(9 * (size_t)n);
    FB_CUDA(cudaMemcpyAsync(c.h_vtx.data(), c.d_vtx, 9 * (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, s));
    FB_CUDA(cudaStreamSynchronize(s));
  }
  std::unordered_map<VKey, int, VKeyHash> vid;
  vid.reserve((size_t)n * 2);
  std::vector<int> pv(3 * (size_t)n);
  for (int i = 0; i < n; i++)
    for (int k = 0; k < 3; k++) {
      const double *x = &c.h_vtx[9 * (size_t)i + 3 * k];
      VKey key{dbits(x[0]), dbits(x[1]), dbits(x[2])};
      auto it = vid.find(key);
      int id;
      if (it == vid.end()) {
        id = (int)vid.size();
        vid.emplace(key, id);
      } else {
        id = it->second;
      }
      pv[3 * (size_t)i + k] = id;
    }
  const int nv = (int)vid.size();
  std::vector<int> vOff(nv + 1, 0), vPan(3 * (size_t)n);
  for (int i = 0; i < 3 * n; i++) vOff[pv[i] + 1]++;
  for (int v = 0; v < nv; v++) vOff[v + 1] += vOff[v];
  {
    std::vector<int> cur(vOff.begin(), vOff.end() - 1);
    for (int i = 0; i < 3 * n; i++) vPan[cur[pv[i]]++] = i / 3;
  }
  std::vector<int> leafOf(n);
  for (int L = 0; L < pt.nLeaves; L++)
    for (int k = 0; k < pt.leafCount[L]; k++) leafOf[pt.leafStart[L] + k] = L;
  // per panel: itself and the panels sharing a vertex with it, ascending,
  // kept when their leaves are near; chunks of panels on host threads, merged
  // in panel order
  std::vector<int> spOff(n + 1, 0), spDst, spSrc;
  const int nth = (int)std::max(1u, std::min(32u, std::thread::hardware_concurrency()));
  std::vector<std::vector<int>> partSrc(nth);
  std::vector<int> cntOf(n, 0);
  auto work_range = [&](int th) {
    const int x0 = (int)((long long)n * th / nth), x1 = (int)((long long)n * (th + 1) / nth);
    std::vector<int> cand;
    std::vector<int> &out = partSrc[th];
    out.reserve(16 * (size_t)(x1 - x0));
    for (int X = x0; X < x1; X++) {
      cand.clear();
      cand.push_back(X);
      for (int k = 0; k < 3; k++) {
        int v = pv[3 * (size_t)X + k];
        for (int e = vOff[v]; e < vOff[v + 1]; e++) cand.push_back(vPan[e]);
      }
      std::sort(cand.begin(), cand.end());
      cand.erase(std::unique(cand.begin(), cand.end()), cand.end());
      const int *nb = nearSortedFlat.data() + pt.nearOff[leafOf[X]];
      const int *ne = nearSortedFlat.data() + pt.nearOff[leafOf[X] + 1];
      int cnt = 0;
      for (int Y : cand)
        if (std::binary_search(nb, ne, leafOf[Y])) {
          out.push_back(Y);
          cnt++;
        }
      cntOf[X] = cnt;
    }
  };
  {
    std::vector<std::thread> pool;
    for (int th = 1; th < nth; th++) pool.emplace_back(work_range, th);
    work_range(0);
    for (auto &th : pool) th.join();
  }
  for (int X = 0; X < n; X++) spOff[X + 1] = spOff[X] + cntOf[X];
  spSrc.reserve(spOff[n]);
  for (int th = 0; th < nth; th++) spSrc.insert(spSrc.end(), partSrc[th].begin(), partSrc[th].end());
  spDst.resize(spSrc.size());
  for (int X = 0; X < n; X++)
    for (int e = spOff[X]; e < spOff[X + 1]; e++) spDst[e] = X;
  c.nSpecial = (long long)spSrc.size();
  if (!c.arena.upload(&c.d_spOff, spOff, s)) return false;
  if (!c.arena.upload(&c.d_spSrc, spSrc, s)) return false;
  if (!c.arena.upload(d_spDst, spDst, s)) return false;
  return true;
}

// The parts that the near-field kernels pair up: the leaves.  A direct context
// pairs everything with everything, so in FP64, where positions need no
// leaf's frame, its parts are equal runs of panels (equal_part_length).
static bool equal_parts(const Context &c) { return c.dense && !c.mixed && c.prm.quad_order == 1; }

// the indices of small non-negative keys, the largest first, equal ones in order (a counting sort)
static std::vector<int> by_decreasing(const std::vector<int> &key) {
  int top = 0;
  for (int k : key) top = std::max(top, k);
  std::vector<int> at(top + 2, 0), out(key.size());
  for (int k : key) at[top - k + 1]++;
  for (int k = 0; k <= top; k++) at[k + 1] += at[k];
  for (size_t i = 0; i < key.size(); i++) out[at[top - key[i]]++] = (int)i;
  return out;
}

static bool setup_near_parts(Context &c) {
  const PanelTree &pt = c.pt;
  cudaStream_t s = c.stream;
  c.partStart = pt.leafStart;
  c.partCount = pt.leafCount;
  c.d_partStart = c.d_leafStart;
  c.d_partCount = c.d_leafCount;
  c.d_partOf = c.d_leafOfPanel;
  c.d_partCtr = c.d_leafCtr;
  std::vector<int> partOf;
  std::vector<double> ctr;
  if (equal_parts(c)) {
    const int len = equal_part_length(c.n);
    c.partStart.clear();
    c.partCount.clear();
    partOf.resize(c.n);
    for (int i = 0; i < c.n; i += len) {
      ctr.insert(ctr.end(), 3, 0.0);   // one frame for all: coincident panels of two parts differ by exactly 0
      for (int j = i; j < std::min(c.n, i + len); j++) partOf[j] = (int)c.partStart.size();
      c.partStart.push_back(i);
      c.partCount.push_back(std::min(len, c.n - i));
    }
    if (!c.arena.upload(&c.d_partStart, c.partStart, s) || !c.arena.upload(&c.d_partCount, c.partCount, s) ||
        !c.arena.upload(&c.d_partOf, partOf, s) || !c.arena.upload(&c.d_partCtr, ctr, s))
      return false;
  }
  // the finishing kernel's blocks: (part, group of 32 targets), the largest parts first
  std::vector<int2> work;
  for (int L : by_decreasing(c.partCount))
    for (int g = 0; g * 32 < c.partCount[L]; g++) work.push_back(make_int2(L, g));
  c.nWork = (int)work.size();
  if (!c.arena.upload(&c.d_work, work, s)) return false;
  FB_CUDA(cudaStreamSynchronize(s));   // the host vectors go out of scope
  return true;
}

// The symmetric near field's tasks: every unordered pair of distinct near
// parts whose smaller one has at least FB_NEAR_SYM_MIN_LEAF panels, the larger
// on the register side, largest tasks first, cut into chunks by
// plan_near_tasks.  FABIPB_B200_NEAR_SYM=0 turns them off (every pair in the
// finishing kernel), as does a plan without tasks.  In FP64 a pair also needs
// FB_NEAR_SYM64_MIN_PAIRS panel pairs -- below that a 16 x 16 tile is so empty
// that two ordered passes cost less -- and the tasks at least half of all
// panel pairs, else their launches cost more than they save (1,280 panels in
// leaves of 5: a GMRES solve took 1.04 ms with tasks on every pair, 1.01 in
// ordered passes).
#ifndef FB_NEAR_SYM_MIN_LEAF
#define FB_NEAR_SYM_MIN_LEAF 4
#endif
#ifndef FB_NEAR_SYM64_MIN_PAIRS
#define FB_NEAR_SYM64_MIN_PAIRS 128
#endif
// cost of a padded pair on a half-warp, percent of that on a warp
#ifndef FB_NEAR_SYM16_COST
#define FB_NEAR_SYM16_COST 110
#endif
static bool setup_near_sym(Context &c) {
  c.nSymTasks = c.nSym32 = 0;
  const PanelTree &pt = c.pt;
  cudaStream_t s = c.stream;
  const char *env = getenv("FABIPB_B200_NEAR_SYM");
  const bool equal = equal_parts(c);
  const int nParts = (int)c.partCount.size();
  const std::vector<int> &count = c.partCount;
  const size_t esz = c.mixed ? sizeof(float2) : sizeof(double2);
  bool off = (env && atoi(env) == 0) || (c.dense && c.prm.quad_order > 1);
  auto on_tasks = [&](int a, int b) {
    return !off && a != b && std::min(count[a], count[b]) >= FB_NEAR_SYM_MIN_LEAF &&
           (c.mixed || (long long)count[a] * count[b] >= FB_NEAR_SYM64_MIN_PAIRS);
  };
  // the near parts of part L
  std::vector<int> all;
  if (equal)
    for (int L = 0; L < nParts; L++) all.push_back(L);
  auto near_begin = [&](int L) { return equal ? all.data() : pt.nearSrc.data() + pt.nearOff[L]; };
  auto near_end = [&](int L) { return equal ? all.data() + nParts : pt.nearSrc.data() + pt.nearOff[L + 1]; };
  if (!off && !c.mixed) {
    long long sum = 0, on = 0;
    for (int L = 0; L < nParts; L++)
      for (const int *p = near_begin(L); p != near_end(L); p++) {
        const long long k = (long long)count[L] * count[*p];
        sum += k;
        if (on_tasks(L, *p)) on += k;
      }
    off = 2 * on < sum;
  }
  NearPlan plan;
  if (!off) {
    const double directLimit = !c.dense ? 0.0 : equal ? equal_part_scratch(c.n) : 1.02 * kNearScratch;
    plan = plan_near_tasks(count, esz, directLimit, [&](auto &&f) {
      for (int L = 0; L < nParts; L++)
        for (const int *p = near_begin(L); p != near_end(L); p++)
          if (*p > L) f(L, *p, on_tasks(L, *p));
    });
    off = !plan.tasks;
  }
  if (!off) {
    const int chunk = plan.chunk;
    constexpr long long kTopCost = 1 << 20;
    std::vector<NearTask> tasks;
    std::vector<int> cost;   // panel pairs, at most kTopCost
    std::vector<char> half;
    int top16 = 0;           // the dearest half-warp task
    std::vector<int> gatOff(nParts + 1, 0);
    long long tot = 0;
    for (int L = 0; L < nParts; L++)
      for (const int *p = near_begin(L); p != near_end(L); p++) {
        const int S = *p;
        if (S <= L || !on_tasks(L, S)) continue;
        const int R = count[L] >= count[S] ? L : S, T = R == L ? S : L;
        const int cr = count[R], ct = count[T];
        // the half-warp where its padding to 16-panel groups and tiles saves more than its cost
        const long long p32 = (long long)((cr + 31) / 32) * ((ct + 31) / 32) * 1024;
        const long long p16 = (long long)((cr + 15) / 16) * ((ct + 15) / 16) * 256;
        const bool small = p16 * FB_NEAR_SYM16_COST < p32 * 100;
        const int nch = (cr + chunk - 1) / chunk;
        const int scrR = (int)tot;
        tot += cr;
        gatOff[R + 1]++;
        gatOff[T + 1] += nch;
        for (int r0 = 0; r0 < cr; r0 += chunk) {
          const int r1 = std::min(cr, r0 + chunk);
          tasks.push_back(NearTask{R, T, r0, r1, scrR, (int)tot});
          tot += ct;
          cost.push_back((int)std::min((long long)(r1 - r0) * ct, kTopCost));
          half.push_back(small);
          if (small) top16 = std::max(top16, cost.back());
          c.nSym32 += small ? 0 : 1;
        }
      }
    c.nSymTasks = (int)tasks.size();
    if (c.nSymTasks > 0) {
      std::vector<NearTask> sorted;
      sorted.reserve(tasks.size());
      // the warp tasks first, then the half-warp ones (two to a warp, so neighbours should cost the same), each by
      // decreasing cost
      for (size_t i = 0; i < tasks.size(); i++)
        if (!half[i]) cost[i] += top16 + 1;
      for (int i : by_decreasing(cost)) sorted.push_back(tasks[i]);
      // every part's slots, in the order of the tasks' making
      for (int L = 0; L < nParts; L++) gatOff[L + 1] += gatOff[L];
      std::vector<int> gatSlot(gatOff[nParts]), at(gatOff.begin(), gatOff.end() - 1);
      for (const NearTask &t : tasks) {
        if (t.r0 == 0) gatSlot[at[t.R]++] = t.scrR;
        gatSlot[at[t.T]++] = t.scrT;
      }
      if (!c.arena.upload(&c.d_symTask, sorted, s) || !c.arena.upload(&c.d_gatOff, gatOff, s) ||
          !c.arena.upload(&c.d_gatSlot, gatSlot, s) || !c.arena.alloc(&c.d_symScr, esz * (size_t)tot) ||
          !c.arena.alloc(&c.d_recA, 2 * esz * (size_t)c.n) || !c.arena.alloc(&c.d_recB, 2 * esz * (size_t)c.n))
        return false;
      FB_CUDA(cudaStreamSynchronize(s));   // the host vectors go out of scope
    }
  }
  if (c.nSymTasks == 0 && !equal) {   // every pair in the finishing kernel
    c.d_ordOff = c.d_nearOff;
    c.d_ordSrc = c.d_nearSrc;
    return true;
  }
  std::vector<int> ordOff(nParts + 1, 0), ordSrc;
  for (int L = 0; L < nParts; L++) {
    for (const int *p = near_begin(L); p != near_end(L); p++)
      if (!on_tasks(L, *p)) ordSrc.push_back(*p);
    ordOff[L + 1] = (int)ordSrc.size();
  }
  if (!c.arena.upload(&c.d_ordOff, ordOff, s) || !c.arena.upload(&c.d_ordSrc, ordSrc, s)) return false;
  FB_CUDA(cudaStreamSynchronize(s));
  return true;
}

// static target geometry relative to the leaf centres
static bool setup_near_targets(Context &c) {
  const int n = c.n;
  cudaStream_t s = c.stream;
  size_t vb = c.mixed ? sizeof(float4) : sizeof(double4);
  if (!c.arena.alloc(&c.d_tgtP, vb * n) || !c.arena.alloc(&c.d_tgtN, vb * n)) return false;
  if (c.mixed) {
    near_targets_kernel<float><<<ceil_div(n, 256), 256, 0, s>>>(
        n, c.d_vtx, c.d_nrm, c.d_area, c.d_partOf, c.d_partCtr, (float4 *)c.d_tgtP, (float4 *)c.d_tgtN);
  } else {
    near_targets_kernel<double><<<ceil_div(n, 256), 256, 0, s>>>(
        n, c.d_vtx, c.d_nrm, c.d_area, c.d_partOf, c.d_partCtr, (double4 *)c.d_tgtP, (double4 *)c.d_tgtN);
  }
  FB_CUDA(cudaGetLastError());
  return setup_near_sym(c);
}

template <bool ADJ>
static void launch_near_f32(Context &c, const double *sgm, double coef, double *out, cudaStream_t s, bool accumulate) {
  const double kap = c.prm.kappa, eps = c.epsilon;
  const NearConstF K{(float)kap, (float)(-kap * 1.4426950408889634), (float)eps, (float)(1.0 / eps),
                     (float)(kap * kap)};
  const float4 *tgtP = (const float4 *)c.d_tgtP, *tgtN = (const float4 *)c.d_tgtN;
  float4 *recA = (float4 *)c.d_recA, *recB = (float4 *)c.d_recB;
  if (c.nSymTasks > 0) {
    near_pack_kernel<float><<<ceil_div(c.n, 256), 256, 0, s>>>(c.n, tgtP, tgtN, c.d_area, sgm, recA, recB);
    const unsigned blocks = ceil_div(c.nSym32, kSymWarps) + ceil_div(c.nSymTasks - c.nSym32, 2 * kSymWarps);
    near_sym_f2_kernel<ADJ><<<blocks, kSymWarps * 32, 0, s>>>(c.nSym32, c.nSymTasks, c.d_symTask, c.d_partStart,
                                                              c.d_partCount, c.d_partCtr, recA, recB, K,
                                                              (float2 *)c.d_symScr);
    c.launches += 2;
  }
  near_apply_f2_kernel<ADJ><<<c.nWork, kNearWarps * 32, 0, s>>>(
      c.d_work, c.d_partStart, c.d_partCount, c.d_ordOff, c.d_ordSrc, c.d_partCtr, tgtP, tgtN, c.d_spOff, c.d_spSrc,
      ADJ ? c.d_spKT : c.d_spK, sgm, c.d_area, c.n, K, coef, accumulate ? 1 : 0, out, c.d_gatOff, c.d_gatSlot,
      (const float2 *)c.d_symScr);
  c.launches += 1;
}

// FP64 contexts, and the FP64 residuals of a mixed context (its own records; the scratch is FP32
// there, so every pair goes to the finishing kernel)
template <bool ADJ>
static void launch_near_f64(Context &c, const double *sgm, double coef, double *out, cudaStream_t s, bool accumulate) {
  const double kap = c.prm.kappa, eps = c.epsilon;
  const NearConstD K{kap, -kap * kExpScale, eps, 1.0 / eps, kap * kap};
  const bool own = !c.mixed, sym = own && c.nSymTasks > 0, meet = equal_parts(c);
  const double4 *tgtP = (const double4 *)(own ? c.d_tgtP : c.d_tgtP64);
  const double4 *tgtN = (const double4 *)(own ? c.d_tgtN : c.d_tgtN64);
  if (sym) {
    double4 *recA = (double4 *)c.d_recA, *recB = (double4 *)c.d_recB;
    near_pack_kernel<double><<<ceil_div(c.n, 256), 256, 0, s>>>(c.n, tgtP, tgtN, c.d_area, sgm, recA, recB);
    const unsigned blocks = ceil_div(c.nSym32, kSymWarps) + ceil_div(c.nSymTasks - c.nSym32, 2 * kSymWarps);
    auto kern = meet ? near_sym_kernel<ADJ, true> : near_sym_kernel<ADJ, false>;
    kern<<<blocks, kSymWarps * 32, 0, s>>>(c.nSym32, c.nSymTasks, c.d_symTask, c.d_partStart, c.d_partCount,
                                           c.d_partCtr, recA, recB, K, (double2 *)c.d_symScr);
    c.launches += 2;
  }
  auto apply = meet ? near_apply_kernel<ADJ, true> : near_apply_kernel<ADJ, false>;
  apply<<<c.nWork, kNearWarps * 32, 0, s>>>(
      c.d_work, c.d_partStart, c.d_partCount, own ? c.d_ordOff : c.d_nearOff, own ? c.d_ordSrc : c.d_nearSrc,
      c.d_partCtr, tgtP, tgtN, c.d_spOff, c.d_spSrc, ADJ ? c.d_spKT : c.d_spK, sgm, c.d_area, c.n, K, coef,
      accumulate ? 1 : 0, out, sym ? c.d_gatOff : nullptr, c.d_gatSlot, (const double2 *)c.d_symScr);
  c.launches += 1;
}

// FP64 records in a mixed context, for the FP64 residuals of iterative
// refinement (built at context set-up)
static bool setup_near_fp64(Context &c) {
  if (c.d_tgtP64) return true;
  const int n = c.n;
  const size_t vb = sizeof(double4) * (size_t)n;
  if (!c.arena.alloc(&c.d_tgtP64, vb) || !c.arena.alloc(&c.d_tgtN64, vb)) return false;
  near_targets_kernel<double><<<ceil_div(n, 256), 256, 0, c.stream>>>(n, c.d_vtx, c.d_nrm, c.d_area, c.d_leafOfPanel,
                                                                      c.d_leafCtr, (double4 *)c.d_tgtP64,
                                                                      (double4 *)c.d_tgtN64);
  FB_CUDA(cudaGetLastError());
  return true;
}

// Transposed special-pair table: entry (X, Y) of row X holds the correction
// of the pair (Y, X) arranged for the ADJ epilogue
// (out_pot += dK3(Y,X) l_dpdn + dK1(Y,X) l_pot, out_dpdn += dK2(Y,X) l_dpdn + dK0(Y,X) l_pot).
__global__ void special_transpose_kernel(long long nSp, const long long *__restrict__ mate, const double4 *__restrict__ spK,
                                         double4 *spKT) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nSp) return;
  const double4 d = spK[mate[e]];
  spKT[e] = make_double4(d.w, d.y, d.z, d.x);
}

// mate[e] of entry e = (X, Y): the index of (Y, X); *bad = X + 1 when missing
__global__ void special_mate_kernel(int n, const int *__restrict__ spOff, const int *__restrict__ spSrc,
                                    long long *mate, int *bad) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x;
  if (X >= n) return;
  for (int e = spOff[X]; e < spOff[X + 1]; e++) {
    const int Y = spSrc[e];
    int lo = spOff[Y], hi = spOff[Y + 1];
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (spSrc[mid] < X) lo = mid + 1;
      else hi = mid;
    }
    if (lo < spOff[Y + 1] && spSrc[lo] == X) mate[e] = lo;
    else atomicExch(bad, X + 1);
  }
}

static bool setup_near_adjoint(Context &c) {
  if (c.d_spKT) return true;
  // the special-pair set is symmetric (shared vertex, near leaf pairs): find
  // for every entry (X, Y) the entry (Y, X), by binary search in the
  // (ascending) row of Y, on the device
  const int n = c.n;
  DevArena tmp;
  ArenaScope scope{tmp};
  long long *d_mate = nullptr;
  int *d_bad = nullptr;
  if (!tmp.alloc_n(&d_mate, (size_t)std::max<long long>(c.nSpecial, 1)) || !tmp.alloc_n(&d_bad, 1)) return false;
  FB_CUDA(cudaMemsetAsync(d_bad, 0, sizeof(int), c.stream));
  special_mate_kernel<<<ceil_div(n, 256), 256, 0, c.stream>>>(n, c.d_spOff, c.d_spSrc, d_mate, d_bad);
  int bad = 0;
  FB_CUDA(cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
  FB_CUDA(cudaStreamSynchronize(c.stream));
  FB_CHECK(bad == 0, "special pair (%d, .) has no mirror entry", bad - 1);
  if (!c.arena.alloc_n(&c.d_spKT, (size_t)std::max<long long>(c.nSpecial, 1))) return false;
  if (c.nSpecial > 0)
    special_transpose_kernel<<<ceil_div(c.nSpecial, 256), 256, 0, c.stream>>>(c.nSpecial, d_mate, c.d_spK, c.d_spKT);
  FB_CUDA(cudaGetLastError());
  FB_CUDA(cudaStreamSynchronize(c.stream));   // the mates are freed on return
  return true;
}

bool launch_near(Context &c, const double *sgm, double coef, double *out, bool adjoint, bool fp64,
                 cudaStream_t stream, bool accumulate) {
  if (adjoint && !setup_near_adjoint(c)) return false;
  cudaStream_t s = stream ? stream : c.stream;
  const bool acc = accumulate;
  if (c.prm.quad_order > 1) {   // every near pair by panelIA0 at order q, in FP64 in every context
    auto kern = adjoint ? near_quad_kernel<true> : near_quad_kernel<false>;
    kern<<<ceil_div(c.n, kQuadWarps), kQuadWarps * 32, 0, s>>>(
        c.n, c.prm.quad_order, c.d_leafOfPanel, c.d_leafStart, c.d_leafCount, c.d_nearOff, c.d_nearSrc, c.d_vtx,
        c.d_nrm, c.d_area, c.d_spOff, c.d_spSrc, adjoint ? c.d_spKT : c.d_spK, c.prm.kappa, c.epsilon, sgm, coef,
        acc ? 1 : 0, out);
    c.launches += 1;
    FB_CUDA(cudaGetLastError());
    return true;
  }
  if (c.mixed && !fp64) {
    if (adjoint) launch_near_f32<true>(c, sgm, coef, out, s, acc);
    else launch_near_f32<false>(c, sgm, coef, out, s, acc);
  } else {
    if (c.mixed && !setup_near_fp64(c)) return false;
    if (adjoint) launch_near_f64<true>(c, sgm, coef, out, s, acc);
    else launch_near_f64<false>(c, sgm, coef, out, s, acc);
  }
  FB_CUDA(cudaGetLastError());
  return true;
}

}  // namespace fb
