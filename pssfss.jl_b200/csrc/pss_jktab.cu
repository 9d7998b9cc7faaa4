// K2, tabulated form of the face-pair integrals for sheets with many pair classes.
//
// jksums (PGF.jl:67-106) adds 168 and more lattice summands at every quadrature point of every
// pair.  Only the images next to the pair vary fast with the offset; the sum over the images of
// ring 2 and beyond is smooth (its nearest singularity lies a whole cell away from every offset
// a sheet can have), so it is tabulated once per phasing and interpolated:
//   * the offsets, a parallelogram of lattice coordinates, are cut into panels of 8 x 8
//     Chebyshev nodes.  A panel's half-width is at most 1/48 of the distance D to the nearest
//     tabulated image: the Bernstein ellipse through that image has radius 96 in both
//     directions, so the interpolation error is about 96^-8 = 1.4e-16 of the far sum, which is
//     itself at most a few tenths of the whole.  Nor is a half-width above 0.15, where e^-d's own
//     change over a panel adds h^8 / (2^7 8!) = 5e-14 of the far sum; panels that wide belong to
//     compact sheets, whose far sum is below 1 % of the whole;
//   * the reference stops a sum at its own ring R (relative change below 1e-8), so R is part of
//     the result.  R depends on the offset alone: a panel stores the far sum through ring R0
//     and through R0 + 1, R0 the first ring that not every point of the panel surely passes over.
//     Panels whose points all surely stop at R0 are taken as a whole; the others carry a map of
//     32 x 32 sub-cells that says R0, R0 + 1 or unknown;
//   * "surely" is a bound, not a sample.  A node speaks for the points within the distance de of
//     it (which together cover the panel) by the sums' Lipschitz constants; in a sub-cell a sum
//     lies within (wa^2 + wb^2)/8 times its second derivative of the convex hull of its four
//     corner values, so its modulus is bounded on both sides.  The constants come from the same
//     summands without their phases.  So zeros of a ring's sum (the reference may stop there
//     early) and of the whole sum are seen however small their surroundings are;
//   * pairs with a point in an unknown sub-cell (at the sweeps' smoothing parameter 0.4-0.9 % of
//     the points, up to 5 % at phasings of pi, whose real ring sums vanish along curves) go to a
//     list and through the direct form (filljk_pair), bit for bit as before.
// What bounds it: the direct form issues about 4200 FP64 operations per quadrature point and is
// bound by the FP64 pipe; this one issues about 400 and reads 64 nodes from L1/L2.  A pair's
// eight lanes own one column of the panel each, so a node row is one 128-byte line, and a lane
// keeps its column in registers while consecutive quadrature points stay in the panel.
// Measured (direct -> tabulated, tables included): 17.6 -> 2.9 ms for the 3.19M classes of the
// N = 3976 meander at normal incidence (nodes 0.22, map 0.11, sums 2.20, list 0.41), 18.1 -> 4.75 ms
// for four phasings of a ring of 1168 faces (0.38, 0.17, 3.47, 0.73).
#include <algorithm>
#include <cmath>

#include "pss_lattice.cuh"

namespace {

constexpr int kND = 8;                  // nodes per panel and direction
constexpr int kSub = 32;                // sub-cells per panel and direction
constexpr int kRMin = 6;                // first ring the reference tests
constexpr int kRec = 9;                 // far sums recorded at a node: through rings kRMin - 1 .. 13
constexpr double kConv = 1e-8;          // its threshold
constexpr double kTol = 1e-6;           // share of the threshold left to rounding on either side
constexpr double kNodeGap = 0.1951;     // a point's distance from a node, in half-widths per direction
// Growth of a derivative bound from where it is formed to the points it speaks for, e^t (1 - t/d)^-3
// for a distance t from there and d to the image: rings 2 and beyond, d at least 48 half-widths and
// t at most 0.39 of them (0.059); ring 1 at a node, d at least 4 t; ring 1 at a corner, d at least 4
// sub-cell sides (0.019).
constexpr double kFar = 1.1, kNear = 2.6;
constexpr int kBounds = 6;
constexpr int kMaxPanels = 8192;

struct TabDev {
  double iv[4];           // u-scaled offset -> lattice coordinates
  double a0, b0, ra, rb;
  double wa, wb;          // sides of a panel, u-scaled
  double q;               // reciprocal of the distance to the nearest image of ring 2
  int na, nb;
  double *val[kJKGroup];          // [panel][R0 / R0+1][node a][J, K][node b] (real: one double each)
  double *ring[kJKGroup];         // ring R0 alone at the nodes, laid out like one slot of val
  // per panel, bounds on second derivatives: ring R0 of J and K, ring R0 + 1, rings 2 .. R0 + 1
  float *bound[kJKGroup];
  unsigned char *flag[kJKGroup];  // per panel: 0 whole, 1 map, 2 direct
  unsigned char *map[kJKGroup];   // [panel][kSub][kSub]
  int *list, *count;              // pairs left to the direct form, per phasing
};

// cos((2k+1) pi / 16) and the reciprocals of prod_{m != k} (x_k - x_m)
__constant__ double c_node[kND] = {0.9807852804032304, 0.8314696123025452, 0.5555702330196023, 0.19509032201612833,
                                   -0.1950903220161282, -0.555570233019602, -0.8314696123025453, -0.9807852804032304};
__constant__ double c_nodew[kND] = {3.121445152258054, -8.889123728313642, 13.30351379684073, -15.692564486451692,
                                    15.692564486451692, -13.303513796840717, 8.889123728313624, -3.121445152258053};

// Sums at a node, ring by ring as in jksums; the far part (rings >= 2) through each ring r in
// 5 .. 13 and the ring's sums without phases (r = 5: of rings 2 .. 5) are handed to rec.
// Returns the first ring that some point within de of the node may stop at (0: beyond the record);
// sure: all of them do.
// Derivatives: |d1 (e^-d / d)| <= e^-d (1/d + 1/d^2), |d2 (e^-d / d)| <= e^-d (1/d + 2/d^2 + 2/d^3),
// |d1 e^-d| <= e^-d, |d2 e^-d| <= e^-d (1 + 1/d).
__device__ __forceinline__ double slope_of(double q) { return 1 + q; }  // per e^-d / d, 1/d <= q
__device__ __forceinline__ double curve_of(double q) { return fma(2 * q, 1 + q, 1.0); }
template <bool REAL, class Rec>
__device__ __forceinline__ int scan_rings(double urx, double ury, double us1x, double us1y, double us2x, double us2y,
                                          const cd *__restrict__ ph1, const cd *__restrict__ ph2,
                                          const double *__restrict__ etab, double de, double q, bool &sure, Rec &&rec) {
  const double arg = sqrt(urx * urx + ury * ury);
  const double rterm = exp_neg(arg, etab);
  cd ksum = mkcd(rterm, 0.0);
  cd jsum = arg <= 1e-5 ? mkcd((-arg / 6 + 0.5) * arg - 1, 0.0) : mkcd((rterm - 1) / arg, 0.0);
  cd jfar = mkcd(0, 0), kfar = jfar;
  double lipj = 0.5, lipk = 1.0, farj = 0, fark = 0;  // Lipschitz constants: of the (0, 0) term
  const double slope = kFar * slope_of(q);
  int R = 0;
  sure = false;
  for (int r = 1; r < kRMin - 1 + kRec; ++r) {
    cd jr = mkcd(0, 0), kr = jr;
    double sj = 0, sk = 0, ramax = 0;
    auto summand = [&](int m, int n, double dm, double dn) {
      const double dx = urx - (dm * us1x + dn * us2x), dy = ury - (dm * us1y + dn * us2y);
      const double d2 = dx * dx + dy * dy, ra = rsqrt(d2), er = exp_neg(d2 * ra, etab), ej = er * ra;
      if constexpr (REAL) {
        jr.x += ej;
        kr.x += er;
      } else {
        const cd f = ph1[m + PSS_JKRINGMAX] * ph2[n + PSS_JKRINGMAX];
        jr = jr + mkcd(er * f.x * ra, er * f.y * ra);
        kr = kr + mkcd(er * f.x, er * f.y);
        sj += ej;
        sk += er;
      }
      if (r == 1) ramax = fmax(ramax, ra);
    };
    const double dr = (double)r;
    double d = -dr;
    for (int i = -r; i <= r; ++i, d += 1.0) {
      summand(r, i, dr, d);
      summand(-r, i, -dr, d);
    }
    d = 1.0 - dr;
    for (int i = 1 - r; i < r; ++i, d += 1.0) {
      summand(i, -r, d, -dr);
      summand(i, r, d, dr);
    }
    if constexpr (REAL) { sj = jr.x; sk = kr.x; }
    lipk += kFar * sk;
    if (r == 1) {
      lipj += 4 * de * ramax < 1 ? kNear * slope_of(ramax) * sj : 1e300;  // no bound beside an image
    } else {
      jfar = jfar + jr;
      kfar = kfar + kr;
      farj += sj;
      fark += sk;
      lipj += slope * sj;
    }
    if (r == kRMin - 1) rec(0, jfar, kfar, farj, fark);
    if (r >= kRMin) rec(r - (kRMin - 1), jfar, kfar, sj, sk);
    if (R) return R;  // one ring past R has been recorded
    jsum = jsum + jr;
    ksum = ksum + kr;
    if (r >= kRMin) {
      const double aj = cabsd(jsum), ak = cabsd(ksum), rj = cabsd(jr), rk = cabsd(kr);
      const double ej = slope * de * sj, ek = kFar * de * sk, dj = de * lipj, dk = de * lipk;
      constexpr double up = kConv * (1 + kTol), dn = kConv * (1 - kTol);
      if (!(rj - ej > up * (aj + dj) || rk - ek > up * (ak + dk))) {
        R = r;
        sure = rj + ej < dn * (aj - dj) && rk + ek < dn * (ak - dk);
      }
    }
  }
  return 0;  // passed over to the last recorded ring, or R + 1 not recorded
}

// Bounds on the modulus over a sub-cell's convex hull of four corner values.
__device__ __forceinline__ double hull_max(const cd (&v)[4]) {
  double m = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) m = fmax(m, v[k].x * v[k].x + v[k].y * v[k].y);
  return sqrt(m);
}
__device__ __forceinline__ double hull_min(const cd (&v)[4]) {  // along the mean's direction
  const double mx = (v[0].x + v[1].x) + (v[2].x + v[3].x), my = (v[0].y + v[1].y) + (v[2].y + v[3].y);
  const double m2 = mx * mx + my * my;
  if (!(m2 > 0)) return 0.0;
  double m = 1e300;
#pragma unroll
  for (int k = 0; k < 4; ++k) m = fmin(m, v[k].x * mx + v[k].y * my);
  return m * rsqrt(m2);
}

// One CTA of 64 threads per panel (x) and phasing (y): node (i, j) = (tid / 8, tid % 8).
template <bool REAL>
__global__ void __launch_bounds__(64) k_jktab_nodes(TabDev T, PsiGroup pg, double us1x, double us1y, double us2x,
                                                    double us2y) {
  __shared__ cd ph1[1][kPhase], ph2[1][kPhase];
  __shared__ double etab[256];
  __shared__ cd rj[kRec][64], rk[kRec][64];
  __shared__ float sj[kRec][64], sk[kRec][64];  // sums without phases
  __shared__ int lo, hi;
  __shared__ unsigned bound[kBounds];  // positive floats, which order as their bits do
  const int p = blockIdx.y, panel = blockIdx.x, tid = threadIdx.x;
  PsiGroup one{};
  one.n = 1;
  one.psi1[0] = pg.psi1[p];
  one.psi2[0] = pg.psi2[p];
  fill_phases<1>(one, 1, ph1, ph2, etab);
  if (tid == 0) { lo = 1000; hi = 0; }
  if (tid < kBounds) bound[tid] = 0;
  for (int r = 0; r < kRec; ++r) {
    rj[r][tid] = rk[r][tid] = mkcd(0, 0);
    sj[r][tid] = sk[r][tid] = 0.f;
  }
  __syncthreads();
  const int i = tid >> 3, j = tid & 7, ia = panel % T.na, ib = panel / T.na;
  const double a = T.a0 + (ia + 0.5 * (1.0 + c_node[i])) / T.ra, b = T.b0 + (ib + 0.5 * (1.0 + c_node[j])) / T.rb;
  bool sure;
  const int R = scan_rings<REAL>(a * us1x + b * us2x, a * us1y + b * us2y, us1x, us1y, us2x, us2y, ph1[0], ph2[0], etab,
                                 kNodeGap * 0.5 * (T.wa + T.wb), T.q, sure, [&](int r, cd jf, cd kf, double vj, double vk) {
                                   rj[r][tid] = jf;
                                   rk[r][tid] = kf;
                                   sj[r][tid] = __double2float_ru(vj);
                                   sk[r][tid] = __double2float_ru(vk);
                                 });
  if (R) atomicMin(&lo, R);
  atomicMax(&hi, sure ? R : 1000);
  __syncthreads();
  const bool direct = lo == 1000;
  if (tid == 0) T.flag[p][panel] = direct ? 2 : hi == lo ? 0 : 1;
  const int r0 = direct ? 1 : lo - (kRMin - 1);
  {
    float far_j = 0, far_k = 0;
    for (int r = 0; r <= r0 + 1; ++r) {
      far_j = __fadd_ru(far_j, sj[r][tid]);
      far_k = __fadd_ru(far_k, sk[r][tid]);
    }
    const float cj = __double2float_ru(curve_of(T.q));
    const float v[kBounds] = {__fmul_ru(cj, sj[r0][tid]),     __fadd_ru(sj[r0][tid], sk[r0][tid]),
                              __fmul_ru(cj, sj[r0 + 1][tid]), __fadd_ru(sj[r0 + 1][tid], sk[r0 + 1][tid]),
                              __fmul_ru(cj, far_j),           __fadd_ru(far_j, far_k)};
#pragma unroll
    for (int k = 0; k < kBounds; ++k) {
      const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(v[k]));
      if ((tid & 31) == 0) atomicMax(&bound[k], m);
    }
    __syncthreads();
    if (tid < kBounds) T.bound[p][panel * kBounds + tid] = __uint_as_float(bound[tid]);
  }
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const cd J = rj[r0 + s][tid], K = rk[r0 + s][tid];
    if constexpr (REAL) {
      double2 *v = (double2 *)T.val[p] + (size_t)(panel * 2 + s) * 64;
      v[i * 8 + j] = make_double2(J.x, K.x);
    } else {
      double2 *v = (double2 *)T.val[p] + (size_t)(panel * 2 + s) * 128;
      v[(i * 2) * 8 + j] = make_double2(J.x, J.y);
      v[(i * 2 + 1) * 8 + j] = make_double2(K.x, K.y);
    }
  }
  // ring R0 itself, for the map
  const cd J = rj[r0][tid] - rj[r0 - 1][tid], K = rk[r0][tid] - rk[r0 - 1][tid];
  double2 *v = (double2 *)T.ring[p] + (size_t)panel * (REAL ? 64 : 128);
  if constexpr (REAL) {
    v[i * 8 + j] = make_double2(J.x, K.x);
  } else {
    v[(i * 2) * 8 + j] = make_double2(J.x, J.y);
    v[(i * 2 + 1) * 8 + j] = make_double2(K.x, K.y);
  }
}

// Lagrange basis of the panel nodes at t, times s.
__device__ __forceinline__ void basis8(double t, double s, double *out) {
  double d[kND], pre[kND];
#pragma unroll
  for (int k = 0; k < kND; ++k) d[k] = t - c_node[k];
  pre[0] = s;
#pragma unroll
  for (int k = 1; k < kND; ++k) pre[k] = pre[k - 1] * d[k - 1];
  double suf = 1.0;
#pragma unroll
  for (int k = kND - 1; k >= 0; --k) {
    out[k] = (pre[k] * suf) * c_nodew[k];
    suf *= d[k];
  }
}

// Sub-cell maps of the panels that need one: the sums and their rings R0 and R0 + 1 at the 33 x 33
// corners, from the nearest images and the panel's own interpolants of the far sums (through R0
// and R0 + 1) and of ring R0: about 400 operations per corner, where summing the rings anew would
// take 5000.  Strips of kStrip sub-cell rows, so that three CTAs fit an SM.
constexpr int kC = kSub + 1, kStrip = 11, kCorners = (kStrip + 1) * kC;
template <bool REAL>
__global__ void __launch_bounds__(256, 2) k_jktab_map(TabDev T, PsiGroup pg, double us1x, double us1y, double us2x,
                                                   double us2y) {
  constexpr int W = REAL ? 6 : 12;  // reals per node: far R0 (J, K), far R0 + 1, ring R0
  __shared__ double etab[256];
  __shared__ cd fnear[9];
  __shared__ double lag[kC][kND];
  __shared__ double node[64][W];
  extern __shared__ __align__(16) unsigned char map_smem[];
  cd *cs = (cd *)map_smem;  // [J, K through R0; ring R0; ring R0 + 1][corner]
  float *cn = (float *)(cs + 6 * kCorners);  // [J, K][corner]: second-derivative bound of the near terms
  double *half = (double *)(cn + 2 * kCorners);  // [corner i][node j][W]
  const int p = blockIdx.y, panel = blockIdx.x, tid = threadIdx.x;
  if (T.flag[p][panel] != 1) return;
  etab[tid] = exp2((double)tid / 256.0);
  if (tid < 9) {
    double s1, c1, s2, c2;
    sincos(-((double)(tid / 3 - 1) * pg.psi1[p]), &s1, &c1);
    sincos(-((double)(tid % 3 - 1) * pg.psi2[p]), &s2, &c2);
    fnear[tid] = mkcd(c1, s1) * mkcd(c2, s2);
  }
  if (tid < kC) basis8(2.0 * tid / kSub - 1.0, 1.0, lag[tid]);
  for (int e = tid; e < 64 * W; e += 256) {
    // value w of node k = 8 i + j: slot w / (W / 3), then J and K (real and imaginary)
    const int k = e / W, w = e % W, sl = w / (W / 3), c = w % (W / 3);
    const double *v = sl < 2 ? T.val[p] + (size_t)(panel * 2 + sl) * 64 * (W / 3) : T.ring[p] + (size_t)panel * 64 * (W / 3);
    node[k][w] = REAL ? v[k * 2 + c] : v[((k / 8 * 2 + c / 2) * 8 + k % 8) * 2 + c % 2];
  }
  __syncthreads();
  for (int e = tid; e < kC * kND * W; e += 256) {
    const int i = e / (kND * W), j = e / W % kND, w = e % W;
    double s = 0;
#pragma unroll
    for (int k = 0; k < kND; ++k) s = fma(lag[i][k], node[k * 8 + j][w], s);
    half[e] = s;
  }
  const int ia = panel % T.na, ib = panel / T.na;
  const double wa = T.wa / kSub, wb = T.wb / kSub, diag = wa + wb, q8 = (wa * wa + wb * wb) / 8;
  const float *bnd = T.bound[p] + panel * kBounds;
  const double fj = kFar * q8 * bnd[0], fk = kFar * q8 * bnd[1], gj = kFar * q8 * bnd[2], gk = kFar * q8 * bnd[3];
  const double sj = kFar * q8 * bnd[4], sk = kFar * q8 * bnd[5];
  for (int i0 = 0; i0 < kSub; i0 += kStrip) {
    const int rows = min(kStrip, kSub - i0);
    __syncthreads();  // half written, the previous strip read
    for (int e = tid; e < (rows + 1) * kC; e += 256) {
      const int i = i0 + e / kC, j = e % kC;
      double v[12];
#pragma unroll
      for (int w = 0; w < W; ++w) {
        double s = 0;
#pragma unroll
        for (int k = 0; k < kND; ++k) s = fma(lag[j][k], half[(i * kND + k) * W + w], s);
        v[w] = s;
      }
      const double a = T.a0 + (ia + (double)i / kSub) / T.ra, b = T.b0 + (ib + (double)j / kSub) / T.rb;
      const double ux = a * us1x + b * us2x, uy = a * us1y + b * us2y;
      const double arg = sqrt(ux * ux + uy * uy), rterm = exp_neg(arg, etab);
      cd js = mkcd(arg <= 1e-5 ? (-arg / 6 + 0.5) * arg - 1 : (rterm - 1) / arg, 0.0), ks = mkcd(rterm, 0.0);
      // the (0, 0) term's kink at the origin: beside it, the Lipschitz constants' equivalent
      const bool off = arg > 2 * diag;
      double nj = off ? 1.0 / 3 + 0.5 / (arg - diag) : 0.5 * diag / q8, nk = off ? 1.0 + 1.0 / (arg - diag) : diag / q8;
      double s1 = 0, s0 = 0, ramax = 0;  // of e^-d / d, of e^-d, the nearest image's 1/d
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        if (q == 4) continue;
        const double m = q / 3 - 1, n = q % 3 - 1;
        const double dx = ux - (m * us1x + n * us2x), dy = uy - (m * us1y + n * us2y);
        const double d2 = dx * dx + dy * dy, ra = rsqrt(d2), er = exp_neg(d2 * ra, etab);
        const cd f = fnear[q];
        js = js + mkcd(er * f.x * ra, er * f.y * ra);
        ks = ks + mkcd(er * f.x, er * f.y);
        s1 = fma(er, ra, s1);
        s0 += er;
        ramax = fmax(ramax, ra);
      }
      nj += 4 * diag * ramax < 1 ? kNear * curve_of(ramax) * s1 : 1e300;  // beside an image: unknown
      nk += 4 * diag * ramax < 1 ? kNear * (s0 + s1) : 1e300;
      auto val = [&](int k) { return REAL ? mkcd(v[k], 0.0) : mkcd(v[2 * k], v[2 * k + 1]); };  // (slot, J / K)
      cs[e] = js + val(0);
      cs[kCorners + e] = ks + val(1);
      cs[2 * kCorners + e] = val(4);
      cs[3 * kCorners + e] = val(5);
      cs[4 * kCorners + e] = val(2) - val(0);
      cs[5 * kCorners + e] = val(3) - val(1);
      cn[e] = __double2float_ru(nj);
      cn[kCorners + e] = __double2float_ru(nk);
    }
    __syncthreads();
    for (int e = tid; e < rows * kSub; e += 256) {
      const int e0 = e / kSub * kC + e % kSub;
      const int c[4] = {e0, e0 + 1, e0 + kC, e0 + kC + 1};
      cd v[6][4];
      float nj = 0, nk = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k][q] = cs[k * kCorners + c[q]];
        nj = fmaxf(nj, cn[c[q]]);
        nk = fmaxf(nk, cn[kCorners + c[q]]);
      }
      constexpr double up = kConv * (1 + kTol), dn = kConv * (1 - kTol);
      const double ej = fma(q8, (double)nj, sj), ek = fma(q8, (double)nk, sk);  // of the whole sums
      int state = 2;
      if (hull_max(v[2]) + fj < dn * (hull_min(v[0]) - ej) && hull_max(v[3]) + fk < dn * (hull_min(v[1]) - ek)) {
        state = 0;
      } else if (hull_min(v[2]) - fj > up * (hull_max(v[0]) + ej) || hull_min(v[3]) - fk > up * (hull_max(v[1]) + ek)) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // through ring R0 + 1
          v[0][q] = v[0][q] + v[4][q];
          v[1][q] = v[1][q] + v[5][q];
        }
        if (hull_max(v[4]) + gj < dn * (hull_min(v[0]) - ej) && hull_max(v[5]) + gk < dn * (hull_min(v[1]) - ek)) state = 1;
      }
      T.map[p][(size_t)panel * kSub * kSub + i0 * kSub + e] = (unsigned char)state;
    }
  }
}
constexpr int kMapSmem = kCorners * (6 * (int)sizeof(cd) + 2 * (int)sizeof(float)) + kC * kND * 12 * (int)sizeof(double);

constexpr int kTabThreads = 128;
// The seven points in a walk around the triangle (vertex, midpoint, ..., centroid): neighbours
// share a panel more often than in the rule's order.
__host__ __device__ constexpr int walk(int t) { return t == 0 ? 3 : t == 1 ? 4 : t == 2 ? 2 : t == 3 ? 6 : t == 4 ? 1 : t == 5 ? 5 : 0; }
constexpr int kBasStride = 7 * 2 * kND + 2;  // doubles per pair: the four pairs of a warp on different banks

// Eight lanes per face pair.  Lane q < 7 owns quadrature point q: its nearest images (rings 0
// and 1) one by one, its panel, and the Lagrange bases of its position, handed to the pair's
// lanes through shared memory.  Then every lane j sums its column j of the panel for all seven
// points into the six moments; a reduce-scatter over the eight lanes leaves moment k in lane k.
template <int NP, bool REAL>
__global__ void __launch_bounds__(kTabThreads, REAL ? 8 : 4) k_filljk_tab(SheetDev G, double ul, PsiGroup pg, double us1x,
                                                               double us1y, double us2x, double us2y, TabDev T,
                                                               JKGroup jk) {
  __shared__ cd fnear[NP][9];
  __shared__ double etab[256];
  __shared__ __align__(16) double bas[kTabThreads / 8][kBasStride];
  // a group's near sums wait in shared memory for their phasing's turn (registers limit the CTAs
  // per SM)
  __shared__ double2 near_sum[NP == 1 ? 1 : NP][2][NP == 1 ? 1 : kTabThreads];
  const int np = NP == 1 ? 1 : pg.n;
  for (int t = threadIdx.x; t < 256; t += blockDim.x) etab[t] = exp2((double)t / 256.0);
  for (int t = threadIdx.x; t < NP * 9; t += blockDim.x) {
    const int p = t / 9, m = t % 9 / 3 - 1, n = t % 3 - 1;
    double s1, co1, s2, co2;
    sincos(-((double)m * (p < np ? pg.psi1[p] : 0.0)), &s1, &co1);
    sincos(-((double)n * (p < np ? pg.psi2[p] : 0.0)), &s2, &co2);
    fnear[p][t % 9] = mkcd(co1, s1) * mkcd(co2, s2);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, q = lane & 7, grp = lane & ~7;
  const long long gid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 3;
  const bool live = gid < G.nufp;
  const int iu = live ? (int)gid : G.nufp - 1;  // idle groups mirror the last pair, write nothing
  const PairGeo g = pair_geo(G, iu);
  double ux, uy;
  quad_offset(g, min(q, 6), ul, ux, uy);
  // nearest images: the regularised (0, 0) term, then ring 1 in ring order
  cd js[NP], ks[NP];
  {
    const double arg = sqrt(ux * ux + uy * uy);
    const double rterm = exp_neg(arg, etab);
    const double j0 = arg <= 1e-5 ? (-arg / 6 + 0.5) * arg - 1 : (rterm - 1) / arg;
#pragma unroll
    for (int p = 0; p < NP; ++p) { js[p] = mkcd(0, 0); ks[p] = mkcd(0, 0); }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int m = e < 3 ? 1 : e < 6 ? -1 : 0, n = e < 6 ? e % 3 - 1 : e == 6 ? -1 : 1;
      const double dx = ux - ((double)m * us1x + (double)n * us2x), dy = uy - ((double)m * us1y + (double)n * us2y);
      const double d2 = dx * dx + dy * dy, ra = rsqrt(d2), er = exp_neg(d2 * ra, etab);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        if constexpr (REAL) {
          js[p].x += er * ra;
          ks[p].x += er;
        } else {
          const cd f = fnear[p][(m + 1) * 3 + n + 1];
          const cd term = mkcd(er * f.x, er * f.y);
          js[p] = js[p] + mkcd(term.x * ra, term.y * ra);
          ks[p] = ks[p] + term;
        }
      }
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      js[p].x += j0;
      ks[p].x += rterm;
      if constexpr (NP > 1) {
        near_sum[p][0][threadIdx.x] = make_double2(js[p].x, js[p].y);
        near_sum[p][1][threadIdx.x] = make_double2(ks[p].x, ks[p].y);
      }
    }
  }
  // panel and sub-cell of this point; bases (the quadrature weight goes into the second one)
  int panel;
  int sub;
  {
    const double fa = (T.iv[0] * ux + T.iv[1] * uy - T.a0) * T.ra, fb = (T.iv[2] * ux + T.iv[3] * uy - T.b0) * T.rb;
    const int ia = max(0, min(T.na - 1, (int)fa)), ib = max(0, min(T.nb - 1, (int)fb));
    const double ta = 2.0 * (fa - ia) - 1.0, tb = 2.0 * (fb - ib) - 1.0;
    panel = ib * T.na + ia;
    const int ca = max(0, min(kSub - 1, (int)((ta + 1.0) * (0.5 * kSub))));
    const int cb = max(0, min(kSub - 1, (int)((tb + 1.0) * (0.5 * kSub))));
    sub = ca * kSub + cb;
    if (q < 7) {
      double *o = &bas[threadIdx.x >> 3][q * 2 * kND];
      basis8(ta, 1.0, o);
      basis8(tb, c_qw[q], o + kND);
    }
  }
  __syncwarp();
  double rr0, rr1, ri;
  edge_terms(g, ul, q, grp, rr0, rr1, ri);
  const double *mybas = bas[threadIdx.x >> 3];
  const double qw = q < 7 ? c_qw[q] : 0.0, qx = q < 7 ? c_qxi[q] : 0.0, qe = q < 7 ? c_qeta[q] : 0.0;
#pragma unroll 1
  for (int p = 0; p < np; ++p) {
    // this point's state under phasing p: 0 / 1 the table slot, 2 the direct form
    int state = T.flag[p][panel];
    if (state == 1) state = T.map[p][(size_t)panel * kSub * kSub + sub];
    const unsigned direct = __ballot_sync(0xffffffffu, state == 2 && q < 7) & (0xffu << grp);
    const int slot = panel * 2 + (state == 1 ? 1 : 0);
    // near part of the moments: lane q's own point
    cd jn, kn;
    if constexpr (NP == 1) {
      jn = js[0];
      kn = ks[0];
    } else {
      const double2 a = near_sum[p][0][threadIdx.x], b = near_sum[p][1][threadIdx.x];
      jn = mkcd(a.x, a.y);
      kn = mkcd(b.x, b.y);
    }
    const JKDev &o = jk.s[p];
    if constexpr (REAL) {
      // J and K together: one double2 per node
      double acc[6] = {qw * jn.x, qx * (qw * jn.x), qe * (qw * jn.x), qw * kn.x, qx * (qw * kn.x), qe * (qw * kn.x)};
      double2 row[kND];
      int held = -1;
      const double2 *val = (const double2 *)T.val[p] + q;
#pragma unroll
      for (int w = 0; w < 7; ++w) {
        const int t = walk(w);
        const int s = __shfl_sync(0xffffffffu, slot, grp + t);
        if (s != held) {
          held = s;
#pragma unroll
          for (int i = 0; i < kND; ++i) row[i] = __ldg(val + (size_t)s * 64 + i * 8);
        }
        const double2 *lx = (const double2 *)(mybas + t * 2 * kND);
        const double ly = mybas[t * 2 * kND + kND + q];
        double jv = 0, kv = 0;
#pragma unroll
        for (int i = 0; i < kND; i += 2) {
          const double2 l = lx[i / 2];
          jv = fma(l.x, row[i].x, fma(l.y, row[i + 1].x, jv));
          kv = fma(l.x, row[i].y, fma(l.y, row[i + 1].y, kv));
        }
        jv *= ly;
        kv *= ly;
        acc[0] += jv;
        acc[1] = fma(c_qxi[t], jv, acc[1]);
        acc[2] = fma(c_qeta[t], jv, acc[2]);
        acc[3] += kv;
        acc[4] = fma(c_qxi[t], kv, acc[4]);
        acc[5] = fma(c_qeta[t], kv, acc[5]);
      }
      // reduce-scatter over the eight lanes: lane k ends with moment k (lanes 6 and 7 with none)
      const bool b4 = q & 4, b2 = q & 2, b1 = q & 1;
      double h[4], h2[2];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double hi = k < 2 ? acc[4 + k] : 0.0;
        h[k] = (b4 ? hi : acc[k]) + __shfl_xor_sync(0xffffffffu, b4 ? acc[k] : hi, 4);
      }
#pragma unroll
      for (int k = 0; k < 2; ++k)
        h2[k] = (b2 ? h[2 + k] : h[k]) + __shfl_xor_sync(0xffffffffu, b2 ? h[k] : h[2 + k], 2);
      const cd out = mkcd((b1 ? h2[1] : h2[0]) + __shfl_xor_sync(0xffffffffu, b1 ? h2[0] : h2[1], 1), 0.0);
      if (live) {
        if (q == 0) o.J[iu] = out;
        else if (q == 1) o.Jxi[iu] = out;
        else if (q == 2) o.Jeta[iu] = out;
        else if (q == 3) o.K[iu] = out;
        else if (q == 4) o.Kxi[iu] = out;
        else if (q == 5) o.Keta[iu] = out;
      }
    } else {
      // J, then K: half the registers of both at once
#pragma unroll 1
      for (int hk = 0; hk < 2; ++hk) {
        const cd own = qw * (hk ? kn : jn);
        cd acc[3] = {own, qx * own, qe * own};
        double2 row[kND];
        int held = -1;
        const double2 *val = (const double2 *)T.val[p] + hk * 8 + q;
#pragma unroll
        for (int w = 0; w < 7; ++w) {
          const int t = walk(w);
          const int s = __shfl_sync(0xffffffffu, slot, grp + t);
          if (s != held) {
            held = s;
#pragma unroll
            for (int i = 0; i < kND; ++i) row[i] = __ldg(val + (size_t)s * 128 + i * 16);
          }
          const double2 *lx = (const double2 *)(mybas + t * 2 * kND);
          const double ly = mybas[t * 2 * kND + kND + q];
          cd v = mkcd(0, 0);
#pragma unroll
          for (int i = 0; i < kND; i += 2) {
            const double2 l = lx[i / 2];
            v.x = fma(l.x, row[i].x, fma(l.y, row[i + 1].x, v.x));
            v.y = fma(l.x, row[i].y, fma(l.y, row[i + 1].y, v.y));
          }
          v = ly * v;
          acc[0] = acc[0] + v;
          acc[1] = mkcd(fma(c_qxi[t], v.x, acc[1].x), fma(c_qxi[t], v.y, acc[1].y));
          acc[2] = mkcd(fma(c_qeta[t], v.x, acc[2].x), fma(c_qeta[t], v.y, acc[2].y));
        }
        // reduce-scatter: lanes 0, 2 and 4 end with moments 0, 1 and 2
        const bool b4 = q & 4, b2 = q & 2;
        cd h[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const cd hi = k == 0 ? acc[2] : mkcd(0, 0), keep = b4 ? hi : acc[k], send = b4 ? acc[k] : hi;
          h[k] = mkcd(keep.x + __shfl_xor_sync(0xffffffffu, send.x, 4), keep.y + __shfl_xor_sync(0xffffffffu, send.y, 4));
        }
        const cd keep = b2 ? h[1] : h[0], send = b2 ? h[0] : h[1];
        cd out = mkcd(keep.x + __shfl_xor_sync(0xffffffffu, send.x, 2), keep.y + __shfl_xor_sync(0xffffffffu, send.y, 2));
        out = mkcd(out.x + __shfl_xor_sync(0xffffffffu, out.x, 1), out.y + __shfl_xor_sync(0xffffffffu, out.y, 1));
        if (live) {
          if (q == 0) (hk ? o.K : o.J)[iu] = out;
          else if (q == 2) (hk ? o.Kxi : o.Jxi)[iu] = out;
          else if (q == 4) (hk ? o.Keta : o.Jeta)[iu] = out;
        }
      }
    }
    if (!live) continue;
    if (q == 6) {
      o.rho_r[2 * iu] = rr0;
      o.rho_r[2 * iu + 1] = rr1;
    } else if (q == 7) {
      o.rinv[iu] = ri;
      if (direct) T.list[(size_t)p * G.nufp + atomicAdd(T.count + p, 1)] = iu;
    }
  }
}

// The listed pairs of phasing blockIdx.y by the direct form, over the values just written.
__global__ void __launch_bounds__(jk_threads<1>(), 3) k_filljk_list(SheetDev G, double ul, PsiGroup pg, double us1x,
                                                                    double us1y, double us2x, double us2y, TabDev T,
                                                                    JKGroup jk, int *nonconv) {
  __shared__ cd ph1[1][kPhase], ph2[1][kPhase];
  __shared__ double etab[256];
  const int p = blockIdx.y, cnt = T.count[p];
  const int per = blockDim.x >> 3;  // pairs of a CTA
  if ((long long)blockIdx.x * per >= cnt) return;
  PsiGroup one{};
  one.n = 1;
  one.psi1[0] = pg.psi1[p];
  one.psi2[0] = pg.psi2[p];
  JKGroup oj{};
  oj.s[0] = jk.s[p];
  fill_phases<1>(one, 1, ph1, ph2, etab);
  __syncthreads();
  const int *list = T.list + (size_t)p * G.nufp;
  const int n = (cnt + 3) & ~3;  // whole warps: four pairs each
  for (int e = blockIdx.x * per + (threadIdx.x >> 3); e < n; e += gridDim.x * per) {
    const bool live = e < cnt;
    filljk_pair<1>(G, ul, one, 1, us1x, us1y, us2x, us2y, oj, nonconv + p, list[live ? e : cnt - 1], live, ph1, ph2,
                   etab);
  }
}

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

}  // namespace

// The panels of a sheet, or false where the direct form is taken:
//   * an image of ring 2 lies inside the parallelogram of offsets (a sheet that reaches over
//     more than a cell), or would need more than 8192 panels;
//   * fewer than 55 pair classes per panel: seven direct evaluations per class then cost less
//     than six per table node, which is what the tables cost with their maps.
bool pss_jktab_plan(const SheetDev &G, double ulocal, const double s1[2], const double s2[2], int np, JKTabPlan &P) {
  P = JKTabPlan{};
  if (G.nufp < 4096 || !(ulocal > 0) || !(G.ext1 > 0) || !(G.ext2 > 0) || !(G.ext1 < 1.5) || !(G.ext2 < 1.5)) return false;
  const double e1[2] = {ulocal * s1[0], ulocal * s1[1]}, e2[2] = {ulocal * s2[0], ulocal * s2[1]};
  const double W1 = G.ext1, W2 = G.ext2;  // |offset| in lattice coordinates (panel indices are clamped)
  // distance from the parallelogram [-W1, W1] x [-W2, W2] to the nearest image of ring >= 2
  double dmin = 1e300;
  for (int m = -5; m <= 5; ++m)
    for (int n = -5; n <= 5; ++n) {
      if (std::max(std::abs(m), std::abs(n)) < 2) continue;
      if (std::fabs(m) <= W1 && std::fabs(n) <= W2) return false;
      for (int e = 0; e < 4; ++e) {  // edges a = +-W1, b = +-W2
        const double sgn = e & 1 ? 1 : -1;
        const double *t = e < 2 ? e2 : e1;                      // edge direction
        const double fa = e < 2 ? sgn * W1 : 0, fb = e < 2 ? 0 : sgn * W2, half = e < 2 ? W2 : W1;
        const double px = (m - fa) * e1[0] + (n - fb) * e2[0], py = (m - fa) * e1[1] + (n - fb) * e2[1];
        const double tt = t[0] * t[0] + t[1] * t[1];
        const double s = std::max(-half, std::min(half, (px * t[0] + py * t[1]) / tt));
        dmin = std::min(dmin, std::hypot(px - s * t[0], py - s * t[1]));
      }
    }
  const double h = std::min(dmin / 48.0, 0.15);  // panel half-width (u-scaled; exp(-R) varies on the scale 1)
  if (!(h > 0)) return false;
  const double ca = std::ceil(W1 * std::hypot(e1[0], e1[1]) / h), cb = std::ceil(W2 * std::hypot(e2[0], e2[1]) / h);
  if (!(ca * cb <= kMaxPanels)) return false;
  P.na = std::max(1, (int)ca);
  P.nb = std::max(1, (int)cb);
  const size_t panels = (size_t)P.na * P.nb;
  if ((size_t)G.nufp < 55 * panels) return false;
  P.dmin = dmin;
  P.a0 = -W1;
  P.b0 = -W2;
  P.ra = P.na / (2 * W1);
  P.rb = P.nb / (2 * W2);
  const size_t per = align256(panels * 3 * 64 * 4 * sizeof(double)) + align256(panels * kBounds * sizeof(float)) +
                     align256(panels) + align256(panels * kSub * kSub);
  P.bytes = (size_t)np * (per + (size_t)G.nufp * sizeof(int)) + 512;
  return true;
}

size_t pss_jktab_bytes(const SheetDev &G, double ulocal, const double s1[2], const double s2[2], int np) {
  JKTabPlan P;
  return pss_jktab_plan(G, ulocal, s1, s2, np, P) ? P.bytes : 0;
}

int pss_jktab_launch(const SheetDev &G, double ulocal, const PsiGroup &pg, const double s1[2], const double s2[2],
                     const JKGroup &jk, int *nonconv, const JKTabPlan &P, void *ws, cudaStream_t st) {
  const double a = ulocal * s1[0], b = ulocal * s1[1], c = ulocal * s2[0], d = ulocal * s2[1];
  const double det = a * d - b * c;
  const int np = pg.n;
  const size_t panels = (size_t)P.na * P.nb;
  TabDev T{};
  T.iv[0] = d / det; T.iv[1] = -c / det; T.iv[2] = -b / det; T.iv[3] = a / det;
  T.a0 = P.a0; T.b0 = P.b0; T.ra = P.ra; T.rb = P.rb; T.na = P.na; T.nb = P.nb;
  T.wa = std::hypot(a, b) / P.ra;
  T.wb = std::hypot(c, d) / P.rb;
  T.q = 1 / P.dmin;
  char *w = (char *)(((uintptr_t)ws + 255) & ~(uintptr_t)255);
  for (int p = 0; p < np; ++p) {
    T.val[p] = (double *)w;
    T.ring[p] = T.val[p] + panels * 2 * 64 * 4;
    w += align256(panels * 3 * 64 * 4 * sizeof(double));
    T.bound[p] = (float *)w; w += align256(panels * kBounds * sizeof(float));
    T.flag[p] = (unsigned char *)w; w += align256(panels);
    T.map[p] = (unsigned char *)w; w += align256(panels * kSub * kSub);
  }
  T.count = (int *)w; w += 64;
  T.list = (int *)w;
  PSS_CUDA_TRY(cudaMemsetAsync(T.count, 0, kJKGroup * sizeof(int), st));
  const bool real = np == 1 && pg.psi1[0] == 0.0 && pg.psi2[0] == 0.0;
  const dim3 gp((unsigned)panels, np);
  const unsigned gt = cdiv_u((long long)G.nufp * 8, kTabThreads);
  static DeviceOnce once;
  if (int rc = device_once(once, [] {
        PSS_CUDA_TRY(cudaFuncSetAttribute(k_jktab_map<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMapSmem));
        PSS_CUDA_TRY(cudaFuncSetAttribute(k_jktab_map<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMapSmem));
        return 0;
      }))
    return rc;
  for (int k = 0; k < 4; ++k) pss_count_launch();
  if (real) {
    k_jktab_nodes<true><<<gp, 64, 0, st>>>(T, pg, a, b, c, d);
    k_jktab_map<true><<<gp, 256, kMapSmem, st>>>(T, pg, a, b, c, d);
    k_filljk_tab<1, true><<<gt, kTabThreads, 0, st>>>(G, ulocal, pg, a, b, c, d, T, jk);
  } else {
    k_jktab_nodes<false><<<gp, 64, 0, st>>>(T, pg, a, b, c, d);
    k_jktab_map<false><<<gp, 256, kMapSmem, st>>>(T, pg, a, b, c, d);
    if (np == 1) k_filljk_tab<1, false><<<gt, kTabThreads, 0, st>>>(G, ulocal, pg, a, b, c, d, T, jk);
    else if (np == 2) k_filljk_tab<2, false><<<gt, kTabThreads, 0, st>>>(G, ulocal, pg, a, b, c, d, T, jk);
    else k_filljk_tab<kJKGroup, false><<<gt, kTabThreads, 0, st>>>(G, ulocal, pg, a, b, c, d, T, jk);
  }
  k_filljk_list<<<dim3(148 * 6, np), jk_threads<1>(), 0, st>>>(G, ulocal, pg, a, b, c, d, T, jk, nonconv);
  PSS_CUDA_TRY(cudaGetLastError());
  return 0;
}
