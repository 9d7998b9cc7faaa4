// Spatial lattice sums of the face-pair integrals: device code shared by the direct kernel
// (pss_fill.cu) and the tabulated one (pss_jktab.cu).
#pragma once
#include "pss_internal.cuh"

namespace {

// Phase factors of the lattice terms, cis(-m psi1) and cis(-n psi2) for |m|, |n| <= 65 (the
// ring budget): kPhase entries each, index m + 65.  A term's factor cis(-(m psi1 + n psi2)) is
// their product, one complex multiply in place of a sincos per summand.
constexpr int kPhase = 2 * PSS_JKRINGMAX + 1;

// exp(-a), a >= 0, by Tang's table-driven method (P. T. P. Tang, "Table-driven implementation
// of the exponential function in IEEE floating-point arithmetic", ACM Trans. Math. Softw. 15
// (1989) 144-157): -a = (256 m + j) ln2/256 + r with |r| <= ln2/512 (k = 256 m + j the nearest
// integer to -a 256/ln2, found by adding 1.5 * 2^52; ln2/256 in two parts, so r keeps its full
// precision), exp(-a) = 2^m * 2^(j/256) * p(r) with p the degree-5 Taylor polynomial of e^r
// (remainder below r^6/720 < 1e-20 relative) and 2^(j/256) from a 256-entry table; 2^m enters
// through the exponent field.  About ten FP64 operations.  a >= 708 gives 0: such summands are
// far below the lattice sums' 1e-8 convergence test.
constexpr double kExpShift = 6755399441055744.0;  // 1.5 * 2^52
constexpr double kExpInvStep = 0x1.71547652b82fep+8;  // 256 / ln2
constexpr double kExpStepHi = 0x1.62e42fefa39efp-9;   // ln2 / 256, nearest double
constexpr double kExpStepLo = 0x1.abc9e3b39803fp-64;  // ln2 / 256 - kExpStepHi
__device__ __forceinline__ double exp_neg(double a, const double *__restrict__ tab) {
  if (!(a < 708.0)) return 0.0;
  const double sh = fma(-a, kExpInvStep, kExpShift);
  const int k = __double2loint(sh);  // nearest integer to -a 256/ln2, two's complement
  const double kf = sh - kExpShift;
  const double r = fma(kf, -kExpStepLo, fma(kf, -kExpStepHi, -a));
  double p = fma(r, 1.0 / 120, 1.0 / 24);
  p = fma(p, r, 1.0 / 6);
  p = fma(p, r, 0.5);
  p = fma(p, r, 1.0);
  p = fma(p, r, 1.0);
  const double t = tab[k & 255] * p;
  return __hiloint2double(__double2hiint(t) + ((k >> 8) << 20), __double2loint(t));
}

// jksums (PGF.jl:67-106): the spatial lattice sums J and K at one observation offset, ring by
// ring in the reference's order (rmin = 5, at most 65 rings, relative change 1e-8), for NP
// phasings at once.  A summand's distance, exp(-u r) and 1/r do not depend on the phasing, so
// they are evaluated once and weighted by each phasing's factor; every phasing keeps its own
// ring partials and stops accumulating at its own convergence ring, so its sums are those of
// a serial evaluation at that phasing alone, bit for bit.  Slots p >= np are idle.  Returns the
// mask of converged phasings.
template <int NP>
__device__ __forceinline__ unsigned jksums_group(double urx, double ury, int np, bool nophase, double us1x,
                                                 double us1y, double us2x, double us2y,
                                                 const cd (*__restrict__ ph1)[kPhase],
                                                 const cd (*__restrict__ ph2)[kPhase], const double *__restrict__ etab,
                                                 cd *jout, cd *kout) {
  const int rmin = 5;
  constexpr int UNR = NP == 1 ? 2 : 1;  // two summands in flight where the registers allow
  const double small = 1e-5, convtest = 1e-8;
  double arg = sqrt(urx * urx + ury * ury);
  double rterm = exp_neg(arg, etab);
  const cd k0 = mkcd(rterm, 0.0);
  const cd j0 = arg <= small ? mkcd((-arg / 6 + 0.5) * arg - 1, 0.0) : mkcd((rterm - 1) / arg, 0.0);
  cd jsum[NP], ksum[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) { jsum[p] = j0; ksum[p] = k0; }
  unsigned live = (1u << np) - 1u, conv = 0;
  for (int r = 1; r <= PSS_JKRINGMAX && live; ++r) {
    cd jring[NP], kring[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) { jring[p] = mkcd(0, 0); kring[p] = mkcd(0, 0); }
    auto summand = [&](int m, int n, double dm, double dn) {
      double dx = urx - (dm * us1x + dn * us2x);
      double dy = ury - (dm * us1y + dn * us2y);
      // one reciprocal square root gives both the distance and the 1/r weight (two FP64
      // divisions fewer per summand than sqrt then term / r)
      const double d2 = dx * dx + dy * dy;
      const double ra = rsqrt(d2);
      const double a = d2 * ra;
      double er = exp_neg(a, etab);
      if (NP == 1 && nophase) {  // real terms: the imaginary parts stay exactly zero
        jring[0].x = jring[0].x + er * ra;
        kring[0].x = kring[0].x + er;
      } else {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          const cd f = ph1[p][m + PSS_JKRINGMAX] * ph2[p][n + PSS_JKRINGMAX];
          const cd term = mkcd(er * f.x, er * f.y);
          jring[p] = jring[p] + mkcd(term.x * ra, term.y * ra);
          kring[p] = kring[p] + term;
        }
      }
    };
    // the ring's 8r lattice points in Ring's order (ring_mn): m = r with n = -r..r, m = -r with
    // n = -r..r, then n = -r and n = r with m = -r+1..r-1; the indices are also counted in
    // FP64 (exact integers), so no summand converts one
    {
      const double dr = (double)r;
      double dn = -dr;
#pragma unroll UNR
      for (int i = -r; i <= r; ++i, dn += 1.0) summand(r, i, dr, dn);
      dn = -dr;
#pragma unroll UNR
      for (int i = -r; i <= r; ++i, dn += 1.0) summand(-r, i, -dr, dn);
      double dm = 1.0 - dr;
#pragma unroll UNR
      for (int i = 1 - r; i < r; ++i, dm += 1.0) summand(i, -r, dm, -dr);
      dm = 1.0 - dr;
#pragma unroll UNR
      for (int i = 1 - r; i < r; ++i, dm += 1.0) summand(i, r, dm, dr);
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      if (!((live >> p) & 1u)) continue;
      jsum[p] = jsum[p] + jring[p];
      ksum[p] = ksum[p] + kring[p];
      if (r > rmin) {
        double c1 = cabsd(jring[p] / jsum[p]), c2 = cabsd(kring[p] / ksum[p]);
        if (fmax(c1, c2) < convtest) { live &= ~(1u << p); conv |= 1u << p; }
      }
    }
  }
#pragma unroll
  for (int p = 0; p < NP; ++p) { jout[p] = jsum[p]; kout[p] = ksum[p]; }
  return conv;
}

__device__ __forceinline__ void face_vtx(const SheetDev &G, int f, double r[3][2], double scale) {
  for (int k = 0; k < 3; ++k) {
    int v = G.fv[3 * f + k];
    r[k][0] = G.rho[2 * v] * scale;
    r[k][1] = G.rho[2 * v + 1] * scale;
  }
}

// The lattice phase factors of np phasings (slots np..NP-1: zero phasing) and the exp table of
// a CTA; the caller synchronises.
template <int NP>
__device__ __forceinline__ void fill_phases(const PsiGroup &pg, int np, cd (*__restrict__ ph1)[kPhase],
                                            cd (*__restrict__ ph2)[kPhase], double *__restrict__ etab) {
  for (int t = threadIdx.x; t < 256; t += blockDim.x) etab[t] = exp2((double)t / 256.0);
  for (int t = threadIdx.x; t < NP * kPhase; t += blockDim.x) {
    const int p = t / kPhase;
    const double k = (double)(t % kPhase - PSS_JKRINGMAX);
    const double a1 = p < np ? pg.psi1[p] : 0.0, a2 = p < np ? pg.psi2[p] : 0.0;
    double s1, c1, s2, c2;
    sincos(-(k * a1), &s1, &c1);
    sincos(-(k * a2), &s2, &c2);
    ph1[p][t % kPhase] = mkcd(c1, s1);
    ph2[p][t % kPhase] = mkcd(c2, s2);
  }
}

// Geometry of a face pair: source triangle (doubled area and orientation) and match centroid.
struct PairGeo {
  double rs[3][2], rmc[2];
  double area2, unz;
};
__device__ __forceinline__ PairGeo pair_geo(const SheetDev &G, int iu) {
  PairGeo g;
  const int fp = G.ufp_rep[iu];
  const int ifm = fp % G.nface, ifs = fp / G.nface;
  double rm[3][2];
  face_vtx(G, ifs, g.rs, 1.0);
  face_vtx(G, ifm, rm, 1.0);
  const double rs32[2] = {g.rs[2][0] - g.rs[1][0], g.rs[2][1] - g.rs[1][1]};
  const double rs12[2] = {g.rs[0][0] - g.rs[1][0], g.rs[0][1] - g.rs[1][1]};
  g.area2 = (-rs32[1]) * rs12[0] + rs32[0] * rs12[1];
  g.unz = 1.0;
  if (g.area2 < 0) { g.area2 = fabs(g.area2); g.unz = -1.0; }
  g.rmc[0] = ((rm[0][0] + rm[1][0]) + rm[2][0]) / 3;
  g.rmc[1] = ((rm[0][1] + rm[1][1]) + rm[2][1]) / 3;
  return g;
}
// Offset (u-scaled) of the match centroid from quadrature point q of the source triangle.
__device__ __forceinline__ void quad_offset(const PairGeo &g, int q, double ul, double &ux, double &uy) {
  const double rs31[2] = {g.rs[2][0] - g.rs[0][0], g.rs[2][1] - g.rs[0][1]};
  const double rs21[2] = {g.rs[1][0] - g.rs[0][0], g.rs[1][1] - g.rs[0][1]};
  const double rtx = (g.rs[0][0] + rs21[0] * c_qxi[q]) + rs31[0] * c_qeta[q];
  const double rty = (g.rs[0][1] + rs21[1] * c_qxi[q]) + rs31[1] * c_qeta[q];
  ux = ul * (g.rmc[0] - rtx);
  uy = ul * (g.rmc[1] - rty);
}

// The phasing-free terms of a pair (the 1/R integral and its gradient over the source
// triangle): one edge per lane of the pair's eight (lane q takes edge q mod 3), summed in edge
// order, so every lane returns the serial evaluation's values.
__device__ __forceinline__ void edge_terms(const PairGeo &g, double ul, int q, int grp, double &rr0, double &rr1,
                                           double &ri) {
  const int i = q % 3, ip1 = (i + 1) % 3;
  // selected by predicates, not by a run-time index into the vertex array
  const double ax = i == 0 ? g.rs[0][0] : i == 1 ? g.rs[1][0] : g.rs[2][0];
  const double ay = i == 0 ? g.rs[0][1] : i == 1 ? g.rs[1][1] : g.rs[2][1];
  const double bx = ip1 == 0 ? g.rs[0][0] : ip1 == 1 ? g.rs[1][0] : g.rs[2][0];
  const double by = ip1 == 0 ? g.rs[0][1] : ip1 == 1 ? g.rs[1][1] : g.rs[2][1];
  double lx = bx - ax, ly = by - ay;
  const double ln = sqrt(lx * lx + ly * ly);
  lx /= ln;
  ly /= ln;
  const double ux = (-g.unz) * (-ly), uy = (-g.unz) * lx;
  const double d0x = ax - g.rmc[0], d0y = ay - g.rmc[1];
  const double d1x = bx - g.rmc[0], d1y = by - g.rmc[1];
  const double p0 = ux * d0x + uy * d0y;
  const double p0sq = p0 * p0;
  const double lp = lx * d1x + ly * d1y;
  const double lm = lx * d0x + ly * d0y;
  const double ledge = lp - lm;
  const double pplus = sqrt(p0sq + lp * lp);
  const double pminus = sqrt(p0sq + lm * lm);
  double factor, rif = 0.0;
  if (fabs(p0 / ledge) < 1e-4) {
    factor = lp * pplus - lm * pminus;
  } else {
    factor = p0 * log((pplus + lp) / (pminus + lm));
    rif = factor;
    factor = (factor * p0 + pplus * lp) - pminus * lm;
  }
  rr0 = rr1 = ri = 0.0;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const double f = __shfl_sync(0xffffffffu, factor, grp + e);
    rr0 += __shfl_sync(0xffffffffu, ux, grp + e) * f;
    rr1 += __shfl_sync(0xffffffffu, uy, grp + e) * f;
    ri += __shfl_sync(0xffffffffu, rif, grp + e);
  }
  rr0 *= 0.5;
  rr1 *= 0.5;
  rr0 /= g.area2;
  rr1 /= g.area2;
  ri /= (g.area2 * ul);
}

template <int NP>
constexpr int jk_threads() { return NP == 1 ? 256 : 128; }

// Eight lanes per unique face pair (four pairs per warp): lane q < 7 computes the lattice
// sums of quadrature point q (jksums, serial in the reference's ring order) for the group's
// np <= NP phasings; the pair's first lane gathers the seven results with warp shuffles and
// accumulates them in the 7-point rule's order, so each pair's integrals are those of a
// serial evaluation bit for bit.  The phasing-free parts (the smooth-term geometry, rho_r and
// the 1/R integral) are computed once and written to every phasing's slot.  Groups that are
// not live mirror the last pair and write nothing; every lane of a warp calls it.
template <int NP>
__device__ __forceinline__ void filljk_pair(const SheetDev &G, double ul, const PsiGroup &pg, int np, double us1x,
                                            double us1y, double us2x, double us2y, const JKGroup &jk, int *nonconv,
                                            long long pair, bool live, const cd (*__restrict__ ph1)[kPhase],
                                            const cd (*__restrict__ ph2)[kPhase], const double *__restrict__ etab) {
  const bool nophase = NP == 1 && pg.psi1[0] == 0.0 && pg.psi2[0] == 0.0;
  const int lane = threadIdx.x & 31, q = lane & 7, grp = lane & ~7;
  const int iu = live ? (int)pair : G.nufp - 1;
  const PairGeo g = pair_geo(G, iu);
  cd js[NP], ks[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) { js[p] = mkcd(0, 0); ks[p] = mkcd(0, 0); }
  unsigned ok = (1u << np) - 1u;
  if (q < 7) {
    double ux, uy;
    quad_offset(g, q, ul, ux, uy);
    ok = jksums_group<NP>(ux, uy, np, nophase, us1x, us1y, us2x, us2y, ph1, ph2, etab, js, ks);
  }
  __syncwarp();
  double rr0, rr1, ri;
  edge_terms(g, ul, q, grp, rr0, rr1, ri);
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    cd aJ = mkcd(0, 0), aJx = aJ, aJe = aJ, aK = aJ, aKx = aJ, aKe = aJ;
    int bad = 0;
#pragma unroll
    for (int i = 0; i < 7; ++i) {  // every lane takes part in the shuffles; the group's lane 0 keeps the sums
      cd jv, kv;
      jv.x = __shfl_sync(0xffffffffu, js[p].x, grp + i);
      jv.y = __shfl_sync(0xffffffffu, js[p].y, grp + i);
      kv.x = __shfl_sync(0xffffffffu, ks[p].x, grp + i);
      kv.y = __shfl_sync(0xffffffffu, ks[p].y, grp + i);
      bad |= !((__shfl_sync(0xffffffffu, ok, grp + i) >> p) & 1u);
      cd jw = c_qw[i] * jv;
      aJx = aJx + c_qxi[i] * jw;
      aJe = aJe + c_qeta[i] * jw;
      aJ = aJ + jw;
      cd kw = c_qw[i] * kv;
      aKx = aKx + c_qxi[i] * kw;
      aKe = aKe + c_qeta[i] * kw;
      aK = aK + kw;
    }
    if (q != 0 || !live || p >= np) continue;
    const JKDev &o = jk.s[p];
    o.J[iu] = aJ; o.Jxi[iu] = aJx; o.Jeta[iu] = aJe;
    o.K[iu] = aK; o.Kxi[iu] = aKx; o.Keta[iu] = aKe;
    o.rho_r[2 * iu] = rr0;
    o.rho_r[2 * iu + 1] = rr1;
    o.rinv[iu] = ri;
    if (bad) atomicAdd(nonconv + p, 1);
  }
}

}  // namespace
