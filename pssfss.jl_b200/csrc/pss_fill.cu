// K2 + K3: face-pair integrals and the MoM matrix fill.
//
// K2 k_filljk   restates Zint.jl:54-179 (filljk!) with PGF.jl:67-106 (jksums): eight
//               lanes per unique face pair, one lattice sum (quadrature point) per lane in
//               the reference's ring order, the seven sums gathered by warp shuffles and
//               accumulated in the 7-point rule's order, FP64; larger sheets take the
//               tabulated form of the same sums (pss_jktab.cu).
// K3a k_pairs   restates Zint.jl:218-245 (zint) and the per-edge algebra of
//               FillZY.jl:141-197 / 362-419: one thread per unique face pair computes
//               the 3x3 unflagged edge-pair terms  zA*(ρc2[iml]·a_isl) - zP*φ.
// K3b k_assemble replaces the spin-locked scatter of FillZY.jl:160-239 by a gather:
//               each Z entry sums, in a fixed order, the <=2x2 face incidences of its
//               test and source basis functions, applying the Floquet/sign flags and the
//               surface-resistance terms of Eqs. 7-34/7-35 (FillZY.jl:221-230).
//               Deterministic, atomic-free; writes FP64 and/or split FP32 planes.
#include <algorithm>

#include "pss_internal.cuh"
#include "pss_lattice.cuh"

namespace {

// Direct form: one launch over every face pair of a sheet (pss_jktab.cu holds the tabulated
// form that larger sheets take, and the rule between the two).
template <int NP>
__global__ void __launch_bounds__(jk_threads<NP>(), 3) k_filljk(SheetDev G, double ul, PsiGroup pg, double us1x, double us1y,
                                                double us2x, double us2y, JKGroup jk, int *nonconv) {
  __shared__ cd ph1[NP][kPhase], ph2[NP][kPhase];
  __shared__ double etab[256];  // 2^(j/256) for exp_neg
  const int np = NP == 1 ? 1 : pg.n;
  fill_phases<NP>(pg, np, ph1, ph2, etab);
  __syncthreads();
  const long long gid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 3;  // pair of this group
  filljk_pair<NP>(G, ul, pg, np, us1x, us1y, us2x, us2y, jk, nonconv, gid, gid < G.nufp, ph1, ph2, etab);
}

__device__ __forceinline__ cd ld_cd(const cd *p) {  // one 16-byte load
  const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
  return mkcd(v.x, v.y);
}

// One thread per class.  Bound by its FP64 operations (about 1200) and the gathers of its 42
// table nodes; what does not belong to the pair is prepared elsewhere: the point's coefficients
// on the host, vertices in metres and centroids per face at the upload, the cell-shift phases
// per CTA, both tables of a node in one 32-byte load.  613 -> 291 us for the 3.19M classes of the
// N = 3976 meander.
__global__ void __launch_bounds__(128, 5) k_pairs(SheetDev G, const PointParams *__restrict__ Pp, JKDev jk,
                                               const cd *__restrict__ tab, int mmax, cd *__restrict__ zb) {
  __shared__ PointParams P;
  __shared__ cd ph[9];
  for (int e = threadIdx.x; e < (int)(sizeof(PointParams) / sizeof(double)); e += blockDim.x)
    ((double *)&P)[e] = ((const double *)Pp)[e];
  __syncthreads();
  if (threadIdx.x < 9) ph[threadIdx.x] = cisd(-((double)((int)threadIdx.x / 3 - 1) * P.psi1 + (double)((int)threadIdx.x % 3 - 1) * P.psi2));
  __syncthreads();
  const int iu = blockIdx.x * blockDim.x + threadIdx.x;
  if (iu >= G.nufp) return;
  const cd *phase = P.psi1 == 0.0 && P.psi2 == 0.0 ? nullptr : ph;
  const int2 pf = __ldg(G.pair_faces + iu);
  const double2 *fm = reinterpret_cast<const double2 *>(G.face_m);
  const double2 rs0 = __ldg(fm + 4 * pf.y), rs1 = __ldg(fm + 4 * pf.y + 1), rs2 = __ldg(fm + 4 * pf.y + 2);
  const double2 rc = __ldg(fm + 4 * pf.x + 3);
  const double2 e1 = make_double2(rs1.x - rs0.x, rs1.y - rs0.y), e2 = make_double2(rs2.x - rs0.x, rs2.y - rs0.y);
  cd I1 = mkcd(0, 0), I1x = I1, I1e = I1, I2 = I1;
#pragma unroll 1
  for (int i = 0; i < 7; ++i) {
    const double xi = c_qxi[i], eta = c_qeta[i], w = c_qw[i];
    const double rtx = (rs0.x + e1.x * xi) + e2.x * eta, rty = (rs0.y + e1.y * xi) + e2.y * eta;
    cd g1, g2;
    sigma_interp(tab, mmax, P, rc.x - rtx, rc.y - rty, phase, g1, g2);
    g1 = w * g1;
    I1x = mkcd(fma(xi, g1.x, I1x.x), fma(xi, g1.y, I1x.y));
    I1e = mkcd(fma(eta, g1.x, I1e.x), fma(eta, g1.y, I1e.y));
    I1 = I1 + g1;
    I2 = mkcd(fma(w, g2.x, I2.x), fma(w, g2.y, I2.y));
  }
  const double u = P.u;
  const double rinv = jk.rinv[iu];
  const double2 rr = __ldg(reinterpret_cast<const double2 *>(jk.rho_r) + iu);
  // cI1*I1 + u*J + cK*K and its xi, eta moments; the third barycentric moment is the rest
  const cd J = ld_cd(jk.J + iu), K = ld_cd(jk.K + iu);
  const cd zphi = P.zP * cmac(cmac(u * mkcd(rinv + J.x, J.y), P.cI2, I2), P.cKP, K);
  const cd A0 = cmac(cmac(u * J, P.cI1, I1), P.cK, K);
  const cd Ax = cmac(cmac(u * ld_cd(jk.Jxi + iu), P.cI1, I1x), P.cK, ld_cd(jk.Kxi + iu));
  const cd Ae = cmac(cmac(u * ld_cd(jk.Jeta + iu), P.cI1, I1e), P.cK, ld_cd(jk.Keta + iu));
  const cd Az = (A0 - Ax) - Ae;
  const double2 rm0 = __ldg(fm + 4 * pf.x), rm1 = __ldg(fm + 4 * pf.x + 1), rm2 = __ldg(fm + 4 * pf.x + 2);
  // rho - r_isl integrated: the moments weighted by the vertices' offsets from vertex isl; subtracting r_isl times
  // the whole from the absolute moments cancels to 1e-14 of the result, this form keeps 1e-16
  double2 *out = reinterpret_cast<double2 *>(zb) + iu;  // plane q at out[q * nufp]: coalesced stores
#pragma unroll
  for (int isl = 0; isl < 3; ++isl) {
    const double2 ri = isl == 0 ? rs0 : isl == 1 ? rs1 : rs2;
    cd av[2];
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const double o = d ? ri.y : ri.x;
      const double d0 = (d ? rs0.y : rs0.x) - o, d1 = (d ? rs1.y : rs1.x) - o, d2 = (d ? rs2.y : rs2.x) - o;
      const double sg = (d ? rr.y : rr.x) + (u * rinv) * ((d ? rc.y : rc.x) - o);
      av[d] = mkcd(fma(d0, Ax.x, fma(d1, Ae.x, fma(d2, Az.x, sg))), fma(d0, Ax.y, fma(d1, Ae.y, d2 * Az.y)));
      av[d] = P.zA * av[d];
    }
#pragma unroll
    for (int iml = 0; iml < 3; ++iml) {
      const double2 rm = iml == 0 ? rm0 : iml == 1 ? rm1 : rm2;
      const double cx = 0.5 * (rc.x - rm.x), cy = 0.5 * (rc.y - rm.y);
      out[(size_t)(3 * isl + iml) * G.nufp] =
          make_double2(fma(cx, av[0].x, fma(cy, av[1].x, -zphi.x)), fma(cx, av[0].y, fma(cy, av[1].y, -zphi.y)));
    }
  }
}

// The incidences of a test basis function, unpacked once per thread: face, slot and conjugated
// signed Floquet factor of each (unused ones repeat the first with factor 0).
struct RowInc {
  int cnt, face[4], loc[4];
  cd flag[4];
};
__device__ __forceinline__ void unpack_inc(int4 v, const cd *ff, int cnt, bool conj, RowInc &r) {
  const int q[4] = {v.x, v.y, v.z, v.w};
  r.cnt = cnt;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int e = a < cnt ? q[a] : q[0];
    r.face[a] = e >> 8;
    r.loc[a] = (e >> 4) & 3;
    cd f = ff[e & 7];
    if (conj) f = conjd(f);
    r.flag[a] = a < cnt ? (e & 8 ? -f : f) : mkcd(0, 0);
  }
}

// Surface-resistance term of incidences (fa, ka) x (fa, kb) of one face (Eqs. 7-34/7-35,
// FillZY.jl:221-230).
__device__ __noinline__ cd resistance_term(const SheetDev &G, int fa, int ka, int kb, cd mflag, cd sflag) {
  const double fr = G.fr[fa];
  if (fr == 0.0) return mkcd(0, 0);
  const double *ls = G.face_ls + 3 * fa;
  const double g = fr / G.face_a48[fa];
  if (ka == kb) {  // the other two edges of the face: next and previous slot
    const double l1 = ls[(kb + 1) % 3], l2 = ls[(kb + 2) % 3], l0 = ls[kb];
    return mkcd(g * (3 * (l1 * l1 + l2 * l2) - l0 * l0), 0.0);
  }
  const double lt = ls[3 - ka - kb];  // the third edge
  const double geo = ls[kb] * ls[kb] + ls[ka] * ls[ka] - 3 * (lt * lt);
  return geo * ((g * sflag) * mflag);
}

// Z[m, n] (m = test / match basis function, n = source) from the pair terms zb: the <= 4 x 4
// face incidences of the two basis functions in a fixed order, with the Floquet / sign flags
// and the surface-resistance terms.  Two by two, the case of every interior edge and of every
// edge pair across the cell boundary, runs without branches so that its loads overlap.
__device__ __forceinline__ cd assemble_entry(const SheetDev &G, const cd *ff, bool res, const cd *__restrict__ zb,
                                             const RowInc &M, int n) {
  const int cn = __ldg(G.inc_cnt + n);
  RowInc S;
  unpack_inc(__ldg(G.inc + n), ff, cn, false, S);
  cd acc = mkcd(0, 0);
  if (M.cnt <= 2 && cn <= 2) {
    int iu[4];
    cd v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t)
      iu[t] = __ldg(G.ufpm + (size_t)M.face[t >> 1] + (size_t)S.face[t & 1] * G.nface);
#pragma unroll
    for (int t = 0; t < 4; ++t)
      v[t] = ld_cd(zb + (size_t)(3 * S.loc[t & 1] + M.loc[t >> 1]) * G.nufp + iu[t]);
#pragma unroll
    for (int t = 0; t < 4; ++t) acc = cmac(acc, M.flag[t >> 1] * S.flag[t & 1], v[t]);
  } else {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        if (a >= M.cnt || b >= cn) continue;
        const int iu = __ldg(G.ufpm + (size_t)M.face[a] + (size_t)S.face[b] * G.nface);
        acc = cmac(acc, M.flag[a] * S.flag[b], ld_cd(zb + (size_t)(3 * S.loc[b] + M.loc[a]) * G.nufp + iu));
      }
  }
  if (res) {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if (a < M.cnt && b < cn && M.face[a] == S.face[b])
          acc = acc + resistance_term(G, M.face[a], M.loc[a], S.loc[b], M.flag[a], S.flag[b]);
  }
  return acc;
}

// Four entries of a row of a sheet without resistance whose basis functions all have at most two
// incidences: no branches, all class numbers and then all pair terms in flight together.
__device__ __forceinline__ void assemble_four(const SheetDev &G, const cd *ff, const cd *__restrict__ zb,
                                              const RowInc &M, const int (&n)[4], cd (&z)[4]) {
  int2 e[4];  // the columns' packed incidences
  bool two[4];
  int iu[4][4];
  cd v[4][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    e[k] = __ldg(reinterpret_cast<const int2 *>(G.inc + n[k]));
    two[k] = __ldg(G.inc_cnt + n[k]) > 1;
    if (!two[k]) e[k].y = e[k].x;
#pragma unroll
    for (int t = 0; t < 4; ++t)
      iu[k][t] = __ldg(G.ufpm + (size_t)M.face[t >> 1] + (size_t)((t & 1 ? e[k].y : e[k].x) >> 8) * G.nface);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int t = 0; t < 4; ++t)
      v[k][t] = ld_cd(zb + (size_t)(3 * (((t & 1 ? e[k].y : e[k].x) >> 4) & 3) + M.loc[t >> 1]) * G.nufp + iu[k][t]);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    cd sf[2] = {ff[e[k].x & 7], ff[e[k].y & 7]};
    if (e[k].x & 8) sf[0] = -sf[0];
    if (e[k].y & 8) sf[1] = -sf[1];
    if (!two[k]) sf[1] = mkcd(0, 0);
    z[k] = mkcd(0, 0);
#pragma unroll
    for (int t = 0; t < 4; ++t) z[k] = cmac(z[k], M.flag[t >> 1] * sf[t & 1], v[k][t]);
  }
}

// Z[m, n], row-major (z64 with leading dimension ld, the FP32 planes with ldf), one 32 x 64
// tile per CTA of 32 x 8 threads.  The gathers run with a warp along the 32 rows of a tile
// column (consecutive match basis functions against one source basis function: consecutive
// match faces, so the class look-ups and most pair-term loads of a warp are contiguous); each
// thread keeps its row's incidences and takes 8 columns; the tile then goes out through shared
// memory row by row, 64 consecutive entries per row.  Bound by the latency of the gathers (4 class
// numbers and 4 pair terms per entry).  TWO, for sheets without resistance whose basis functions
// all have at most two incidences: the gathers of four columns are issued together, class
// numbers first (336 -> 210 us at N = 3976); the general form takes one entry after the other.
template <bool TWO>
__global__ void __launch_bounds__(256, TWO ? 2 : 3) k_assemble(SheetDev G, const PointParams *__restrict__ Pp,
                                                  const cd *__restrict__ zb, cd *__restrict__ z64,
                                                  float *__restrict__ zr, float *__restrict__ zi, long long ld,
                                                  long long ldf) {
  __shared__ __align__(16) cd tile[32][65];
  __shared__ cd ff[8];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int m0 = blockIdx.y * 32, n0 = blockIdx.x * 64;
  if (ty == 0 && tx < 5) ff[tx] = Pp->ff[tx];
  __syncthreads();
  const int m = min(m0 + tx, G.nbf - 1);  // rows past the end repeat the last, written nowhere
  const bool res = G.has_res && !Pp->magnetic;
  RowInc M;
  unpack_inc(__ldg(G.inc + m), ff, __ldg(G.inc_cnt + m), true, M);
  if constexpr (TWO) {
#pragma unroll
    for (int k0 = 0; k0 < 8; k0 += 4) {
      int n[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) n[k] = min(n0 + ty + 8 * (k0 + k), G.nbf - 1);
      cd z[4];
      assemble_four(G, ff, zb, M, n, z);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        *reinterpret_cast<double2 *>(&tile[tx][ty + 8 * (k0 + k)]) = make_double2(z[k].x, z[k].y);
    }
  } else {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int c = ty + 8 * k;
    const cd v = assemble_entry(G, ff, res, zb, M, min(n0 + c, G.nbf - 1));
    *reinterpret_cast<double2 *>(&tile[tx][c]) = make_double2(v.x, v.y);
  }
  }
  __syncthreads();
#pragma unroll
  for (int rr = 0; rr < 4; ++rr) {
    const int r = ty * 4 + rr, mm = m0 + r;
    if (mm >= G.nbf) break;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = tx + 32 * h, n = n0 + c;
      if (n >= G.nbf) continue;
      const double2 v = *reinterpret_cast<const double2 *>(&tile[r][c]);
      if (z64) *reinterpret_cast<double2 *>(z64 + (size_t)mm * ld + n) = v;
      if (zr) {
        zr[(size_t)mm * ldf + n] = (float)v.x;
        zi[(size_t)mm * ldf + n] = (float)v.y;
      }
    }
  }
}

// Adjoint contraction of one perturbed input set, without its matrix.  CTA (x, y) takes the 32
// rows m = 32x .. 32x+31 (threadIdx.x) and column chunk y of gridDim.y; its 8 warps split the
// chunk's columns (n = chunk start + threadIdx.y + 8j);
// each thread assembles Z_k[m, n] on the fly from the set's pair terms (recomputed
// Green's-function values, never stored) - a warp gathers one column's 32 rows, consecutive
// match faces, so its class look-ups are contiguous - and accumulates Z_k[m, n] X[n, b].  The
// 8 column shares of a row are added in a fixed order to form the chunk's part of
//     y[m, b] = R_k[m, b] - sum_n Z_k[m, n] X[n, b]
// (R_k in chunk 0's part) for the right-hand sides b0 .. b0+NB-1, and the CTA writes its share
// of G[a + b*nm] = sum_m Lam[m, a] y[m, b] to part[x + y*gridDim.x] (rows in a fixed order, no
// atomics: the shares are added in a fixed order by k_adj_reduce, so the result is deterministic).
// Vectors are nbf x nm column-major.
template <int kAdjNB, bool TWO>
__global__ void __launch_bounds__(256, 2) k_adj_contract(SheetDev G, const PointParams *__restrict__ Pp,
                                                      const cd *__restrict__ zb, const cd *__restrict__ X,
                                                      const cd *__restrict__ R, const cd *__restrict__ Lam, int nm,
                                                      int b0, cd *__restrict__ part) {
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int m = blockIdx.x * 32 + tx;
  const int nb = min(kAdjNB, nm - b0);
  const int nbf = G.nbf;
  const int csz = (nbf + gridDim.y - 1) / gridDim.y, c0 = blockIdx.y * csz, c1 = min(nbf, c0 + csz);
  __shared__ cd red[8][32][kAdjNB];
  __shared__ cd yrow[32][kAdjNB];
  __shared__ cd ff[8];
  cd acc[kAdjNB];
#pragma unroll
  for (int b = 0; b < kAdjNB; ++b) acc[b] = mkcd(0, 0);
  if (ty == 0 && tx < 5) ff[tx] = Pp->ff[tx];
  __syncthreads();
  {
    const bool res = G.has_res && !Pp->magnetic;
    const int mc = min(m, nbf - 1);  // rows past the end repeat the last and are dropped below
    RowInc M;
    unpack_inc(__ldg(G.inc + mc), ff, __ldg(G.inc_cnt + mc), true, M);
    if constexpr (TWO) {
      for (int nn = c0 + ty; nn < c1; nn += 32) {
        int n[4];
        cd z[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) n[k] = min(nn + 8 * k, c1 - 1);
        assemble_four(G, ff, zb, M, n, z);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (nn + 8 * k >= c1) break;
#pragma unroll
          for (int b = 0; b < kAdjNB; ++b)
            if (b < nb) acc[b] = cmac(acc[b], z[k], X[(size_t)(b0 + b) * nbf + n[k]]);
        }
      }
    } else {
#pragma unroll 2
      for (int n = c0 + ty; n < c1; n += 8) {
        const cd z = assemble_entry(G, ff, res, zb, M, n);
#pragma unroll
        for (int b = 0; b < kAdjNB; ++b)
          if (b < nb) acc[b] = cmac(acc[b], z, X[(size_t)(b0 + b) * nbf + n]);
      }
    }
  }
#pragma unroll
  for (int b = 0; b < kAdjNB; ++b) red[ty][tx][b] = acc[b];
  __syncthreads();
  if (ty == 0) {
    for (int b = 0; b < kAdjNB; ++b) {
      cd sdot = mkcd(0, 0);
      for (int w = 0; w < 8; ++w) sdot = sdot + red[w][tx][b];
      // rows past the last and right-hand sides past nm lie outside R: they are not read
      const bool ok = m < nbf && b < nb;
      const cd rb = ok && blockIdx.y == 0 ? R[(size_t)(b0 + b) * nbf + m] : mkcd(0, 0);
      yrow[tx][b] = ok ? rb - sdot : mkcd(0, 0);
    }
  }
  __syncthreads();
  // this CTA's share of G: thread e of the 256 covers entries e, e + 256, ...
  const int tid = ty * 32 + tx;
  for (int e = tid; e < nm * nb; e += 256) {
    const int a = e % nm, b = e / nm;
    cd sum = mkcd(0, 0);
    for (int r = 0; r < 32; ++r) {
      const int mr = blockIdx.x * 32 + r;
      if (mr < nbf) sum = sum + Lam[(size_t)a * nbf + mr] * yrow[r][b];
    }
    part[((size_t)blockIdx.y * gridDim.x + blockIdx.x) * nm * nm + a + (size_t)(b0 + b) * nm] = sum;
  }
}

// G[e] = sum over the CTAs' shares, in a fixed order (strided partial sums, then a tree).
__global__ void __launch_bounds__(256) k_adj_reduce(int nparts, int ne, const cd *__restrict__ part, cd *__restrict__ G) {
  const int e = blockIdx.x;
  __shared__ cd red[256];
  cd s = mkcd(0, 0);
  for (int q = threadIdx.x; q < nparts; q += 256) s = s + part[(size_t)q * ne + e];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] = red[threadIdx.x] + red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) G[e] = red[0];
}

}  // namespace

constexpr int kAdjChunks = 8;  // column chunks of the contraction grid
size_t pss_adj_part_bytes(int nbf, int nm) { return (size_t)cdiv_u(nbf, 32) * kAdjChunks * nm * nm * sizeof(cd); }

void pss_adj_contract(const SheetDev &G, const PointParams *dP1, const cd *zb, const cd *X, const cd *R,
                      const cd *Lam, int nm, cd *part, cd *Gout, cudaStream_t st) {
  const int nblk = cdiv_u(G.nbf, 32);
  for (int b0 = 0; b0 < nm;) {  // four right-hand sides at a time where that is all there is
    const int nb = nm - b0 <= 4 ? 4 : 8;
    const bool two = G.two_inc && !G.has_res;
    auto kern = nb == 4 ? (two ? k_adj_contract<4, true> : k_adj_contract<4, false>)
                        : (two ? k_adj_contract<8, true> : k_adj_contract<8, false>);
    pss_count_launch();
    kern<<<dim3(nblk, kAdjChunks), dim3(32, 8), 0, st>>>(G, dP1, zb, X, R, Lam, nm, b0, part);
    b0 += nb;
  }
  pss_count_launch();
  k_adj_reduce<<<nm * nm, 256, 0, st>>>(nblk * kAdjChunks, nm * nm, part, Gout);
}

int pss_filljk_group(const SheetDev &G, double ulocal, int np, const double *psi1, const double *psi2,
                     const double s1[2], const double s2[2], const JKDev *jk, int *nonconv, void *ws, size_t ws_bytes,
                     cudaStream_t st) {
  if (G.nufp == 0 || np <= 0) return 0;
  PsiGroup pg{};
  JKGroup jg{};
  pg.n = std::min(np, kJKGroup);
  for (int p = 0; p < pg.n; ++p) {
    pg.psi1[p] = psi1[p];
    pg.psi2[p] = psi2[p];
    jg.s[p] = jk[p];
  }
  const double a = ulocal * s1[0], b = ulocal * s1[1], c = ulocal * s2[0], d = ulocal * s2[1];
  JKTabPlan plan;
  if (pss_jktab_plan(G, ulocal, s1, s2, pg.n, plan) && ws_bytes >= plan.bytes)
    return pss_jktab_launch(G, ulocal, pg, s1, s2, jg, nonconv, plan, ws, st);
  const long long lanes = (long long)G.nufp * 8;
  pss_count_launch();
  if (pg.n == 1)
    k_filljk<1><<<cdiv_u(lanes, jk_threads<1>()), jk_threads<1>(), 0, st>>>(G, ulocal, pg, a, b, c, d, jg, nonconv);
  else if (pg.n == 2)
    k_filljk<2><<<cdiv_u(lanes, jk_threads<2>()), jk_threads<2>(), 0, st>>>(G, ulocal, pg, a, b, c, d, jg, nonconv);
  else
    k_filljk<kJKGroup><<<cdiv_u(lanes, jk_threads<kJKGroup>()), jk_threads<kJKGroup>(), 0, st>>>(G, ulocal, pg, a, b,
                                                                                             c, d, jg, nonconv);
  PSS_CUDA_TRY(cudaGetLastError());
  return 0;
}

int pss_filljk(const SheetDev &G, double ulocal, double psi1, double psi2, const double s1[2], const double s2[2],
               JKDev jk, int *nonconv, void *ws, size_t ws_bytes, cudaStream_t st) {
  return pss_filljk_group(G, ulocal, 1, &psi1, &psi2, s1, s2, &jk, nonconv, ws, ws_bytes, st);
}

void pss_fill_pairs(const SheetDev &G, const PointParams *dP1, const JKDev &jk, const TableDev &tab, cd *zb,
                    cudaStream_t st) {
  if (G.nufp == 0) return;
  pss_count_launch();
  k_pairs<<<cdiv_u(G.nufp, 128), 128, 0, st>>>(G, dP1, jk, tab.t, tab.mmax, zb);
}

void pss_fill_assemble(const SheetDev &G, const PointParams *dP1, const cd *zb, cd *z64, float *zr, float *zi,
                       long long ld, long long ldf, cudaStream_t st) {
  dim3 blk(32, 8);
  dim3 grd(cdiv_u(G.nbf, 64), cdiv_u(G.nbf, 32));
  pss_count_launch();
  auto kern = G.two_inc && !G.has_res ? k_assemble<true> : k_assemble<false>;
  kern<<<grd, blk, 0, st>>>(G, dP1, zb, z64, zr, zi, ld, ldf);
}
