// Internal declarations shared by the library's translation units.
#pragma once
#include <atomic>
#include <mutex>

#include "pss_common.cuh"
#include "pssfss_b200.h"

// The current device and the identifier of its current CUDA context (pss_mem.cu).  A context's
// handle comes back after a reset of the device, its identifier does not.
constexpr int kMaxDevices = 64;
int pss_context_id(int *dev, unsigned long long *id);

// One-time set-up per device and context (kernel attributes and the like), safe to reach from
// several host threads: f() runs once for each context it is first called in (that context
// current), so what it sets is set again after a device reset.
struct DeviceOnce {
  std::atomic<unsigned long long> done[kMaxDevices] = {};  // the context's identifier (from 1 on)
  std::mutex mu;
};
template <class F>
int device_once(DeviceOnce &o, F &&f) {
  int dev = -1;
  unsigned long long id = 0;
  if (int rc = pss_context_id(&dev, &id)) return rc;
  if (o.done[dev].load(std::memory_order_acquire) == id) return 0;
  std::lock_guard<std::mutex> lk(o.mu);
  if (o.done[dev].load(std::memory_order_relaxed) == id) return 0;
  const int rc = f();
  if (!rc) o.done[dev].store(id, std::memory_order_release);
  return rc;
}

// Layer stack of one Gblock region (same for every frequency point of a batch).
struct StackParams {
  int nl, s;  // number of layers, 1-based interface index of the sheet
  cd eps[PSS_MAXLAYERS], mu[PSS_MAXLAYERS];
  double width[PSS_MAXLAYERS];  // metres
};

// Per frequency-point scalars (computed on the host, read by the kernels).
struct PointParams {
  double k0, u, psi1, psi2, omega;
  double b1[2], b2[2], b00[2];  // reciprocal lattice (1/m) and principal Floquet vector
  double area;                  // 4π²/|β1×β2|  (m²)
  double k0sq, b2min;
  cd mutilde, epsbar, c3, d3;       // electric (PGF.jl:205-210, FillZY.jl:60-61)
  cd f1, f3, p1, p3;                // magnetic summand factors (PGF.jl:496-499)
  cd I1fact, KFfact, I2fact, KPfact;  // filly factors (FillZY.jl:319-322)
  cd ff[5];                         // Floquet factors by edge code (FillZY.jl:72-77)
  // coefficients of the pair terms (k_pairs): a_isl = cI1*I1_i + sing + u*J_i + cK*K_i,
  // phi = cI2*I2 + u*(rinv + J) + cKP*K, term(isl, iml) = zA*(rc2[iml] . a_isl) - zP*phi
  cd cI1, cK, cI2, cKP, zA, zP;
  int magnetic;
};

// Device-resident sheet topology (0-based indices).
struct SheetDev {
  int nface, nbf, nufp, nnode;
  double upm;  // sheet units per metre
  const double *rho;     // 2*nnode, sheet units
  const int *fv;         // 3*nface
  const int *ufpm;       // nface*nface, 0-based class of (match fa, source fb) at fa + fb*nface
  const int *ufp_rep;    // nufp, 0-based column-major face pair of the class representative
  // pair terms zb (pss_fill_pairs): 9 planes of nufp complex, term 3*isl + iml of class iu at
  // zb[(3*isl + iml)*nufp + iu]
  const double *fr;      // nface
  const double *face_ls; // 3*nface edge lengths (m): |r3-r2|, |r1-r3|, |r1-r2|
  const double *face_a48;// nface: 48*|area| (m²)
  const int *inc_cnt;    // nbf
  const int *inc_face;   // 4*nbf
  const int *inc_loc;    // 4*nbf local edge slot 0..2
  const int *inc_sgn;    // 4*nbf +1 plus / -1 minus
  const int *inc_eci;    // 4*nbf edge boundary code 0..4
  const double *face_m;  // 8 per face, metres: the three vertices and the centroid (k_pairs)
  const int2 *pair_faces;// nufp: (match face, source face) of the class representative
  const int4 *inc;       // nbf: packed incidences, face << 8 | slot << 4 | minus << 3 | edge code
  int has_res;           // some face has a surface resistance
  int two_inc;           // no basis function has more than two incidences
  double ext1, ext2;     // extents of the vertices in lattice coordinates (along s1 and s2)
};

// J/K cache (Zint.jl:54-179), SoA over unique face pairs.
struct JKDev {
  cd *J, *Jxi, *Jeta, *K, *Kxi, *Keta;
  double *rho_r;  // 2*nufp
  double *rinv;   // nufp
};

// Face-pair integrals of up to kJKGroup phasings (psi1, psi2) of one sheet in one launch: the
// phasing-free part of every lattice summand is shared, each phasing keeps its own sums.
constexpr int kJKGroup = 4;
struct PsiGroup {
  double psi1[kJKGroup], psi2[kJKGroup];
  int n;
};
struct JKGroup {
  JKDev s[kJKGroup];
};

// Modal tables of one point: padded (mmax+2)^2 column-major, index (m,n) in -1..mmax, both
// tables of a node side by side (entry e: t[2e] and t[2e + 1], one 32-byte sector).
struct TableDev {
  cd *t;
  int mmax;
};

// Both tables of one node by one 32-byte load.
__device__ __forceinline__ void ld_node(const cd *p, double (&v)[4]) {
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}

// a / 2 pi, correctly rounded: quotient estimate and one fused correction with the correctly
// rounded reciprocal (P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34 (1990) 111-119).  The rounding matters: the stencil
// below is not continuous across its cells, and mesh offsets fall on cell boundaries.
__device__ __forceinline__ double over_twopi(double a) {
  constexpr double y = 1.0 / PSS_TWOPI;
  const double q = a * y;
  return fma(fma(-q, PSS_TWOPI, a), y, q);
}

// Six-point interpolation of both padded tables (PGF.jl:396-441) at offset (rx, ry); ph: the
// phase factors cis(-(ms psi1 + ns psi2)) for ms, ns in -1..1 (null: no phasing).
__device__ __forceinline__ void sigma_interp(const cd *__restrict__ T, int mmax, const PointParams &P, double rx,
                                             double ry, const cd *__restrict__ ph, cd &s1, cd &s2) {
  double x1o = over_twopi(P.b1[0] * rx + P.b1[1] * ry);
  if (fabs(x1o) < 1e-8) x1o = 0.0;
  double x2o = over_twopi(P.b2[0] * rx + P.b2[1] * ry);
  if (fabs(x2o) < 1e-8) x2o = 0.0;
  // Julia's mod(x, 1) in [0, 1] is x - floor(x); the cell shift is floor(x)
  const double ms = floor(x1o), ns = floor(x2o);
  const double x1 = x1o - ms, x2 = x2o - ns;
  int m = (int)(mmax * x1);
  int n = (int)(mmax * x2);
  // x <= 1, and mmax*x can round up to mmax; the stencil then must stay inside the padded
  // table (same point, one cell to the left).
  if (m >= mmax) m = mmax - 1;
  if (n >= mmax) n = mmax - 1;
  const double p = mmax * x1 - m, q = mmax * x2 - n;
  const double p2 = p * p, q2 = q * q, pq = p * q;
  const int L = mmax + 2;
  const cd *c = T + 2 * ((size_t)(m + 1) + (size_t)(n + 1) * L);
  const double w[6] = {0.5 * (q2 - q),  0.5 * (p2 - p),              ((1.0 + pq) - p2) - q2,
                       0.5 * ((p2 - 2.0 * pq) + p), 0.5 * ((q2 - 2.0 * pq) + q), pq};
  double v[6][4];
  ld_node(c - 2 * L, v[0]);
  ld_node(c - 2, v[1]);
  ld_node(c, v[2]);
  ld_node(c + 2, v[3]);
  ld_node(c + 2 * L, v[4]);
  ld_node(c + 2 * L + 2, v[5]);
  double s[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    s[e] = w[0] * v[0][e];
#pragma unroll
    for (int k = 1; k < 6; ++k) s[e] = fma(w[k], v[k][e], s[e]);
  }
  s1 = mkcd(s[0], s[1]);
  s2 = mkcd(s[2], s[3]);
  if (ph) {
    cd f;
    if (fabs(ms) <= 1.0 && fabs(ns) <= 1.0) f = ph[((int)ms + 1) * 3 + (int)ns + 1];
    else f = cisd(-(ms * P.psi1 + ns * P.psi2));
    s1 = s1 * f;
    s2 = s2 * f;
  }
}

// The device a context runs on (0, or -1 for a null context with a message).
extern "C" int pss_ctx_device(const pss_ctx *c, int *dev);

// Device memory (pss_mem.cu): a bounded pool per device with cudaMalloc / cudaFree semantics.
int pss_dev_alloc(void **p, size_t bytes);
void pss_dev_free(void *p);
int pss_dev_trim();  // gives the current device's kept memory back

// Counts every kernel the library launches (reported by pss_kernel_launches()).
void pss_count_launch();
// Optional CUDA-event timing of the Schur-complement GEMM launches (pss_profile): returns
// a token (-1 when profiling is off) to pass to pss_prof_end with the launch's flops.
int pss_prof_begin(cudaStream_t st);
void pss_prof_end(int token, cudaStream_t st, int kind, double work);

// ---- host launchers (return 0 or a negative error code; errors via pss_set_error) ----
// Modal tables (pss_tables.cu)
void pss_tables_ring_fill(const StackParams &S, const PointParams *dP, int npts, int R, cd *dense,
                          size_t point_stride, cudaStream_t st);
void pss_tables_ring_sums(const PointParams *dP, int npts, int R, const cd *dense, size_t point_stride,
                          double convtest, unsigned char *conv, cudaStream_t st);
void pss_tables_find_mmax(int npts, int R, const unsigned char *conv, int *mmax, int *flag, cudaStream_t st);
// Up to kTableChunk points of one mmax (their slots in the chunk) finished together.
constexpr int kTableChunk = 32;
struct TableGroup {
  int n;
  int q[kTableChunk];
};
int pss_tables_finish(const cd *dense, size_t pstride, int R, int mmax, const PointParams *dP, const TableGroup &g,
                      cd *stage, cd *t, size_t tstride, cudaStream_t st);
size_t pss_table_cap(int mmax);  // (mmax+2)^2 entries per padded table

// Face-pair integrals and matrix fill (pss_fill.cu)
// ws: scratch of at least pss_jktab_bytes; in a smaller one every pair's lattice sums run ring by ring.
int pss_filljk(const SheetDev &G, double ulocal, double psi1, double psi2, const double s1[2], const double s2[2],
               JKDev jk, int *nonconv, void *ws, size_t ws_bytes, cudaStream_t st);
// np <= kJKGroup phasings at once into jk[0..np), non-convergence counts into nonconv[0..np)
int pss_filljk_group(const SheetDev &G, double ulocal, int np, const double *psi1, const double *psi2,
                     const double s1[2], const double s2[2], const JKDev *jk, int *nonconv, void *ws,
                     size_t ws_bytes, cudaStream_t st);
// Tabulated lattice sums (pss_jktab.cu): the panels that cover a sheet's offsets, and the bytes
// of the tables, maps and the list of pairs left to the direct form for np phasings.
struct JKTabPlan {
  int na = 0, nb = 0;  // panels along the two lattice vectors
  double a0 = 0, b0 = 0, ra = 0, rb = 0;  // first panel's corner; panels per unit lattice coordinate
  double dmin = 0;     // distance of the offsets to the nearest image of ring 2 (u-scaled)
  size_t bytes = 0;
};
bool pss_jktab_plan(const SheetDev &G, double ulocal, const double s1[2], const double s2[2], int np, JKTabPlan &P);
size_t pss_jktab_bytes(const SheetDev &G, double ulocal, const double s1[2], const double s2[2], int np);
int pss_jktab_launch(const SheetDev &G, double ulocal, const PsiGroup &pg, const double s1[2], const double s2[2],
                     const JKGroup &jk, int *nonconv, const JKTabPlan &P, void *ws, cudaStream_t st);
void pss_fill_pairs(const SheetDev &G, const PointParams *dP1, const JKDev &jk, const TableDev &tab, cd *zb,
                    cudaStream_t st);
// Assemble Z (row-major): z64 with leading dimension ld, the FP32 planes (zr, zi) with ldf.
// z64 and/or (zr, zi) may be null.
void pss_fill_assemble(const SheetDev &G, const PointParams *dP1, const cd *zb, cd *z64, float *zr, float *zi,
                       long long ld, long long ldf, cudaStream_t st);

// Basis-function transforms, right-hand sides, projection (pss_bfft.cu)
void pss_bfft(const SheetDev &G, int nmodes, const double *kvec, double psi1, double psi2, cd *bf,
              cudaStream_t st);
void pss_rhs(int nbf, int nmodes, const cd *bf, const cd *src, cd *rhs, cudaStream_t st);
void pss_project(int nbf, int nmodes, const cd *bf, const double *tobs, const cd *wobs, const cd *X, cd *dS,
                 cudaStream_t st);
// PT (nbf x nmodes, column-major): row i of the projection, t_i · F_i[n], for the adjoint solve.
void pss_proj_rows(int nbf, int nmodes, const cd *bf, const double *tobs, cd *PT, cudaStream_t st);
// Adjoint contraction of a perturbed set from its pair terms zb (no matrix stored):
//   Gout[a + b*nm] = sum_m Lam[m, a] (R[m, b] - sum_n Z[m, n] X[n, b]);
// part: scratch of pss_adj_part_bytes(nbf, nm).
size_t pss_adj_part_bytes(int nbf, int nm);
void pss_adj_contract(const SheetDev &G, const PointParams *dP1, const cd *zb, const cd *X, const cd *R,
                      const cd *Lam, int nm, cd *part, cd *Gout, cudaStream_t st);

// Dense complex LU and solves (pss_lu.cu); matrices row-major with leading dimension ld.
// Batched forms factor nb matrices of order n at A + b*ms (elements), pivots at ipiv + b*n,
// info words at info + b; all matrices advance together, one launch per step.
int pss_lu64(int n, cd *A, long long ld, int *ipiv, int *info, void *ws, size_t ws_bytes, cudaStream_t st);
int pss_lu32(int n, float *Ar, float *Ai, long long ld, int *ipiv, int *info, void *ws, size_t ws_bytes,
             cudaStream_t st);
int pss_lu64_batched(int n, int nb, cd *A, long long ld, long long ms, int *ipiv, int *info, void *ws,
                     size_t ws_bytes, cudaStream_t st);
// FP32 tile shape: panel_w in {8, 16, 32} columns per cluster panel, outer_nb in {64, 128}
// columns per outer block (the tensor-core update's K); 0 picks 32 / 128.
int pss_lu32_batched(int n, int nb, float *Ar, float *Ai, long long ld, long long ms, int *ipiv, int *info,
                     void *ws, size_t ws_bytes, cudaStream_t st, int panel_w = 0, int outer_nb = 0);
size_t pss_lu_ws_bytes(int n, int precision, int nb = 1);

// Tensor-core (tcgen05, 3xTF32) complex Schur update on FP32 planes (pss_gemm_tc.cu), for
// each of nb matrices A_b = A + b*ms (elements):
//   A_b[m0:m0+M, n0:n0+N] -= A_b[m0:m0+M, k0:k0+K] * A_b[k0:k0+K, n0:n0+N],
// row-major, leading dimension ld; ws holds the split operands
// (pss_tc_ws_bytes(M, N, K rounded up to 16, nb)).  A bounded pipeline wait that gives up
// writes -1 to err[b].
size_t pss_tc_ws_bytes(int Mmax, int Nmax, int KP, int nb = 1);
int pss_cgemm_tc(float *Ar, float *Ai, long long ld, long long ms, int nb, int m0, int M, int n0, int N, int k0,
                 int K, void *ws, size_t ws_bytes, int *err, cudaStream_t st);

// Triangular solves and refinement (pss_trsv.cu).  The factor is either FP64 (LU64) or
// FP32 planes (Lr, Li); pass the other as null.
struct SolveWS {
  int n = 0, nblk = 0, nb = 0, epoch = 0;
  long long dstride = 0;   // elements between the matrices' diagonal-block inverses
  int cstride = 0;         // ints between the matrices' control words
  cd *Dinv = nullptr;      // inverses of the 64x64 diagonal blocks (L and U), per matrix
  int *perm = nullptr;     // pivot permutations
  int *ctrl = nullptr;     // per matrix: ticket, error flag, converged flag, per-block epoch flags
  double *norms = nullptr; // refinement norms, per matrix
  void bind(void *base, int n_, int nb_ = 1);
};
// Batched over nb matrices: factors at LU64 (or Lr/Li) + b*ms, ipiv + b*n, right-hand sides
// and solutions (n x nrhs column-major) at B/X + b*vs, status[b].
size_t pss_solve_ws_bytes(int n, int nb = 1);
int pss_solve_prepare(SolveWS &ws, int nb, const cd *LU64, const float *Lr, const float *Li, long long ld,
                      long long ms, const int *ipiv, cudaStream_t st);
int pss_solve_lu(SolveWS &ws, int nb, const cd *LU64, const float *Lr, const float *Li, long long ld, long long ms,
                 int nrhs, const cd *B, cd *X, long long vs, int use_done, cudaStream_t st);
int pss_refine(SolveWS &ws, int nb, const cd *A, long long ld, long long ms, const float *Lr, const float *Li,
               long long ldf, long long msf, int nrhs, const cd *B, cd *X, cd *R, cd *D, long long vs, int maxit, int *status, cudaStream_t st);
void pss_solve_status(SolveWS &ws, int nb, int *status, cudaStream_t st);
// Adjoint (transposed) solves on the same factors: Y = Z^-T B (W: scratch like B), and their
// FP64 refinement against A (FP32 factors) with a scratch of pss_refine_trans_ws_bytes.
int pss_solve_lu_trans(SolveWS &ws, int nb, const cd *LU64, const float *Lr, const float *Li, long long ld,
                       long long ms, int nrhs, const cd *B, cd *Y, cd *W, long long vs, int use_done,
                       cudaStream_t st);
size_t pss_refine_trans_ws_bytes(int n, int nrhs, int nb);
int pss_refine_trans(SolveWS &ws, int nb, const cd *A, long long ld, long long ms, const float *Lr, const float *Li,
                     long long ldf, long long msf, int nrhs, const cd *B, cd *Y, cd *R, cd *D, cd *W, void *scratch, size_t scratch_bytes,
                     long long vs, int maxit, int *status, cudaStream_t st);
