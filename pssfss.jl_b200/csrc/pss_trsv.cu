// K5: triangular solves with the LU factors, FP64 residuals and iterative refinement.
//
// Replaces LAPACK zgetrs (ldiv!, PSSFSS.jl:439,566) for the small right-hand-side sets
// of a sweep point (n_rhs = number of incident modes, 4 at normal incidence).
//
// Chained block substitution: the factor is cut into 64-row blocks; CTA tickets are
// taken in start order (atomicAdd), CTA b solves block b and only waits (bounded spin on
// a per-block epoch flag) for blocks that started before it, so it never waits on a CTA
// that is not resident.  Every CTA streams its share of the triangle (the bulk of the
// bytes) concurrently; the serial chain per block is the product with its predecessor's tile
// and the one with the precomputed inverse of the diagonal block.  FP32 arithmetic for FP32
// factors, FP64 for FP64 factors.
//
// Refinement (LAPACK zcgesv's scheme): r = b - A x with the FP64 matrix, stop when
// max|r_j| <= max|x_j| * ||A||_inf * eps * sqrt(n) for every rhs j (cabs1 norms).
#include <cuda/atomic>
#include "pss_internal.cuh"

namespace {

constexpr int BS = 64;        // block rows
constexpr int NJ = 4;         // right-hand sides of one chain
constexpr int kChains = 16;   // chains (groups of NJ right-hand sides) of a matrix in one launch
constexpr int kMaxRefRhs = 1024;          // right-hand sides of one refinement
constexpr int kNX = kMaxRefRhs;           // norms layout: [max|r_j|] [max|x_j|] [||A||]
constexpr int kNA = 2 * kMaxRefRhs;
constexpr int kNormCount = 2 * kMaxRefRhs + 1;
constexpr long long kSpinCap = 1LL << 24;

struct Fac {  // row-major factor access: FP64 interleaved or FP32 planes
  const cd *a64;
  const float *ar, *ai;
  long long ld;
  long long ms;  // elements between the factors of a batch
  __device__ __forceinline__ cd at(long long r, long long c) const {
    if (a64) return a64[r * ld + c];
    return mkcd((double)ar[r * ld + c], (double)ai[r * ld + c]);
  }
  __device__ __forceinline__ Fac of(int b) const {  // factor b of the batch
    return Fac{a64 ? a64 + b * ms : nullptr, ar ? ar + b * ms : nullptr, ai ? ai + b * ms : nullptr, ld, ms};
  }
};

// Per-matrix control words of a batch: [1] error, [2] converged; from word 8 on, for each of up
// to kChains chains, its ticket and its blocks' flags.
struct Ctrl {
  int *base;
  int stride;
  __device__ __forceinline__ int *of(int b) const { return base + (long long)b * stride; }
};

__device__ __forceinline__ double cabs1(cd z) { return fabs(z.x) + fabs(z.y); }

// L2-only (L1-bypassing) access to blocks of X that other CTAs produce or consume.
__device__ __forceinline__ cd ldcg(const cd *p) {
  const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
  return mkcd(v.x, v.y);
}
__device__ __forceinline__ void stcg(cd *p, cd v) { __stcg(reinterpret_cast<double2 *>(p), make_double2(v.x, v.y)); }

// Spin until flags[c] >= epoch (acquire).  Returns false (and records an error) at the cap.
__device__ __forceinline__ bool wait_flag(int *flags, int c, int epoch, int *err) {
  cuda::atomic_ref<int, cuda::thread_scope_device> f(flags[c]);
  long long it = 0;
  while (f.load(cuda::memory_order_acquire) < epoch) {
    if (++it > kSpinCap) {
      atomicExch(err, 1);
      return false;
    }
    if (it > 512) __nanosleep(64);  // hot spin first: the chain's step time is a few microseconds
  }
  return true;
}

__device__ __forceinline__ void post_flag(int *flags, int b, int epoch) {
  cuda::atomic_ref<int, cuda::thread_scope_device> f(flags[b]);
  f.store(epoch, cuda::memory_order_release);
}

// Inverses of the 64x64 diagonal blocks: Dinv[(2*blk + 0)] = L_bb^{-1} (unit lower),
// Dinv[(2*blk + 1)] = U_bb^{-1}; each 64x64 row-major FP64.  Four lanes per column of the inverse,
// each with 16 interleaved rows in registers; a finished entry goes to the other three by a
// shuffle and the rows still open take it off at once (the one-thread-per-column form, a chain of
// 64 dot products with both matrices in shared memory, took 1130 us for 12 factors of N = 3976).
__global__ void __launch_bounds__(256) k_diag_inv(Fac F0, int n, cd *Dinv0, long long dstride) {
  const int blk = blockIdx.x, upper = blockIdx.y;
  const Fac F = F0.of(blockIdx.z);
  const int r0 = blk * BS, nb = min(BS, n - r0);
  constexpr int LD = BS + 1;
  extern __shared__ __align__(16) unsigned char dinv_smem[];
  cd *T = (cd *)dinv_smem;  // 64 rows of LD
  __shared__ cd rdiag[BS];
  const int tid = threadIdx.x;
  for (int e = tid; e < BS * BS; e += 256) {
    const int i = e / BS, k = e % BS;
    T[i * LD + k] = (i < nb && k < nb) ? F.at(r0 + i, r0 + k) : mkcd(i == k, 0);
  }
  __syncthreads();
  if (upper && tid < BS) rdiag[tid] = mkcd(1.0, 0.0) / T[tid * LD + tid];
  __syncthreads();
  const int k = tid >> 2, p = tid & 3;  // column k, rows p + 4 i
  cd x[BS / 4];
#pragma unroll
  for (int i = 0; i < BS / 4; ++i) x[i] = mkcd(p + 4 * i == k, 0);
  if (!upper) {
#pragma unroll
    for (int j = 0; j < BS - 1; ++j) {
      cd v;
      v.x = __shfl_sync(0xffffffffu, x[j / 4].x, j % 4, 4);
      v.y = __shfl_sync(0xffffffffu, x[j / 4].y, j % 4, 4);
#pragma unroll
      for (int i = j / 4; i < BS / 4; ++i)
        if (p + 4 * i > j) x[i] = cmsub(x[i], T[(p + 4 * i) * LD + j], v);
    }
  } else {
#pragma unroll
    for (int j = BS - 1; j >= 0; --j) {
      if (p == j % 4) x[j / 4] = x[j / 4] * rdiag[j];
      cd v;
      v.x = __shfl_sync(0xffffffffu, x[j / 4].x, j % 4, 4);
      v.y = __shfl_sync(0xffffffffu, x[j / 4].y, j % 4, 4);
#pragma unroll
      for (int i = 0; i <= j / 4; ++i)
        if (p + 4 * i < j) x[i] = cmsub(x[i], T[(p + 4 * i) * LD + j], v);
    }
  }
  cd *D = Dinv0 + blockIdx.z * dstride + (size_t)(2 * blk + upper) * BS * BS;
#pragma unroll
  for (int i = 0; i < BS / 4; ++i) D[(p + 4 * i) * BS + k] = x[i];
}
constexpr int kDinvSmem = BS * (BS + 1) * (int)sizeof(cd);

// perm[i] = original row that ends in position i after the LAPACK swap sequence ipiv.
__global__ void __launch_bounds__(1024) k_ipiv_to_perm(int n, const int *ipiv0, int *perm0) {
  extern __shared__ int sp[];
  const int *ipiv = ipiv0 + (long long)blockIdx.x * n;
  int *perm = perm0 + (long long)blockIdx.x * n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) sp[i] = i;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 0; k < n; ++k) {
      int p = ipiv[k];
      int t = sp[k]; sp[k] = sp[p]; sp[p] = t;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) perm[i] = sp[i];
}

// Arithmetic of a chained pass: FP64 for FP64 factors; FP32 for FP32 factors, as LAPACK
// zcgesv solves its corrections in single precision (cgetrs) before the FP64 update.
template <bool F32>
struct SolveT;
template <>
struct SolveT<false> {
  using C = cd;
  __device__ static C fac(const Fac &F, long long r, long long c) { return F.a64[r * F.ld + c]; }
  __device__ static C from(cd v) { return v; }
  __device__ static cd to(C v) { return v; }
};
template <>
struct SolveT<true> {
  using C = cf;
  __device__ static C fac(const Fac &F, long long r, long long c) { return cf{F.ar[r * F.ld + c], F.ai[r * F.ld + c]}; }
  __device__ static C from(cd v) { return cf{(float)v.x, (float)v.y}; }
  __device__ static cd to(C v) { return mkcd(v.x, v.y); }
};
__device__ __forceinline__ cf operator-(cf a, cf b) { return cf{a.x - b.x, a.y - b.y}; }
template <class C>
__device__ __forceinline__ C czero() { return C{0, 0}; }

// One chained substitution pass, a chain of NJ right-hand sides per (matrix, chain) of the grid:
//   lower: X[rows_b] = Linv_b (B[perm[rows_b]] - sum_{c<b} L[b,c] X[c])
//   upper: X[rows_b] = Uinv_b (X[rows_b] - sum_{c>b} U[b,c] X[c])   (in place)
// TRANS (the adjoint system Z^T y = b, Z = P^T L U, so U^T L^T (P y) = b): the lower pass
// runs with U^T (block (b, c) read as the transpose of block (c, b) of the factor, the
// diagonal inverse transposed) on B unpermuted, the upper pass with L^T in place; the
// caller applies P^T to the result (pss_solve_lu_trans).
//
// One CTA per 64-row block b (ticket order).  The blocks of a chain finish one after another, so
// what a step takes between its predecessor's flag and its own is the pass's time (63 steps at
// N = 3976); everything else happens before that flag:
//   * the tiles of all blocks but the predecessor's: a warp reads whole 128-byte row segments,
//     looks up 32 flags at a time, and its partial sums are reduced across the CTA before the
//     last wait;
//   * the predecessor's tile waits in registers, the diagonal inverse in shared memory.
// After the flag: x of the predecessor to shared memory, one 64 x 64 product from registers, one
// with the inverse, the result and the flag.  The release of the flag after the block barrier
// orders the block's stores; no further fence is needed.  660 -> 390 us per triangle of 12 factors
// (N = 3976, four right-hand sides, FP32, cold caches).  Chains of more right-hand sides run side
// by side.  A row's products, the predecessor's among them, are summed on their own and
// subtracted from its right-hand side once.
template <bool F32>
struct TrsvT {
  static constexpr int T = F32 ? 256 : 512;    // threads
  static constexpr int RW = 64 / (T / 32);     // tile rows of a warp
  static constexpr int Q = T / 64;             // lanes of a row in the predecessor's product
  static constexpr int LD = BS + 1;
  using C = typename SolveT<F32>::C;
  static constexpr int SMEM = BS * LD * (int)sizeof(C);                            // diagonal inverse
  static constexpr int SMEM_T = SMEM + T / 32 * BS * NJ * (int)sizeof(C);          // + the warps' sums (TRANS)
};
template <bool LOWER, bool F32, bool TRANS>
__global__ void __launch_bounds__(TrsvT<F32>::T, F32 ? 2 : 1)
    k_trsv(Fac F0, int n, const int *__restrict__ perm0, const cd *__restrict__ B0, cd *__restrict__ X0, long long vs,
           int nrhs, int j00, int nchain, const cd *__restrict__ Dinv0, long long dstride, Ctrl ctrl, int epoch,
           int use_done) {
  using S = SolveT<F32>;
  using P = TrsvT<F32>;
  using C = typename S::C;
  // the grid runs (matrix, chain) fastest, so the CTAs start block row by block row across all of
  // them and every chain advances in the same waves
  const int bm = blockIdx.x / nchain, ch = blockIdx.x % nchain;
  int *cw = ctrl.of(bm);
  if (use_done && cw[2]) return;
  const Fac F = F0.of(bm);
  const int *perm = perm0 + (long long)bm * n;
  const int j0 = j00 + ch * NJ, nj = min(NJ, nrhs - j0);
  const cd *B = B0 + bm * vs + (size_t)j0 * n;
  cd *X = X0 + bm * vs + (size_t)j0 * n;
  const int nblk = (n + BS - 1) / BS;
  int *ticket = cw + 8 + ch * (nblk + 1), *flags = ticket + 1, *err = cw + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  C *Ds = (C *)smraw;
  C *part = Ds + BS * P::LD;  // TRANS: [warp][64][NJ]
  __shared__ C y[BS][NJ];
  __shared__ C ya[BS][NJ];  // products of all tiles but the predecessor's
  __shared__ C xs[BS][NJ];
  __shared__ C xw[P::T / 32][P::RW][NJ];
  __shared__ int s_b;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    const int t = atomicAdd(ticket, 1);
    if (t == nblk - 1) *ticket = 0;  // every block has its ticket: ready for the next launch
    s_b = t;
  }
  __syncthreads();
  const int b = LOWER ? s_b : nblk - 1 - s_b;
  const int r0 = b * BS, nr = min(BS, n - r0);
  // diagonal block: L_bb^-1 (lower pass) or U_bb^-1 (upper pass); transposed, U_bb^-T for the
  // lower pass of the adjoint system and L_bb^-T for its upper pass
  const cd *D = Dinv0 + bm * dstride + (size_t)(2 * b + ((LOWER != TRANS) ? 0 : 1)) * BS * BS;
  for (int e = tid; e < BS * BS; e += P::T) {
    const int r = e / BS, c = e % BS;
    if constexpr (TRANS) Ds[c * P::LD + r] = S::from(D[e]);
    else Ds[r * P::LD + c] = S::from(D[e]);
  }
  if (tid < BS * NJ) {
    const int r = tid / NJ, j = tid % NJ;
    cd v = mkcd(0, 0);
    if (r < nr && j < nj)
      v = LOWER ? B[(size_t)j * n + (TRANS ? r0 + r : perm[r0 + r])] : ldcg(&X[(size_t)j * n + r0 + r]);
    y[r][j] = S::from(v);
    ya[r][j] = czero<C>();
  }
  // tiles in the order their blocks finish; the last one, the predecessor's, apart
  const int nt = LOWER ? b : nblk - 1 - b;
  auto block_of = [&](int t) { return LOWER ? t : nblk - 1 - t; };
  // the predecessor's tile in registers: Q lanes per row, 64 / Q columns each
  constexpr int CQ = 64 / P::Q;
  const int pi = tid / P::Q, pq = tid % P::Q;
  // ---- tiles 0 .. nt-2 ----
  C acc[TRANS ? 2 : P::RW][NJ];
#pragma unroll
  for (int r = 0; r < (TRANS ? 2 : P::RW); ++r)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[r][j] = czero<C>();
  int ready = 0;  // tiles known to be finished
#pragma unroll 1
  for (int t = 0; t < nt - 1; ++t) {
    const int t0 = block_of(t) * BS, ntc = min(BS, n - t0);
    C lv[P::RW][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int col = lane + 32 * h;
#pragma unroll
      for (int rr = 0; rr < P::RW; ++rr) {
        const int row = warp * P::RW + rr;
        if constexpr (TRANS) lv[rr][h] = (col < nr && row < ntc) ? S::fac(F, t0 + row, r0 + col) : czero<C>();
        else lv[rr][h] = (row < nr && col < ntc) ? S::fac(F, r0 + row, t0 + col) : czero<C>();
      }
    }
    if (t >= ready) {  // look up the flags of the next 32 tiles; wait for this one's
      const int u = t + lane;
      bool up = false;
      if (u < nt - 1) {
        cuda::atomic_ref<int, cuda::thread_scope_device> f(flags[block_of(u)]);
        up = f.load(cuda::memory_order_acquire) >= epoch;
      }
      const unsigned m = __ballot_sync(0xffffffffu, up);
      ready = t + (m == 0xffffffffu ? 32 : __ffs(~m) - 1);
      if (ready == t) {
        if (lane == 0) wait_flag(flags, block_of(t), epoch, err);
        ready = t + 1;
      }
      __syncwarp();
    }
    if constexpr (TRANS) {
      if (lane < P::RW * NJ) {
        const int rr = lane / NJ, j = lane % NJ, row = warp * P::RW + rr;
        xw[warp][rr][j] = (row < ntc && j < nj) ? S::from(ldcg(&X[(size_t)j * n + t0 + row])) : czero<C>();
      }
      __syncwarp();
#pragma unroll
      for (int rr = 0; rr < P::RW; ++rr)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const C xv = xw[warp][rr][j];
#pragma unroll
          for (int h = 0; h < 2; ++h) acc[h][j] = cmac(acc[h][j], lv[rr][h], xv);
        }
      __syncwarp();
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int col = lane + 32 * h;
        C xv[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          xv[j] = (col < ntc && j < nj) ? S::from(ldcg(&X[(size_t)j * n + t0 + col])) : czero<C>();
#pragma unroll
        for (int rr = 0; rr < P::RW; ++rr)
#pragma unroll
          for (int j = 0; j < NJ; ++j) acc[rr][j] = cmac(acc[rr][j], lv[rr][h], xv[j]);
      }
    }
  }
  if (nt > 1) {
    if constexpr (TRANS) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < NJ; ++j) part[(warp * BS + lane + 32 * h) * NJ + j] = acc[h][j];
      __syncthreads();
      if (tid < BS * NJ) {
        C v = czero<C>();
        for (int w = 0; w < P::T / 32; ++w) {
          const C q = part[w * BS * NJ + tid];
          v = C{v.x + q.x, v.y + q.y};
        }
        ya[tid / NJ][tid % NJ] = v;
      }
    } else {
      __syncthreads();  // ya cleared
#pragma unroll
      for (int rr = 0; rr < P::RW; ++rr)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          for (int o = 16; o > 0; o >>= 1) {
            acc[rr][j].x += __shfl_xor_sync(0xffffffff, acc[rr][j].x, o);
            acc[rr][j].y += __shfl_xor_sync(0xffffffff, acc[rr][j].y, o);
          }
          if (lane == 0) ya[warp * P::RW + rr][j] = acc[rr][j];
        }
    }
  }
  // ---- the predecessor's tile ----
  if (nt > 0) {
    const int c = block_of(nt - 1), t0 = c * BS, ntc = min(BS, n - t0);
    C lv[CQ];
#pragma unroll
    for (int q = 0; q < CQ; ++q) {
      const int col = pq + P::Q * q;
      lv[q] = (pi < nr && col < ntc) ? (TRANS ? S::fac(F, t0 + col, r0 + pi) : S::fac(F, r0 + pi, t0 + col)) : czero<C>();
    }
    if (lane == 0) wait_flag(flags, c, epoch, err);
    __syncwarp();
    if (tid < BS * NJ) {
      const int r = tid % BS, j = tid / BS;
      xs[r][j] = (r < ntc && j < nj) ? S::from(ldcg(&X[(size_t)j * n + t0 + r])) : czero<C>();
    }
    __syncthreads();
    C s[NJ];
#pragma unroll
    for (int j = 0; j < NJ; ++j) s[j] = czero<C>();
#pragma unroll
    for (int q = 0; q < CQ; ++q)
#pragma unroll
      for (int j = 0; j < NJ; ++j) s[j] = cmac(s[j], lv[q], xs[pq + P::Q * q][j]);
#pragma unroll
    for (int o = 1; o < P::Q; o <<= 1)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        s[j].x += __shfl_xor_sync(0xffffffff, s[j].x, o);
        s[j].y += __shfl_xor_sync(0xffffffff, s[j].y, o);
      }
    if (pq == 0)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {  // all products first, then one rounding at y's size
        const C q = ya[pi][j];
        y[pi][j] = y[pi][j] - C{q.x + s[j].x, q.y + s[j].y};
      }
  }
  __syncthreads();
  // X[rows] = Dinv_b * y: one entry per T / 256 lanes
  {
    constexpr int H = P::T / (BS * NJ);
    const int h = tid % H, e = tid / H, r = e / NJ, j = e % NJ;
    C s0 = czero<C>(), s1 = czero<C>();
#pragma unroll 8
    for (int k = h; k < BS; k += 2 * H) {
      s0 = cmac(s0, Ds[r * P::LD + k], y[k][j]);
      s1 = cmac(s1, Ds[r * P::LD + k + H], y[k + H][j]);
    }
    s0 = C{s0.x + s1.x, s0.y + s1.y};
    if constexpr (H == 2) {
      s0.x += __shfl_xor_sync(0xffffffff, s0.x, 1);
      s0.y += __shfl_xor_sync(0xffffffff, s0.y, 1);
    }
    if (h == 0 && r < nr && j < nj) stcg(&X[(size_t)j * n + r0 + r], S::to(s0));
  }
  __syncthreads();
  if (tid == 0) post_flag(flags, b, epoch);
}

// R = B - A X with max|r_j| (norms[j]), max|x_j| (norms[kNX + j]) and ||A||_inf (norms[kNA]), for
// M right-hand sides from j0 = M * blockIdx.x on (4, the sweep's usual case; 8 at a time for
// more, the groups of one row block side by side so that they share its rows in L2): a CTA of 8
// warps takes 16 rows, each warp 2 of them; the columns go in chunks whose X block (M x 4096 / M
// entries) is staged in shared memory and reused by the rows of every warp, so the matrix rows
// are the only HBM stream (streaming loads).  The column loop has no early exit (the ragged last
// chunk is predicated); rows past n are clamped to row n-1 for their loads and dropped at the end.
// A lane takes kResG columns at a time and sums their products on their own before it adds them to
// the running sum: 5 operations a component for two products and one rounding at the running
// sum's size, where adding each takes 6 and two, and nested multiply-adds take 4 and four.  The
// residual's own rounding is what limits a refined solution: order 1501, error against 64 bits
// 4.0e-16 with nested multiply-adds.  593 us for 12 matrices of N = 3976 (nested 594, each 770).
constexpr int kResRows = 2, kResG = 2;
constexpr int kResSmem = 4096 * (int)sizeof(cd);  // 64 KB
__device__ __forceinline__ cd ldcs(const cd *p) {
  const double2 v = __ldcs(reinterpret_cast<const double2 *>(p));
  return cd{v.x, v.y};
}
template <int M>
__global__ void __launch_bounds__(256, M == 4 ? 3 : 2) k_resid(int n, const cd *__restrict__ A0, long long ld, long long ms, int nrhs0,
                                               const cd *__restrict__ X0, const cd *__restrict__ B0,
                                               cd *__restrict__ R0, long long vs, double *norms0, Ctrl ctrl) {
  constexpr int CH = 4096 / M;
  const int bm = blockIdx.z;
  if (ctrl.of(bm)[2]) return;
  const int j0 = blockIdx.x * M, nrhs = min(M, nrhs0 - j0);
  const cd *A = A0 + bm * ms, *X = X0 + bm * vs + (size_t)j0 * n, *B = B0 + bm * vs + (size_t)j0 * n;
  cd *R = R0 + bm * vs + (size_t)j0 * n;
  double *norms = norms0 + (long long)bm * kNormCount;
  extern __shared__ __align__(16) unsigned char res_smem[];
  double2(*xs)[CH] = reinterpret_cast<double2(*)[CH]>(res_smem);  // [M][CH]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = blockIdx.y * (8 * kResRows) + warp * kResRows;
  const cd *arow[kResRows];
  cd acc[kResRows][M];
  double rs[kResRows];
#pragma unroll
  for (int i = 0; i < kResRows; ++i) {
    arow[i] = A + (long long)min(r0 + i, n - 1) * ld;
    rs[i] = 0.0;
#pragma unroll
    for (int j = 0; j < M; ++j) acc[i][j] = mkcd(0, 0);
  }
  for (int t0 = 0; t0 < n; t0 += CH) {
    const int len = min(CH, n - t0);
    __syncthreads();
#pragma unroll 4
    for (int e = threadIdx.x; e < M * CH; e += 256) {
      const int j = e / CH, t = e % CH;
      xs[j][t] = (j < nrhs && t < len) ? *reinterpret_cast<const double2 *>(&X[(size_t)j * n + t0 + t]) : make_double2(0, 0);
    }
    __syncthreads();
    const int qn = (len + 31) >> 5;
#pragma unroll 2
    for (int q0 = 0; q0 < qn; q0 += kResG) {  // the staged block's rows past len are zero
      cd av[kResG][kResRows];
#pragma unroll
      for (int g = 0; g < kResG; ++g) {
        const int t = (q0 + g) * 32 + lane;
        const bool ok = t < len;
#pragma unroll
        for (int i = 0; i < kResRows; ++i) {
          av[g][i] = ok ? ldcs(arow[i] + t0 + t) : mkcd(0, 0);
          rs[i] += cabs1(av[g][i]);
        }
      }
#pragma unroll
      for (int j = 0; j < M; ++j) {
        cd p[kResRows];
#pragma unroll
        for (int g = 0; g < kResG; ++g) {
          const double2 v = xs[j][(q0 + g) * 32 + lane];
#pragma unroll
          for (int i = 0; i < kResRows; ++i)
            p[i] = g == 0 ? av[g][i] * mkcd(v.x, v.y) : cmac_nested(p[i], av[g][i], mkcd(v.x, v.y));
        }
#pragma unroll
        for (int i = 0; i < kResRows; ++i) acc[i][j] = acc[i][j] + p[i];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kResRows; ++i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      rs[i] += __shfl_xor_sync(0xffffffff, rs[i], o);
#pragma unroll
      for (int j = 0; j < M; ++j) {
        acc[i][j].x += __shfl_xor_sync(0xffffffff, acc[i][j].x, o);
        acc[i][j].y += __shfl_xor_sync(0xffffffff, acc[i][j].y, o);
      }
    }
    const int row = r0 + i;
    if (row >= n) continue;
    if (lane == 0 && j0 == 0)
      atomicMax((unsigned long long *)&norms[kNA], (unsigned long long)__double_as_longlong(rs[i]));
#pragma unroll
    for (int j = 0; j < M; ++j) {
      if (j < nrhs && lane == j) {
        const cd r = B[(size_t)j * n + row] - acc[i][j];
        R[(size_t)j * n + row] = r;
        atomicMax((unsigned long long *)&norms[j0 + j], (unsigned long long)__double_as_longlong(cabs1(r)));
        const double xv = cabs1(X[(size_t)j * n + row]);
        atomicMax((unsigned long long *)&norms[kNX + j0 + j], (unsigned long long)__double_as_longlong(xv));
      }
    }
  }
}

__global__ void k_ir_check(int n, int nrhs, double *norms0, Ctrl ctrl, int *status0, int last) {
  int *cw = ctrl.of(blockIdx.x);
  int *done = cw + 2, *err = cw + 1, *status = status0 + blockIdx.x;
  double *norms = norms0 + (long long)blockIdx.x * kNormCount;
  if (*done) return;
  const double cte = 1.1102230246251565e-16 * sqrt((double)n) * norms[kNA];
  int ok = 1, bad = 0;
  for (int j = 0; j < nrhs; ++j) {
    double rn = norms[j], xn = norms[kNX + j];
    if (!(isfinite(rn) && isfinite(xn))) bad = 1;
    else if (rn > xn * cte) ok = 0;
  }
  if (*err) { bad = 1; *status |= PSS_ST_DEVICE_TIMEOUT; }
  if (bad) { *status |= PSS_ST_NONFINITE; *done = 1; }
  else if (ok) *done = 1;
  else if (last) { *status |= PSS_ST_REFINE_NOCONV; *done = 1; }
  for (int j = 0; j < nrhs; ++j) norms[j] = norms[kNX + j] = 0.0;
  norms[kNA] = 0.0;
}

__global__ void k_err_status(Ctrl ctrl, int *status0) {
  int *err = ctrl.of(blockIdx.x) + 1;
  if (*err) status0[blockIdx.x] |= PSS_ST_DEVICE_TIMEOUT;
  *err = 0;
}

__global__ void k_axpy(long long total, cd *X0, const cd *D0, long long vs, Ctrl ctrl) {
  const int bm = blockIdx.y;
  if (ctrl.of(bm)[2]) return;
  cd *X = X0 + bm * vs;
  const cd *D = D0 + bm * vs;
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < total) X[i] = X[i] + D[i];
}

// y[perm[r]] = w[r] for every right-hand side: applies P^T after the adjoint passes.
__global__ void k_unpermute(int n, int nrhs, const int *__restrict__ perm0, const cd *__restrict__ W0,
                            cd *__restrict__ Y0, long long vs, Ctrl ctrl, int use_done) {
  const int bm = blockIdx.y;
  if (use_done && ctrl.of(bm)[2]) return;
  const int *perm = perm0 + (long long)bm * n;
  const cd *W = W0 + bm * vs;
  cd *Y = Y0 + bm * vs;
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)n * nrhs) return;
  const int r = (int)(e % n), j = (int)(e / n);
  Y[(size_t)j * n + perm[r]] = W[e];
}

// Adjoint residual R = B - A^T Y, first stage: CTA (column block cb of 128, row chunk q of
// kTrRows) sums its rows for each column j and right-hand side, and the column's |a| sums
// (the infinity norm of A^T is the largest column sum of A), into part[q] (fixed order, no
// atomics; the second stage adds the chunks in order).  A thread owns a column, so every row
// of the chunk is read coalesced across the CTA.
constexpr int kTrRows = 256, kTrCols = 128;
__global__ void __launch_bounds__(kTrCols) k_resid_t1(int n, const cd *__restrict__ A0, long long ld, long long ms,
                                                      int nrhs, const cd *__restrict__ Y0, long long vs,
                                                      cd *__restrict__ part0, double *__restrict__ cabs0,
                                                      long long pstride, Ctrl ctrl) {
  const int bm = blockIdx.z;
  if (ctrl.of(bm)[2]) return;
  const cd *A = A0 + bm * ms, *Y = Y0 + bm * vs;
  const int j = blockIdx.x * kTrCols + threadIdx.x, q = blockIdx.y;
  const int i0 = q * kTrRows, i1 = min(n, i0 + kTrRows);
  const int nch = (int)gridDim.y;
  cd *part = part0 + (long long)bm * pstride;
  double *cabs = cabs0 + (long long)bm * nch * n;
  __shared__ double2 ys[kTrRows][NJ];
  for (int j0 = 0; j0 < nrhs; j0 += NJ) {
    const int nj = min(NJ, nrhs - j0);
    __syncthreads();
    for (int e = threadIdx.x; e < kTrRows * NJ; e += kTrCols) {
      const int t = e / kTrRows, i = e % kTrRows;
      const cd v = (t < nj && i0 + i < i1) ? Y[(size_t)(j0 + t) * n + i0 + i] : mkcd(0, 0);
      ys[i][t] = make_double2(v.x, v.y);
    }
    __syncthreads();
    if (j >= n) continue;
    cd acc[NJ];
#pragma unroll
    for (int t = 0; t < NJ; ++t) acc[t] = mkcd(0, 0);
    double cs = 0.0;
#pragma unroll 8
    for (int i = i0; i < i1; ++i) {
      const cd a = ldcs(A + (long long)i * ld + j);
      cs += cabs1(a);
#pragma unroll
      for (int t = 0; t < NJ; ++t) {
        const double2 v = ys[i - i0][t];
        acc[t] = cmac(acc[t], a, mkcd(v.x, v.y));
      }
    }
    if (j0 == 0) cabs[(long long)q * n + j] = cs;
#pragma unroll
    for (int t = 0; t < NJ; ++t)
      if (t < nj) part[((long long)q * nrhs + j0 + t) * n + j] = acc[t];
  }
}

// Second stage: R = B - sum of the chunks (in chunk order), with the refinement norms of
// k_resid: max|r_j| (norms[j]), max|y_j| (norms[kNX + j]) and ||A^T||_inf (norms[kNA]).
__global__ void k_resid_t2(int n, int nch, int nrhs, const cd *__restrict__ part0, const double *__restrict__ cabs0,
                           long long pstride, const cd *__restrict__ Y0, const cd *__restrict__ B0, cd *__restrict__ R0,
                           long long vs, double *norms0, Ctrl ctrl) {
  const int bm = blockIdx.y;
  if (ctrl.of(bm)[2]) return;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const cd *part = part0 + (long long)bm * pstride;
  const double *cabs = cabs0 + (long long)bm * nch * n;
  const cd *Y = Y0 + bm * vs, *B = B0 + bm * vs;
  cd *R = R0 + bm * vs;
  double *norms = norms0 + (long long)bm * kNormCount;
  double cs = 0.0;
  for (int q = 0; q < nch; ++q) cs += cabs[(long long)q * n + j];
  atomicMax((unsigned long long *)&norms[kNA], (unsigned long long)__double_as_longlong(cs));
  for (int t = 0; t < nrhs; ++t) {
    cd s = mkcd(0, 0);
    for (int q = 0; q < nch; ++q) s = s + part[((long long)q * nrhs + t) * n + j];
    const cd r = B[(size_t)t * n + j] - s;
    R[(size_t)t * n + j] = r;
    atomicMax((unsigned long long *)&norms[t], (unsigned long long)__double_as_longlong(cabs1(r)));
    atomicMax((unsigned long long *)&norms[kNX + t],
              (unsigned long long)__double_as_longlong(cabs1(Y[(size_t)t * n + j])));
  }
}

template <bool LOWER, bool F32, bool TRANS>
cudaError_t set_trsv_smem() {
  return cudaFuncSetAttribute(k_trsv<LOWER, F32, TRANS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              TRANS ? TrsvT<F32>::SMEM_T : TrsvT<F32>::SMEM);
}

// Both passes of a solve for every group of kChains chains.
template <bool F32, bool TRANS>
int trsv_passes(SolveWS &ws, int nb, const Fac &F, int nrhs, const cd *B, cd *X, long long vs, int use_done,
                cudaStream_t st) {
  static DeviceOnce once;
  if (int rc = device_once(once, [] {
        PSS_CUDA_TRY((set_trsv_smem<true, F32, TRANS>()));
        PSS_CUDA_TRY((set_trsv_smem<false, F32, TRANS>()));
        return 0;
      }))
    return rc;
  const Ctrl ctrl{ws.ctrl, ws.cstride};
  const int smem = TRANS ? TrsvT<F32>::SMEM_T : TrsvT<F32>::SMEM;
  for (int pass = 0; pass < 2; ++pass)
    for (int j0 = 0; j0 < nrhs; j0 += NJ * kChains) {
      const int nchain = min(kChains, (nrhs - j0 + NJ - 1) / NJ);
      ++ws.epoch;
      pss_count_launch();
      auto kern = pass == 0 ? k_trsv<true, F32, TRANS> : k_trsv<false, F32, TRANS>;
      kern<<<dim3(nb * nchain, ws.nblk), TrsvT<F32>::T, smem, st>>>(F, ws.n, ws.perm, B, X, vs, nrhs, j0, nchain,
                                                                    ws.Dinv, ws.dstride, ctrl, ws.epoch, use_done);
    }
  PSS_CUDA_TRY(cudaGetLastError());
  return 0;
}

}  // namespace

// ------------------------------- host side -------------------------------

size_t pss_solve_ws_bytes(int n, int nb) {
  int nblk = (n + BS - 1) / BS;
  return (size_t)nb * ((size_t)nblk * 2 * BS * BS * sizeof(cd) + (size_t)n * sizeof(int) +
                       (size_t)(8 + kChains * (nblk + 1)) * sizeof(int) + kNormCount * sizeof(double)) + 512;
}

void SolveWS::bind(void *base, int n_, int nb_) {
  n = n_;
  nb = nb_;
  nblk = (n + BS - 1) / BS;
  dstride = (long long)nblk * 2 * BS * BS;
  cstride = 8 + kChains * (nblk + 1);
  char *p = (char *)base;
  Dinv = (cd *)p;
  p += (size_t)nb * dstride * sizeof(cd);
  perm = (int *)p;
  p += (size_t)nb * n * sizeof(int);
  ctrl = (int *)p;
  p += (size_t)nb * cstride * sizeof(int);
  p = (char *)(((uintptr_t)p + 15) & ~(uintptr_t)15);
  norms = (double *)p;
}

// After the LU of nb matrices: pivot permutations and diagonal-block inverses; control
// words and norms cleared, epoch reset.
int pss_solve_prepare(SolveWS &ws, int nb, const cd *LU64, const float *Lr, const float *Li, long long ld,
                      long long ms, const int *ipiv, cudaStream_t st) {
  if (nb > ws.nb) { pss_set_error("solve workspace holds %d matrices, %d asked", ws.nb, nb); return -4; }
  Fac F{LU64, Lr, Li, ld, ms};
  pss_count_launch();
  k_ipiv_to_perm<<<nb, 1024, ws.n * sizeof(int), st>>>(ws.n, ipiv, ws.perm);
  static DeviceOnce once;
  if (int rc = device_once(once, [] {
        PSS_CUDA_TRY(
            cudaFuncSetAttribute(k_diag_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, kDinvSmem));
        return 0;
      }))
    return rc;
  pss_count_launch();
  k_diag_inv<<<dim3(ws.nblk, 2, nb), 256, kDinvSmem, st>>>(F, ws.n, ws.Dinv, ws.dstride);
  PSS_CUDA_TRY(cudaMemsetAsync(ws.ctrl, 0, (size_t)nb * ws.cstride * sizeof(int), st));
  PSS_CUDA_TRY(cudaMemsetAsync(ws.norms, 0, (size_t)nb * kNormCount * sizeof(double), st));
  ws.epoch = 0;
  return 0;
}

// X = (LU)^{-1} P B for each of nb matrices (B and X distinct, n x nrhs column-major, vs
// elements apart).  use_done: skip matrices whose refinement has converged.
int pss_solve_lu(SolveWS &ws, int nb, const cd *LU64, const float *Lr, const float *Li, long long ld, long long ms,
                 int nrhs, const cd *B, cd *X, long long vs, int use_done, cudaStream_t st) {
  const Fac F{LU64, Lr, Li, ld, ms};
  return LU64 ? trsv_passes<false, false>(ws, nb, F, nrhs, B, X, vs, use_done, st)
              : trsv_passes<true, false>(ws, nb, F, nrhs, B, X, vs, use_done, st);
}

// A timed-out wait in a solve (never expected) marks the point (status[b]).
void pss_solve_status(SolveWS &ws, int nb, int *status, cudaStream_t st) {
  pss_count_launch();
  k_err_status<<<nb, 1, 0, st>>>(Ctrl{ws.ctrl, ws.cstride}, status);
}

// Iterative refinement of each X_b against its FP64 matrix A_b (FP32 factors), up to
// maxit steps; matrices that converge drop out (their converged word).
int pss_refine(SolveWS &ws, int nb, const cd *A, long long ld, long long ms, const float *Lr, const float *Li,
               long long ldf, long long msf, int nrhs, const cd *B, cd *X, cd *R, cd *D, long long vs, int maxit, int *status, cudaStream_t st) {
  if (nrhs > kMaxRefRhs) { pss_set_error("refinement supports at most %d right-hand sides", kMaxRefRhs); return -1; }
  const Ctrl ctrl{ws.ctrl, ws.cstride};
  static DeviceOnce once;
  if (int rc = device_once(once, [] {
        PSS_CUDA_TRY(cudaFuncSetAttribute(k_resid<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem));
        PSS_CUDA_TRY(cudaFuncSetAttribute(k_resid<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem));
        return 0;
      }))
    return rc;
  // converged words of every matrix cleared
  PSS_CUDA_TRY(cudaMemset2DAsync(ws.ctrl + 2, ws.cstride * sizeof(int), 0, sizeof(int), nb, st));
  const long long total = (long long)ws.n * nrhs;
  for (int it = 0; it <= maxit; ++it) {
    pss_count_launch();
    const unsigned rows = cdiv_u(ws.n, 8 * kResRows);
    if (nrhs <= 4)
      k_resid<4><<<dim3(1, rows, nb), 256, kResSmem, st>>>(ws.n, A, ld, ms, nrhs, X, B, R, vs, ws.norms, ctrl);
    else
      k_resid<8><<<dim3(cdiv_u(nrhs, 8), rows, nb), 256, kResSmem, st>>>(ws.n, A, ld, ms, nrhs, X, B, R, vs, ws.norms,
                                                                         ctrl);
    pss_count_launch();
    k_ir_check<<<nb, 1, 0, st>>>(ws.n, nrhs, ws.norms, ctrl, status, it == maxit);
    if (it == maxit) break;
    int rc = pss_solve_lu(ws, nb, nullptr, Lr, Li, ldf, msf, nrhs, R, D, vs, 1, st);
    if (rc) return rc;
    pss_count_launch();
    k_axpy<<<dim3(cdiv_u(total, 256), nb), 256, 0, st>>>(total, X, D, vs, ctrl);
  }
  PSS_CUDA_TRY(cudaGetLastError());
  return 0;
}

// Adjoint solves Y = Z^-T B with the factors of P Z = L U (the same factors as pss_solve_lu,
// after pss_solve_prepare): U^T V = B, L^T W = V (both chained passes into W), Y = P^T W.
// W: scratch of the size of B.  use_done: skip matrices whose refinement has converged.
int pss_solve_lu_trans(SolveWS &ws, int nb, const cd *LU64, const float *Lr, const float *Li, long long ld,
                       long long ms, int nrhs, const cd *B, cd *Y, cd *W, long long vs, int use_done,
                       cudaStream_t st) {
  const Fac F{LU64, Lr, Li, ld, ms};
  const Ctrl ctrl{ws.ctrl, ws.cstride};
  if (int rc = LU64 ? trsv_passes<false, true>(ws, nb, F, nrhs, B, W, vs, use_done, st)
                    : trsv_passes<true, true>(ws, nb, F, nrhs, B, W, vs, use_done, st))
    return rc;
  pss_count_launch();
  k_unpermute<<<dim3(cdiv_u((long long)ws.n * nrhs, 256), nb), 256, 0, st>>>(ws.n, nrhs, ws.perm, W, Y, vs, ctrl,
                                                                          use_done);
  PSS_CUDA_TRY(cudaGetLastError());
  return 0;
}

// Scratch of the adjoint residual for nb matrices and nrhs right-hand sides (row-chunk partial
// sums and column sums).
size_t pss_refine_trans_ws_bytes(int n, int nrhs, int nb) {
  const size_t nch = (size_t)(n + kTrRows - 1) / kTrRows;
  return (size_t)nb * nch * ((size_t)nrhs * n * sizeof(cd) + (size_t)n * sizeof(double)) + 256;
}

// Iterative refinement of the adjoint solutions Y_b (Z_b^T Y_b = B_b) against the FP64
// matrices, as pss_refine: r = B - Z^T Y in FP64 (two-stage, fixed order), correction from the
// FP32 factors (pss_solve_lu_trans), the same stopping rule with ||Z^T||_inf.
int pss_refine_trans(SolveWS &ws, int nb, const cd *A, long long ld, long long ms, const float *Lr, const float *Li,
                     long long ldf, long long msf, int nrhs, const cd *B, cd *Y, cd *R, cd *D, cd *W, void *scratch, size_t scratch_bytes,
                     long long vs, int maxit, int *status, cudaStream_t st) {
  if (nrhs > kMaxRefRhs) { pss_set_error("refinement supports at most %d right-hand sides", kMaxRefRhs); return -1; }
  if (scratch_bytes < pss_refine_trans_ws_bytes(ws.n, nrhs, nb)) {
    pss_set_error("adjoint refinement scratch too small");
    return -4;
  }
  const Ctrl ctrl{ws.ctrl, ws.cstride};
  const int nch = (ws.n + kTrRows - 1) / kTrRows;
  const long long pstride = (long long)nch * nrhs * ws.n;
  cd *part = (cd *)scratch;
  double *cabs = (double *)(part + (size_t)nb * pstride);
  PSS_CUDA_TRY(cudaMemset2DAsync(ws.ctrl + 2, ws.cstride * sizeof(int), 0, sizeof(int), nb, st));
  const long long total = (long long)ws.n * nrhs;
  for (int it = 0; it <= maxit; ++it) {
    pss_count_launch();
    k_resid_t1<<<dim3(cdiv_u(ws.n, kTrCols), nch, nb), kTrCols, 0, st>>>(ws.n, A, ld, ms, nrhs, Y, vs, part, cabs,
                                                                        pstride, ctrl);
    pss_count_launch();
    k_resid_t2<<<dim3(cdiv_u(ws.n, 256), nb), 256, 0, st>>>(ws.n, nch, nrhs, part, cabs, pstride, Y, B, R, vs,
                                                            ws.norms, ctrl);
    pss_count_launch();
    k_ir_check<<<nb, 1, 0, st>>>(ws.n, nrhs, ws.norms, ctrl, status, it == maxit);
    if (it == maxit) break;
    int rc = pss_solve_lu_trans(ws, nb, nullptr, Lr, Li, ldf, msf, nrhs, R, D, W, vs, 1, st);
    if (rc) return rc;
    pss_count_launch();
    k_axpy<<<dim3(cdiv_u(total, 256), nb), 256, 0, st>>>(total, Y, D, vs, ctrl);
  }
  PSS_CUDA_TRY(cudaGetLastError());
  return 0;
}
