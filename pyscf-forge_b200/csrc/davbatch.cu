// Device-resident lockstep Davidson-Liu for a batch of independent CSF-FCI
// problems (csffci_batch_plan_*).
//
// Every step of an iteration runs on the device for all problems at once,
// driven by a per-problem state record (subspace size, number of new
// vectors, convergence flags, Ritz values) that the kernels read and write,
// so an iteration is a fixed launch sequence with no host synchronisation
// and is captured once as a CUDA graph and replayed:
//
//   k_db_proj<0>   partial dots T.V and |T|^2 over 256-element chunks
//   k_db_sproj<0>  reduce -> projection coefficients
//   k_db_proj<1>   T -= coef.V, partial dots T.V        (second projection)
//   k_db_sproj<1>
//   k_db_proj<2>   T -= coef.V, partial Gram T.T
//   k_db_sproj<2>  orthonormal combinations (Jacobi on the small Gram)
//   k_db_new       W = c.T, V[m..] = W
//   CSF -> det (batched block GEMMs), sigma per orbital count (gated
//   persistent job table), det -> CSF into AW
//   k_db_hv        AV[m..] = AW, partial dots V.AW
//   k_db_sritz     subspace matrix update, Jacobi eigensolver, root
//                  selection (overlap following once a root converged)
//   k_db_ritz      X = cc.V, AX = cc.AV, R = AX - e X, partial |R|^2 and
//                  the Olsen dots x.P r, x.P x
//   k_db_sconv     convergence, correction bookkeeping, restart decision
//   k_db_pre       T = (R - e1 X) P  (Olsen correction over the diagonal),
//                  restart copies V[:k] = X, AV[:k] = AX
//
// The per-problem algorithm is that of the one-problem solver (role of
// pyscf lib.davidson1 via fci.eig at pyscf/csf_fci/csf.py:487-490, with the
// diagonal Olsen preconditioner of fci.make_precond, csf.py:433).  Every
// reduction runs in a fixed order (chunk partials summed in unit order), so
// a batch is bit-reproducible up to the atomic scatter of sigma.  No
// counterpart in the reference, which solves one problem per call.
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#include "batch_internal.cuh"
#include "common.cuh"
#include "profile.cuh"
#include "sigma_rr_kernel.cuh"

namespace csffci {

constexpr int DB_KMAX = 8;     // roots per problem
constexpr int DB_CAPMAX = 64;  // subspace capacity max_space + 2*nroots
constexpr int DB_NT = 256;     // threads of the streaming kernels
constexpr int DB_EPT = 1;      // elements per thread
constexpr int DB_CH = DB_NT * DB_EPT;
constexpr int DB_NW = DB_NT / 32;
constexpr int DB_ST = 128;  // threads of the small per-problem kernels
constexpr int DB_RT = 256;  // threads of the subspace eigenproblem

// shared memory of the subspace eigenproblem, matrices of ld columns; the
// kernel is allowed the most of any plan (see MAX_SMEM)
constexpr size_t db_ritz_smem(size_t ld) {
  return sizeof(double) * (2 * ld * ld + (2 * DB_KMAX + 1) * ld) + sizeof(int) * ld;
}
constexpr int DB_RITZ_SMEM = (int)db_ritz_smem(DB_CAPMAX | 1);

struct DBProb {
  int64_t n;
  int32_t k, cap, space, unit0, nunits, pad;
  double *V, *AV, *X, *AX, *R, *T, *W, *AW;
  const double* hdiag;
  double *h, *coef, *cc, *xprev;
  double *qprev, *dprev;  // eigenvectors (cap x cap) and eigenvalues of the last subspace matrix
};

struct DBState {
  int32_t m, m_old, kT, knew, kk, done, restart, niter, any_conv, have_e, kk_prev;
  int32_t mq;  // size of the basis qprev/dprev diagonalise (0: none)
  int32_t todo[DB_KMAX];
  int32_t conv[DB_KMAX];
  double e[DB_KMAX], e_prev[DB_KMAX], rnorm[DB_KMAX], e1[DB_KMAX], es[DB_KMAX], tnorm[DB_KMAX];
};

struct DBArgs {
  const DBProb* prob;
  DBState* st;
  const int32_t* unit_prob;
  double* partial;
  int nslot, capb, kb, nprob;
  long long nunits;
  double tol, toloose, lindep, shift;
  int* count;
};

__device__ __forceinline__ double db_pinv(double h, double es) {
  double v = 1.0 / (h - es);
  if (fabs(v) > 1e8) v = 1e8;
  return v;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// slot of dot (row i, column j) and of the per-row extras
__device__ __forceinline__ int slot_dot(const DBArgs& a, int i, int j) { return i * a.capb + j; }
__device__ __forceinline__ int slot_x(const DBArgs& a, int which, int i) {
  return a.kb * a.capb + which * a.kb + i;
}

// ---------------------------------------------------------------------------
// streaming kernels: one unit = one 256-element chunk of one problem; KM
// is the largest root count of the batch (register arrays).  The problem
// record is copied to registers first (stores through its pointers could
// alias it), and loops over the subspace keep several rows in flight: for the
// few chunks of a small problem the time is the latency of those loops.
// ---------------------------------------------------------------------------

// Dot products of the k rows of xs (shared, DB_CH each, zero past n) with m
// rows of V: each warp takes every DB_NW-th row of V, so no sum crosses
// warps; put(i, j, sum).  Against all warps on every row with a block
// reduction (and chunks of 1024): 9.8 -> 3.7 us per projection of an
// 1800-element problem.
template <int KM, typename PutF>
__device__ __forceinline__ void db_dots(const double* xs, int k, const double* __restrict__ V, int64_t n, int64_t c0,
                                        int m, int lane, int w, PutF put) {
  const int len = (int)min((int64_t)DB_CH, n - c0);
  constexpr int RB = 2, EL = DB_CH / 32;  // rows together, elements of a lane
  for (int j0 = w; j0 < m; j0 += RB * DB_NW) {
    double x[RB][EL];
#pragma unroll
    for (int r = 0; r < RB; ++r)
#pragma unroll
      for (int q = 0; q < EL; ++q) {
        const int j = j0 + r * DB_NW, e = lane + 32 * q;
        x[r][q] = (j < m && e < len) ? V[j * n + c0 + e] : 0.0;
      }
#pragma unroll
    for (int i = 0; i < KM; ++i) {
      if (i >= k) continue;
#pragma unroll
      for (int r = 0; r < RB; ++r) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < EL; ++q) s = fma(xs[i * DB_CH + lane + 32 * q], x[r][q], s);
        s = warp_sum(s);
        if (lane == 0 && j0 + r * DB_NW < m) put(i, j0 + r * DB_NW, s);
      }
    }
  }
}

template <int KM, int PASS>
__global__ void __launch_bounds__(DB_NT) k_db_proj(DBArgs a) {
  extern __shared__ double sm[];
  double* const ts = sm;                // T of the chunk
  double* const cs = sm + KM * DB_CH;   // coefficients
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (long long u = blockIdx.x; u < a.nunits; u += gridDim.x) {
    const int p = a.unit_prob[u];
    const int kT = a.st[p].kT, m = a.st[p].m;
    if (a.st[p].done || kT == 0) continue;
    const DBProb P = a.prob[p];
    const int64_t n = P.n, c0 = (int64_t)(u - P.unit0) * DB_CH;
    __syncthreads();  // ts and cs of the previous unit are consumed
    if (PASS >= 1)
      for (int i = tid; i < kT * m; i += DB_NT) cs[i] = P.coef[i / m * P.cap + i % m];
    if (PASS >= 1) __syncthreads();
#pragma unroll
    for (int q = 0; q < DB_EPT; ++q) {
      const int l = tid + q * DB_NT;
      const int64_t e = c0 + l;
      double t[KM];
#pragma unroll
      for (int i = 0; i < KM; ++i) t[i] = (i < kT && e < n) ? P.T[i * n + e] : 0.0;
      if (PASS >= 1 && e < n) {
#pragma unroll 8
        for (int j = 0; j < m; ++j) {
          const double v = P.V[j * n + e];
#pragma unroll
          for (int i = 0; i < KM; ++i)
            if (i < kT) t[i] = fma(-cs[i * m + j], v, t[i]);
        }
#pragma unroll
        for (int i = 0; i < KM; ++i)
          if (i < kT) P.T[i * n + e] = t[i];
      }
#pragma unroll
      for (int i = 0; i < KM; ++i) ts[i * DB_CH + l] = t[i];
    }
    __syncthreads();
    double* const out = a.partial + u * a.nslot;
    if (PASS <= 1) {
      db_dots<KM>(ts, kT, P.V, n, c0, m, lane, w, [&](int i, int j, double v) { out[slot_dot(a, i, j)] = v; });
      if (PASS == 0)
        for (int i = w; i < kT; i += DB_NW) {
          double v = 0.0;
          for (int e = lane; e < DB_CH; e += 32) v = fma(ts[i * DB_CH + e], ts[i * DB_CH + e], v);
          v = warp_sum(v);
          if (lane == 0) out[slot_x(a, 0, i)] = v;
        }
    } else {
      for (int i = w; i < kT * kT; i += DB_NW) {
        const int r = i / kT, c = i % kT;
        if (c > r) continue;
        double v = 0.0;
        for (int e = lane; e < DB_CH; e += 32) v = fma(ts[r * DB_CH + e], ts[c * DB_CH + e], v);
        v = warp_sum(v);
        if (lane == 0) out[slot_dot(a, r, c)] = v;
      }
    }
  }
}

// W = corth . T (knew rows), V[m_old + r] = W[r]
template <int KM>
__global__ void __launch_bounds__(DB_NT) k_db_new(DBArgs a) {
  const int tid = threadIdx.x;
  for (long long u = blockIdx.x; u < a.nunits; u += gridDim.x) {
    const int p = a.unit_prob[u];
    const int kT = a.st[p].kT, knew = a.st[p].knew, m0 = a.st[p].m_old;
    if (a.st[p].done || knew == 0) continue;
    const DBProb P = a.prob[p];
    const int64_t n = P.n;
    const int64_t e0 = (int64_t)(u - P.unit0) * DB_CH + tid;
    double t[KM][DB_EPT];
#pragma unroll
    for (int i = 0; i < KM; ++i)
#pragma unroll
      for (int q = 0; q < DB_EPT; ++q) t[i][q] = (i < kT && e0 + q * DB_NT < n) ? P.T[i * n + e0 + q * DB_NT] : 0.0;
    for (int r = 0; r < knew; ++r) {
      double c[KM];
#pragma unroll
      for (int i = 0; i < KM; ++i) c[i] = i < kT ? P.coef[r * P.cap + i] : 0.0;
#pragma unroll
      for (int q = 0; q < DB_EPT; ++q) {
        const int64_t e = e0 + q * DB_NT;
        if (e >= n) continue;
        double v = 0.0;
#pragma unroll
        for (int i = 0; i < KM; ++i) v = fma(c[i], t[i][q], v);
        P.W[r * n + e] = v;
        P.V[(m0 + r) * n + e] = v;
      }
    }
  }
}

// AV[m_old + r] = AW[r]; partial dots V[j] . AW[r], j < m_old + knew
template <int KM>
__global__ void __launch_bounds__(DB_NT) k_db_hv(DBArgs a) {
  extern __shared__ double sm[];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (long long u = blockIdx.x; u < a.nunits; u += gridDim.x) {
    const int p = a.unit_prob[u];
    const int knew = a.st[p].knew, m0 = a.st[p].m_old;
    if (a.st[p].done || knew == 0) continue;
    const DBProb P = a.prob[p];
    const int64_t n = P.n, c0 = (int64_t)(u - P.unit0) * DB_CH;
    __syncthreads();  // the previous unit is consumed
    for (int r = 0; r < knew; ++r)
#pragma unroll
      for (int q = 0; q < DB_EPT; ++q) {
        const int l = tid + q * DB_NT;
        double v = 0.0;
        if (c0 + l < n) {
          v = P.AW[r * n + c0 + l];
          P.AV[(m0 + r) * n + c0 + l] = v;
        }
        sm[r * DB_CH + l] = v;
      }
    __syncthreads();
    double* const out = a.partial + u * a.nslot;
    db_dots<KM>(sm, knew, P.V, n, c0, m0 + knew, lane, w,
                [&](int i, int j, double v) { out[slot_dot(a, i, j)] = v; });
  }
}

// X = cc.V, AX = cc.AV, R = AX - e X; partial |R|^2, x.P r, x.P x
template <int KM>
__global__ void __launch_bounds__(DB_NT) k_db_ritz(DBArgs a) {
  extern __shared__ double sm[];
  double* const cs = sm;                          // Ritz coefficients, row j: KM
  double* const red = sm + KM * DB_CAPMAX;        // [warp][3 KM]
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (long long u = blockIdx.x; u < a.nunits; u += gridDim.x) {
    const int p = a.unit_prob[u];
    const DBState& S = a.st[p];
    const int kk = S.kk, m = S.m;
    if (S.done || S.knew == 0) continue;
    const DBProb P = a.prob[p];
    const int64_t n = P.n;
    const int64_t e0 = (int64_t)(u - P.unit0) * DB_CH + tid;
    __syncthreads();  // cs and red of the previous unit are consumed
    for (int i = tid; i < KM * m; i += DB_NT) cs[i] = i % KM < kk ? P.cc[i % KM * P.cap + i / KM] : 0.0;
    __syncthreads();
    double rr[KM], xpr[KM], xpx[KM];
#pragma unroll
    for (int i = 0; i < KM; ++i) rr[i] = xpr[i] = xpx[i] = 0.0;
#pragma unroll 1
    for (int q = 0; q < DB_EPT; ++q) {
      const int64_t e = e0 + q * DB_NT;
      if (e >= n) break;
      double x[KM], ax[KM];
#pragma unroll
      for (int i = 0; i < KM; ++i) x[i] = ax[i] = 0.0;
#pragma unroll 8
      for (int j = 0; j < m; ++j) {
        const double v = P.V[j * n + e], av = P.AV[j * n + e];
#pragma unroll
        for (int i = 0; i < KM; ++i) {
          const double c = cs[j * KM + i];
          x[i] = fma(c, v, x[i]);
          ax[i] = fma(c, av, ax[i]);
        }
      }
      const double hd = P.hdiag[e];
#pragma unroll
      for (int i = 0; i < KM; ++i)
        if (i < kk) {
          const double ei = S.e[i];
          const double r = fma(-ei, x[i], ax[i]);
          P.X[i * n + e] = x[i];
          P.AX[i * n + e] = ax[i];
          P.R[i * n + e] = r;
          const double pw = db_pinv(hd, ei - a.shift);
          rr[i] = fma(r, r, rr[i]);
          xpr[i] = fma(x[i] * pw, r, xpr[i]);
          xpx[i] = fma(x[i] * pw, x[i], xpx[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < KM; ++i)
      if (i < kk) {
        const double s0 = warp_sum(rr[i]), s1 = warp_sum(xpr[i]), s2 = warp_sum(xpx[i]);
        if (lane == 0) {
          red[w * 3 * KM + i] = s0;
          red[w * 3 * KM + KM + i] = s1;
          red[w * 3 * KM + 2 * KM + i] = s2;
        }
      }
    __syncthreads();
    if (tid < 3 * KM && tid % KM < kk) {
      double v = 0.0;
#pragma unroll
      for (int i = 0; i < DB_NW; ++i) v += red[i * 3 * KM + tid];
      a.partial[u * a.nslot + slot_x(a, tid / KM, tid % KM)] = v;
    }
  }
}

// T[row] = (R[i] - e1 X[i]) P for the unconverged roots; restart copies
__global__ void __launch_bounds__(DB_NT) k_db_pre(DBArgs a) {
  const int tid = threadIdx.x;
  for (long long u = blockIdx.x; u < a.nunits; u += gridDim.x) {
    const int p = a.unit_prob[u];
    const DBState& S = a.st[p];
    if (S.done) continue;
    const DBProb P = a.prob[p];
    const int kT = S.kT, kk = S.kk, restart = S.restart;
    const int64_t n = P.n;
    const int64_t e0 = (int64_t)(u - P.unit0) * DB_CH + tid;
    double hd[DB_EPT];
#pragma unroll
    for (int q = 0; q < DB_EPT; ++q) hd[q] = e0 + q * DB_NT < n ? P.hdiag[e0 + q * DB_NT] : 0.0;
    for (int row = 0; row < kT; ++row) {
      const int i = S.todo[row];
      const double e1 = S.e1[row], es = S.es[row];
      double r[DB_EPT], x[DB_EPT];
#pragma unroll
      for (int q = 0; q < DB_EPT; ++q) {
        const int64_t e = e0 + q * DB_NT;
        r[q] = e < n ? P.R[i * n + e] : 0.0;
        x[q] = e < n ? P.X[i * n + e] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < DB_EPT; ++q)
        if (e0 + q * DB_NT < n) P.T[row * n + e0 + q * DB_NT] = (r[q] - e1 * x[q]) * db_pinv(hd[q], es);
    }
    if (restart)
      for (int i = 0; i < kk; ++i)
#pragma unroll
        for (int q = 0; q < DB_EPT; ++q) {
          const int64_t e = e0 + q * DB_NT;
          if (e >= n) continue;
          const double x = P.X[i * n + e], ax = P.AX[i * n + e];
          P.V[i * n + e] = x;
          P.AV[i * n + e] = ax;
        }
  }
}

// ---------------------------------------------------------------------------
// small per-problem kernels (one block of DB_ST threads per problem)
// ---------------------------------------------------------------------------
// count sums over the problem's chunk partials: put(i, sum of slot(i)), for
// i in first, first + 1, ..., first + 31, first + step, ...  A thread per sum
// for up to 16 chunks; else the warps take every nw-th chunk of 32 sums at a
// time (consecutive slots: coalesced) and the warps' sums are added in warp
// order.  Every thread of the block calls this.
template <typename SlotF, typename PutF>
__device__ __forceinline__ void db_reduce_slots(const DBArgs& a, const DBProb& P, int count, SlotF slot, PutF put,
                                                int first = 0, int step = 32) {
  __shared__ double red[DB_RT / 32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const double* const base = a.partial + (long long)P.unit0 * a.nslot;
  const long long ns = a.nslot;
  const bool few = P.nunits <= 16;
  for (int b = first + (few ? warp * step : 0); b < count; b += few ? nw * step : step) {
    const int i = b + lane;
    double v = 0.0;
    if (i < count) {
      const double* src = base + slot(i);
#pragma unroll 8
      for (int u = few ? 0 : warp; u < P.nunits; u += few ? 1 : nw) v += src[u * ns];
    }
    if (few) {
      if (i < count) put(i, v);
      continue;
    }
    __syncthreads();  // red of the previous round is consumed
    red[warp][lane] = v;
    __syncthreads();
    if (warp == 0 && i < count) {
      v = 0.0;
      for (int w = 0; w < nw; ++w) v += red[w][lane];
      put(i, v);
    }
  }
}

// Cyclic Jacobi eigensolver for the symmetric n x n matrix A (shared
// memory, leading dimension ld), round-robin parallel ordering: each step
// rotates n/2 disjoint pairs (Golub & Van Loan, Matrix Computations,
// sections 8.5.2 and 8.5.5).  On return diag(A) holds the eigenvalues and
// the columns of Q the eigenvectors; w/perm give them in ascending order.
// n <= 64 and at least two warps.
//
// Latency-bound (one block per problem, n around 30), so a step is two
// barriers: the two-sided update of the 2 x 2 blocks of A, one block and its
// mirror a thread, and then, side by side, the next step's rotations (warp
// 0) and this step's columns of Q (the other warps).  With rows, columns and
// rotations in turn, three barriers and an integer division per element, a
// subspace of 30 took 165 us; this takes 58.
struct DBRot {
  double c[2][32], s[2][32];
  unsigned char p[2][32], q[2][32];
  unsigned short blk[528];  // 2 x 2 blocks (t1, t2), t1 <= t2
  double off[DB_RT / 32], dia[DB_RT / 32];
};

__device__ __noinline__ void db_jacobi(double* A, double* Q, int n, int ld, DBRot* R, double* w, int* perm,
                                       bool qinit) {
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  if (!qinit)  // else Q holds a starting basis the rotations are applied to
    for (int i = warp; i < n; i += nw)
      for (int j = lane; j < n; j += 32) Q[i * ld + j] = i == j ? 1.0 : 0.0;
  const int nn = n + (n & 1), np = nn / 2, nblk = np * (np + 1) / 2;
  for (int t1 = warp; t1 < np; t1 += nw)
    for (int t2 = t1 + lane; t2 < np; t2 += 32) R->blk[t1 * np - t1 * (t1 - 1) / 2 + t2 - t1] = (unsigned short)(t1 << 8 | t2);
  auto rotations = [&](int step, int buf) {  // warp 0, lane t = pair t
    if (lane >= np) return;
    auto wrap = [&](int v) { return (v >= nn - 1 ? v - (nn - 1) : v) + 1; };
    const int i0 = lane == 0 ? 0 : wrap(lane - 1 + step), i1 = wrap(nn - 2 - lane + step);
    const int pp = min(i0, i1), qq = max(i0, i1);
    double c = 1.0, s = 0.0;
    if (qq < n) {
      const double apq = A[pp * ld + qq], app = A[pp * ld + pp], aqq = A[qq * ld + qq];
      // negligible against the diagonal: left to the block update, which
      // sets a pair's own entry to zero
      const double q2 = apq * apq;
      if (!(q2 <= 1e-36 * fabs(app * aqq) || q2 == 0.0)) {
        // tan = sign(tau) / (|tau| + sqrt(1 + tau^2)), tau = d / (2 apq)
        const double d = aqq - app, f = 2.0 * fabs(apq);
        double tt = f / (fabs(d) + sqrt(fma(d, d, 4.0 * q2)));
        if (d != 0.0 && (d < 0.0) != (apq < 0.0)) tt = -tt;
        c = rsqrt(fma(tt, tt, 1.0));
        s = tt * c;
      }
    }
    R->p[buf][lane] = (unsigned char)pp;
    R->q[buf][lane] = (unsigned char)qq;
    R->c[buf][lane] = c;
    R->s[buf][lane] = s;
  };
  __syncthreads();
  for (int sweep = 0; sweep < 60 && n > 1; ++sweep) {
    // convergence: off-diagonal Frobenius norm vs the diagonal
    double off = 0.0, dia = 0.0;
    for (int r = warp; r < n; r += nw)
      for (int c = lane; c < n; c += 32) {
        const double v = A[r * ld + c];
        if (r == c) dia += v * v;
        else off += v * v;
      }
    off = warp_sum(off);
    dia = warp_sum(dia);
    if (lane == 0) {
      R->off[warp] = off;
      R->dia[warp] = dia;
    }
    __syncthreads();
    double so = 0.0, sd = 0.0;
    for (int i = 0; i < nw; ++i) {
      so += R->off[i];
      sd += R->dia[i];
    }
    if (so == 0.0 || so <= 1e-32 * sd) break;
    if (warp == 0) rotations(0, 0);
    __syncthreads();
    for (int step = 0; step < nn - 1; ++step) {
      const int buf = step & 1;
      // A <- J^T A J by 2 x 2 blocks
      for (int i = tid; i < nblk; i += nt) {
        const int t1 = R->blk[i] >> 8, t2 = R->blk[i] & 255;
        const int p1 = R->p[buf][t1], q1 = R->q[buf][t1], p2 = R->p[buf][t2], q2 = R->q[buf][t2];
        const double c1 = R->c[buf][t1], s1 = R->s[buf][t1], c2 = R->c[buf][t2], s2 = R->s[buf][t2];
        const bool e1 = q1 < n, e2 = q2 < n;  // the odd one out has no partner
        const double app = A[p1 * ld + p2], apq = e2 ? A[p1 * ld + q2] : 0.0;
        const double aqp = e1 ? A[q1 * ld + p2] : 0.0, aqq = e1 && e2 ? A[q1 * ld + q2] : 0.0;
        const double rpp = c1 * app - s1 * aqp, rpq = c1 * apq - s1 * aqq;
        const double rqp = s1 * app + c1 * aqp, rqq = s1 * apq + c1 * aqq;
        const double npp = c2 * rpp - s2 * rpq, npq = s2 * rpp + c2 * rpq;
        const double nqp = c2 * rqp - s2 * rqq, nqq = s2 * rqp + c2 * rqq;
        A[p1 * ld + p2] = npp;
        if (t1 == t2) {
          if (e1) {
            A[q1 * ld + q1] = nqq;
            A[p1 * ld + q1] = 0.0;
            A[q1 * ld + p1] = 0.0;
          }
        } else {
          A[p2 * ld + p1] = npp;
          if (e2) A[p1 * ld + q2] = A[q2 * ld + p1] = npq;
          if (e1) A[q1 * ld + p2] = A[p2 * ld + q1] = nqp;
          if (e1 && e2) A[q1 * ld + q2] = A[q2 * ld + q1] = nqq;
        }
      }
      __syncthreads();
      if (warp == 0) {
        if (step + 1 < nn - 1) rotations(step + 1, buf ^ 1);
      } else {
        for (int t = warp - 1; t < np; t += nw - 1) {
          const int pp = R->p[buf][t], qq = R->q[buf][t];
          const double c = R->c[buf][t], s = R->s[buf][t];
          if (qq >= n || s == 0.0) continue;
          for (int row = lane; row < n; row += 32) {
            const double qp = Q[row * ld + pp], qv = Q[row * ld + qq];
            Q[row * ld + pp] = c * qp - s * qv;
            Q[row * ld + qq] = s * qp + c * qv;
          }
        }
      }
      __syncthreads();
    }
  }
  // ascending order (ties by index)
  for (int i = tid; i < n; i += nt) {
    const double di = A[i * ld + i];
    int r = 0;
    for (int j = 0; j < n; ++j) {
      const double dj = A[j * ld + j];
      r += (dj < di) || (dj == di && j < i);
    }
    perm[r] = i;
    w[r] = di;
  }
  __syncthreads();
}

// orthonormal combinations of the projected corrections; the Gram matrix
// is scaled by the norms before projection so that the linear-dependence
// cut is relative
__device__ void db_orth(const DBArgs& a, const DBProb& P, DBState& S, int kT) {
  const int tid = threadIdx.x;
  __shared__ double G[DB_KMAX * DB_KMAX], Q[DB_KMAX * DB_KMAX], w[DB_KMAX];
  __shared__ double sc[DB_KMAX];
  __shared__ int perm[DB_KMAX];
  __shared__ DBRot rot;
  for (int i = tid; i < kT; i += DB_ST) sc[i] = 1.0 / sqrt(fmax(S.tnorm[i], 1e-300));
  __syncthreads();
  // the lower half (the upper slots were not formed)
  db_reduce_slots(
      a, P, kT * kT, [&](int idx) { return slot_dot(a, max(idx / kT, idx % kT), min(idx / kT, idx % kT)); },
      [&](int idx, double v) { G[idx / kT * DB_KMAX + idx % kT] = v * sc[idx / kT] * sc[idx % kT]; });
  __syncthreads();
  db_jacobi(G, Q, kT, DB_KMAX, &rot, w, perm, false);
  if (tid == 0) {
    double wmax = 0.0;
    for (int i = 0; i < kT; ++i) wmax = fmax(wmax, w[i]);
    const double cut = fmax(a.lindep, 1e-14 * wmax);
    int first = 0;
    while (first < kT && !(w[first] > cut)) ++first;
    int nkeep = kT - first;
    if (S.m + nkeep > P.cap) {
      nkeep = P.cap - S.m;
      if (nkeep < 0) nkeep = 0;
      first = kT - nkeep;
    }
    for (int r = 0; r < nkeep; ++r) {
      const int col = perm[first + r];
      const double f = 1.0 / sqrt(w[first + r]);
      for (int i = 0; i < kT; ++i) P.coef[r * P.cap + i] = Q[i * DB_KMAX + col] * f * sc[i];
    }
    S.knew = nkeep;
    S.m_old = S.m;
    if (nkeep == 0) S.done = 1;
  }
}

// blockIdx.y: every gridDim.y-th group of 32 sums (passes 0 and 1)
template <int PASS>
__global__ void __launch_bounds__(PASS <= 1 ? DB_RT : DB_ST) k_db_sproj(DBArgs a) {
  const int p = blockIdx.x;
  DBState& S = a.st[p];
  if (S.done || S.kT == 0) return;
  const DBProb P = a.prob[p];
  const int kT = S.kT, m = S.m;
  if constexpr (PASS <= 1) {
    db_reduce_slots(
        a, P, kT * m, [&](int idx) { return slot_dot(a, idx / m, idx % m); },
        [&](int idx, double v) { P.coef[idx / m * P.cap + idx % m] = v; }, 32 * blockIdx.y, 32 * gridDim.y);
    if (PASS == 0 && blockIdx.y == 0)
      db_reduce_slots(
          a, P, kT, [&](int i) { return slot_x(a, 0, i); }, [&](int i, double v) { S.tnorm[i] = v; });
  } else {
    db_orth(a, P, S, kT);
  }
}

__global__ void __launch_bounds__(DB_RT) k_db_sritz(DBArgs a) {
  extern __shared__ double sm[];
  const int p = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  DBState& S = a.st[p];
  if (S.done || S.knew == 0) return;
  const DBProb& P = a.prob[p];
  const int cap = P.cap, ld = a.capb | 1;  // odd: rows of a column in different banks
  const int knew = S.knew, m0 = S.m_old, m = m0 + knew;
  double* A = sm;
  double* Q = A + ld * ld;
  double* hn = Q + ld * ld;  // the new columns of the subspace matrix
  double* w = hn + DB_KMAX * ld;
  double* ov = w + ld;
  int* perm = (int*)(ov + DB_KMAX * ld);
  __shared__ int idx_s[DB_KMAX];
  __shared__ DBRot rot;
  // Warm start: the first m0 basis vectors were diagonalised at the last
  // iteration (eigenvectors qprev, eigenvalues dprev; after a restart the
  // identity and the Ritz values).  In the basis diag(qprev, I) the matrix
  // is diag(dprev) bordered by the new rows and columns, which the Jacobi
  // sweeps then clear in a few sweeps instead of diagonalising from scratch
  // (the off-diagonal entries dropped there are below the Jacobi tolerance
  // of the last solve).  Both border halves take the same sum, so A stays
  // exactly symmetric.
  const bool warm = S.mq == m0 && m0 > 0;
  db_reduce_slots(
      a, P, knew * m, [&](int idx) { return slot_dot(a, idx / m, idx % m); },
      [&](int idx, double v) { hn[idx / m * ld + idx % m] = v; });
  for (int i = warp; i < m; i += DB_RT / 32)
    for (int j = lane; j < m; j += 32) {
      if (warm) {
        Q[i * ld + j] = (i < m0 && j < m0) ? P.qprev[i * cap + j] : (i == j ? 1.0 : 0.0);
        if (i < m0 && j < m0) A[i * ld + j] = i == j ? P.dprev[i] : 0.0;
      } else if (i < m0 && j < m0) {
        A[i * ld + j] = P.h[i * cap + j];
      }
    }
  __syncthreads();
  // the new rows and columns; the square of both takes the symmetric part of
  // its two computed halves
  for (int r = warp; r < knew; r += DB_RT / 32)
    for (int j = lane; j < m; j += 32) {
      double v = hn[r * ld + j];
      if (j >= m0) v = 0.5 * (v + hn[(j - m0) * ld + m0 + r]);
      P.h[(m0 + r) * cap + j] = v;
      P.h[j * cap + m0 + r] = v;
      if (warm && j < m0) {
        v = 0.0;
        for (int l = 0; l < m0; ++l) v = fma(Q[l * ld + j], hn[r * ld + l], v);
      }
      A[(m0 + r) * ld + j] = v;
      A[j * ld + m0 + r] = v;
    }
  __syncthreads();
  db_jacobi(A, Q, m, ld, &rot, w, perm, warm);
  // the eigenpairs of this basis, for the next iteration's warm start
  for (int idx = tid; idx < m * m; idx += DB_RT) {
    const int i = idx / m, j = idx % m;
    P.qprev[i * cap + j] = Q[i * ld + j];
  }
  for (int i = tid; i < m; i += DB_RT) P.dprev[i] = A[i * ld + i];
  const int kk = m < P.k ? m : P.k;
  const bool follow = S.have_e && S.any_conv;
  if (follow) {
    for (int idx = tid; idx < S.kk_prev * m; idx += DB_RT) {
      const int i = idx / m, j = idx % m;
      double s = 0.0;
      for (int l = 0; l < m; ++l) s = fma(P.xprev[i * cap + l], Q[l * ld + perm[j]], s);
      ov[i * ld + j] = fabs(s);
    }
  }
  __syncthreads();
  if (tid == 0) {
    int sel[DB_KMAX];
    int nsel = 0;
    if (follow) {
      // for each previous root the unused Ritz vector of largest overlap,
      // then the chosen ones by energy
      for (int i = 0; i < S.kk_prev; ++i) {
        int best = -1;
        double bv = -1.0;
        for (int j = 0; j < m; ++j) {
          bool used = false;
          for (int t = 0; t < nsel; ++t) used |= sel[t] == j;
          if (!used && ov[i * ld + j] > bv) {
            bv = ov[i * ld + j];
            best = j;
          }
        }
        if (best >= 0) sel[nsel++] = best;
      }
      for (int i = 1; i < nsel; ++i)
        for (int j = i; j > 0 && sel[j] < sel[j - 1]; --j) {
          const int x = sel[j];
          sel[j] = sel[j - 1];
          sel[j - 1] = x;
        }
      if (nsel > kk) nsel = kk;
    }
    if (nsel < kk) {
      nsel = kk;
      for (int i = 0; i < kk; ++i) sel[i] = i;
    }
    for (int i = 0; i < DB_KMAX; ++i) S.e_prev[i] = S.e[i];
    S.kk_prev = S.have_e ? S.kk : 0;
    for (int i = 0; i < kk; ++i) {
      idx_s[i] = sel[i];
      S.e[i] = w[sel[i]];
    }
    S.kk = kk;
    S.m = m;
  }
  __syncthreads();
  for (int idx = tid; idx < kk * cap; idx += DB_RT) {
    const int i = idx / cap, j = idx % cap;
    P.cc[i * cap + j] = j < m ? Q[j * ld + perm[idx_s[i]]] : 0.0;
  }
}

__global__ void __launch_bounds__(DB_ST) k_db_sconv(DBArgs a) {
  const int p = blockIdx.x, tid = threadIdx.x;
  DBState& S = a.st[p];
  if (S.done || S.knew == 0) return;
  const DBProb& P = a.prob[p];
  const int kk = S.kk, cap = P.cap;
  __shared__ double rr[DB_KMAX], xpr[DB_KMAX], xpx[DB_KMAX];
  __shared__ int restart_s, done_s;
  db_reduce_slots(
      a, P, 3 * kk, [&](int idx) { return slot_x(a, idx / kk, idx % kk); },
      [&](int idx, double v) { (idx / kk == 0 ? rr : idx / kk == 1 ? xpr : xpx)[idx % kk] = v; });
  __syncthreads();
  if (tid == 0) {
    const bool have_prev = S.have_e && S.kk_prev == kk;
    bool all = true, any = false;
    for (int i = 0; i < kk; ++i) {
      S.rnorm[i] = sqrt(fmax(rr[i], 0.0));
      const double de = have_prev ? S.e[i] - S.e_prev[i] : INFINITY;
      const bool c = fabs(de) < a.tol && S.rnorm[i] < a.toloose;
      S.conv[i] = c;
      all &= c;
      any |= c;
    }
    S.any_conv = any;
    S.have_e = 1;
    S.niter += 1;
    int kT = 0;
    if (all && kk == P.k) {
      S.done = 1;
    } else {
      for (int i = 0; i < kk; ++i) {
        if (S.conv[i]) continue;
        S.todo[kT] = i;
        S.e1[kT] = xpx[i] != 0.0 ? xpr[i] / xpx[i] : 0.0;
        S.es[kT] = S.e[i] - a.shift;
        ++kT;
      }
    }
    if (kT == 0) S.done = 1;  // nothing left to correct
    S.kT = kT;
    S.knew = 0;  // set again by the next orthonormalisation
    S.restart = !S.done && (S.m + kT > P.space);
    if (S.restart) S.m = kk;
    S.mq = S.restart ? kk : S.m;  // the basis the stored eigenpairs belong to
    restart_s = S.restart;
    done_s = S.done;
  }
  __syncthreads();
  if (done_s) return;
  // the previous Ritz coefficients for root following (identity after a
  // restart, whose basis is the Ritz vectors themselves) and, on restart,
  // the subspace matrix diag(e)
  const int restart = restart_s;
  for (int idx = tid; idx < kk * cap; idx += DB_ST) {
    const int i = idx / cap, j = idx % cap;
    P.xprev[idx] = restart ? (i == j ? 1.0 : 0.0) : P.cc[idx];
  }
  if (restart) {
    // the basis is the Ritz vectors: h = diag(e), eigenvectors the identity
    for (int idx = tid; idx < cap * cap; idx += DB_ST) {
      const int i = idx / cap, j = idx % cap;
      P.h[idx] = (i == j && i < kk) ? S.e[i] : 0.0;
      P.qprev[idx] = (i == j && i < kk) ? 1.0 : 0.0;
    }
    for (int i = tid; i < kk; i += DB_ST) P.dprev[i] = S.e[i];
  }
}

__global__ void k_db_init(DBArgs a, const double* const* x0) {
  const int p = blockIdx.x;
  DBState& S = a.st[p];
  const DBProb& P = a.prob[p];
  for (int64_t i = threadIdx.x; i < (int64_t)P.k * P.n; i += blockDim.x) P.T[i] = x0[p][i];
  if (threadIdx.x == 0) {
    memset(&S, 0, sizeof(S));
    S.kT = P.k;
  }
}

__global__ void k_db_count(DBArgs a) {
  __shared__ int c;
  if (threadIdx.x == 0) c = 0;
  __syncthreads();
  int mine = 0;
  for (int p = threadIdx.x; p < a.nprob; p += blockDim.x) mine += a.st[p].done ? 0 : 1;
  atomicAdd(&c, mine);
  __syncthreads();
  if (threadIdx.x == 0) *a.count = c;
}

}  // namespace csffci

using namespace csffci;

struct csffci_batch_plan {
  int nprob = 0, kb = 0, capb = 0, nslot = 0;
  long long nunits = 0;
  csffci_batch_options_t opt{};
  std::vector<csffci_batch_problem_t> in;
  std::vector<std::vector<csffci_block_t>> blocks;
  std::vector<DBProb> prob;
  std::vector<int64_t> ndet;
  std::vector<int64_t> off_cdet;  // byte offsets of the det buffers
  std::vector<int32_t> unit_prob;
  // sigma groups by orbital count
  std::vector<int> group_norb;
  std::vector<std::vector<csffci_sigma_job_t>> group_jobs;
  std::vector<SigmaBatchInfo> group_info;
  std::vector<csffci_sigma_job_t*> group_dev;
  std::vector<csffci_transform_job_t> jrev, jfwd, jdet;
  int64_t trev = 0, tfwd = 0, tdet = 0;
  csffci_transform_job_t *drev = nullptr, *dfwd = nullptr, *ddet = nullptr;
  csffci_sigma_job_t* dtune = nullptr;
  size_t arena_bytes = 0;
  char* arena = nullptr;
  DBArgs args{};
  double** dx0 = nullptr;
  int* hcount = nullptr;
  size_t smem_stream = 0, smem_ritz = 0;
  bool bound = false;
  cudaStream_t cap_stream = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int iterations = 0;
};

namespace {

size_t al(size_t b) { return (b + 255) & ~(size_t)255; }

template <int KM>
int enqueue_iteration_km(csffci_batch_plan_t* P, cudaStream_t s) {
  const DBArgs& a = P->args;
  const int gs = grid_for(a.nunits, 1, 148 * 8);
  const int np = P->nprob;
  const dim3 gsum(np, (P->kb * P->capb + 31) / 32);
  int st;
#define DB_CHECK(what)                 \
  if ((st = check_launch(what)) != 0) \
    return st;
  // one profiler scope per launch (timed only while profiling is enabled)
#define DB_LAUNCH(name, what, ...)  \
  {                                 \
    ProfScope ps_(name, s);         \
    __VA_ARGS__;                    \
  }                                 \
  DB_CHECK(what)
  DB_LAUNCH("k_db_proj", "batch solver: projection 0", (k_db_proj<KM, 0><<<gs, DB_NT, P->smem_stream, s>>>(a)));
  DB_LAUNCH("k_db_sproj", "batch solver: projection 0 reduce", (k_db_sproj<0><<<gsum, DB_RT, 0, s>>>(a)));
  DB_LAUNCH("k_db_proj", "batch solver: projection 1", (k_db_proj<KM, 1><<<gs, DB_NT, P->smem_stream, s>>>(a)));
  DB_LAUNCH("k_db_sproj", "batch solver: projection 1 reduce", (k_db_sproj<1><<<gsum, DB_RT, 0, s>>>(a)));
  DB_LAUNCH("k_db_proj", "batch solver: projection 2", (k_db_proj<KM, 2><<<gs, DB_NT, P->smem_stream, s>>>(a)));
  DB_LAUNCH("k_db_sproj", "batch solver: orthonormalisation", (k_db_sproj<2><<<np, DB_ST, 0, s>>>(a)));
  DB_LAUNCH("k_db_new", "batch solver: new vectors", (k_db_new<KM><<<gs, DB_NT, 0, s>>>(a)));
  if ((st = transform_batch_launch(1, P->drev, (int)P->jrev.size(), P->trev, s)) != 0) return st;
  for (size_t g = 0; g < P->group_info.size(); ++g)
    if ((st = sigma_batch_launch(P->group_info[g], P->group_dev[g], s)) != 0) return st;
  if ((st = transform_batch_launch(0, P->dfwd, (int)P->jfwd.size(), P->tfwd, s)) != 0) return st;
  DB_LAUNCH("k_db_hv", "batch solver: H v", (k_db_hv<KM><<<gs, DB_NT, P->smem_stream, s>>>(a)));
  DB_LAUNCH("k_db_sritz", "batch solver: subspace eigenproblem", (k_db_sritz<<<np, DB_RT, P->smem_ritz, s>>>(a)));
  DB_LAUNCH("k_db_ritz", "batch solver: Ritz vectors", (k_db_ritz<KM><<<gs, DB_NT, P->smem_stream, s>>>(a)));
  DB_LAUNCH("k_db_sconv", "batch solver: convergence", (k_db_sconv<<<np, DB_ST, 0, s>>>(a)));
  DB_LAUNCH("k_db_pre", "batch solver: preconditioner", (k_db_pre<<<gs, DB_NT, 0, s>>>(a)));
#undef DB_LAUNCH
#undef DB_CHECK
  return CSFFCI_OK;
}

int enqueue_iteration(csffci_batch_plan_t* P, cudaStream_t s) {
  return P->kb <= 4 ? enqueue_iteration_km<4>(P, s) : enqueue_iteration_km<DB_KMAX>(P, s);
}

}  // namespace

extern "C" {

int csffci_batch_plan_create(int nprob, const csffci_batch_problem_t* probs, const csffci_batch_options_t* opt,
                             csffci_batch_plan_t** plan, size_t* arena_bytes) {
  CSF_REQUIRE(plan && arena_bytes && opt, "batch_plan_create: NULL argument");
  *plan = nullptr;
  CSF_REQUIRE(nprob > 0 && probs, "batch_plan_create: empty batch");
  CSF_REQUIRE(opt->max_space >= 1 && opt->max_cycle >= 0, "batch_plan_create: bad options");
  for (int i = 0; i < nprob && opt->deterministic; ++i)
    CSF_REQUIRE(probs[i].norb >= 4 && probs[i].norb <= 16,
                "batch_plan_create: the deterministic scatter covers 4 <= norb <= 16, not %d", probs[i].norb);
  auto* P = new csffci_batch_plan();
  P->nprob = nprob;
  P->opt = *opt;
  if (P->opt.check_every < 1) P->opt.check_every = 1;
  P->in.assign(probs, probs + nprob);
  P->blocks.resize(nprob);
  P->prob.resize(nprob);
  P->ndet.resize(nprob);
  int kb = 1, capb = 1;
  long long nunits = 0;
  for (int i = 0; i < nprob; ++i) {
    const csffci_batch_problem_t& q = probs[i];
    if (!(q.norb >= 4 && q.norb <= 16 && q.neleca >= 0 && q.nelecb >= 0 && q.neleca <= q.norb &&
          q.nelecb <= q.norb && q.nroots >= 1 && q.nroots <= DB_KMAX && q.ncsf >= q.nroots &&
          q.nblocks >= 0 && (q.nblocks == 0 || q.blocks) && q.csd_mask && q.h2e && q.link_a && q.link_b &&
          q.hdiag && q.x0 && (q.eta == 0 || ((q.eta == 1 || q.eta == -1) && q.neleca == q.nelecb)))) {
      delete P;
      set_error("batch_plan_create: problem %d is invalid (norb 4..16, 1..%d roots <= ncsf, eta 0 or +-1 "
                "with neleca == nelecb, device pointers set)",
                i, DB_KMAX);
      return CSFFCI_ERR_INVALID;
    }
    const int cap = opt->max_space + 2 * q.nroots;
    if (cap > DB_CAPMAX) {
      delete P;
      set_error("batch_plan_create: max_space + 2*nroots = %d exceeds %d", cap, DB_CAPMAX);
      return CSFFCI_ERR_INVALID;
    }
    for (int b = 0; b < q.nblocks; ++b)
      if (q.blocks[b].conf_sel != nullptr) {
        delete P;
        set_error("batch_plan_create: problem %d: point-group-restricted CSF blocks are not supported", i);
        return CSFFCI_ERR_INVALID;
      }
    P->blocks[i].assign(q.blocks, q.blocks + q.nblocks);
    DBProb& d = P->prob[i];
    memset(&d, 0, sizeof(d));
    d.n = q.ncsf;
    d.k = q.nroots;
    d.cap = cap;
    d.space = opt->max_space + q.nroots;
    d.unit0 = (int32_t)nunits;
    d.nunits = (int32_t)((q.ncsf + DB_CH - 1) / DB_CH);
    d.hdiag = q.hdiag;
    nunits += d.nunits;
    P->ndet[i] = (int64_t)host_binom(q.norb, q.neleca) * (int64_t)host_binom(q.norb, q.nelecb);
    if (q.nroots > kb) kb = q.nroots;
    if (cap > capb) capb = cap;
  }
  P->kb = kb;
  P->capb = capb;
  P->nslot = kb * capb + 3 * kb;
  P->nunits = nunits;
  // arena: per-problem vectors, then the tables (offsets until bind)
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off += al(bytes);
    return o;
  };
  std::vector<size_t> o_vec(nprob), o_det(nprob), o_small(nprob);
  for (int i = 0; i < nprob; ++i) {
    const DBProb& d = P->prob[i];
    o_vec[i] = take(sizeof(double) * (size_t)d.n * (2 * d.cap + 6 * d.k));
    // det buffers: k vectors, k sigmas, and per root the spin-symmetric
    // scratch (ndet doubles) or, with the deterministic scatter, the three
    // int64 digit planes (3 ndet)
    const int nscr = opt->deterministic ? 3 : (probs[i].eta ? 1 : 0);
    o_det[i] = take(sizeof(double) * (size_t)P->ndet[i] * d.k * (2 + nscr));
    o_small[i] = take(sizeof(double) * (2 * (size_t)d.cap * d.cap + 3 * (size_t)d.k * d.cap + d.cap));
  }
  const size_t o_partial = take(sizeof(double) * (size_t)nunits * P->nslot);
  const size_t o_prob = take(sizeof(DBProb) * nprob);
  const size_t o_state = take(sizeof(DBState) * nprob);
  const size_t o_units = take(sizeof(int32_t) * nunits);
  const size_t o_x0 = take(sizeof(double*) * nprob);
  const size_t o_count = take(sizeof(int));
  // sigma groups (one job per problem and root) and transform jobs
  std::vector<int> norbs;
  for (int i = 0; i < nprob; ++i) {
    bool seen = false;
    for (int v : norbs) seen |= v == probs[i].norb;
    if (!seen) norbs.push_back(probs[i].norb);
  }
  P->group_norb = norbs;
  std::vector<size_t> o_group(norbs.size());
  size_t max_group = 1;
  for (size_t g = 0; g < norbs.size(); ++g) {
    size_t nj = 0;
    for (int i = 0; i < nprob; ++i)
      if (probs[i].norb == norbs[g]) nj += probs[i].nroots;
    o_group[g] = take(sizeof(csffci_sigma_job_t) * nj);
    if (nj > max_group) max_group = nj;
  }
  const size_t o_tune = take(sizeof(csffci_sigma_job_t) * max_group);  // ungated copy for the autotuner
  size_t ntj = 0;
  for (int i = 0; i < nprob; ++i)
    for (int b = 0; b < probs[i].nblocks; ++b)
      if (probs[i].blocks[b].ncsf > 0 && probs[i].blocks[b].nconf > 0) ++ntj;
  const size_t o_rev = take(sizeof(csffci_transform_job_t) * (ntj ? ntj : 1));
  const size_t o_fwd = take(sizeof(csffci_transform_job_t) * (ntj ? ntj : 1));
  const size_t o_det_jobs = take(sizeof(csffci_transform_job_t) * (ntj ? ntj : 1));
  P->arena_bytes = off;
  for (int i = 0; i < nprob; ++i) {
    DBProb& d = P->prob[i];
    d.V = (double*)o_vec[i];
    d.h = (double*)o_small[i];
  }
  P->off_cdet.assign(o_det.begin(), o_det.end());
  P->args.partial = (double*)o_partial;
  P->args.prob = (const DBProb*)o_prob;
  P->args.st = (DBState*)o_state;
  P->args.unit_prob = (const int32_t*)o_units;
  P->dx0 = (double**)o_x0;
  P->args.count = (int*)o_count;
  P->group_dev.resize(norbs.size());
  for (size_t g = 0; g < norbs.size(); ++g) P->group_dev[g] = (csffci_sigma_job_t*)o_group[g];
  P->drev = (csffci_transform_job_t*)o_rev;
  P->dfwd = (csffci_transform_job_t*)o_fwd;
  P->ddet = (csffci_transform_job_t*)o_det_jobs;
  P->dtune = (csffci_sigma_job_t*)o_tune;
  *plan = P;
  *arena_bytes = P->arena_bytes;
  return CSFFCI_OK;
}

int csffci_batch_plan_bind(csffci_batch_plan_t* P, void* arena, size_t arena_bytes, cudaStream_t stream) {
  CSF_REQUIRE(P && !P->bound, "batch_plan_bind: plan missing or already bound");
  CSF_REQUIRE(arena && arena_bytes >= P->arena_bytes && ((uintptr_t)arena & 255) == 0,
              "batch_plan_bind: arena of %zu bytes (need %zu, 256-byte aligned)", arena_bytes, P->arena_bytes);
  char* base = (char*)arena;
  P->arena = base;
  auto rel = [&](const void* o) { return base + (size_t)(uintptr_t)o; };
  const int nprob = P->nprob;
  for (int i = 0; i < nprob; ++i) {
    DBProb& d = P->prob[i];
    double* v = (double*)rel(d.V);
    double* sm = (double*)rel(d.h);
    const size_t n = (size_t)d.n;
    d.V = v;
    d.AV = v + (size_t)d.cap * n;
    d.X = d.AV + (size_t)d.cap * n;
    d.AX = d.X + (size_t)d.k * n;
    d.R = d.AX + (size_t)d.k * n;
    d.T = d.R + (size_t)d.k * n;
    d.W = d.T + (size_t)d.k * n;
    d.AW = d.W + (size_t)d.k * n;
    d.h = sm;
    d.coef = sm + (size_t)d.cap * d.cap;
    d.cc = d.coef + (size_t)d.k * d.cap;
    d.xprev = d.cc + (size_t)d.k * d.cap;
    d.qprev = d.xprev + (size_t)d.k * d.cap;
    d.dprev = d.qprev + (size_t)d.cap * d.cap;
  }
  P->args.partial = (double*)rel(P->args.partial);
  P->args.prob = (const DBProb*)rel(P->args.prob);
  P->args.st = (DBState*)rel(P->args.st);
  P->args.unit_prob = (const int32_t*)rel(P->args.unit_prob);
  P->dx0 = (double**)rel(P->dx0);
  P->args.count = (int*)rel(P->args.count);
  for (auto& g : P->group_dev) g = (csffci_sigma_job_t*)rel(g);
  P->drev = (csffci_transform_job_t*)rel(P->drev);
  P->dfwd = (csffci_transform_job_t*)rel(P->dfwd);
  P->ddet = (csffci_transform_job_t*)rel(P->ddet);
  P->dtune = (csffci_sigma_job_t*)rel(P->dtune);
  P->args.nslot = P->nslot;
  P->args.capb = P->capb;
  P->args.kb = P->kb;
  P->args.nprob = nprob;
  P->args.nunits = P->nunits;
  P->args.tol = P->opt.conv_tol;
  P->args.toloose = P->opt.conv_tol_residual > 0 ? P->opt.conv_tol_residual : sqrt(P->opt.conv_tol);
  P->args.lindep = P->opt.lindep;
  P->args.shift = P->opt.level_shift;
  P->unit_prob.resize(P->nunits);
  for (int i = 0; i < nprob; ++i)
    for (int u = 0; u < P->prob[i].nunits; ++u) P->unit_prob[P->prob[i].unit0 + u] = i;
  // sigma job tables: job (problem i, root v) gated by knew of problem i
  P->group_jobs.assign(P->group_norb.size(), {});
  P->group_info.assign(P->group_norb.size(), SigmaBatchInfo());
  DBState* st = P->args.st;
  for (size_t g = 0; g < P->group_norb.size(); ++g) {
    for (int i = 0; i < nprob; ++i) {
      const csffci_batch_problem_t& q = P->in[i];
      if (q.norb != P->group_norb[g]) continue;
      double* det = (double*)(base + P->off_cdet[i]);
      const size_t nd = (size_t)P->ndet[i];
      for (int v = 0; v < q.nroots; ++v) {
        csffci_sigma_job_t J;
        memset(&J, 0, sizeof(J));
        J.h2e = q.h2e;
        J.link_a = q.link_a;
        J.link_b = q.link_b;
        J.ci = det + (size_t)v * nd;
        J.sigma = det + (size_t)(q.nroots + v) * nd;
        if (P->opt.deterministic) {
          J.scratch = det + (size_t)(2 * q.nroots + 3 * v) * nd;
          J.flags = CSFFCI_SIGMA_JOB_DETERMINISTIC;
        } else {
          J.scratch = q.eta ? det + (size_t)(2 * q.nroots + v) * nd : nullptr;
        }
        J.neleca = q.neleca;
        J.nelecb = q.nelecb;
        J.sym = q.eta ? 1 : 0;
        J.eta = q.eta ? q.eta : 1;
        J.live = &st[i].knew;
        J.live_index = v;
        P->group_jobs[g].push_back(J);
      }
    }
    int stt = sigma_batch_prepare(P->group_norb[g], (int)P->group_jobs[g].size(), P->group_jobs[g].data(),
                                  &P->group_info[g]);
    if (stt) return stt;
  }
  // transform tables: W -> cdet (gated by knew), sdet -> AW (gated by
  // knew), X -> cdet (gated by kk, for the final vectors)
  P->jrev.clear();
  P->jfwd.clear();
  P->jdet.clear();
  for (int i = 0; i < nprob; ++i) {
    const csffci_batch_problem_t& q = P->in[i];
    const DBProb& d = P->prob[i];
    double* det = (double*)(base + P->off_cdet[i]);
    const int64_t nd = P->ndet[i];
    for (const csffci_block_t& b : P->blocks[i]) {
      if (b.ncsf <= 0 || b.nconf <= 0) continue;
      csffci_transform_job_t J;
      memset(&J, 0, sizeof(J));
      J.mask = q.csd_mask;
      J.umat = b.umat;
      J.csd_offset = b.csd_offset;
      J.csf_offset = b.csf_offset;
      J.nconf = b.nconf;
      J.ndet = b.ndet;
      J.ncsf = b.ncsf;
      J.nvec = q.nroots;
      J.sign = b.sign;
      csffci_transform_job_t r = J, f = J, x = J;
      r.x = d.W;
      r.ldx = d.n;
      r.y = det;
      r.ldy = nd;
      r.live = &st[i].knew;
      f.x = det + (size_t)q.nroots * nd;
      f.ldx = nd;
      f.y = d.AW;
      f.ldy = d.n;
      f.live = &st[i].knew;
      x.x = d.X;
      x.ldx = d.n;
      x.y = det;
      x.ldy = nd;
      x.live = &st[i].kk;
      P->jrev.push_back(r);
      P->jfwd.push_back(f);
      P->jdet.push_back(x);
    }
  }
  int stt = transform_batch_prepare(1, (int)P->jrev.size(), P->jrev.data(), &P->trev);
  if (!stt) stt = transform_batch_prepare(0, (int)P->jfwd.size(), P->jfwd.data(), &P->tfwd);
  if (!stt) stt = transform_batch_prepare(1, (int)P->jdet.size(), P->jdet.data(), &P->tdet);
  if (stt) return stt;
  // uploads
  std::vector<const double*> x0(nprob);
  for (int i = 0; i < nprob; ++i) x0[i] = P->in[i].x0;
  CSF_CUDA(cudaMemcpyAsync((void*)P->args.prob, P->prob.data(), sizeof(DBProb) * nprob, cudaMemcpyHostToDevice,
                           stream));
  CSF_CUDA(cudaMemcpyAsync((void*)P->args.unit_prob, P->unit_prob.data(), sizeof(int32_t) * P->nunits,
                           cudaMemcpyHostToDevice, stream));
  CSF_CUDA(cudaMemcpyAsync(P->dx0, x0.data(), sizeof(double*) * nprob, cudaMemcpyHostToDevice, stream));
  for (size_t g = 0; g < P->group_jobs.size(); ++g)
    CSF_CUDA(cudaMemcpyAsync(P->group_dev[g], P->group_jobs[g].data(),
                             sizeof(csffci_sigma_job_t) * P->group_jobs[g].size(), cudaMemcpyHostToDevice, stream));
  if (!P->jrev.empty()) {
    const size_t nb = sizeof(csffci_transform_job_t) * P->jrev.size();
    CSF_CUDA(cudaMemcpyAsync(P->drev, P->jrev.data(), nb, cudaMemcpyHostToDevice, stream));
    CSF_CUDA(cudaMemcpyAsync(P->dfwd, P->jfwd.data(), nb, cudaMemcpyHostToDevice, stream));
    CSF_CUDA(cudaMemcpyAsync(P->ddet, P->jdet.data(), nb, cudaMemcpyHostToDevice, stream));
  }
  // determinant vectors read as zero outside the CSF blocks: clear once
  for (int i = 0; i < nprob; ++i)
    CSF_CUDA(cudaMemsetAsync(base + P->off_cdet[i], 0,
                             sizeof(double) * (size_t)P->ndet[i] * P->in[i].nroots, stream));
  // autotuner: every tile variant timed on each group's jobs (ungated
  // copy; the outputs are scratch at this point)
  if (P->opt.autotune) {
    for (size_t g = 0; g < P->group_jobs.size(); ++g) {
      std::vector<csffci_sigma_job_t> ung = P->group_jobs[g];
      for (auto& J : ung) J.live = nullptr;
      CSF_CUDA(cudaMemcpyAsync(P->dtune, ung.data(), sizeof(csffci_sigma_job_t) * ung.size(),
                               cudaMemcpyHostToDevice, stream));
      SigmaBatchInfo t = P->group_info[g];
      t.job0.live = nullptr;
      int stt2 = sigma_batch_tune(t, ung.data(), P->dtune, stream);
      if (stt2) return stt2;
      P->group_info[g].variant = t.variant;
      CSF_CUDA(cudaStreamSynchronize(stream));  // ung is released below
    }
  }
  k_db_init<<<nprob, 256, 0, stream>>>(P->args, (const double* const*)P->dx0);
  int st2 = check_launch("batch solver: init");
  if (st2) return st2;
  // shared memory of the streaming and subspace kernels
  // a chunk of the roots' vectors and their coefficients
  const int km = P->kb <= 4 ? 4 : DB_KMAX;
  P->smem_stream = sizeof(double) * km * (DB_CH + DB_CAPMAX);
  const size_t ldr = P->capb | 1;
  P->smem_ritz = db_ritz_smem(ldr);
  if (P->smem_ritz > 48 * 1024)
    CSF_CUDA(cudaFuncSetAttribute(k_db_sritz, cudaFuncAttributeMaxDynamicSharedMemorySize, DB_RITZ_SMEM));
  CSF_CUDA(cudaMallocHost(&P->hcount, sizeof(int)));
  CSF_CUDA(cudaStreamSynchronize(stream));
  P->bound = true;
  return CSFFCI_OK;
}

int csffci_batch_plan_run(csffci_batch_plan_t* P, cudaStream_t stream, int* iterations) {
  CSF_REQUIRE(P && P->bound, "batch_plan_run: plan not bound");
  int it = 0, st = 0;
  const int maxc = P->opt.max_cycle;
  if (maxc > 0 && P->opt.use_graph && !P->exec) {
    // first iteration eagerly (sets kernel attributes, validates the
    // launch sequence), then one iteration captured as a graph
    if ((st = enqueue_iteration(P, stream)) != 0) return st;
    ++it;
    if (!P->cap_stream) CSF_CUDA(cudaStreamCreateWithFlags(&P->cap_stream, cudaStreamNonBlocking));
    CSF_CUDA(cudaStreamSynchronize(stream));
    CSF_CUDA(cudaStreamBeginCapture(P->cap_stream, cudaStreamCaptureModeRelaxed));
    st = enqueue_iteration(P, P->cap_stream);
    cudaGraph_t g = nullptr;
    cudaError_t ce = cudaStreamEndCapture(P->cap_stream, &g);
    if (st) {
      if (g) cudaGraphDestroy(g);
      return st;
    }
    CSF_CUDA(ce);
    P->graph = g;
    CSF_CUDA(cudaGraphInstantiate(&P->exec, P->graph, 0));
  }
  while (it < maxc) {
    int n = P->opt.check_every;
    if (n > maxc - it) n = maxc - it;
    for (int r = 0; r < n; ++r) {
      if (P->exec) {
        CSF_CUDA(cudaGraphLaunch(P->exec, stream));
      } else if ((st = enqueue_iteration(P, stream)) != 0) {
        return st;
      }
    }
    it += n;
    k_db_count<<<1, 256, 0, stream>>>(P->args);
    if ((st = check_launch("batch solver: count")) != 0) return st;
    CSF_CUDA(cudaMemcpyAsync(P->hcount, P->args.count, sizeof(int), cudaMemcpyDeviceToHost, stream));
    CSF_CUDA(cudaStreamSynchronize(stream));
    if (*P->hcount == 0) break;
  }
  P->iterations = it;
  if (iterations) *iterations = it;
  return CSFFCI_OK;
}

int csffci_batch_plan_max_roots(const csffci_batch_plan_t* P) { return P ? P->kb : 0; }

int csffci_batch_plan_tile_variants(const csffci_batch_plan_t* P, int32_t* norb, int32_t* variant, int cap) {
  if (!P) return 0;
  const int n = (int)P->group_norb.size();
  for (int g = 0; g < n && g < cap; ++g) {
    if (norb) norb[g] = P->group_norb[g];
    if (variant)
      variant[g] = (g < (int)P->group_info.size() && P->group_info[g].variant >= 0)
                       ? P->group_info[g].variant
                       : rr_default_variant(P->group_norb[g]);
  }
  return n;
}

int csffci_batch_plan_results(csffci_batch_plan_t* P, double* energies, int32_t* converged, int32_t* niter,
                              int32_t* nfound, cudaStream_t stream) {
  CSF_REQUIRE(P && P->bound, "batch_plan_results: plan not bound");
  std::vector<DBState> st(P->nprob);
  CSF_CUDA(cudaMemcpyAsync(st.data(), P->args.st, sizeof(DBState) * P->nprob, cudaMemcpyDeviceToHost, stream));
  CSF_CUDA(cudaStreamSynchronize(stream));
  const int kb = P->kb;
  for (int i = 0; i < P->nprob; ++i) {
    for (int r = 0; r < kb; ++r) {
      const bool have = r < st[i].kk;
      if (energies) energies[i * kb + r] = have ? st[i].e[r] : NAN;
      if (converged) converged[i * kb + r] = have ? st[i].conv[r] : 0;
    }
    if (niter) niter[i] = st[i].niter;
    if (nfound) nfound[i] = st[i].kk;
  }
  return CSFFCI_OK;
}

int csffci_batch_plan_to_det(csffci_batch_plan_t* P, cudaStream_t stream) {
  CSF_REQUIRE(P && P->bound, "batch_plan_to_det: plan not bound");
  for (int i = 0; i < P->nprob; ++i)
    CSF_CUDA(cudaMemsetAsync(P->arena + P->off_cdet[i], 0, sizeof(double) * (size_t)P->ndet[i] * P->in[i].nroots,
                             stream));
  return transform_batch_launch(1, P->ddet, (int)P->jdet.size(), P->tdet, stream);
}

int csffci_batch_plan_vectors(const csffci_batch_plan_t* P, int iprob, const double** csf, const double** det) {
  CSF_REQUIRE(P && P->bound && iprob >= 0 && iprob < P->nprob, "batch_plan_vectors: bad problem index");
  if (csf) *csf = P->prob[iprob].X;
  if (det) *det = (const double*)(P->arena + P->off_cdet[iprob]);
  return CSFFCI_OK;
}

void csffci_batch_plan_destroy(csffci_batch_plan_t* P) {
  if (!P) return;
  if (P->exec) cudaGraphExecDestroy(P->exec);
  if (P->graph) cudaGraphDestroy(P->graph);
  if (P->cap_stream) cudaStreamDestroy(P->cap_stream);
  if (P->hcount) cudaFreeHost(P->hcount);
  delete P;
}

}  // extern "C"
