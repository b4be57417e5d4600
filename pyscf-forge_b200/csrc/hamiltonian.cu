// Hamiltonian building blocks: absorb_h1e, the determinant diagonal, the
// p-space Slater-Condon block and the one-electron contraction.
#include <mutex>

#include "common.cuh"
#include "profile.cuh"

namespace csffci {

// f(j,k) = (h1e[j][k] - 1/2 sum_i (ji|ik)) / nelec, evaluated on the fly
__device__ __forceinline__ double absorb_f(int norb, int npair, const double* h1e,
                                           const double* eri, double inv_n, int j, int k) {
  double s = 0.0;
  for (int i = 0; i < norb; ++i) s += eri[(int64_t)pair_index(j, i) * npair + pair_index(i, k)];
  return (h1e[j * norb + k] - 0.5 * s) * inv_n;
}

__device__ __forceinline__ void unpair(int pq, int* p, int* q) {
  int h = (int)((sqrt(8.0 * pq + 1.0) - 1.0) * 0.5);
  while (h * (h + 1) / 2 > pq) --h;
  while ((h + 1) * (h + 2) / 2 <= pq) ++h;
  *p = h;
  *q = pq - h * (h + 1) / 2;
}

// h2e[pq][rs] = fac*(eri[pq][rs] + delta_pq f[r][s] + delta_rs f[p][q]),
// pair (p,q) with p >= q
__global__ void k_absorb_h2e(int norb, int npair, const double* h1e, const double* eri,
                             double inv_n, double fac, double* h2e) {
  int64_t n = (int64_t)npair * npair;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    int pq = (int)(t / npair), rs = (int)(t - (int64_t)pq * npair);
    int p, q, r, s;
    unpair(pq, &p, &q);
    unpair(rs, &r, &s);
    double v = eri[t];
    if (p == q) v += absorb_f(norb, npair, h1e, eri, inv_n, r, s);
    if (r == s) v += absorb_f(norb, npair, h1e, eri, inv_n, p, q);
    h2e[t] = v * fac;
  }
}

// per-string pieces of the determinant diagonal:
//   e1[I] = sum_{i in I} h[i][i] + 1/2 sum_{i,j in I} (J_ij - K_ij)
//   jv[I][q] = sum_{i in I} J_iq          (only for the alpha strings)
// with J_ij = (ii|jj) = eri[ii][jj], K_ij = (ij|ji) = eri[ij][ij].
//
// LANES 32: a warp per string of either spin, its lanes over q.  The sums are
// chains of loads, so what counts is how many run at once (one thread per
// string left most of the GPU idle: 45 us a spin at 14 orbitals and 7 electrons,
// now 10 us for both in one launch).  LANES 1: a thread per string, for as many
// strings as fill the GPU that way: 32 lanes then only multiply the work of
// finding a string and its orbitals (see hdiag_det_run).
template <int LANES>
__global__ void __launch_bounds__(128) k_string_energy(int norb, int neleca, int nelecb, int npair,
                                                       unsigned long long na, unsigned long long nb,
                                                       const double* __restrict__ ha, const double* __restrict__ hb,
                                                       const double* __restrict__ eri, double* ea, double* ja,
                                                       double* eb, uint64_t* sb) {
  const int lane = threadIdx.x & (LANES - 1);
  const unsigned long long nw = (unsigned long long)gridDim.x * (blockDim.x / LANES);
  for (unsigned long long w = blockIdx.x * (unsigned long long)(blockDim.x / LANES) + threadIdx.x / LANES; w < na + nb;
       w += nw) {
    const bool alpha = w < na;
    const unsigned long long I = alpha ? w : w - na;
    const unsigned long long s = str_unrank(norb, alpha ? neleca : nelecb, I);
    const double* const h = alpha ? ha : hb;
    double e = 0.0;
    for (int q = lane; q < norb; q += LANES) {
      const bool occ = (s >> q) & 1ull;
      if (LANES == 1 && !alpha && !occ) continue;
      const int qq = pair_index(q, q);
      double j = 0.0, k = 0.0;
      if (LANES == 1) {
        for (unsigned long long b = s; b; b &= b - 1) {
          const int i = __ffsll((long long)b) - 1;
          const int iq = pair_index(i, q);
          j += eri[(int64_t)pair_index(i, i) * npair + qq];
          if (occ) k += eri[(int64_t)iq * npair + iq];
        }
      } else {
#pragma unroll 4
        for (int i = 0; i < norb; ++i)
          if ((s >> i) & 1ull) {
            const int iq = pair_index(i, q);
            j += eri[(int64_t)pair_index(i, i) * npair + qq];
            k += eri[(int64_t)iq * npair + iq];
          }
      }
      if (occ) e += h[q * norb + q] + 0.5 * (j - k);
      if (alpha) ja[I * norb + q] = j;
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
    if (lane == 0) {
      if (alpha) {
        ea[I] = e;
      } else {
        eb[I] = e;
        sb[I] = s;
      }
    }
  }
}

// hdiag[ia][ib] = ea + eb + sum over the orbitals q of ib of ja[ia][q], by
// tables of the sums over HD_BITS orbitals at a time, for HD_ROWS rows ia a
// block: two table reads an element at 14 orbitals instead of a loop over 7
// electrons (110 -> 26 us for 94 MB, which take 15 us to write).
constexpr int HD_BITS = 7, HD_ROWS = 4;
constexpr long long HD_WARPS = 20000;
__global__ void __launch_bounds__(256) k_hdiag_det_table(int norb, unsigned long long Na, unsigned long long Nb,
                                                         const double* __restrict__ ea, const double* __restrict__ eb,
                                                         const double* __restrict__ ja, const uint64_t* __restrict__ sb,
                                                         double* hdiag) {
  extern __shared__ double hd_tab[];  // [chunk][row][2^HD_BITS]
  constexpr int TS = 1 << HD_BITS;
  const int nch = (norb + HD_BITS - 1) / HD_BITS;
  const unsigned long long r0 = (unsigned long long)blockIdx.x * HD_ROWS;
  for (int t = threadIdx.x; t < nch * HD_ROWS * TS; t += blockDim.x) {
    const int m = t & (TS - 1), r = (t >> HD_BITS) % HD_ROWS, c = (t >> HD_BITS) / HD_ROWS;
    const int q0 = c * HD_BITS;
    double v = 0.0;
    if (r0 + r < Na && q0 + (32 - __clz(m)) <= norb)
      for (int b = m; b; b &= b - 1) v += ja[(r0 + r) * norb + q0 + __ffs(b) - 1];
    hd_tab[t] = v;
  }
  double e[HD_ROWS];
#pragma unroll
  for (int r = 0; r < HD_ROWS; ++r) e[r] = r0 + r < Na ? ea[r0 + r] : 0.0;
  __syncthreads();
  for (unsigned long long ib = blockIdx.y * (unsigned long long)blockDim.x + threadIdx.x; ib < Nb;
       ib += (unsigned long long)gridDim.y * blockDim.x) {
    const double x = eb[ib];
    double v[HD_ROWS];
#pragma unroll
    for (int r = 0; r < HD_ROWS; ++r) v[r] = e[r] + x;
    unsigned long long s = sb[ib];
    for (int c = 0; c < nch; ++c, s >>= HD_BITS) {
      const double* const tab = hd_tab + c * HD_ROWS * TS + ((int)s & (TS - 1));
#pragma unroll
      for (int r = 0; r < HD_ROWS; ++r) v[r] += tab[r * TS];
    }
#pragma unroll
    for (int r = 0; r < HD_ROWS; ++r)
      if (r0 + r < Na) hdiag[(r0 + r) * Nb + ib] = v[r];
  }
}

// the same, element by element
__global__ void k_hdiag_det(int norb, unsigned long long Na, unsigned long long Nb,
                            const double* __restrict__ ea, const double* __restrict__ eb,
                            const double* __restrict__ ja, const uint64_t* __restrict__ sb,
                            double* hdiag) {
  unsigned long long n = Na * Nb;
  for (unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; t < n;
       t += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long ia = t / Nb, ib = t - ia * Nb;
    unsigned long long s = sb[ib];
    const double* j = ja + ia * norb;
    double v = ea[ia] + eb[ib];
    while (s) {
      int q = __ffsll((long long)s) - 1;
      s &= s - 1;
      v += j[q];
    }
    hdiag[t] = v;
  }
}

// both launches of the determinant diagonal; ea, ja, eb and sb are scratch
static int hdiag_det_run(int norb, int neleca, int nelecb, unsigned long long Na, unsigned long long Nb,
                         const double* h1a, const double* h1b, const double* eri, double* ea, double* ja, double* eb,
                         uint64_t* sb, double* hdiag, cudaStream_t stream) {
  const int npair = norb * (norb + 1) / 2;
  // a warp per string up to HD_WARPS strings (us, warps against threads: 13 000
  // strings 40 and 57, 18 600 36 and 40, 26 000 56 and 45, 78 000 155 and 45,
  // 735 000 1580 and 214)
  const long long nstr = (long long)(Na + Nb);
  auto kern = nstr <= HD_WARPS ? k_string_energy<32> : k_string_energy<1>;
  kern<<<grid_for(nstr <= HD_WARPS ? nstr * 32 : nstr, 128), 128, 0, stream>>>(norb, neleca, nelecb, npair, Na, Nb, h1a,
                                                                               h1b, eri, ea, ja, eb, sb);
  const int st = check_launch("hdiag_det strings");
  if (st) return st;
  ProfScope ps_("k_hdiag_det", stream);
  const unsigned long long nx = (Na + HD_ROWS - 1) / HD_ROWS;
  // a row has to be longer than a table for the tables to pay
  if (Nb >= (1u << HD_BITS) && nx <= 0x7fffffffull) {
    // the columns are split where the rows leave the GPU idle (8 blocks a SM)
    unsigned long long ny = (148 * 8 + nx - 1) / nx, most = (Nb + 1023) / 1024;
    if (ny > most) ny = most;
    const size_t smem = (size_t)((norb + HD_BITS - 1) / HD_BITS) * HD_ROWS * (1 << HD_BITS) * sizeof(double);
    k_hdiag_det_table<<<dim3((unsigned)nx, (unsigned)ny), 256, smem, stream>>>(norb, Na, Nb, ea, eb, ja, sb, hdiag);
  } else {
    k_hdiag_det<<<grid_for((long long)(Na * Nb), 256, 148 * 32), 256, 0, stream>>>(norb, Na, Nb, ea, eb, ja, sb,
                                                                                  hdiag);
  }
  return check_launch("hdiag_det");
}

// ---------------------------------------------------------------------------
// Slater-Condon matrix elements <a1 b1|H|a2 b2> for distinct determinants
// ---------------------------------------------------------------------------
__device__ __forceinline__ double eri_at(const double* eri, int npair, int p, int q, int r, int s) {
  return eri[(int64_t)pair_index(p, q) * npair + pair_index(r, s)];
}

__device__ __forceinline__ int between_sign(unsigned long long s, int p, int q) {
  int hi = p > q ? p : q, lo = p > q ? q : p;
  unsigned long long mask = (1ull << hi) - (1ull << (lo + 1));
  return (__popcll(s & mask) & 1) ? -1 : 1;
}

__device__ double sc_element(int norb, int npair, const double* ha, const double* hb,
                             const double* eri, unsigned long long a1, unsigned long long b1,
                             unsigned long long a2, unsigned long long b2) {
  unsigned long long da = a1 ^ a2, db = b1 ^ b2;
  int nxa = __popcll(da) / 2, nxb = __popcll(db) / 2;
  if (nxa + nxb > 2) return 0.0;
  if (nxa + nxb == 1) {
    bool alpha = nxa == 1;
    unsigned long long sf = alpha ? a2 : b2, st = alpha ? a1 : b1, so = alpha ? b2 : a2;
    const double* h = alpha ? ha : hb;
    int q = __ffsll((long long)(sf & ~st)) - 1;
    int p = __ffsll((long long)(st & ~sf)) - 1;
    double v = h[p * norb + q];
    unsigned long long k = sf;
    while (k) {
      int kk = __ffsll((long long)k) - 1;
      k &= k - 1;
      v += eri_at(eri, npair, p, q, kk, kk) - eri_at(eri, npair, p, kk, kk, q);
    }
    k = so;
    while (k) {
      int kk = __ffsll((long long)k) - 1;
      k &= k - 1;
      v += eri_at(eri, npair, p, q, kk, kk);
    }
    return between_sign(sf, p, q) * v;
  }
  if (nxa == 1 && nxb == 1) {
    int q = __ffsll((long long)(a2 & ~a1)) - 1, p = __ffsll((long long)(a1 & ~a2)) - 1;
    int s = __ffsll((long long)(b2 & ~b1)) - 1, r = __ffsll((long long)(b1 & ~b2)) - 1;
    return between_sign(a2, p, q) * between_sign(b2, r, s) * eri_at(eri, npair, p, q, r, s);
  }
  // double excitation within one spin
  unsigned long long sf = nxa == 2 ? a2 : b2, st = nxa == 2 ? a1 : b1;
  unsigned long long qs = sf & ~st, ps = st & ~sf;
  int q1 = __ffsll((long long)qs) - 1;
  int q2 = 63 - __clzll((long long)qs);
  int p1 = __ffsll((long long)ps) - 1;
  int p2 = 63 - __clzll((long long)ps);
  int sgn = between_sign(sf, p1, q1);
  unsigned long long mid = (sf ^ (1ull << q1)) | (1ull << p1);
  sgn *= between_sign(mid, p2, q2);
  return sgn * (eri_at(eri, npair, p1, q1, p2, q2) - eri_at(eri, npair, p1, q2, p2, q1));
}

__global__ void k_pspace_h0(int norb, int npair, unsigned long long Nb, const double* ha,
                            const double* hb, const double* eri, const double* hd,
                            const uint32_t* addr, int neleca, int nelecb, int n, double* h0) {
  int64_t tot = (int64_t)n * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < tot;
       t += (int64_t)gridDim.x * blockDim.x) {
    int i = (int)(t / n), j = (int)(t - (int64_t)i * n);
    double v;
    if (i == j) {
      v = hd[addr[i]];
    } else {
      unsigned long long ai = addr[i] / Nb, bi = addr[i] - ai * Nb;
      unsigned long long aj = addr[j] / Nb, bj = addr[j] - aj * Nb;
      v = sc_element(norb, npair, ha, hb, eri, str_unrank(norb, neleca, ai),
                     str_unrank(norb, nelecb, bi), str_unrank(norb, neleca, aj),
                     str_unrank(norb, nelecb, bj));
    }
    h0[t] = v;
  }
}

// sigma[K] += sum over links of K: s * h[i][a] * c[target]  (gather form of
// sum_pq h_pq E_pq c; one thread owns one output element)
__global__ void k_contract_1e(int norb, unsigned long long Na, unsigned long long Nb, int nla,
                              int nlb, const double* __restrict__ ha, const double* __restrict__ hb,
                              const csffci_link_t* __restrict__ la,
                              const csffci_link_t* __restrict__ lb, const double* __restrict__ ci,
                              double* sigma) {
  unsigned long long n = Na * Nb;
  for (unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; t < n;
       t += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long ka = t / Nb, kb = t - ka * Nb;
    double acc = 0.0;
    const csffci_link_t* L = la + ka * nla;
    for (int l = 0; l < nla; ++l) {
      csffci_link_t e = L[l];
      int a = e.op & 0xff, i = e.op >> 8;
      acc += e.sign * ha[i * norb + a] * ci[(unsigned long long)e.addr * Nb + kb];
    }
    L = lb + kb * nlb;
    for (int l = 0; l < nlb; ++l) {
      csffci_link_t e = L[l];
      int a = e.op & 0xff, i = e.op >> 8;
      acc += e.sign * hb[i * norb + a] * ci[ka * Nb + e.addr];
    }
    sigma[t] += acc;
  }
}

// The same for C1_ROWS rows ka a block: their rows of c, their alpha links
// (coefficient and row) and hb in shared memory, and every beta link read once
// for all of them.  Element by element each of the nla + nlb links cost two
// dependent loads and a look at h, at 11% of the issue slots.  11 orbitals
// (6,5): 41 us, now 20 us, most of it the latency of the rows of c that the
// alpha links read from L2.
constexpr int C1_ROWS = 4;
struct C1Link {
  double v;
  long long off;
};
__global__ void __launch_bounds__(256) k_contract_1e_rows(int norb, long long Na, int Nb, int nla, int nlb,
                                                          const double* __restrict__ ha, const double* __restrict__ hb,
                                                          const csffci_link_t* __restrict__ la,
                                                          const csffci_link_t* __restrict__ lb,
                                                          const double* __restrict__ ci, double* sigma) {
  extern __shared__ __align__(16) unsigned char c1_smem[];
  double* const crow = (double*)c1_smem;                          // [C1_ROWS][Nb]
  C1Link* const al = (C1Link*)(c1_smem + (((size_t)C1_ROWS * Nb * sizeof(double) + 15) & ~(size_t)15));
  double* const hs = (double*)(al + (size_t)C1_ROWS * nla);       // [norb][norb]
  const long long r0 = (long long)blockIdx.x * C1_ROWS;
  const int nr = (int)min((long long)C1_ROWS, Na - r0);
  for (int t = threadIdx.x; t < C1_ROWS * Nb; t += blockDim.x) crow[t] = t < nr * Nb ? ci[r0 * Nb + t] : 0.0;
  for (int t = threadIdx.x; t < C1_ROWS * nla; t += blockDim.x) {
    C1Link x{0.0, 0};
    if (t < nr * nla) {
      const csffci_link_t e = la[r0 * nla + t];
      x.v = e.sign * ha[(e.op >> 8) * norb + (e.op & 0xff)];
      x.off = (long long)e.addr * Nb;
    }
    al[t] = x;
  }
  for (int t = threadIdx.x; t < norb * norb; t += blockDim.x) hs[t] = hb[t];
  __syncthreads();
  for (int kb = blockIdx.y * blockDim.x + threadIdx.x; kb < Nb; kb += gridDim.y * blockDim.x) {
    double acc[C1_ROWS];
#pragma unroll
    for (int r = 0; r < C1_ROWS; ++r) acc[r] = 0.0;
    // loads in batches of 16: left to itself the compiler waits for each
    const double* const cb = ci + kb;
    for (int l0 = 0; l0 < nla; l0 += 4) {
      double x[4][C1_ROWS];
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int r = 0; r < C1_ROWS; ++r) x[k][r] = l0 + k < nla ? __ldg(&cb[al[r * nla + l0 + k].off]) : 0.0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int r = 0; r < C1_ROWS; ++r)
          if (l0 + k < nla) acc[r] += al[r * nla + l0 + k].v * x[k][r];
    }
    // a link is two loads, not one per field: address; op, sign and pad
    const unsigned* const L = reinterpret_cast<const unsigned*>(lb + (long long)kb * nlb);
    for (int l0 = 0; l0 < nlb; l0 += 8) {
      unsigned to[8], w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        to[k] = l0 + k < nlb ? __ldg(&L[2 * (l0 + k)]) : 0u;
        w[k] = l0 + k < nlb ? __ldg(&L[2 * (l0 + k) + 1]) : 0u;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const double v = (double)((int)(w[k] << 8) >> 24) * hs[((w[k] >> 8) & 0xffu) * norb + (w[k] & 0xffu)];
#pragma unroll
        for (int r = 0; r < C1_ROWS; ++r)
          if (l0 + k < nlb) acc[r] += v * crow[r * Nb + to[k]];
      }
    }
#pragma unroll
    for (int r = 0; r < C1_ROWS; ++r)
      if (r < nr) sigma[(r0 + r) * Nb + kb] += acc[r];
  }
}

}  // namespace csffci

using namespace csffci;

extern "C" {

int csffci_absorb_h1e(int norb, int nelec, const double* h1e, const double* eri, double fac,
                      double* h2e, cudaStream_t stream) {
  CSF_REQUIRE(norb >= 1 && norb <= 63, "absorb_h1e: bad norb %d", norb);
  CSF_REQUIRE(h2e != eri, "absorb_h1e: h2e must not alias eri");
  int npair = norb * (norb + 1) / 2;
  k_absorb_h2e<<<grid_for((int64_t)npair * npair, 128), 128, 0, stream>>>(
      norb, npair, h1e, eri, 1.0 / (nelec + 1e-100), fac, h2e);
  return check_launch("absorb_h1e");
}

size_t csffci_hdiag_det_workspace(int norb, int neleca, int nelecb) {
  unsigned long long Na = host_binom(norb, neleca), Nb = host_binom(norb, nelecb);
  return (size_t)(Na * (norb + 1) + Nb) * sizeof(double) + (size_t)Nb * sizeof(uint64_t) + 256;
}

int csffci_hdiag_det(int norb, int neleca, int nelecb, const double* h1a, const double* h1b,
                     const double* eri, double* hdiag, void* work, size_t work_bytes,
                     cudaStream_t stream) {
  CSF_REQUIRE(norb >= 1 && norb <= 63 && neleca >= 0 && nelecb >= 0 && neleca <= norb &&
                  nelecb <= norb,
              "hdiag_det: bad (norb=%d, nelec=(%d,%d))", norb, neleca, nelecb);
  size_t need = csffci_hdiag_det_workspace(norb, neleca, nelecb);
  if (work == nullptr || work_bytes < need) {
    set_error("hdiag_det: workspace of %zu bytes < %zu required", work_bytes, need);
    return CSFFCI_ERR_MEMORY;
  }
  unsigned long long Na = host_binom(norb, neleca), Nb = host_binom(norb, nelecb);
  double* ea = (double*)work;
  double* ja = ea + Na;
  double* eb = ja + Na * norb;
  uint64_t* sb = (uint64_t*)(eb + Nb);
  return hdiag_det_run(norb, neleca, nelecb, Na, Nb, h1a, h1b, eri, ea, ja, eb, sb, hdiag, stream);
}

int csffci_pspace_h0(int norb, int neleca, int nelecb, const double* h1a, const double* h1b,
                     const double* eri, const double* hdiag_det, const uint32_t* det_addr, int n,
                     double* h0, cudaStream_t stream) {
  CSF_REQUIRE(norb >= 1 && norb <= 63 && n >= 0, "pspace_h0: bad arguments");
  if (n == 0) return CSFFCI_OK;
  int npair = norb * (norb + 1) / 2;
  unsigned long long Nb = host_binom(norb, nelecb);
  {
    ProfScope ps_("k_pspace_h0", stream);
    k_pspace_h0<<<grid_for((long long)n * n, 128, 148 * 32), 128, 0, stream>>>(
        norb, npair, Nb, h1a, h1b, eri, hdiag_det, det_addr, neleca, nelecb, n, h0);
  }
  return check_launch("pspace_h0");
}

int csffci_contract_1e(int norb, int neleca, int nelecb, const double* h1a, const double* h1b,
                       const csffci_link_t* link_a, const csffci_link_t* link_b, const double* ci,
                       double* sigma, cudaStream_t stream) {
  CSF_REQUIRE(norb >= 1 && norb <= 63, "contract_1e: bad norb %d", norb);
  unsigned long long Na = host_binom(norb, neleca), Nb = host_binom(norb, nelecb);
  int nla = neleca * (norb - neleca + 1), nlb = nelecb * (norb - nelecb + 1);
  // Rows that fit in shared memory (7000 columns at 16 orbitals), not for
  // narrow or flat vectors: a block has a thread per column and four rows, so
  // most of it would be idle (element-wise against by rows, us: 184756 x 1 121
  // and 644, 38760 x 20 135 and 218, 10626 x 24 65 and 75, 1 x 3432 20 and 23;
  // but 2024 x 24 25 and 20, 1770 x 60 56 and 30, 20 x 4845 46 and 36).
  const size_t smem = (((size_t)C1_ROWS * Nb * sizeof(double) + 15) & ~(size_t)15) +
                      (size_t)C1_ROWS * nla * sizeof(C1Link) + (size_t)norb * norb * sizeof(double);
  const bool wide = Nb >= 32 || (Nb >= 24 && Na <= 4096);
  if (Na >= 14 && wide && Na < (1ull << 31) && Nb < (1ull << 24) && smem <= MAX_SMEM) {
    if (smem > 48 * 1024)
      CSF_CUDA(cudaFuncSetAttribute(k_contract_1e_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM));
    const long long nx = ((long long)Na + C1_ROWS - 1) / C1_ROWS;
    // few rows: the columns are split as well
    long long ny = (2 * 148 + nx - 1) / nx, most = ((long long)Nb + 255) / 256;
    if (ny > most) ny = most;
    k_contract_1e_rows<<<dim3((unsigned)nx, (unsigned)ny), 256, smem, stream>>>(
        norb, (long long)Na, (int)Nb, nla, nlb, h1a, h1b, link_a, link_b, ci, sigma);
    return check_launch("contract_1e");
  }
  k_contract_1e<<<grid_for((long long)(Na * Nb), 256, 148 * 32), 256, 0, stream>>>(
      norb, Na, Nb, nla, nlb, h1a, h1b, link_a, link_b, ci, sigma);
  return check_launch("contract_1e");
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Determinant diagonal without any allocation and without a caller
// workspace.
//
// Some callers cannot call cudaMalloc: a host program whose device memory
// is owned entirely by another allocator (a framework's caching pool with a
// fixed budget, where a raw cudaMalloc would grow memory behind its back),
// or a latency-sensitive loop where cudaMalloc/cudaFree would synchronise
// the device.  Such callers also have no spare buffer to hand over as the
// workspace that csffci_hdiag_det needs.  This variant keeps that
// workspace in a fixed array that is part of the library image instead.
//
// The array below is CSFFCI_HDIAG_NOALLOC_MAX_DOUBLES doubles (2 MiB).  Every
// GPU that loads the library holds it until the process exits.  It fits the
// per-string tables of up to norb = 16 at half filling: Na*(norb+1) + Nb
// doubles plus Nb 64-bit strings.  Larger spaces are rejected.
// ---------------------------------------------------------------------------
static __device__ __align__(256) double g_hdiag_noalloc_scratch[CSFFCI_HDIAG_NOALLOC_MAX_DOUBLES];

namespace csffci {
namespace {
std::mutex g_noalloc_mutex;
// device address of the array per device ordinal, valid for the context
// whose unique id is g_noalloc_ctx[dev] (0: not looked up yet)
void* g_noalloc_ptr[256] = {nullptr};
unsigned long long g_noalloc_ctx[256] = {0};

// Unique id of the calling thread's current context (cuCtxGetId, reached
// through the runtime's driver entry points so that libcuda is not linked);
// 0 when it cannot be had.  Context ids are never reused within a process,
// so an id that differs from the cached one means the cached address
// belongs to a context that no longer is current (a cudaDeviceReset, or a
// context created by another library).
unsigned long long current_context_id() {
  typedef int (*get_current_fn)(void**);
  typedef int (*get_id_fn)(void*, unsigned long long*);
  static get_current_fn get_current = nullptr;
  static get_id_fn get_id = nullptr;
  static bool resolved = false;
  if (!resolved) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = (get_current_fn)f;
    f = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = (get_id_fn)f;
    resolved = true;
  }
  void* ctx = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&ctx) != 0 || ctx == nullptr || get_id(ctx, &id) != 0) return 0;
  return id;
}
}  // namespace
}  // namespace csffci

extern "C" int csffci_hdiag_det_noalloc(int norb, int neleca, int nelecb, const double* h1a,
                                        const double* h1b, const double* eri, double* hdiag,
                                        cudaStream_t stream) {
  CSF_REQUIRE(norb >= 1 && norb <= 63 && neleca >= 0 && nelecb >= 0 && neleca <= norb &&
                  nelecb <= norb,
              "hdiag_det_noalloc: bad (norb=%d, nelec=(%d,%d))", norb, neleca, nelecb);
  const unsigned long long Na = host_binom(norb, neleca), Nb = host_binom(norb, nelecb);
  const unsigned long long need = Na * (unsigned long long)(norb + 1) + 2ull * Nb;
  if (need > (unsigned long long)CSFFCI_HDIAG_NOALLOC_MAX_DOUBLES) {
    set_error("hdiag_det_noalloc: (norb=%d, nelec=(%d,%d)) needs %llu doubles of scratch, more "
              "than the fixed %d; use csffci_hdiag_det with a workspace",
              norb, neleca, nelecb, need, CSFFCI_HDIAG_NOALLOC_MAX_DOUBLES);
    return CSFFCI_ERR_MEMORY;
  }
  // The symbol's name is a host-side stand-in, not a device address: look
  // the address up once per device and context, with that device current.
  int dev = 0;
  CSF_CUDA(cudaGetDevice(&dev));
  CSF_REQUIRE(dev >= 0 && dev < 256, "hdiag_det_noalloc: device ordinal %d out of range", dev);
  void* base = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    const unsigned long long ctx = current_context_id();
    if (g_noalloc_ptr[dev] == nullptr || ctx == 0 || ctx != g_noalloc_ctx[dev]) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_hdiag_noalloc_scratch);
      if (e != cudaSuccess || p == nullptr) {
        set_error("hdiag_det_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev,
                  cudaGetErrorString(e));
        return CSFFCI_ERR_CUDA;
      }
      g_noalloc_ptr[dev] = p;
      g_noalloc_ctx[dev] = current_context_id();
    }
    base = g_noalloc_ptr[dev];
  }
  // Every entry of the scratch that the kernels read is written first by the
  // same call (ea, ja, eb and the beta strings), so nothing needs clearing.
  double* ea = (double*)base;
  double* ja = ea + Na;
  double* eb = ja + Na * norb;
  uint64_t* sb = (uint64_t*)(eb + Nb);
  return hdiag_det_run(norb, neleca, nelecb, Na, Nb, h1a, h1b, eri, ea, ja, eb, sb, hdiag, stream);
}
