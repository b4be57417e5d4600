// Warp tiles of the det <-> CSF transforms and of the CSF diagonal, shared by
// transform.cu (the blocks of one space) and batch.cu (job tables).
//
// Per npair block the transform is a product with umat (ndet x ncsf): rows are
// configurations of one vector, det->CSF gathers a row's determinants through
// csd_mask, CSF->det scatters the product through it.  A warp takes 16 rows (or
// two times 16) x up to 64 columns on the FP64 tensor pipe and loads its A
// fragments itself, straight from global memory: eight (or sixteen)
// independent 8-byte gathers a lane and step of 16 k, the mask of the next
// step already in flight; no shared memory and no barrier.  Consecutive warps
// work on consecutive configurations, so the sectors that neighbours share
// are likely still in L2.
// Blocks with few rows and a long K (few pairs) split K over the 8 warps of
// the CTA, partial sums added in warp order.
//
// The products of one output run over k in the same order for every column,
// so determinants whose spin functions are equal up to a sign get bitwise
// equal coefficients up to that sign (singlet vectors stay exactly symmetric).
#pragma once
#include "common.cuh"

namespace csffci {

enum { XF_DET2CSF = 0, XF_CSF2DET = 1, XF_HDIAG = 2 };

constexpr int XF_W = 8;  // warps of a CTA

// one block of one problem
struct XfTile {
  const double* x;
  double* y;
  const uint32_t* mask;  // of the block's first configuration
  const double* u;       // [ndet][ncsf]
  const double* z;       // exchange table (diagonal only)
  const int32_t* sel;    // selected configurations or NULL
  int64_t ldx, ldy, csf_off, nconf;
  int ndet, ncsf, nvec;
  double sign;
};

// what the diagonal needs of the orbitals: K_pq = (pq|qp) in shared memory and
// the strings of the block (norb <= 16)
struct XfOrb {
  const double* kx;  // [16][16]
  int norb, npair, nspin;
  int64_t sconf;
};

// Tile shape of a block: (row tiles, column tiles) of a warp, or one row tile
// x kcols column tiles of a CTA with K split over its warps.
struct XfShape {
  int cls, nchunk;  // class, column chunks
  int vper;         // vectors of a warp's tile (classes below 4)
  int64_t ntask;    // CTA tasks
};

__host__ __device__ inline int xf_rows(int cls) { return cls <= 1 ? 2 : 1; }
__host__ __device__ inline int xf_cols(int cls) {
  return cls == 0 || cls == 4 ? 1 : cls == 1 || cls == 5 ? 2 : cls == 3 ? 8 : 4;
}

constexpr int XF_WARPS = 148 * 2 * XF_W;  // of two CTAs an SM
constexpr int XF_VMAX = (1 << 14) - 1;  // vectors of a tile, as job tables hold it

inline int xf_vper(int64_t warps, int nvec) {
  const int64_t groups = warps > 0 && warps < XF_WARPS ? (XF_WARPS + warps - 1) / warps : 1;
  const int64_t per = (nvec + groups - 1) / groups;
  return (int)(per < 1 ? 1 : per > XF_VMAX ? XF_VMAX : per);
}

// nconf configurations of nvec vectors, N columns, K terms.  Up to 16 columns
// two row tiles a warp (the gathers of 32 rows in flight hide the latency of
// the few k-steps), else one row tile x 32 or 64 columns.  A tile goes over
// the vectors one by one; where the tiles are fewer than XF_WARPS, the vectors
// are dealt out among the warps (256 vectors of a 7-orbital space one after
// another took 660 us, now 20).  Where the tiles make
// fewer than four warps an SM and K is long, a CTA shares one tile: columns
// are then cut until the tiles cover the SMs twice.
inline XfShape xf_shape(int64_t nconf, int nvec, int N, int K) {
  XfShape s;
  const int64_t mt = (nconf + 15) / 16;
  const int nt = (N + 7) / 8;
  s.cls = nt <= 1 ? 0 : nt <= 2 ? 1 : nt <= 4 ? 2 : 3;
  s.nchunk = (nt + xf_cols(s.cls) - 1) / xf_cols(s.cls);
  const int64_t warps = (mt + xf_rows(s.cls) - 1) / xf_rows(s.cls) * s.nchunk;
  s.vper = xf_vper(warps, nvec);
  s.ntask = (warps * ((nvec + s.vper - 1) / s.vper) + XF_W - 1) / XF_W;
  if (warps < 148 * 4 && K >= 64) {
    const int64_t ms = (nconf * nvec + 15) / 16;
    for (s.cls = 6; s.cls > 4 && ms * ((nt + xf_cols(s.cls) - 1) / xf_cols(s.cls)) < 2 * 148; --s.cls) {
    }
    s.nchunk = (nt + xf_cols(s.cls) - 1) / xf_cols(s.cls);
    s.ntask = ms * s.nchunk;
  }
  return s;
}

// A element i = row g + 8 (i & 1), k = t + 4 (i / 2) of the step
__device__ __forceinline__ void xf_mma(double (&c)[4], const double (&a0)[4], const double (&a1)[4],
                                       const double (&b)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, "
      "{%12,%13,%14,%15}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0[0]), "d"(a1[0]), "d"(a0[1]), "d"(a1[1]), "d"(a0[2]), "d"(a1[2]), "d"(a0[3]), "d"(a1[3]), "d"(b[0]),
        "d"(b[1]), "d"(b[2]), "d"(b[3]));
}

// singly occupied orbitals of a configuration, 4 bits each
__device__ __forceinline__ unsigned long long xf_somos(const XfOrb& o, int64_t conf) {
  const int64_t dc = conf / o.sconf, sc = conf - dc * o.sconf;
  const unsigned long long dstr = str_unrank(o.norb, o.npair, (unsigned long long)dc);
  const unsigned long long sstr = str_unrank(o.norb - o.npair, o.nspin, (unsigned long long)sc);
  unsigned long long out = 0;
  int ns = 0, is = 0;
  for (int p = 0; p < o.norb; ++p) {
    if ((dstr >> p) & 1ull) continue;
    if ((sstr >> is) & 1ull) out |= (unsigned long long)p << (4 * ns++);
    ++is;
  }
  return out;
}

// B fragment of columns n0 + 8 t + g, k = kb + t + 4 j.  umat is indexed in 32
// bits without sign: at most 2^32 determinants leave a block at most 65535 spin
// determinants and no more CSFs, but 25 orbitals (20,5) have 2.15e9 entries.
template <int MODE>
__device__ __forceinline__ void xf_bfrag(const XfTile& B, const double* u, int n, int N, int kb, int k1, int tq,
                                         double (&b)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int k = kb + tq + 4 * j;
    double v = 0.0;
    if (k < k1 && n < N) v = u[MODE == XF_CSF2DET ? (uint32_t)n * (uint32_t)B.ncsf + k : (uint32_t)k * (uint32_t)B.ncsf + n];
    b[j] = MODE == XF_HDIAG ? v * v : v;
  }
}

// determinants of the rows at step kb (det->CSF and diagonal)
template <int R>
__device__ __forceinline__ void xf_load_mask(const XfTile& B, const uint32_t (&mo)[R][2], int kb, int k1, int tq,
                                             uint32_t (&d)[R][2][4]) {
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = kb + tq + 4 * j;
        d[r][h][j] = k < k1 ? B.mask[mo[r][h] + k] : 0u;
      }
}

// One vector: acc[R][NT] += the rows' products over k in [0, k1).  mo: offset
// of a row in the block's mask and d: its determinants at the first step, left
// so if more vectors follow (det->CSF), co: of its CSFs in x (CSF->det).
template <int MODE, int R, int NT>
__device__ __forceinline__ void xf_accumulate(const XfTile& B, const double* __restrict__ x, const uint32_t (&mo)[R][2],
                                              const uint32_t (&co)[R][2], int n0, int k1, bool more, int lane,
                                              uint32_t (&d)[R][2][4], double (&acc)[R][NT][4]) {
  const int gq = lane >> 2, tq = lane & 3;
  const int N = MODE == XF_CSF2DET ? B.ndet : B.ncsf;
  const double* __restrict__ u = B.u;
  for (int kb = 0; kb < k1; kb += 16) {
    double a[R][2][4];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int k = kb + tq + 4 * j;
          a[r][h][j] = k >= k1 ? 0.0 : MODE == XF_CSF2DET ? x[co[r][h] + k] : __ldcg(x + d[r][h][j]);
        }
    if (MODE != XF_CSF2DET && k1 > 16 && (kb + 16 < k1 || more))
      xf_load_mask<R>(B, mo, kb + 16 < k1 ? kb + 16 : 0, k1, tq, d);
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      double b[4];
      xf_bfrag<MODE>(B, u, n0 + 8 * t + gq, N, kb, k1, tq, b);
#pragma unroll
      for (int r = 0; r < R; ++r) xf_mma(acc[r][t], a[r][0], a[r][1], b);
    }
  }
}

// the exchange part of the diagonal: K(somo a, somo b) Z[ab][n]
template <int R, int NT>
__device__ __forceinline__ void xf_exchange(const XfTile& B, const XfOrb& o, const uint32_t (&conf)[R][2], int n0,
                                            int lane, double (&acc)[R][NT][4]) {
  const int gq = lane >> 2, tq = lane & 3;
  const int nq = o.nspin * (o.nspin - 1) / 2;
  unsigned long long so[R][2];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int h = 0; h < 2; ++h) so[r][h] = xf_somos(o, conf[r][h]);
  for (int kb = 0; kb < nq; kb += 16) {
    double a[R][2][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // ab = b (b - 1) / 2 + a, a < b
      const int k = min(kb + tq + 4 * j, nq - 1);
      int b = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)k)) * 0.5f);
      while (b * (b - 1) / 2 > k) --b;
      while ((b + 1) * b / 2 <= k) ++b;
      const int sb = 4 * b, sa = 4 * (k - b * (b - 1) / 2);
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          a[r][h][j] = kb + tq + 4 * j < nq ? o.kx[((so[r][h] >> sa) & 15) * 16 + ((so[r][h] >> sb) & 15)] : 0.0;
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      double b[4];
      xf_bfrag<XF_DET2CSF>(B, B.z, n0 + 8 * t + gq, B.ncsf, kb, nq, tq, b);
#pragma unroll
      for (int r = 0; r < R; ++r) xf_mma(acc[r][t], a[r][0], a[r][1], b);
    }
  }
}

// A warp's own tile: R times 16 configurations x 8 NT columns, vector after
// vector (nvec of them), so that a CSF->det tile reads its addresses once,
// before the first product.  cf: configuration of a row in the block's mask,
// c: its position in the (packed) CSF vector; rows that are not in repeat
// another and are not stored.
template <int MODE, int R, int NT>
__device__ __forceinline__ void xf_rows_tile(const XfTile& B, const XfOrb* orb, const uint32_t (&cf)[R][2],
                                             const uint32_t (&c)[R][2], const bool (&in)[R][2], int n0, int lane) {
  const int tq = lane & 3;
  const int N = MODE == XF_CSF2DET ? B.ndet : B.ncsf, K = MODE == XF_CSF2DET ? B.ncsf : B.ndet;
  uint32_t mo[R][2], co[R][2];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      mo[r][h] = cf[r][h] * (uint32_t)B.ndet;
      co[r][h] = c[r][h] * (uint32_t)B.ncsf;
    }
  uint32_t d[R][2][NT][2];
  if (MODE == XF_CSF2DET) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int n = n0 + 8 * t + 2 * tq + i;
            d[r][h][t][i] = n < N ? B.mask[mo[r][h] + n] : 0u;
          }
  }
  uint32_t dk[R][2][4];
  if (MODE == XF_DET2CSF) xf_load_mask<R>(B, mo, 0, K, tq, dk);
  for (int v = 0; v < B.nvec; ++v) {
    if (MODE == XF_HDIAG) xf_load_mask<R>(B, mo, 0, K, tq, dk);  // one vector
    double acc[R][NT][4];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[r][t][0] = acc[r][t][1] = acc[r][t][2] = acc[r][t][3] = 0.0;
    const double* const x = B.x + v * B.ldx + (MODE == XF_CSF2DET ? B.csf_off : 0);
    xf_accumulate<MODE, R, NT>(B, x, mo, co, n0, K, MODE == XF_DET2CSF && v + 1 < B.nvec, lane, dk, acc);
    if (MODE == XF_HDIAG && orb->nspin >= 2) xf_exchange<R, NT>(B, *orb, cf, n0, lane, acc);
    double* const y = B.y + v * B.ldy + (MODE == XF_CSF2DET ? 0 : B.csf_off);
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!in[r][h]) continue;
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int n = n0 + 8 * t + 2 * tq + i;
            const double q = MODE == XF_HDIAG ? acc[r][t][2 * h + i] : B.sign * acc[r][t][2 * h + i];
            if (n < N) y[MODE == XF_CSF2DET ? d[r][h][t][i] : co[r][h] + n] = q;
          }
      }
  }
}

// vectors v0 to v0 + n - 1 of a block alone
__device__ __forceinline__ void xf_vectors(XfTile& B, int v0, int n) {
  B.x += v0 * B.ldx;
  B.y += v0 * B.ldy;
  B.nvec = n;
}

// the w-th warp tile of a block in configuration order
template <int MODE, int R, int NT>
__device__ __forceinline__ void xf_warp(const XfTile& B, const XfOrb* orb, int64_t w, int nchunk, int lane) {
  const int64_t mt = w / nchunk * R;
  if (mt * 16 >= B.nconf) return;
  uint32_t cf[R][2], c[R][2];
  bool in[R][2];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t m = (uint32_t)(mt + r) * 16 + 8 * h + (lane >> 2);
      in[r][h] = m < (uint32_t)B.nconf;
      c[r][h] = min(m, (uint32_t)B.nconf - 1);
      cf[r][h] = B.sel ? (uint32_t)B.sel[c[r][h]] : c[r][h];
    }
  xf_rows_tile<MODE, R, NT>(B, orb, cf, c, in, (int)(w % nchunk) * 8 * NT, lane);
}

// A tile of 16 (configuration, vector) rows x 8 NT columns shared by the CTA,
// K split over its warps (red: XF_W * NT * 128 doubles of shared memory).
template <int MODE, int NT>
__device__ __forceinline__ void xf_shared(const XfTile& B, const XfOrb* orb, int64_t task, int nchunk, int lane,
                                          int warp, double* red) {
  const int64_t M = (int64_t)B.nvec * B.nconf;
  const int64_t mt = task / nchunk;
  if (mt * 16 >= M) return;  // uniform over the CTA
  const int n0 = (int)(task % nchunk) * 8 * NT;
  const int gq = lane >> 2;
  const int N = MODE == XF_CSF2DET ? B.ndet : B.ncsf, K = MODE == XF_CSF2DET ? B.ncsf : B.ndet;
  const int kw = ((K + XF_W - 1) / XF_W + 15) / 16 * 16;
  const int k0 = min(K, warp * kw), k1 = min(K, k0 + kw);
  double acc[1][NT][4];
#pragma unroll
  for (int t = 0; t < NT; ++t) acc[0][t][0] = acc[0][t][1] = acc[0][t][2] = acc[0][t][3] = 0.0;
  uint32_t mo[1][2], co[1][2], cf[1][2];
  const double* xr[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int64_t m = min(mt * 16 + 8 * h + gq, M - 1);
    const uint32_t c = (uint32_t)(m / B.nvec);
    const int v = (int)(m - (int64_t)c * B.nvec);
    cf[0][h] = B.sel ? (uint32_t)B.sel[c] : c;
    mo[0][h] = cf[0][h] * (uint32_t)B.ndet;
    co[0][h] = c * (uint32_t)B.ncsf;
    xr[h] = B.x + v * B.ldx + (MODE == XF_CSF2DET ? B.csf_off + co[0][h] : 0);
  }
  const int tq = lane & 3;
  for (int kb = k0; kb < k1; kb += 16) {
    double a[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = kb + tq + 4 * j;
        a[h][j] = k >= k1 ? 0.0 : MODE == XF_CSF2DET ? xr[h][k] : __ldcg(xr[h] + B.mask[mo[0][h] + k]);
      }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      double b[4];
      xf_bfrag<MODE>(B, B.u, n0 + 8 * t + gq, N, kb, k1, tq, b);
      xf_mma(acc[0][t], a[0], a[1], b);
    }
  }
  if (MODE == XF_HDIAG && orb->nspin >= 2 && warp == XF_W - 1) xf_exchange<1, NT>(B, *orb, cf, n0, lane, acc);
  __syncthreads();  // red of the previous task is consumed
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) red[(warp * NT * 4 + t * 4 + i) * 32 + lane] = acc[0][t][i];
  __syncthreads();
  for (int e = threadIdx.x; e < NT * 128; e += XF_W * 32) {
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < XF_W; ++q) v += red[q * NT * 128 + e];
    const int ln = e & 31, i = (e >> 5) & 3, t = e >> 7;
    const int64_t m = mt * 16 + (ln >> 2) + 8 * (i >> 1);
    const int n = n0 + 8 * t + 2 * (ln & 3) + (i & 1);
    if (m < M && n < N) {
      const int64_t c = m / B.nvec;
      double* const y = B.y + (m - c * B.nvec) * B.ldy;
      if (MODE == XF_CSF2DET)
        y[B.mask[(B.sel ? B.sel[c] : c) * B.ndet + n]] = B.sign * v;
      else
        y[B.csf_off + c * B.ncsf + n] = MODE == XF_HDIAG ? v : B.sign * v;
    }
  }
}

// A CTA task.  DEAL: B's vectors may be dealt out among the warps, group by
// group (B is changed to those of the group)
template <int MODE, bool DEAL>
__device__ __forceinline__ void xf_run(XfTile& B, const XfOrb* orb, int cls, int64_t task, int nchunk, int vper,
                                       int lane, int warp, double* red) {
  int64_t w = task * XF_W + warp;
  if (DEAL && cls < 4 && B.nvec > vper) {
    const int rows = 16 * xf_rows(cls);
    const int64_t n = (B.nconf + rows - 1) / rows * nchunk, q = w / n;
    if (q * vper >= B.nvec) return;
    w -= q * n;
    xf_vectors(B, (int)q * vper, min(vper, B.nvec - (int)q * vper));
  }
  switch (cls) {
    case 0: return xf_warp<MODE, 2, 1>(B, orb, w, nchunk, lane);
    case 1: return xf_warp<MODE, 2, 2>(B, orb, w, nchunk, lane);
    case 2: return xf_warp<MODE, 1, 4>(B, orb, w, nchunk, lane);
    case 3: return xf_warp<MODE, 1, 8>(B, orb, w, nchunk, lane);
    case 4: return xf_shared<MODE, 1>(B, orb, task, nchunk, lane, warp, red);
    case 5: return xf_shared<MODE, 2>(B, orb, task, nchunk, lane, warp, red);
    default: return xf_shared<MODE, 4>(B, orb, task, nchunk, lane, warp, red);
  }
}

constexpr int XF_RED = XF_W * 4 * 128;  // doubles of shared memory for the K split

}  // namespace csffci
