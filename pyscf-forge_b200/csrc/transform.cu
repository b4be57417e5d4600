// det <-> CSF transforms and the CSF diagonal of one space.
//
// The reference works npair block by npair block: it gathers x[:, csd_mask
// block] into a (nvec*nconf, ndet) matrix, multiplies it by +-umat and scatters
// into the CSF vector (pyscf/csf_fci/csfstring.py:641-658).  Here one launch
// takes every block (transform_tile.cuh): its CTAs walk over the tasks of all
// blocks, those that share a tile (long K, few rows) first.
//
// What bounds it: the random 8-byte accesses through csd_mask (one 32-byte
// sector each), then latency.  Measured, block by block launches of 64 x 64
// GEMM tiles and a thread per configuration -> this:
//   CAS(14,14) triplet, 2 vectors  CSF->det 0.91 -> 0.34 ms, det->CSF 1.01 -> 0.25 ms
//   CAS(12,12) singlet, 3 vectors  CSF->det 0.38 -> 0.04 ms, det->CSF 0.42 -> 0.03 ms
//   CAS(16,16) singlet, 1 vector   CSF->det 4.9 -> 3.1 ms, det->CSF 3.4 -> 2.15 ms
//   CAS(14,14) triplet diagonal    2.75 -> 0.33 ms
#include <string.h>

#include "common.cuh"
#include "profile.cuh"
#include "transform_tile.cuh"

namespace csffci {

constexpr int XF_MAXB = 24;  // blocks of a launch (npair = 0..22 at norb 22)

struct XfBlock {
  const uint32_t* mask;
  const double* u;
  const double* z;
  const int32_t* sel;
  int64_t csf_off, nconf, sconf, task0;
  double sign;
  int ndet, ncsf, nspin, npair, cls, nchunk, vper;
};

struct XfArgs {
  const double* x;
  double* y;
  const double* eri;
  int64_t ldx, ldy, ntask;
  int nvec, nb, norb;
  XfBlock b[XF_MAXB];
};

// DEAL: some block's vectors are dealt out (without, one vector of 16 orbitals
// (5,4) 93 us, with 101: registers)
template <int MODE, bool DEAL>
__global__ void __launch_bounds__(XF_W * 32, 2) k_transform(const __grid_constant__ XfArgs g) {
  __shared__ double red[XF_RED];
  __shared__ double kx[MODE == XF_HDIAG ? 256 : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (MODE == XF_HDIAG) {
    const int np = g.norb * (g.norb + 1) / 2;
    for (int i = threadIdx.x; i < 256; i += XF_W * 32) {
      const int p = i >> 4, q = i & 15;
      const int pq = pair_index(p, q);
      kx[i] = p < g.norb && q < g.norb ? g.eri[(int64_t)pq * np + pq] : 0.0;
    }
    __syncthreads();
  }
  int j = 0;
  for (int64_t task = blockIdx.x; task < g.ntask; task += gridDim.x) {
    while (j + 1 < g.nb && g.b[j + 1].task0 <= task) ++j;
    const XfBlock& b = g.b[j];
    XfTile B;
    B.x = g.x;
    B.y = g.y;
    B.mask = b.mask;
    B.u = b.u;
    B.z = b.z;
    B.sel = b.sel;
    B.ldx = g.ldx;
    B.ldy = g.ldy;
    B.csf_off = b.csf_off;
    B.nconf = b.nconf;
    B.ndet = b.ndet;
    B.ncsf = b.ncsf;
    B.nvec = g.nvec;
    B.sign = b.sign;
    XfOrb o;
    o.kx = kx;
    o.norb = g.norb;
    o.npair = b.npair;
    o.nspin = b.nspin;
    o.sconf = b.sconf;
    xf_run<MODE, DEAL>(B, &o, b.cls, task - b.task0, b.nchunk, b.vper, lane, warp, red);
  }
}

// Spaces whose vectors outgrow the L2: the same tiles in an order that keeps a
// configuration's neighbours together.  All configurations with the same
// occupation (empty, single, double) of the norb / 2 upper orbitals touch the
// same small sub-matrices of the determinant vector: alpha and beta strings
// are in ascending order, so a fixed upper part is a contiguous range of
// each, tens of determinants long.  The configurations of such a group are,
// in every npair block, a rectangle of (doubly occupied string, singly
// occupied string) ranks, since both are ranked in ascending order too, and
// its size depends on the numbers of doubly and singly occupied upper
// orbitals alone; so a warp finds its group and tile from its number with a
// table of those numbers (XfUp), group after group.  Sectors are then read
// once, or completed, while they are in L2.  In block order every 8-byte
// access beyond the L2 costs its own sector: a probe with a random
// permutation gives 155 G stores/s and 210 G loads/s in 40 MB, 35 and 73 in
// 188 MB, 29 and 63 in 640 MB.
constexpr int XF_UP_MAX = 45;     // (doubly, singly) counts of up to 8 upper orbitals
constexpr int XF_UP_BLOCKS = 12;  // npair blocks
constexpr int64_t XF_UP_ELEMENTS = 8 << 20;  // 64 MiB: half of the L2
constexpr int64_t XF_L2_BYTES = 126ll << 20;
constexpr int64_t XF_TOGETHER = 12 << 20;    // 96 MiB of vectors in a launch

struct XfUp {
  int n, low, nk;  // counts in the table; lower orbitals; blocks with shared tiles (first in XfArgs)
  int64_t nkt;     // their tasks
  int64_t start[XF_UP_MAX + 1];                  // first warp task
  unsigned char d[XF_UP_MAX], s[XF_UP_MAX];      // doubly, singly occupied
  uint32_t tile[XF_UP_MAX][XF_UP_BLOCKS + 1];    // first tile of each block within a group
};

__global__ void __launch_bounds__(XF_W * 32, 2) k_csf2det_up(const __grid_constant__ XfArgs g,
                                                             const __grid_constant__ XfUp up) {
  __shared__ double red[XF_RED];
  __shared__ uint32_t bn[17][18];  // binomials (16 orbitals)
  for (int i = threadIdx.x; i < 17 * 18; i += XF_W * 32) bn[i / 18][i % 18] = (uint32_t)binom(i / 18, i % 18);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto tile_of = [&](const XfBlock& b) {
    XfTile B;
    B.x = g.x;
    B.y = g.y;
    B.mask = b.mask;
    B.u = b.u;
    B.z = nullptr;
    B.sel = nullptr;
    B.ldx = g.ldx;
    B.ldy = g.ldy;
    B.csf_off = b.csf_off;
    B.nconf = b.nconf;
    B.ndet = b.ndet;
    B.ncsf = b.ncsf;
    B.nvec = g.nvec;
    B.sign = b.sign;
    return B;
  };
  int64_t t = blockIdx.x;
  for (; t < up.nkt; t += gridDim.x) {
    int j = 0;
    while (j + 1 < up.nk && g.b[j + 1].task0 <= t) ++j;
    const XfBlock& b = g.b[j];
    const XfTile B = tile_of(b);
    if (b.cls == 4) xf_shared<XF_CSF2DET, 1>(B, nullptr, t - b.task0, b.nchunk, lane, warp, red);
    else if (b.cls == 5) xf_shared<XF_CSF2DET, 2>(B, nullptr, t - b.task0, b.nchunk, lane, warp, red);
    else xf_shared<XF_CSF2DET, 4>(B, nullptr, t - b.task0, b.nchunk, lane, warp, red);
  }
  const int nh = g.norb - up.low;
  int e = 0;
  for (int64_t w = (t - up.nkt) * XF_W + warp; w < up.start[up.n]; w += (int64_t)gridDim.x * XF_W) {
    while (up.start[e + 1] <= w) ++e;
    // group number q among those with these counts: upper strings
    const uint32_t per = up.tile[e][g.nb - up.nk];
    const uint32_t rest = (uint32_t)(w - up.start[e]);
    const uint32_t q = rest / per;
    uint32_t tl = rest - q * per;
    const int cd = up.d[e], cs = up.s[e];
    int j = 0;
    while (up.tile[e][j + 1] <= tl) ++j;
    tl -= up.tile[e][j];
    const XfBlock& b = g.b[up.nk + j];
    const int pd = b.npair - cd, ps = b.nspin - cs;
    // upper orbitals from the top: the strings of rank qd (doubly occupied)
    // and qs (singly, among the others), and with them the colex ranks of the
    // block's strings whose lower part is the first of its kind
    const uint32_t nsing = bn[nh - cd][cs];
    uint32_t qd = q / nsing, qs = q - qd * nsing, d0 = 0, s0 = 0;
    int i = cd, k = cs, f = nh - cd;
    for (int p = nh - 1; p >= 0; --p) {
      const uint32_t c = bn[p][i];
      if (i > 0 && c <= qd) {
        qd -= c;
        d0 += bn[up.low + p][pd + i--];
      } else {
        --f;
        const uint32_t cq = bn[f][k];
        if (k > 0 && cq <= qs) {
          qs -= cq;
          s0 += bn[up.low - pd + f][ps + k--];
        }
      }
    }
    const uint32_t ns = bn[up.low - pd][ps], rows = bn[up.low][pd] * ns;
    // chunks of a row tile on neighbouring warps: walking over them in one warp
    // left its sectors incomplete for longer (12.8 ms against 3.6 at CAS(16,16))
    const uint32_t mt = tl / b.nchunk, chunk = tl - mt * b.nchunk;
    uint32_t cf[1][2];
    bool in[1][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t m = mt * 16 + 8 * h + (lane >> 2);
      in[0][h] = m < rows;
      m = min(m, rows - 1);
      const uint32_t di = m / ns;
      cf[0][h] = (d0 + di) * (uint32_t)b.sconf + s0 + (m - di * ns);
    }
    const XfTile B = tile_of(b);
    if (b.cls == 0) xf_rows_tile<XF_CSF2DET, 1, 1>(B, nullptr, cf, cf, in, chunk * 8, lane);
    else if (b.cls == 1) xf_rows_tile<XF_CSF2DET, 1, 2>(B, nullptr, cf, cf, in, chunk * 16, lane);
    else xf_rows_tile<XF_CSF2DET, 1, 4>(B, nullptr, cf, cf, in, chunk * 32, lane);
  }
}

// the orbital count behind the blocks' configuration counts (0: not to be had)
static int xf_norb(const csffci_block_t* blocks, int nblock) {
  for (int n = 1; n <= 22; ++n) {
    bool ok = true, fixed = false;
    for (int b = 0; b < nblock && ok; ++b) {
      const csffci_block_t& S = blocks[b];
      if (S.npair < 0 || S.nspin < 0 || S.npair + S.nspin > n || S.conf_sel != nullptr)
        ok = false;
      else
        ok = (int64_t)(host_binom(n, S.npair) * host_binom(n - S.npair, S.nspin)) == S.nconf;
      fixed = fixed || S.npair > 0 || S.nspin > 0;
    }
    if (ok && fixed) return n;
  }
  return 0;
}

// whether the CSF->det launch of these blocks takes the upper-orbital order
// (*norb: its orbitals): vectors that outgrow the L2, and row tiles for all
// warps, since the order does not deal the vectors out (10 orbitals, 256
// vectors: 670 us, in block order 220)
static bool xf_upper(const csffci_block_t* blocks, int nblock, int nvec, int* norb) {
  int64_t ndet = 0, rows = 0;
  for (int b = 0; b < nblock; ++b) {
    ndet += blocks[b].nconf * blocks[b].ndet;
    rows += (blocks[b].nconf + 15) / 16;
  }
  if (ndet * nvec < XF_UP_ELEMENTS || nblock > XF_UP_BLOCKS || rows < XF_WARPS) return false;
  *norb = xf_norb(blocks, nblock);
  return *norb >= 8 && *norb <= 16;
}

// the table of a launch whose blocks nk.. are in the upper-orbital order
static void xf_up(XfUp& up, const XfArgs& g) {
  const int nh = g.norb / 2;
  up.low = g.norb - nh;
  up.nk = 0;
  while (up.nk < g.nb && g.b[up.nk].cls >= 4) ++up.nk;
  up.nkt = up.nk < g.nb ? g.b[up.nk].task0 : g.ntask;
  up.n = 0;
  up.start[0] = 0;
  for (int cd = 0; cd <= nh; ++cd)
    for (int cs = 0; cs + cd <= nh; ++cs) {
      const int e = up.n;
      uint32_t t = 0;
      for (int j = up.nk; j < g.nb; ++j) {
        const XfBlock& b = g.b[j];
        const int pd = b.npair - cd, ps = b.nspin - cs;
        up.tile[e][j - up.nk] = t;
        if (pd >= 0 && ps >= 0 && pd + ps <= up.low)
          t += (uint32_t)((host_binom(up.low, pd) * host_binom(up.low - pd, ps) + 15) / 16) * b.nchunk;
      }
      up.tile[e][g.nb - up.nk] = t;
      if (t == 0) continue;
      up.d[e] = (unsigned char)cd;
      up.s[e] = (unsigned char)cs;
      up.start[e + 1] = up.start[e] + (int64_t)(host_binom(nh, cd) * host_binom(nh - cd, cs)) * t;
      up.n = e + 1;
    }
}

template <int MODE>
static int run_blocks(int nvec, const double* x, int64_t ldx, double* y, int64_t ldy, const uint32_t* mask,
                      const csffci_block_t* blocks, int nblock, cudaStream_t stream, bool zeroed, int norb = 0,
                      const double* eri = nullptr) {
  int bi = 0;
  while (bi < nblock) {  // one launch unless a caller lists more than XF_MAXB blocks
    XfArgs g;
    memset(&g, 0, sizeof(g));
    g.x = x;
    g.y = y;
    g.eri = eri;
    g.ldx = ldx;
    g.ldy = ldy;
    g.nvec = nvec;
    g.norb = norb;
    const int b0 = bi;
    bi = nblock - b0 < XF_MAXB ? nblock : b0 + XF_MAXB;
    int64_t ndet = 0;
    for (int b = b0; b < bi; ++b) ndet += blocks[b].nconf * blocks[b].ndet;
    bool deal = false;
    const bool upper = MODE == XF_CSF2DET && xf_upper(blocks + b0, bi - b0, nvec, &g.norb);
    for (int pass = 0; pass < 2; ++pass)  // tiles shared by a CTA first
      for (int b = b0; b < bi; ++b) {
        const csffci_block_t& S = blocks[b];
        if (S.nconf == 0 || S.ndet == 0) continue;
        // CSF -> det writes the zeros of a block without CSFs as well, unless
        // everything has been zeroed
        if (S.ncsf == 0 && (MODE != XF_CSF2DET || zeroed)) continue;
        CSF_REQUIRE(S.umat != nullptr || S.ncsf == 0, "transform: block %d has no umat", b);
        CSF_REQUIRE(MODE != XF_HDIAG || S.nspin < 2 || S.zmat != nullptr, "hdiag_csf: block %d has no zmat", b);
        XfShape sh = xf_shape(S.nconf, nvec, MODE == XF_CSF2DET ? S.ndet : S.ncsf,
                                    MODE == XF_CSF2DET ? S.ncsf : S.ndet);
        if ((sh.cls >= 4) != (pass == 0)) continue;
        if (upper && sh.cls < 4) {  // one row tile x up to 32 columns
          const int nt = ((MODE == XF_CSF2DET ? S.ndet : S.ncsf) + 7) / 8;
          sh.cls = nt <= 1 ? 0 : nt <= 2 ? 1 : 2;
          sh.nchunk = (nt + xf_cols(sh.cls) - 1) / xf_cols(sh.cls);
          sh.ntask = 1;  // found through the table
        }
        XfBlock& d = g.b[g.nb++];
        d.mask = mask + S.csd_offset;
        d.u = S.umat;
        d.z = S.zmat;
        d.sel = S.conf_sel;
        d.csf_off = S.csf_offset;
        d.nconf = S.nconf;
        d.sconf = g.norb > 0 ? (int64_t)host_binom(g.norb - S.npair, S.nspin) : 1;
        d.sign = S.sign;
        d.ndet = S.ndet;
        d.ncsf = S.ncsf;
        d.nspin = S.nspin;
        d.npair = S.npair;
        d.cls = sh.cls;
        d.nchunk = sh.nchunk;
        d.vper = sh.vper;
        deal = deal || (sh.cls < 4 && sh.vper < nvec);
        d.task0 = g.ntask;
        g.ntask += sh.ntask;
      }
    if (g.ntask == 0) continue;
    const char* name = MODE == XF_HDIAG ? "k_hdiag_csf" : MODE == XF_CSF2DET ? "k_csf2det" : "k_det2csf";
    if (upper) {
      XfUp up;
      xf_up(up, g);
      const int64_t tasks = up.nkt + (up.start[up.n] + XF_W - 1) / XF_W;
      ProfScope ps_(name, stream);
      // beyond the L2 one CTA per SM: fewer tiles in flight, fewer sectors left
      // incomplete (CAS(16,16) 3.6 -> 3.2 ms; CAS(14,14) is faster with two)
      const int ctas = ndet * (int64_t)sizeof(double) > XF_L2_BYTES ? 1 : 2;
      k_csf2det_up<<<grid_for(tasks, 1, 148 * ctas), XF_W * 32, 0, stream>>>(g, up);
    } else {
      ProfScope ps_(name, stream);
      auto kern = MODE != XF_HDIAG && deal ? k_transform<MODE, MODE != XF_HDIAG> : k_transform<MODE, false>;
      kern<<<grid_for(g.ntask, 1, 148 * 2), XF_W * 32, 0, stream>>>(g);
    }
    const int st = check_launch("det/csf transform");
    if (st) return st;
  }
  return CSFFCI_OK;
}

__global__ void k_zero_rows(double* y, int64_t ldy, int nvec, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (int64_t)nvec * n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t v = i / n;
    y[v * ldy + (i - v * n)] = 0.0;
  }
}

// ---------------------------------------------------------------------------
// CSF diagonal: per configuration c and CSF k
//   hdiag_csf[c,k] = sum_x U[x,k]^2 hdiag_det[x] + sum_{a<b} K(S_a,S_b) Z[ab,k]
// which equals sum_xy U[x,k] H_xy U[y,k] over the within-configuration block
// of pyscf/lib/csf/csfstring.c:295-362 (H_xy = (-1)^(somos between)
// (pq|qp) for two dets that differ by exchanging the spins of SOMOs p,q);
// K(p,q) = (pq|qp) = eri[pq][pq].
// ---------------------------------------------------------------------------

struct HdiagCsfArgs {
  const double* hd;
  const double* eri;
  const uint32_t* mask;
  const double* umat;
  const double* zmat;
  double* out;
  int64_t csd_off, csf_off, nconf, sconf;
  const int32_t* conf_sel;
  int ndet, ncsf, nspin, npair, norb, npair_orb;
};

__global__ void k_hdiag_csf(HdiagCsfArgs g) {
  const int64_t n = g.nconf * g.ncsf;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ic = i / g.ncsf;  // position in the (packed) CSF vector
    const int k = (int)(i - ic * g.ncsf);
    const int64_t conf = g.conf_sel ? g.conf_sel[ic] : ic;  // configuration within the block
    double acc = 0.0;
    const uint32_t* m = g.mask + g.csd_off + conf * g.ndet;
    for (int x = 0; x < g.ndet; ++x) {
      double u = g.umat[(int64_t)x * g.ncsf + k];
      acc = fma(u * u, g.hd[m[x]], acc);
    }
    if (g.nspin >= 2) {
      int64_t dc = conf / g.sconf, sc = conf - dc * g.sconf;
      unsigned long long dstr = str_unrank(g.norb, g.npair, (unsigned long long)dc);
      unsigned long long sstr = str_unrank(g.norb - g.npair, g.nspin, (unsigned long long)sc);
      int somo[64];
      int ns = 0, isorb = 0;
      for (int iorb = 0; iorb < g.norb; ++iorb) {
        if ((dstr >> iorb) & 1ull) continue;
        if ((sstr >> isorb) & 1ull) somo[ns++] = iorb;
        ++isorb;
      }
      int ab = 0;
      for (int b = 1; b < ns; ++b)
        for (int a = 0; a < b; ++a, ++ab) {
          int pq = pair_index(somo[a], somo[b]);
          acc = fma(g.eri[(int64_t)pq * g.npair_orb + pq], g.zmat[(int64_t)ab * g.ncsf + k], acc);
        }
    }
    g.out[g.csf_off + ic * g.ncsf + k] = acc;
  }
}

}  // namespace csffci

using namespace csffci;

extern "C" {

int csffci_det2csf(int nvec, const double* x_det, int64_t ld_det, double* x_csf, int64_t ld_csf,
                   const uint32_t* csd_mask, const csffci_block_t* blocks, int nblock,
                   cudaStream_t stream) {
  CSF_REQUIRE(nvec >= 0 && blocks != nullptr && nblock >= 0, "det2csf: bad arguments");
  if (nvec == 0) return CSFFCI_OK;
  return run_blocks<XF_DET2CSF>(nvec, x_det, ld_det, x_csf, ld_csf, csd_mask, blocks, nblock,
                                  stream, false);
}

int csffci_csf2det(int nvec, const double* x_csf, int64_t ld_csf, double* x_det, int64_t ld_det,
                   int64_t ndet, const uint32_t* csd_mask, const csffci_block_t* blocks,
                   int nblock, cudaStream_t stream) {
  CSF_REQUIRE(nvec >= 0 && blocks != nullptr && nblock >= 0, "csf2det: bad arguments");
  if (nvec == 0) return CSFFCI_OK;
  // Determinants outside a selection start from zero.  Those of blocks without
  // CSFs are written as zeros by the blocks' own tasks, one sector each, unless
  // they are many and a fourth of all: a pass over the vector writes eight in
  // the time of one (18 orbitals (15,3) 2S+1 = 17, where they are 94 %, 16
  // vectors: 80 us, with the pass 37).
  bool zeroed = false;
  int64_t without = 0;
  for (int b = 0; b < nblock; ++b) {
    if (blocks[b].conf_sel != nullptr || (blocks[b].ncsf == 0 && blocks[b].nconf > 0 && blocks[b].ndet == 0))
      zeroed = true;
    if (blocks[b].ncsf == 0) without += blocks[b].nconf * blocks[b].ndet;
  }
  if (4 * without >= ndet && without * nvec >= 1 << 18) zeroed = true;
  if (zeroed) {
    {
      ProfScope ps_("k_zero_rows", stream);
      k_zero_rows<<<grid_for((int64_t)nvec * ndet, 256, 148 * 16), 256, 0, stream>>>(x_det, ld_det,
                                                                                       nvec, ndet);
    }
    int st = check_launch("csf2det zero");
    if (st) return st;
  }
  // How many vectors in a launch.  A sector is shared by several blocks, and one
  // that leaves the L2 before it is complete costs a read and a second write:
  // a vector larger than the L2 goes by itself (CAS(16,16), 4 vectors: 15.9 ms
  // together, 13.5 ms one by one), many smaller ones in launches of 64 to 96
  // MiB (12 orbitals (8,4), 64 vectors: 422 -> 160 us; 14 (10,4), 64: 1.68 ->
  // 0.92 ms; 18 (15,3), 32: 0.53 -> 0.31 ms).  Up to 192 MiB in the
  // upper-orbital order few vectors are faster together (12 (6,6), 16 vectors:
  // 160 us against 186 in halves).
  int64_t chunk = nvec;
  const int64_t all = ndet * nvec;
  int norb;
  if (ndet * (int64_t)sizeof(double) > XF_L2_BYTES) {
    chunk = 1;
  } else if (ndet < XF_UP_ELEMENTS && all > XF_TOGETHER &&
             (nvec > 32 || all > 2 * XF_TOGETHER || !xf_upper(blocks, nblock, nvec, &norb))) {
    const int64_t most = (8 * ndet <= XF_UP_ELEMENTS ? XF_UP_ELEMENTS : XF_TOGETHER) / ndet;
    const int64_t launches = (nvec + most - 1) / most;
    chunk = (nvec + launches - 1) / launches;
  }
  for (int64_t v = 0; v < nvec; v += chunk) {
    const int st = run_blocks<XF_CSF2DET>((int)(nvec - v < chunk ? nvec - v : chunk), x_csf + v * ld_csf, ld_csf,
                                          x_det + v * ld_det, ld_det, csd_mask, blocks, nblock, stream, zeroed);
    if (st) return st;
  }
  return CSFFCI_OK;
}

int csffci_hdiag_csf(int norb, int neleca, int nelecb, const double* hdiag_det, const double* eri,
                     const uint32_t* csd_mask, const csffci_block_t* blocks, int nblock,
                     double* hdiag_csf, cudaStream_t stream) {
  CSF_REQUIRE(norb >= 0 && norb <= 63 && blocks != nullptr, "hdiag_csf: bad arguments");
  if (norb <= 16)
    return run_blocks<XF_HDIAG>(1, hdiag_det, 0, hdiag_csf, 0, csd_mask, blocks, nblock, stream, false, norb, eri);
  // more than 16 orbitals (4 bits no longer name one): a thread per CSF
  int npair_orb = norb * (norb + 1) / 2;
  for (int b = 0; b < nblock; ++b) {
    const csffci_block_t& B = blocks[b];
    if (B.ncsf == 0 || B.nconf == 0) continue;
    CSF_REQUIRE(B.umat != nullptr, "hdiag_csf: block %d has no umat", b);
    CSF_REQUIRE(B.nspin < 2 || B.zmat != nullptr, "hdiag_csf: block %d has no zmat", b);
    HdiagCsfArgs g;
    g.hd = hdiag_det;
    g.eri = eri;
    g.mask = csd_mask;
    g.umat = B.umat;
    g.zmat = B.zmat;
    g.out = hdiag_csf;
    g.csd_off = B.csd_offset;
    g.csf_off = B.csf_offset;
    g.nconf = B.nconf;
    g.conf_sel = B.conf_sel;
    g.sconf = (int64_t)host_binom(norb - B.npair, B.nspin);
    g.ndet = B.ndet;
    g.ncsf = B.ncsf;
    g.nspin = B.nspin;
    g.npair = B.npair;
    g.norb = norb;
    g.npair_orb = npair_orb;
    {
      ProfScope ps_("k_hdiag_csf", stream);
      k_hdiag_csf<<<grid_for(B.nconf * B.ncsf, 128, 148 * 32), 128, 0, stream>>>(g);
    }
    int st = check_launch("hdiag_csf");
    if (st) return st;
  }
  return CSFFCI_OK;
}

}  // extern "C"
