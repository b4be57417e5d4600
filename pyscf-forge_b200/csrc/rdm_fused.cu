// Fused RDM kernel: the excitation rows of a tile of determinants are built
// in shared memory and contracted there, so that T(pq, J) = <J|E_pq|c> never
// goes through global memory (norb 2..16; rdm.cu keeps the slab form for the
// rest, and for vectors of few columns or few determinants: take_fused).
//
// Rows.  For a real vector with bra == ket the ordered rows T_pq are replaced
// by S_pq = T_pq + T_qp (p > q; S_pp = T_pp) and A_pq = T_pq - T_qp.  By
// dm2[pqrs] = dm2[rspq] = dm2[qpsr] the products S.A follow from the 1-RDM
// alone (k_rdm_assemble_sa), so two triangles (npair and npair - norb rows)
// take the place of one of norb^2 rows: 0.40 of the multiplications of the
// 64 x 64 tiles of k_gram_dmma at 16 orbitals.  When moreover c = +-c^T (exactly;
// k_rdm_sym_check), T_pq of (Ja, Jb) and (Jb, Ja) agree up to that sign and
// only Jb <= Ja is formed, the diagonal scaled by sqrt(1/2).
//
// What bounds it: the FP64 tensor pipe, then the shared-memory queue that the
// movers share with it.  8 MMA warps keep every m16n8 output tile of the pass
// in registers over all determinants (a Gram matrix: the A and the B fragment
// of a row block are the same shared-memory words), and 8 mover warps fill
// the next of three stages (two at 16 orbitals): alpha rows by coalesced
// loads, beta rows from row Ja of c in shared memory.  Per 16 columns at 14
// orbitals: 98 m16n8 tiles x 4 k-steps x 32 cycles / 4 pipes = 3136 cycles of
// MMA against about 2100 of shared-memory wavefronts.
//
// Every CTA takes an equal share of the 16-column tiles; the partial sums of
// the CTAs are added in a fixed order (k_rdm_reduce), so results repeat bit
// for bit.
//
// Measured (2-RDM of one symmetric vector, slab form -> this): CAS(14,14)
// 51.2 -> 5.6 ms (74 % of the DMMA peak; without the movers' work the MMA
// warps take 4.7 ms, without the MMA the movers 3.9 ms), CAS(16,16) 900 ->
// 115 ms; spin-resolved transition densities of a norb-11 doublet 1.37 ->
// 0.86 ms.  Slower or no better: 12 MMA warps and 4 movers (6.2 ms), two
// stages (5.9 ms), 16-byte fragment loads, B fragments fetched one tile ahead
// (spills at 16 orbitals, 132 ms), m16n8k16 in place of four m16n8k4 (the
// same).
#include <math.h>
#include <string.h>

#include "rdm_fused.cuh"
#include "sigma_ws.cuh"

namespace csffci {

constexpr int RF_NB = 16;     // determinants per tile
constexpr int RF_DS = 20;     // row stride (doubles): = 4 (mod 16), conflict-free fragment loads
constexpr int RF_NMW = 8;     // MMA warps
constexpr int RF_NMOV = 8;    // mover warps
constexpr int RF_MAXT = 152;  // output tiles per pass: 19 per MMA warp
constexpr int RF_MAXCTA = 148;  // one CTA per SM
constexpr int RF_XST = 3;       // row stages (2 where shared memory is short)
constexpr int RF_LST = 4;       // link stages (3 where shared memory is short)
constexpr int RF_POLLS = 1 << 22;  // try_wait polls before a stage counts as lost

struct RFArgs {
  const csffci_link_t* la;
  const csffci_link_t* lb;
  uint2* pack;           // beta links packed per tile: [tile][link][16]
  const double* src[2];  // vector of each row set
  int spin[2];           // 1 alpha, 2 beta, 3 both
  int nsrc, sa;          // row sets; 1: S/A rows, 0: ordered rows T_pq
  long long Na, Nb;
  int norb, nla, nlb;           // nla, nlb: 0 when no set has that spin
  int rows_s, rows_e, setrows;  // first A row, end of the rows and stride of a set
  int ntile, base;              // output tiles of the pass, tiles of every MMA warp
  int xst, lst;                 // row and link stages
  const int* sym;               // device: [0] c != c^T, [1] c != -c^T (NULL: all determinants)
  double* part;
  unsigned off_l, off_crow, off_al, off_zl, off_rf, off_tab, off_bar;
  unsigned char ta[RF_MAXT], tb[RF_MAXT];  // row blocks (ta, ta + 1) x tb
};

// A link (target; creation and annihilation orbital, sign) by its documented
// fields alone and in 4-byte loads: csffci_rdm12 takes tables that are aligned
// like csffci_link_t and whose padding byte holds anything.
__device__ __forceinline__ uint2 rf_link(const csffci_link_t* p) {
  const unsigned* const w = reinterpret_cast<const unsigned*>(p);
  return make_uint2(__ldg(w), __ldg(w + 1));
}

// A link as the movers use it.  x: offset in crow (bytes) of a beta link, or
// Ka * Nb of an alpha link; y: offsets of the S (or T) row in bits 0-13 and
// of the A row in bits 14-27 (elements of a set; the spare row behind the
// set where there is no A row), sign of S in bit 31, of A in bit 30.
// T[i][a] = sign * c[target] for the link a+ i.
__device__ __forceinline__ unsigned rf_pack_rows(const RFArgs& g, uint2 e) {
  const int a = e.y & 0xff, i = (e.y >> 8) & 0xff;
  unsigned neg = rr_lneg(e);
  int rs, ra = g.rows_e;
  if (g.sa) {
    rs = pair_index(a, i);
    if (a != i) ra = g.rows_s + rs - max(a, i);
  } else {
    rs = i * g.norb + a;
  }
  return (unsigned)(rs * RF_DS) | (unsigned)(ra * RF_DS) << 14 | neg | (i < a ? neg ^ 0x80000000u : neg) >> 1;
}
__device__ __forceinline__ int rf_srow(unsigned y) { return (int)(y & 0x3fffu); }
__device__ __forceinline__ int rf_arow(unsigned y) { return (int)((y >> 14) & 0x3fffu); }
__device__ __forceinline__ unsigned rf_sneg(unsigned y) { return y & 0x80000000u; }
__device__ __forceinline__ unsigned rf_aneg(unsigned y) { return (y << 1) & 0x80000000u; }

// beta links of every 16-column tile in the order the movers read them
// (columns innermost: conflict-free reads, one contiguous copy per tile)
__global__ void k_rdm_pack_links(const __grid_constant__ RFArgs g) {
  const long long nct = (g.Nb + RF_NB - 1) / RF_NB, n = nct * g.nlb * RF_NB;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int jl = (int)(t % RF_NB), m = (int)(t / RF_NB % g.nlb);
    const long long J = t / ((long long)RF_NB * g.nlb) * RF_NB + jl;
    uint2 p = make_uint2(0u, 0u);  // past the last column: never used
    if (J < g.Nb) {
      const uint2 e = rf_link(&g.lb[J * g.nlb + m]);
      p = make_uint2(e.x * (unsigned)sizeof(double), rf_pack_rows(g, e));
    }
    g.pack[t] = p;
  }
}

__device__ __forceinline__ void rf_mma(double (&c)[4], double a0, double a1, double b) {
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b));
}

// the four k-steps of a row of this lane
__device__ __forceinline__ void rf_frag(double (&f)[4], const double* x) {
#pragma unroll
  for (int k = 0; k < 4; ++k) f[k] = x[4 * k];
}

__device__ __forceinline__ void rf_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(ws_smem_addr(bar)) : "memory");
}

// bounded wait; false when the phase never completed
__device__ __forceinline__ bool rf_wait(unsigned long long* bar, unsigned parity) {
  for (int i = 0; i < RF_POLLS; ++i)
    if (ws_mbar_try_wait(bar, parity)) return true;
  return false;
}

// tiles of rows 0..Na-1 with Jb <= Ja: rows 16m..16m+15 have m+1 tiles each
__device__ __forceinline__ long long rf_tri_tiles(long long na) {
  const long long m = na / RF_NB, r = na - m * RF_NB;
  return (RF_NB / 2) * m * (m + 1) + r * (m + 1);
}

__device__ __forceinline__ void rf_locate(long long L, bool sym, long long nct, long long* ja, int* ct) {
  if (!sym) {
    *ja = L / nct;
    *ct = (int)(L - *ja * nct);
    return;
  }
  long long m = (long long)((sqrt(1.0 + 0.5 * (double)L) - 1.0) * 0.5);
  while ((RF_NB / 2) * m * (m + 1) > L) --m;
  while ((RF_NB / 2) * (m + 1) * (m + 2) <= L) ++m;
  const long long rem = L - (RF_NB / 2) * m * (m + 1);
  *ja = RF_NB * m + rem / (m + 1);
  *ct = (int)(rem % (m + 1));
}

// The mover warps.  A shared-memory load of theirs waits 200 to 400 cycles
// behind the fragment loads of the MMA warps, so each lane keeps what it needs
// of a row's alpha links in registers, and the alpha values (global) and the
// beta links with their values of row Ja (shared) of the next tile are loaded
// before this tile's hand-over: between two hand-overs only the stores, one
// round of row loads and one barrier remain.  The packed links of a tile come
// by one bulk copy, issued lst - 1 tiles ahead (they depend on the columns
// alone).  RU links of each spin are held per lane, further ones take a plain
// loop.  Barriers (bar): stage full, stage empty (RF_XST each), links of a
// tile arrived (RF_LST); named barrier 5 among the movers.
template <int RU, int NS>
__device__ __forceinline__ bool rf_movers(const RFArgs& g, unsigned char* smraw, bool sym, long long L0, long long L1,
                                          int mtid, int lane, int mw) {
  constexpr int MTH = RF_NMOV * 32, MPASS = RF_NMOV * 2;
  constexpr int RZ = 4;  // zero rows a lane handles together
  constexpr int RB = 3;  // beta links whose rows are updated together
  double* const X = (double*)smraw;
  unsigned char* const Lb = smraw + g.off_l;
  unsigned char* const crow = smraw + g.off_crow;
  uint2* const al = (uint2*)(smraw + g.off_al);
  int* const zl = (int*)(smraw + g.off_zl);
  int* const rf = (int*)(smraw + g.off_rf);
  unsigned long long* const bar = (unsigned long long*)(smraw + g.off_bar);
  __shared__ int nz_s;
  const int xset = g.setrows * RF_DS, xs = NS * xset;
  const int nla = g.nla, nlb = g.nlb, sa = g.sa;
  const unsigned lbytes = RF_NB * nlb * (unsigned)sizeof(uint2);
  const int jl = mtid & (RF_NB - 1), ml = mtid / RF_NB;
  const int zrow = mtid >> 3, zc = 2 * (mtid & 7);  // 16-byte zero stores
  const long long Nb = g.Nb;
  const long long nct = (Nb + RF_NB - 1) / RF_NB;
  const bool a0 = g.spin[0] & 1, a1 = NS == 2 && (g.spin[1] & 1);
  const bool b0 = g.spin[0] & 2, b1 = NS == 2 && (g.spin[1] & 2);
  const bool one = g.src[0] == g.src[NS - 1];
  const double* const src0 = g.src[0];
  const double* const src1 = g.src[NS - 1];
  // row Ja of the second set's vector behind the first's, or the same
  const unsigned c1 = b0 && b1 && !one ? (unsigned)(Nb * sizeof(double)) : 0u;
  bool ok = true;
  long long ja;
  int ct;
  rf_locate(L0, sym, nct, &ja, &ct);
  int it = 0;
  // thread 0 walks over the tiles ahead of the others: tile pc of row pja is
  // the next whose links are copied, into link stage ps
  long long pL = L0, pja = ja;
  int pc = ct, ps = 0;
  auto issue_links = [&]() {
    if (mtid != 0 || nlb == 0 || pL >= L1) return;
    ws_mbar_expect_tx(&bar[2 * RF_XST + ps], lbytes);
    ws_bulk_g2s(Lb + ps * lbytes, g.pack + (long long)pc * RF_NB * nlb, lbytes, &bar[2 * RF_XST + ps]);
    ++pL;
    if (++ps == g.lst) ps = 0;
    if ((long long)(++pc) * RF_NB >= (sym ? pja + 1 : Nb)) {
      pc = 0;
      ++pja;
    }
  };
  for (int i = 1; i < g.lst; ++i) issue_links();
  int s = 0;         // row stage of the current tile
  unsigned sph = 0;  // and its phase
  int ls = 0, lcur = 0;  // link stage of the next tile and of this one
  unsigned lph = 0;      // phase of the next tile's stage
  unsigned ax[RU], ay[RU], by[RU];
  double va[NS][RU], bv[NS][RU];
#pragma unroll
  for (int k = 0; k < RU; ++k) by[k] = 0u;
  for (long long L = L0; L < L1; ++ja, ct = 0) {
    const long long jend = sym ? ja + 1 : Nb;
    const int nrow = (int)((jend + RF_NB - 1) / RF_NB);
    const int cend = (int)min((long long)nrow, ct + (L1 - L));
    L += cend - ct;
    ws_bar_sync(5, MTH);  // the previous row is consumed
    for (int r = mtid; r < g.rows_e; r += MTH) rf[r] = 0;
    // row Ja of the vectors whose beta excitations are formed
    if (b0 || b1) {
      const double* const r0 = (b0 ? src0 : src1) + ja * Nb;
      for (long long i = mtid; i < Nb; i += MTH) cp_async8(crow + i * sizeof(double), &r0[i]);
      if (c1)
        for (long long i = mtid; i < Nb; i += MTH) cp_async8(crow + c1 + i * sizeof(double), &src1[ja * Nb + i]);
    }
    cp_async_commit();
    ws_bar_sync(5, MTH);
    for (int l = mtid; l < nla; l += MTH) {
      const uint2 e = rf_link(&g.la[ja * nla + l]);
      const unsigned y = rf_pack_rows(g, e);
      rf[rf_srow(y) / RF_DS] = 1;
      if (rf_arow(y) < g.rows_e * RF_DS) rf[rf_arow(y) / RF_DS] = 1;
      al[l] = make_uint2(e.x * (unsigned)Nb, y);
    }
    ws_bar_sync(5, MTH);  // row flags and alpha links
#pragma unroll
    for (int k = 0; k < RU; ++k) {
      const int l = ml + k * MPASS;
      const uint2 e = l < nla ? al[l] : make_uint2(0u, 0u);
      ax[k] = e.x;
      ay[k] = e.y;
    }
    auto load_alpha = [&](int c) {
      const long long j = (long long)c * RF_NB + jl;
#pragma unroll
      for (int k = 0; k < RU; ++k) {
        const bool in = ml + k * MPASS < nla && j < jend;
        if (a0) va[0][k] = in ? src0[ax[k] + j] : 0.0;
        if (a1) va[NS - 1][k] = in ? src1[ax[k] + j] : 0.0;
      }
    };
    load_alpha(ct);
    if (mw == 0) {  // the rows of a set without an alpha link
      int n = 0;
      for (int b = 0; b < g.rows_e; b += 32) {
        const int r = b + lane;
        const bool z = r < g.rows_e && !rf[r];
        const unsigned bal = __ballot_sync(0xffffffffu, z);
        if (z) zl[n + __popc(bal & ((1u << lane) - 1u))] = r * RF_DS;
        n += __popc(bal);
      }
      if (lane == 0) nz_s = n;
    }
    cp_async_wait_all();
    ws_bar_sync(5, MTH);
    const int nzero = nz_s;
    // links of the next tile and their values of row Ja
    auto load_beta = [&]() {
      if (nlb == 0) return;
      if (ok) ok = rf_wait(&bar[2 * RF_XST + ls], lph);
      const uint2* const Lt = (const uint2*)(Lb + ls * lbytes) + jl;
      unsigned bx[RU];
#pragma unroll
      for (int k = 0; k < RU; ++k) {
        const uint2 e = ml + k * MPASS < nlb ? Lt[(ml + k * MPASS) * RF_NB] : make_uint2(0u, 0u);
        bx[k] = e.x;
        by[k] = e.y;
      }
#pragma unroll
      for (int k = 0; k < RU; ++k) {
        bv[0][k] = *reinterpret_cast<const double*>(crow + bx[k]);
        if (b1 && c1) bv[NS - 1][k] = *reinterpret_cast<const double*>(crow + c1 + bx[k]);
      }
      lcur = ls;
      if (++ls == g.lst) {
        ls = 0;
        lph ^= 1;
      }
    };
    load_beta();
    for (int c = ct; c < cend; ++c, ++it) {
      const long long j0 = (long long)c * RF_NB;
      const int nc = (int)min((long long)RF_NB, jend - j0);
      int zr[RZ];
#pragma unroll
      for (int k = 0; k < RZ; ++k) {
        const int i = zrow + k * (RF_NMOV * 4);
        zr[k] = i < nzero ? zl[i] : -1;
      }
      if (it >= g.xst && ok) ok = rf_wait(&bar[RF_XST + s], sph ^ 1);  // the MMA warps are done with this stage
      double* const Xt = X + s * xs;
#pragma unroll
      for (int q = 0; q < NS; ++q) {
        double* const D = Xt + q * xset;
        if (q ? a1 : a0) {
          auto put = [&](unsigned y, double v) {
            D[rf_srow(y) + jl] = rr_flip(v, rf_sneg(y));
            if (sa) D[rf_arow(y) + jl] = rr_flip(v, rf_aneg(y));
          };
#pragma unroll
          for (int k = 0; k < RU; ++k)
            if (ml + k * MPASS < nla) put(ay[k], va[q][k]);
          for (int l = ml + RU * MPASS; l < nla; l += MPASS) {
            const uint2 e = al[l];
            put(e.y, jl < nc ? (q ? src1 : src0)[e.x + j0 + jl] : 0.0);
          }
#pragma unroll
          for (int k = 0; k < RZ; ++k)
            if (zr[k] >= 0) *reinterpret_cast<double2*>(&D[zr[k] + zc]) = make_double2(0.0, 0.0);
          for (int i = zrow + RZ * (RF_NMOV * 4); i < nzero; i += RF_NMOV * 4)
            *reinterpret_cast<double2*>(&D[zl[i] + zc]) = make_double2(0.0, 0.0);
        } else {
          for (int r = zrow; r < g.rows_e; r += RF_NMOV * 4)
            *reinterpret_cast<double2*>(&D[r * RF_DS + zc]) = make_double2(0.0, 0.0);
        }
      }
      if (c + 1 < cend) load_alpha(c + 1);
      ws_bar_sync(5, MTH);  // alpha rows and zeros are in place, links of tile it-1 consumed
      issue_links();
#pragma unroll
      for (int q = 0; q < NS; ++q) {
        if (!(q ? b1 : b0) || jl >= nc) continue;
        double* const D = Xt + q * xset + jl;
        const unsigned cq = q ? c1 : 0u;
        // distinct links of a column have distinct pairs, so the
        // read-modify-writes of a pass do not overlap (but for the spare
        // row): every load is issued before the first store
#pragma unroll
        for (int k0 = 0; k0 < RU; k0 += RB) {
          double ds[RB], da[RB];
#pragma unroll
          for (int k = 0; k < RB; ++k)
            if (k0 + k < RU) {
              ds[k] = D[rf_srow(by[k0 + k])];
              if (sa) da[k] = D[rf_arow(by[k0 + k])];
            }
#pragma unroll
          for (int k = 0; k < RB; ++k)
            if (k0 + k < RU && ml + (k0 + k) * MPASS < nlb) {
              const unsigned y = by[k0 + k];
              const double v = (q && c1 ? bv[NS - 1] : bv[0])[k0 + k];
              D[rf_srow(y)] = ds[k] + rr_flip(v, rf_sneg(y));
              if (sa) D[rf_arow(y)] = da[k] + rr_flip(v, rf_aneg(y));
            }
        }
        const uint2* const Lt = (const uint2*)(Lb + lcur * lbytes) + jl;
        for (int m = ml + RU * MPASS; m < nlb; m += MPASS) {
          const uint2 e = Lt[m * RF_NB];
          const double v = *reinterpret_cast<const double*>(crow + cq + e.x);
          D[rf_srow(e.y)] += rr_flip(v, rf_sneg(e.y));
          if (sa) D[rf_arow(e.y)] += rr_flip(v, rf_aneg(e.y));
        }
      }
      if (sym && ja >= j0 && ja < j0 + RF_NB) {
        // the diagonal determinant (Ja, Ja) counts once, the others twice:
        // the sums are doubled at the end, so its column gets sqrt(1/2)
        ws_bar_sync(5, MTH);
        double* const D = Xt + (int)(ja - j0);
        for (int r = mtid; r < g.rows_e; r += MTH) D[r * RF_DS] *= 0.70710678118654752440;
      }
      __syncwarp();
      if (lane == 0) rf_arrive(&bar[s]);  // this warp's part of the tile is ready
      if (++s == g.xst) {
        s = 0;
        sph ^= 1;
      }
      if (c + 1 < cend) load_beta();
    }
  }
  return ok;
}

// BASE tiles per MMA warp, one more for the first ntile - RF_NMW * BASE
// warps.  The MMA warps wait for a stage one by one (mbarrier), so a warp
// that is done early starts the next tile while the others finish.  SPLIT:
// registers re-split between the roles (setmaxnreg): launched with 128 per
// thread, 512 threads, MMA warps 8 (BASE + 1) + 40 and at most 184, movers the
// rest of 256 (144 and 112 at 14 orbitals, 184 and 72 at 16).
template <int BASE, bool SPLIT, int NS>
__global__ void __launch_bounds__((RF_NMW + RF_NMOV) * 32, 1) k_rdm_fused(const __grid_constant__ RFArgs g) {
  constexpr int NTH = (RF_NMW + RF_NMOV) * 32;
  constexpr int NT = BASE + 1;
  // the accumulators, one strip's A and B fragments and addresses; the movers get the rest
  constexpr int REG_MMA = 8 * NT + 40 > 184 ? 184 : (8 * NT + 40 + 7) / 8 * 8, REG_MOV = 256 - REG_MMA;
  static_assert(!SPLIT || (NTH == 512 && RF_NMW * 32 * REG_MMA + RF_NMOV * 32 * REG_MOV <= NTH * 128 &&
                           REG_MMA >= 128 && REG_MOV >= 24),
                "the re-split registers fit in the launch's allocation");
  extern __shared__ __align__(16) unsigned char smraw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* const X = (double*)smraw;
  int2* const tab = (int2*)(smraw + g.off_tab);
  unsigned long long* const bar = (unsigned long long*)(smraw + g.off_bar);
  __shared__ int bad_s;
  const int xs = NS * g.setrows * RF_DS;
  for (int i = tid; i < g.xst * xs; i += NTH) X[i] = 0.0;  // pad rows stay zero
  const int extra = g.ntile - RF_NMW * BASE;
  for (int i = tid; i < RF_NMW * NT; i += NTH) {
    const int w = i / NT, t = i - w * NT;
    const int k = w * BASE + min(w, extra) + t;
    int2 o = make_int2(-1, 0);
    if (t < BASE + (w < extra ? 1 : 0)) {
      o.x = (t > 0 && g.ta[k] == g.ta[k - 1]) ? -1 : g.ta[k] * 8 * RF_DS;
      o.y = g.tb[k] * 8 * RF_DS;
    }
    tab[i] = o;
  }
  if (tid == 0) {
    bad_s = 0;
    for (int i = 0; i < RF_XST; ++i) {
      ws_mbar_init(&bar[i], RF_NMOV);
      ws_mbar_init(&bar[RF_XST + i], RF_NMW);
    }
    for (int i = 0; i < RF_LST; ++i) ws_mbar_init(&bar[2 * RF_XST + i], 1);
    ws_mbar_init_fence();
  }
  const bool sym = g.sym != nullptr && (g.sym[0] == 0 || g.sym[1] == 0);
  const long long total = sym ? rf_tri_tiles(g.Na) : g.Na * ((g.Nb + RF_NB - 1) / RF_NB);
  const long long L0 = total * blockIdx.x / gridDim.x, L1 = total * (blockIdx.x + 1) / gridDim.x;
  __syncthreads();

  if (warp < RF_NMW) {
    if constexpr (SPLIT) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(REG_MMA));
    const int gq = lane >> 2, tq = lane & 3;
    const bool more = warp < extra;
    double acc[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0;
    const int2* const wt = tab + warp * NT;
    const int n = (int)(L1 - L0);
    bool ok = true;
    int s = 0;
    unsigned ph = 0;
    for (int it = 0; it < n; ++it) {
      if (ok) ok = rf_wait(&bar[s], ph);
      const double* Xs = X + s * xs + gq * RF_DS + tq;
      double a0[4], a1[4];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        if (t < BASE || more) {
          const int2 o = wt[t];
          if (t == 0 || o.x >= 0) {  // a new strip
            rf_frag(a0, Xs + o.x);
            rf_frag(a1, Xs + o.x + 8 * RF_DS);
          }
          double b[4];
          rf_frag(b, Xs + o.y);
#pragma unroll
          for (int k = 0; k < 4; ++k) rf_mma(acc[t], a0[k], a1[k], b[k]);
        }
      }
      __syncwarp();
      if (lane == 0) rf_arrive(&bar[RF_XST + s]);  // this warp is done with the stage
      if (++s == g.xst) {
        s = 0;
        ph ^= 1;
      }
    }
    // a lost stage (its copies never arrived) shows as NaN
    const double scale = ok ? (sym ? 2.0 : 1.0) : __longlong_as_double(0x7ff8000000000000ll);
    double* P = g.part + ((size_t)blockIdx.x * g.ntile + warp * BASE + min(warp, extra)) * 128 + 4 * lane;
#pragma unroll
    for (int t = 0; t < NT; ++t)
      if (t < BASE || more) {
        double2* q = reinterpret_cast<double2*>(P + t * 128);
        q[0] = make_double2(scale * acc[t][0], scale * acc[t][1]);
        q[1] = make_double2(scale * acc[t][2], scale * acc[t][3]);
      }
  } else {
    if constexpr (SPLIT) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(REG_MOV));
    // groups of 16 links a lane holds: five for one row set at 13 to 15 orbitals,
    // where a spin has up to 49, 56 and 64 links (four would hold them; not
    // measured), else three, and the plain loops take the links beyond
    if (!rf_movers<(NS == 1 && BASE >= 8 && BASE < 16) ? 5 : 3, NS>(g, smraw, sym, L0, L1, tid - RF_NMW * 32, lane, warp - RF_NMW)) bad_s = 1;
  }
  __syncthreads();  // the partial sums of this CTA are written
  if (bad_s && tid == 0) g.part[(size_t)blockIdx.x * g.ntile * 128] = __longlong_as_double(0x7ff8000000000000ll);
}

// out[i][j] = sum over the CTAs of the partial tiles, in CTA order; with
// mirror also out[j][i].  The second row block of a strip at the end of a
// row group belongs to the next group (or the spare block): not written.
__global__ void k_rdm_reduce(const __grid_constant__ RFArgs g, int ncta, int ld, int mirror, double* out) {
  const int nel = g.ntile * 128;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nel; e += gridDim.x * blockDim.x) {
    const int k = e >> 7, lane = (e & 127) >> 2, v = e & 3;
    const int row0 = g.ta[k] * 8, row = row0 + (lane >> 2) + 8 * (v >> 1);
    const int col = g.tb[k] * 8 + 2 * (lane & 3) + (v & 1);
    const int set = row0 / g.setrows, in = row0 - set * g.setrows;
    if (row >= set * g.setrows + (in < g.rows_s ? g.rows_s : g.rows_e)) continue;
    double s = 0.0;
    const double* p = g.part + e;
#pragma unroll 8
    for (int b = 0; b < ncta; ++b) s += p[(size_t)b * nel];
    out[(size_t)row * ld + col] = s;
    if (mirror) out[(size_t)col * ld + row] = s;
  }
}

// bad[0] |= (c != c^T), bad[1] |= (c != -c^T), 32 x 32 tiles on and above
// the diagonal; a block stops once both are set.  One thread of a block
// stores a flag, and only when it reads it clear: with a store by every warp
// and tile, the stores to the one word took 0.45 ms at 14 orbitals.
__global__ void __launch_bounds__(256) k_rdm_sym_check(const double* __restrict__ c, long long n, int* bad) {
  __shared__ double tile[32][33];
  __shared__ int known[2];
  const long long nt = (n + 31) / 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (long long t = blockIdx.x; t < nt * nt; t += gridDim.x) {
    const long long ti = t / nt, tj = t - ti * nt;
    if (tj < ti) continue;
    if (ty == 0 && tx < 2) known[tx] = *(volatile int*)&bad[tx];
    double x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long row = tj * 32 + ty + 8 * k, col = ti * 32 + tx;
      tile[ty + 8 * k][tx] = (row < n && col < n) ? c[row * n + col] : 0.0;
      const long long r2 = ti * 32 + ty + 8 * k, c2 = tj * 32 + tx;
      x[k] = (r2 < n && c2 < n) ? c[r2 * n + c2] : 0.0;
    }
    __syncthreads();
    const bool kp = known[0] != 0, km = known[1] != 0;
    if (kp && km) return;
    bool bp = false, bm = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double y = tile[tx][ty + 8 * k];
      bp |= !(x[k] == y);
      bm |= !(x[k] == -y);
    }
    const int anyp = __syncthreads_or(bp), anym = __syncthreads_or(bm);
    if (tx == 0 && ty == 0) {
      if (anyp && !kp && *(volatile int*)&bad[0] == 0) bad[0] = 1;
      if (anym && !km && *(volatile int*)&bad[1] == 0) bad[1] = 1;
    }
  }
}

// Assembly of one same-kind block (spin-summed, alpha-alpha or beta-beta,
// bra == ket) from its S/A Gram matrices, N electrons of that kind:
//   D_pq   = <E_pq> = 1/(2N) sum_r f_pq S_pq.S_rr          (f_pp = 2, else 1)
//   dm2[x][y][r][s] = (f_yx f_rs S_yx.S_rs + t_yx t_rs A_yx.A_rs) / 4
//                     - (d_yr D_xs + d_xs D_yr) / 2        (t = +-1: p > q or not)
// which follows from T_pq.T_rs = dm2[qprs] + d_pr D_qs and
// dm2[qprs] = dm2[pqsr].
__device__ __forceinline__ double rf_d1(const double* M, int ld, int n, double half_inv_n, int p, int q) {
  const double* row = M + (size_t)pair_index(p, q) * ld;
  double v = 0.0;
  for (int r = 0; r < n; ++r) v += row[pair_index(r, r)];
  return v * half_inv_n * (p == q ? 2.0 : 1.0);
}

// one: a block of one spin, whose x+ r+ s y vanishes for x = r and for y = s.
// pairs: 0 below two electrons of that kind, else 1.  Such terms cancel but for
// rounding and are set to zero (NaN stays).
__global__ void k_rdm_assemble_sa(int n, const double* __restrict__ M, int ld, int rows_s, double half_inv_n, bool one,
                                  double pairs, double* dm1, double* dm2) {
  const int n2 = n * n;
  const long long tot = (long long)n2 * n2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < tot;
       t += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(t / ((long long)n * n2)), y = (int)((t / n2) % n), r = (int)((t / n) % n), s = (int)(t % n);
    const int a = pair_index(x, y), b = pair_index(r, s);
    double v = M[(size_t)a * ld + b] * (x == y ? 2.0 : 1.0) * (r == s ? 2.0 : 1.0);
    if (x != y && r != s) {
      const double w = M[(size_t)(rows_s + a - max(x, y)) * ld + rows_s + b - max(r, s)];
      v += ((y > x) == (r > s)) ? w : -w;
    }
    v *= 0.25;
    if (y == r) v -= 0.5 * rf_d1(M, ld, n, half_inv_n, x, s);
    if (x == s) v -= 0.5 * rf_d1(M, ld, n, half_inv_n, y, r);
    dm2[t] = (one && (x == r || y == s) ? 0.0 : pairs) * v;
    if (t < n2) dm1[t] = rf_d1(M, ld, n, half_inv_n, (int)(t / n), (int)(t % n));
  }
}

// alpha-beta block of one vector: E^a and E^b commute, so no 1-RDM terms
// and S.A = 0
__global__ void k_rdm_assemble_sa_ab(int n, const double* __restrict__ M, int ld, int rows_s, int col0, double* dm2) {
  const int n2 = n * n;
  const long long tot = (long long)n2 * n2;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < tot;
       t += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(t / ((long long)n * n2)), y = (int)((t / n2) % n), r = (int)((t / n) % n), s = (int)(t % n);
    const int a = pair_index(x, y), b = pair_index(r, s);
    double v = M[(size_t)a * ld + col0 + b] * (x == y ? 2.0 : 1.0) * (r == s ? 2.0 : 1.0);
    if (x != y && r != s) {
      const double w = M[(size_t)(rows_s + a - max(x, y)) * ld + col0 + rows_s + b - max(r, s)];
      v += ((y > x) == (r > s)) ? w : -w;
    }
    dm2[t] = 0.25 * v;
  }
}

// ---- host side ----------------------------------------------------------

// rows of a set and the shared-memory carve-up; returns the bytes, 0 when
// the tiles do not fit
static size_t rf_layout(RFArgs& g) {
  const int n = g.norb, npair = n * (n + 1) / 2;
  auto up8 = [](int v) { return (v + 7) & ~7; };
  g.rows_s = g.sa ? up8(npair) : up8(n * n);
  g.rows_e = g.rows_s + (g.sa ? up8(npair - n) : 0);
  g.setrows = g.rows_e + 8;  // a spare block: links without an A row, second block of an odd strip
  int nrowc = 0;
  for (int q = 0; q < g.nsrc; ++q)
    if ((g.spin[q] & 2) && !(q && (g.spin[0] & 2) && g.src[q] == g.src[0])) ++nrowc;
  size_t off = 0;
  auto take = [&](size_t b) {
    const size_t o = off;
    off += (b + 15) & ~(size_t)15;
    return (unsigned)o;
  };
  static const int stages[][2] = {{3, 4}, {3, 3}, {2, 4}, {2, 3}, {2, 2}};
  for (const auto& st : stages) {
    g.xst = st[0];
    g.lst = st[1];
    off = 0;
    take((size_t)g.xst * g.nsrc * g.setrows * RF_DS * sizeof(double));
    g.off_l = take((size_t)g.lst * RF_NB * g.nlb * sizeof(uint2));
    g.off_crow = take((size_t)nrowc * g.Nb * sizeof(double));
    g.off_al = take((size_t)(g.nla > 0 ? g.nla : 1) * sizeof(uint2));
    g.off_zl = take((size_t)g.rows_e * sizeof(int));
    g.off_rf = take((size_t)g.rows_e * sizeof(int));
    g.off_tab = take((size_t)(RF_MAXT + RF_NMW) * sizeof(int2));
    g.off_bar = take((2 * RF_XST + RF_LST) * sizeof(unsigned long long));
    if (off <= MAX_SMEM) return off;
  }
  return 0;
}

static RFArgs rf_args(const RdmFusedJob& j) {
  RFArgs g;
  memset(&g, 0, sizeof(g));
  g.la = j.la;
  g.lb = j.lb;
  g.nsrc = j.nsrc;
  g.sa = j.sa;
  int spins = 0;
  for (int q = 0; q < 2; ++q) {
    g.src[q] = j.src[q];
    g.spin[q] = j.spin[q];
    if (q < j.nsrc) spins |= j.spin[q];
  }
  g.Na = j.Na;
  g.Nb = j.Nb;
  g.norb = j.norb;
  g.nla = (spins & 1) ? j.nla : 0;
  g.nlb = (spins & 2) ? j.nlb : 0;
  g.sym = j.sym;
  return g;
}

template <int BASE, int NS>
static int rf_launch(const RFArgs& g, int grid, size_t smem, cudaStream_t stream) {
  // from 10 tiles per warp the accumulators need the re-split registers
  constexpr bool SPLIT = BASE >= 10;
  auto kern = k_rdm_fused<BASE, SPLIT, NS>;
  if (SPLIT) {
    // the raise of the MMA warps needs the 128 registers per thread that
    // the launch is sized for; with fewer it would wait forever
    cudaFuncAttributes fa;
    CSF_CUDA(cudaFuncGetAttributes(&fa, kern));
    if (fa.numRegs != 128) {
      set_error("rdm: fused kernel compiled to %d registers per thread, not 128", fa.numRegs);
      return CSFFCI_ERR_INVALID;
    }
  }
  CSF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM));
  ProfScope ps("k_rdm_fused", stream);
  kern<<<grid, (RF_NMW + RF_NMOV) * 32, smem, stream>>>(g);
  return check_launch("rdm (fused)");
}

static int rf_dispatch(RFArgs& g, int grid, size_t smem, cudaStream_t stream) {
  g.base = g.ntile / RF_NMW;
#define RF_CASE(B, N) \
  case B: return rf_launch<B, N>(g, grid, smem, stream)
  if (g.nsrc == 1) switch (g.base) {  // one triangle pair per orbital count
      RF_CASE(0, 1);   // up to 6
      RF_CASE(1, 1);   // 7, 8
      RF_CASE(2, 1);   // 9
      RF_CASE(3, 1);   // 10
      RF_CASE(5, 1);   // 11
      RF_CASE(6, 1);   // 12
      RF_CASE(9, 1);   // 13
      RF_CASE(12, 1);  // 14
      RF_CASE(15, 1);  // 15
      RF_CASE(18, 1);  // 16
      default: break;
    }
  else switch (g.base) {  // those of one, two, three or four passes at 2 to 16 orbitals
      RF_CASE(0, 2);
      RF_CASE(1, 2);
      RF_CASE(2, 2);
      RF_CASE(3, 2);
      RF_CASE(4, 2);
      RF_CASE(5, 2);
      RF_CASE(8, 2);
      RF_CASE(9, 2);
      RF_CASE(10, 2);
      RF_CASE(11, 2);
      RF_CASE(13, 2);
      RF_CASE(15, 2);
      RF_CASE(16, 2);
      RF_CASE(17, 2);
      RF_CASE(18, 2);
      default: break;
    }
#undef RF_CASE
  set_error("rdm: no fused kernel for %d tiles of %d row sets", g.ntile, g.nsrc);
  return CSFFCI_ERR_INVALID;
}

struct RFTile {
  unsigned char a, b;
};

// strips of two row blocks [a, a + 1] x b over a group of blocks [a0, a1) x
// [b0, b1); tri: b from a on (a0 == b0, a1 == b1)
static int rf_strips(RFTile* t, int n, int a0, int a1, int b0, int b1, bool tri) {
  for (int a = a0; a < a1; a += 2)
    for (int b = tri ? a : b0; b < b1; ++b) {
      t[n].a = (unsigned char)a;
      t[n++].b = (unsigned char)b;
    }
  return n;
}

constexpr int RF_MAX_ALL = 1200;  // tiles of one Gram: 32 x 64 / 2 and spare

// the output tiles of a Gram, after rf_layout
static int rf_tiles(const RFArgs& g, RFTile* tiles) {
  int n = 0;
  const int bs = g.rows_s / 8, be = g.rows_e / 8, bw = g.setrows / 8;
  if (g.nsrc == 1) {  // S.S and A.A (or T.T), upper triangles
    n = rf_strips(tiles, n, 0, bs, 0, bs, true);
    if (g.sa) n = rf_strips(tiles, n, bs, be, bs, be, true);
  } else if (g.sa) {  // S1.S2 and A1.A2
    n = rf_strips(tiles, n, 0, bs, bw, bw + bs, false);
    n = rf_strips(tiles, n, bs, be, bw + bs, bw + be, false);
  } else {
    n = rf_strips(tiles, n, 0, be, bw, bw + be, false);
  }
  return n;
}

// workspace: partial sums, the matrix M with the two flags behind it, the
// packed links
static size_t rf_m_bytes(int norb) {
  const size_t rows = 2 * ((size_t)norb * norb + 24);
  return (rows * rows + 64) * sizeof(double);
}

// the caller's workspace may start at any double; the kernel stores pairs
static double* rf_base(void* work) { return (double*)(((uintptr_t)work + 15) & ~(uintptr_t)15); }

double* rdm_fused_m(void* work) { return rf_base(work) + (size_t)RF_MAXCTA * RF_MAXT * 128; }

size_t rdm_fused_workspace(int norb, long long Nb, int nlb) {
  if (norb < 2 || norb > 16) return 0;
  return (size_t)RF_MAXCTA * RF_MAXT * 128 * sizeof(double) + rf_m_bytes(norb) +
         (size_t)(Nb + RF_NB) * nlb * sizeof(uint2) + 256;
}

bool rdm_fused_fits(const RdmFusedJob& j) {
  // 16 orbitals at most: C(16, 8)^2 determinants, which index a vector in 32 bits
  if (j.norb < 2 || j.norb > 16) return false;
  RFArgs g = rf_args(j);
  return rf_layout(g) != 0;
}

RdmFusedSize rdm_fused_size(const RdmFusedJob& j) {
  RFArgs g = rf_args(j);
  RFTile tiles[RF_MAX_ALL];
  rf_layout(g);
  RdmFusedSize s;
  s.out_tiles = rf_tiles(g, tiles);
  s.passes = (s.out_tiles + RF_MAXT - 1) / RF_MAXT;
  s.cta_rows = (g.Na + RF_MAXCTA - 1) / RF_MAXCTA;
  s.cta_tiles = (g.Na * ((g.Nb + RF_NB - 1) / RF_NB) + RF_MAXCTA - 1) / RF_MAXCTA;
  return s;
}

int rdm_fused_rows_s(const RdmFusedJob& j) {
  const int n = j.norb, r = j.sa ? n * (n + 1) / 2 : n * n;
  return (r + 7) & ~7;
}

int rdm_fused_ld(const RdmFusedJob& j) {
  const int n = j.norb;
  return j.nsrc * (rdm_fused_rows_s(j) + (j.sa ? (n * (n - 1) / 2 + 7) & ~7 : 0) + 8);
}

int rdm_fused_run(const RdmFusedJob& j, void* work, cudaStream_t stream) {
  RFArgs g = rf_args(j);
  double* M = rdm_fused_m(work);
  g.part = rf_base(work);
  g.pack = (uint2*)(((uintptr_t)M + rf_m_bytes(j.norb) + 15) & ~(uintptr_t)15);
  const size_t smem = rf_layout(g);
  if (smem == 0) {
    set_error("rdm: fused tiles exceed shared memory (norb %d)", j.norb);
    return CSFFCI_ERR_INVALID;
  }
  int st;
  const long long nct = (g.Nb + RF_NB - 1) / RF_NB;
  if (g.nlb > 0) {
    k_rdm_pack_links<<<grid_for(nct * RF_NB * g.nlb, 256, 148 * 8), 256, 0, stream>>>(g);
    if ((st = check_launch("rdm pack links"))) return st;
  }
  RFTile tiles[RF_MAX_ALL];
  const int n = rf_tiles(g, tiles);
  const long long all = g.Na * nct;
  const int grid = all < RF_MAXCTA ? (int)all : RF_MAXCTA;
  // equal passes of at most RF_MAXT tiles
  const int npass = (n + RF_MAXT - 1) / RF_MAXT;
  for (int p = 0; p < npass; ++p) {
    const int k0 = (int)((long long)n * p / npass), k1 = (int)((long long)n * (p + 1) / npass);
    g.ntile = k1 - k0;
    for (int k = k0; k < k1; ++k) {
      g.ta[k - k0] = tiles[k].a;
      g.tb[k - k0] = tiles[k].b;
    }
    if ((st = rf_dispatch(g, grid, smem, stream))) return st;
    k_rdm_reduce<<<grid_for(g.ntile * 128, 128), 128, 0, stream>>>(g, grid, j.nsrc * g.setrows, j.nsrc == 1, M);
    if ((st = check_launch("rdm reduce"))) return st;
  }
  return CSFFCI_OK;
}

int rdm_sym_check(const double* c, long long n, int* bad, cudaStream_t stream) {
  CSF_CUDA(cudaMemsetAsync(bad, 0, 2 * sizeof(int), stream));
  const long long nt = (n + 31) / 32;
  k_rdm_sym_check<<<grid_for(nt * nt, 1, 148 * 8), dim3(32, 8), 0, stream>>>(c, n, bad);
  return check_launch("rdm symmetry check");
}

int rdm_assemble_sa(const RdmFusedJob& j, const double* M, int nelec, double* dm1, double* dm2,
                    cudaStream_t stream) {
  const long long n2 = (long long)j.norb * j.norb;
  k_rdm_assemble_sa<<<grid_for(n2 * n2, 128, 148 * 8), 128, 0, stream>>>(
      j.norb, M, rdm_fused_ld(j), rdm_fused_rows_s(j), nelec > 0 ? 0.5 / nelec : 0.0, j.spin[0] != 3,
      nelec < 2 ? 0.0 : 1.0, dm1, dm2);
  return check_launch("rdm assemble");
}

int rdm_assemble_sa_ab(const RdmFusedJob& j, const double* M, double* dm2, cudaStream_t stream) {
  const long long n2 = (long long)j.norb * j.norb;
  k_rdm_assemble_sa_ab<<<grid_for(n2 * n2, 128, 148 * 8), 128, 0, stream>>>(
      j.norb, M, rdm_fused_ld(j), rdm_fused_rows_s(j), rdm_fused_ld(j) / 2, dm2);
  return check_launch("rdm assemble (alpha-beta)");
}

}  // namespace csffci
