// sigma for 4 to 13 orbitals: MMA warps in pairs of column tiles, mover warps
// by pair rows (tile variant 4 of these sizes; one problem or a job table).
//
// As in k_sigma_ws, MMA warps hold h2e fragments in registers and mover warps
// form D and scatter V.  What differs, and why:
//
//   - D and V are separate buffers (two stages each) and every hand-over is an
//     mbarrier per stage, so no MMA warp waits for another one: in k_sigma_ws V
//     overwrites D behind a barrier of all MMA warps, and the warps of a
//     scheduler, which owns one FP64 tensor pipe, stop together.
//   - A tile is 32 columns.  Warps 0.. take 16 pair rows x 16 columns (two of
//     them share a row tile), four more the last 16 (or 8) rows x 8 columns
//     each, so that every scheduler carries the same number of MMAs.
//   - The movers work by pair rows, lanes over the 32 columns.  The beta links
//     of a column tile become a table [pair row][column] -> (target, sign) (a
//     column has at most one link per pair row), so that a row of D =
//     +-c[Ka][J] +- c[Ja][K] is made in registers and stored once: no zero
//     rows, no read-modify-write, no order between alpha and beta, and every
//     access of D and V is a row.  k_sigma_ws went link by link: random rows,
//     four shared accesses a link with bank conflicts.
//   - The tiles are listed column tile by column tile, so the table is made
//     once for many rows Ja and each mover keeps its pair rows' entries in
//     registers.  Row by row it was made for every tile (12 orbitals (6,6)
//     singlet 265 us a call, now 249; 20 problems of 10 orbitals 0.36 ms, now
//     0.27).  What a tile brings is row Ja of c, its alpha entries (two tiles
//     ahead) and its alpha values (in registers, one ahead).
//   - The shares of the CTAs are tiles, not rows: the small spaces have fewer
//     rows than the GPU has SMs.
//
// What bounds it: the movers.  Their shared-memory accesses depend on one
// another and take 200 to 400 cycles under the MMA warps' load, so there are
// 12 of them (4: 478 us a call at 12 orbitals, 12: 298 us), and after that their
// issue slots (65% of all in use with a table whose entries carried a tag, now
// 53%).  12 orbitals (6,6) singlet, kernel: 226 us, the DMMA pipe 74% active
// (k_sigma_ws 340 us, 46%); 8 orbitals (4,4) singlet 12.4 -> 5 us, 13 (7,6) 2580
// (k_sigma_rr) -> 1815 us a call.
//
// The CTAs (one per SM) take equal, contiguous shares of the tiles of all rows
// of all live jobs, in rounds (see MPArgs::rounds).
#include <math.h>
#include <string.h>

#include "sigma_ws.cuh"

namespace csffci {

constexpr int MP_NB = 32;    // columns of a tile
constexpr int MP_DD = 36;    // row stride of D: = 4 (mod 16), conflict-free B fragments
constexpr int MP_DV = 40;    // row stride of V: = 8 (mod 16), conflict-free 16-byte stores
constexpr int MP_TS = 33;    // row stride of the link table
constexpr unsigned MP_LINK = 0x40000000u, MP_OFF = 0x1ffffu;  // table: a link is there; byte offset of its target
constexpr int MP_AL = 8;     // slots of the ring of alpha entries (five are in use)
constexpr int MP_POLLS = 1 << 22;
constexpr long long MP_ROUND = 48ll << 20;  // bytes of c and sigma that a round goes through

struct MPArgs {
  const csffci_sigma_job_t* jobs;  // device table (BATCH) ...
  csffci_sigma_job_t job0;         // ... or the one job
  int njobs;
  // The list of tiles is cut into rounds and each round among the CTAs.  In
  // one round a CTA would stay with its own problems, and all of a large
  // table's vectors (20 problems of 12 orbitals: 270 MB) would be in use at
  // once, their random adds past the L2 cache.
  int rounds;
  unsigned off_v, off_a, off_t, off_crow, off_al, off_job, off_bar;
  int crow_ld;  // elements between the two row buffers
};

// PT row tiles in pairs of column tiles, TAIL: 0 none, 1 a 16-row tile, 2 an
// 8-row tile split over four warps; 12 movers
template <int NORB, int PT, int TAIL, bool BATCH>
struct MPLayout {
  static constexpr int NP = NORB * (NORB + 1) / 2, KS = (NP + 3) / 4;  // pair rows, k-steps of 4
  static constexpr int NPAIRW = 2 * PT;
  static constexpr int NMMA = NPAIRW + (TAIL ? 4 : 0);
  static constexpr int NMOV = 12;
  static constexpr int NTH = (NMMA + NMOV) * 32;
  static constexpr int ROWS = 16 * PT + (TAIL == 1 ? 16 : TAIL == 2 ? 8 : 0);  // rows of V
  static constexpr int RPM = (ROWS + NMOV - 1) / NMOV;                         // pair rows of a mover
  // Registers.  With 12 MMA warps the launch has 80 a thread, split again by
  // setmaxnreg; the k-steps from KR on are then read from shared memory.  The
  // movers of a job table hold what for one problem is in constant memory or
  // in uniform registers: 56 spilled (20 problems of 12 orbitals 8.28 ms, in an
  // earlier form), 72 do not (6.83 ms).  At 13 orbitals a table has 56 and does
  // not spill; 12 k-steps in registers there would need 196 KB of shared memory
  // in place of 181 and have not been measured.
  static constexpr bool SPLIT = NMMA == 12;
  static constexpr int KR = KS <= 14 ? KS : KS > 20 ? 17 : BATCH ? 12 : 17;
  static constexpr int AT = (KS - KR) * (PT + (TAIL ? 1 : 0)) * 64;  // elements of that part of h2e
  static constexpr int REG_LAUNCH = 65536 / NTH / 8 * 8;
  static constexpr int REG_MMA = BATCH && KS <= 20 ? 88 : 104, REG_MOV = 160 - REG_MMA;
  static constexpr int DR = ROWS > 4 * KS ? ROWS : 4 * KS;  // rows of D
  static constexpr int DSZ = DR * MP_DD, VSZ = ROWS * MP_DV, TSZ = NP * MP_TS;
  static_assert(ROWS >= NP, "rows");
  static_assert(NPAIRW % 4 == 0, "equal MMA shares on the four schedulers");
  static_assert(!SPLIT || NMMA * 32 * REG_MMA + NMOV * 32 * REG_MOV <= NTH * REG_LAUNCH, "fits the launch's registers");
};

__device__ __forceinline__ void mp_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(ws_smem_addr(bar)) : "memory");
}

__device__ __forceinline__ bool mp_wait(unsigned long long* bar, unsigned parity) {
  for (int i = 0; i < MP_POLLS; ++i)
    if (ws_mbar_try_wait(bar, parity)) return true;
  return false;
}

// tiles of a job: all columns, or those up to the diagonal (rows 32m..32m+31
// have m + 1 tiles)
__device__ __forceinline__ long long mp_tri(long long rows) {
  const long long m = rows / MP_NB, r = rows - m * MP_NB;
  return (MP_NB / 2) * m * (m + 1) + r * (m + 1);
}
__device__ __forceinline__ long long mp_job_tiles(const csffci_sigma_job_t& J) {
  if (J.live != nullptr && J.live_index >= *J.live) return 0;
  return J.sym ? mp_tri(J.Na) : J.Na * ((J.Nb + MP_NB - 1) / MP_NB);
}

// what the movers read of a job of a table
struct MPJob {
  const double* ci;
  double* out;
  const csffci_link_t *link_a, *link_b;
  int nla, nlb;
};

struct MPShared {
  double* D;
  double* V;
  double* A;  // k-steps from KR on: [step][row tile][row][4]
  unsigned* T;
  double* crow;
  uint2* al;
  MPJob* job;
  unsigned long long* bar;  // D full, D empty, V full, V empty, two each
};

// the job of tile *t of the list, by a warp (32 jobs at a time); *t becomes its
// number in the job
template <bool BATCH>
__device__ __forceinline__ int mp_find(const MPArgs& g, int lane, long long* t) {
  if constexpr (BATCH) {
    for (int j0 = 0; j0 < g.njobs; j0 += 32) {
      const long long own = j0 + lane < g.njobs ? mp_job_tiles(g.jobs[j0 + lane]) : 0;
      long long upto = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long x = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += x;
      }
      const unsigned past = __ballot_sync(0xffffffffu, *t < upto);
      if (past) {
        const int l = __ffs(past) - 1;
        *t -= __shfl_sync(0xffffffffu, upto - own, l);
        return j0 + l;
      }
      *t -= __shfl_sync(0xffffffffu, upto, 31);
    }
    return g.njobs - 1;
  }
  return 0;
}

// Tile *t of a job, whose tiles are listed column tile by column tile: its
// column tile; *t becomes its row
__device__ __forceinline__ int mp_column(const csffci_sigma_job_t& Q, long long* t) {
  int ct = 0;
  if (Q.sym) {
    while (*t >= Q.Na - (long long)ct * MP_NB) *t -= Q.Na - (long long)(ct++) * MP_NB;
    *t += (long long)ct * MP_NB;
  } else {
    ct = (int)(*t / Q.Na);
    *t -= ct * Q.Na;
  }
  return ct;
}

// Tiles it0 .. it0 + n - 1 of the CTA: rows ja0, ja0 + 1, ... of column tile ct
// of job Q.  ok: false once a wait of this warp has run out (it then waits no
// more, in later calls either).
template <int NORB, int PT, int TAIL, bool BATCH>
__device__ __forceinline__ void mp_movers(const MPArgs& g, const MPShared& S, const csffci_sigma_job_t& Q, int ct,
                                          int ja0, int it0, int n, int mtid, int lane, int mw, bool& ok) {
  using L = MPLayout<NORB, PT, TAIL, BATCH>;
  constexpr int NMOV = L::NMOV, MTH = NMOV * 32, RPM = L::RPM, NP = L::NP;
  constexpr int RB = 4, RS = BATCH ? 2 : 4;  // pair rows gathered and scattered together
  // row i of this warp is pair row mw + i NMOV
  auto in = [&](int i) { return i < RPM && (i * NMOV + NMOV <= NP || mw + i * NMOV < NP); };
  const unsigned empty = (unsigned)(g.crow_ld - 1) * 8u;  // no link: the zero behind row Ja of c
  const int Nb = (int)Q.Nb, sym = Q.sym, end = it0 + n, first = ja0 - it0;
  // what one problem has in constant memory is for a job table kept in shared
  // memory: held in registers it would make the movers spill
  if (BATCH && mtid == 0) *S.job = MPJob{Q.ci, sym ? Q.scratch : Q.sigma, Q.link_a, Q.link_b, Q.nla, Q.nlb};
  for (int i = mtid; i < L::TSZ; i += MTH) S.T[i] = empty;
  for (int i = mtid; i < MP_AL * NP; i += MTH) S.al[i] = make_uint2(0u, 0u);
  ws_bar_sync(5, MTH);
  auto ci = [&]() { return BATCH ? S.job->ci : Q.ci; };
  auto out = [&]() { return BATCH ? S.job->out : sym ? Q.scratch : Q.sigma; };
  auto link_a = [&]() { return BATCH ? S.job->link_a : Q.link_a; };
  auto nla = [&]() { return BATCH ? S.job->nla : Q.nla; };
  // row Ja of c of tile it
  auto load_row = [&](int it) {
    double* const cr = S.crow + (it & 1) * g.crow_ld;
    const double* const row = ci() + (first + it) * Nb;
    for (int i = mtid; i < Nb; i += MTH) cp_async8(&cr[i], &row[i]);
    cp_async_commit();
  };
  // the alpha links of tile it: link (if any) of this thread, and its entry
  // (byte offset of row Ka, sign) by pair row; the ring's slot is empty
  auto alpha_link = [&](int it) { return rr_link(&link_a()[(first + it) * nla() + mtid]); };
  auto put_alpha = [&](int it, uint2 e) {
    S.al[(it & (MP_AL - 1)) * NP + rr_lpair(e)] = make_uint2(e.x * (unsigned)Nb * 8u, 1u | rr_lneg(e));
  };
  load_row(it0);
  for (int i = it0; i < it0 + 2 && i < end; ++i)
    if (mtid < nla()) put_alpha(i, alpha_link(i));
  {
    // the beta links of the column tile: link e % nlb of column e / nlb
    const int nlb = BATCH ? S.job->nlb : Q.nlb;
    const int ne = min(MP_NB, Nb - ct * MP_NB) * nlb;
    const csffci_link_t* const src = (BATCH ? S.job->link_b : Q.link_b) + ct * MP_NB * nlb;
    const unsigned inv = (1u << 20) / (unsigned)max(nlb, 1) + 1u;
    for (int e = mtid; e < ne; e += MTH) {
      const uint2 l = rr_link(&src[e]);
      S.T[rr_lpair(l) * MP_TS + (int)(((unsigned)e * inv) >> 20)] = l.x * 8u | MP_LINK | rr_lneg(l);
    }
  }
  cp_async_wait_all();
  ws_bar_sync(5, MTH);
  unsigned t[RPM];
#pragma unroll
  for (int i = 0; i < RPM; ++i) t[i] = in(i) ? S.T[(mw + i * NMOV) * MP_TS + lane] : empty;
  const int j = ct * MP_NB + lane;
  double va[RPM];  // alpha values of the next tile
  unsigned sa;     // their signs
  auto load_alpha = [&](int it) {
    const uint2* const al = S.al + (it & (MP_AL - 1)) * NP + mw;
    const char* const src = reinterpret_cast<const char*>(ci() + j);
    const bool inj = j < (sym ? first + it + 1 : Nb);
    sa = 0u;
#pragma unroll
    for (int i = 0; i < RPM; ++i) {
      const uint2 a = in(i) ? al[i * NMOV] : make_uint2(0u, 0u);
      va[i] = (a.y && inj) ? __ldg(reinterpret_cast<const double*>(src + a.x)) : 0.0;
      sa |= (a.y >> 31) << i;
    }
  };
  load_alpha(it0);
  for (int it = it0; it <= end; ++it) {
    uint2 next = make_uint2(0u, 0u);
    const bool more = it + 2 < end && mtid < nla();
    if (it < end) {
      const int s = it & 1;
      if (it + 1 < end) load_row(it + 1);
      if (more) next = alpha_link(it + 2);
      for (int r = mtid; r < NP; r += MTH) S.al[((it + 3) & (MP_AL - 1)) * NP + r] = make_uint2(0u, 0u);
      if (it >= 2 && ok) ok = mp_wait(&S.bar[2 + s], ((it >> 1) & 1) ^ 1);  // D of tile it-2 is consumed
      const char* const cr = reinterpret_cast<const char*>(S.crow + s * g.crow_ld);
      double* const D = S.D + s * L::DSZ + mw * MP_DD + lane;
#pragma unroll
      for (int i0 = 0; i0 < RPM; i0 += RB) {
        double vb[RB];
#pragma unroll
        for (int k = 0; k < RB; ++k)
          vb[k] = i0 + k < RPM ? *reinterpret_cast<const double*>(cr + (t[i0 + k < RPM ? i0 + k : 0] & MP_OFF)) : 0.0;
#pragma unroll
        for (int k = 0; k < RB; ++k)
          if (in(i0 + k)) {
            const int i = i0 + k < RPM ? i0 + k : 0;
            D[i * NMOV * MP_DD] =
                rr_flip(va[i], (sa << (31 - i)) & 0x80000000u) + rr_flip(vb[k], t[i] & 0x80000000u);
          }
      }
      __syncwarp();
      if (lane == 0) mp_arrive(&S.bar[s]);  // this warp's rows of D are there
      if (it + 1 < end) load_alpha(it + 1);
    }
    if (it > it0) {
      // scatter V of the previous tile
      const int s = (it - 1) & 1, pja = first + it - 1;
      if (ok) ok = mp_wait(&S.bar[4 + s], ((it - 1) >> 1) & 1);
      const uint2* const al = S.al + ((it - 1) & (MP_AL - 1)) * NP + mw;
      const double* const V = S.V + s * L::VSZ + mw * MP_DV + lane;
      char* const orow = reinterpret_cast<char*>(out() + pja * Nb);
      char* const ocol = reinterpret_cast<char*>(out() + j);
      const bool inb = j < (sym ? pja + 1 : Nb), ina = sym ? j < pja : inb;
#pragma unroll
      for (int i0 = 0; i0 < RPM; i0 += RS) {
        uint2 a[RS];
        double v[RS];
#pragma unroll
        for (int k = 0; k < RS; ++k) {
          a[k] = in(i0 + k) ? al[(i0 + k) * NMOV] : make_uint2(0u, 0u);
          v[k] = in(i0 + k) ? V[(i0 + k) * NMOV * MP_DV] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < RS; ++k)
          if (in(i0 + k)) {
            const unsigned tt = t[i0 + k < RPM ? i0 + k : 0];
            if (inb && (tt & MP_LINK))
              rr_red(reinterpret_cast<double*>(orow + (tt & MP_OFF)), rr_flip(v[k], tt & 0x80000000u));
            if (ina && a[k].y) rr_red(reinterpret_cast<double*>(ocol + a[k].x), rr_flip(v[k], a[k].y & 0x80000000u));
          }
      }
      __syncwarp();
      if (lane == 0) mp_arrive(&S.bar[6 + s]);  // V of the previous tile is consumed
    }
    if (more) put_alpha(it + 2, next);
    cp_async_wait_all();
    ws_bar_sync(5, MTH);  // row Ja of tile it+1 and the alpha entries of tile it+2 are there
  }
}

// A hand-over that never came shows as NaN in every job that this CTA has had
// tiles of: with two stages in flight the values lost may be those of an
// earlier job than the one at hand when a wait ran out.  By one warp.
template <bool BATCH>
__device__ __forceinline__ void mp_poison(const MPArgs& g, long long total, int lane) {
  const long long shares = (long long)gridDim.x * g.rounds;
  for (int r = 0; r < g.rounds; ++r) {
    const long long q = (long long)r * gridDim.x + blockIdx.x;
    long long t0 = total * q / shares, n = total * (q + 1) / shares - t0;
    if (n == 0) continue;
    for (int jb = mp_find<BATCH>(g, lane, &t0); n > 0; ++jb) {
      const csffci_sigma_job_t& Q = BATCH ? g.jobs[jb] : g.job0;
      const long long m = BATCH ? min(n, mp_job_tiles(Q) - t0) : n;
      if (m > 0 && lane == 0) rr_red(Q.sym ? Q.scratch : Q.sigma, __longlong_as_double(0x7ff8000000000000ll));
      n -= m;
      t0 = 0;
    }
  }
}

template <int NORB, int PT, int TAIL, bool BATCH>
__global__ void __launch_bounds__(MPLayout<NORB, PT, TAIL, BATCH>::NTH, 1) k_sigma_mp(const __grid_constant__ MPArgs g) {
  using L = MPLayout<NORB, PT, TAIL, BATCH>;
  constexpr int NTH = L::NTH, KS = L::KS, npair = L::NP;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  MPShared S;
  S.D = (double*)smraw;
  S.V = (double*)(smraw + g.off_v);
  S.A = (double*)(smraw + g.off_a);
  S.T = (unsigned*)(smraw + g.off_t);
  S.crow = (double*)(smraw + g.off_crow);
  S.al = (uint2*)(smraw + g.off_al);
  S.job = (MPJob*)(smraw + g.off_job);
  S.bar = (unsigned long long*)(smraw + g.off_bar);
  __shared__ long long total_s;
  __shared__ int bad_s;
  for (int i = tid; i < 2 * L::DSZ; i += NTH) S.D[i] = 0.0;  // rows past npair stay zero
  if (tid < 2) S.crow[tid * g.crow_ld + g.crow_ld - 1] = 0.0;
  if (tid == 0) {
    total_s = 0;
    bad_s = 0;
    for (int i = 0; i < 2; ++i) {
      ws_mbar_init(&S.bar[i], L::NMOV);
      ws_mbar_init(&S.bar[2 + i], L::NMMA);
      ws_mbar_init(&S.bar[4 + i], L::NMMA);
      ws_mbar_init(&S.bar[6 + i], L::NMOV);
    }
    ws_mbar_init_fence();
  }
  __syncthreads();
  if (BATCH) {
    long long t = 0;
    for (int i = tid; i < g.njobs; i += NTH) t += mp_job_tiles(g.jobs[i]);
    if (t) atomicAdd((unsigned long long*)&total_s, (unsigned long long)t);
    __syncthreads();
  }
  const long long total = BATCH ? total_s : mp_job_tiles(g.job0);
  const long long shares = (long long)gridDim.x * g.rounds;

  if (warp < L::NMMA) {
    if constexpr (L::SPLIT) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(L::REG_MMA));
    const int gq = lane >> 2, tq = lane & 3;
    const bool pair = warp < L::NPAIRW;
    // pair warps: row tile warp / 2, columns 16 (warp & 1)..; tail warps: the
    // last rows, columns 8 (warp - NPAIRW)..
    const int r0 = (pair ? warp / 2 : PT) * 16 + gq, r1 = r0 + 8;
    const int c0 = pair ? 16 * (warp & 1) : 8 * (warp - L::NPAIRW);
    constexpr int KR = L::KR, NRT = PT + (TAIL ? 1 : 0);
    double a0[KR], a1[KR];
    const int rt = pair ? warp / 2 : PT;
    double* const as = S.A + rt * 64 + lane;
    auto load_a = [&](const double* h2e) {
      auto at = [&](int r, int k) {
        const int c = 4 * k + tq;
        return r < npair && c < npair ? h2e[(long long)r * npair + c] : 0.0;
      };
#pragma unroll
      for (int k = 0; k < KR; ++k) {
        a0[k] = at(r0, k);
        a1[k] = at(r1, k);
      }
      if constexpr (KS > KR) {  // shared by the warps of a row tile
        const int nth = pair ? 64 : 128;
        ws_bar_sync(6 + rt, nth);
        for (int k = KR; k < KS; ++k) {
          as[(k - KR) * NRT * 64] = at(r0, k);
          as[(k - KR) * NRT * 64 + 32] = at(r1, k);
        }
        ws_bar_sync(6 + rt, nth);
      }
    };
    bool ok = true;
    int it = 0;
    for (int r = 0; r < g.rounds; ++r) {
      const long long q = (long long)r * gridDim.x + blockIdx.x;
      long long t0 = total * q / shares;
      const int n = it + (int)(total * (q + 1) / shares - t0);
      if (it == n) continue;
      for (int jb = mp_find<BATCH>(g, lane, &t0); it < n; ++jb) {  // job by job
        const csffci_sigma_job_t& Q = BATCH ? g.jobs[jb] : g.job0;
        const int end = BATCH ? it + (int)min((long long)(n - it), mp_job_tiles(Q) - t0) : n;
        t0 = 0;
        if (end == it) continue;
        load_a(Q.h2e);
        for (; it < end; ++it) {
          const int s = it & 1;
          const unsigned ph = (it >> 1) & 1;
          if (ok) ok = mp_wait(&S.bar[s], ph);
          const double* Db = S.D + s * L::DSZ + tq * MP_DD + gq + c0;
          double acc[2][4];
#pragma unroll
          for (int t = 0; t < 2; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0;
          if (pair) {
#pragma unroll
            for (int k = 0; k < KS; ++k) {
              const double x0 = k < KR ? a0[k < KR ? k : 0] : as[(k - KR) * NRT * 64];
              const double x1 = k < KR ? a1[k < KR ? k : 0] : as[(k - KR) * NRT * 64 + 32];
              rr_dmma16(acc[0], x0, x1, Db[4 * k * MP_DD]);
              rr_dmma16(acc[1], x0, x1, Db[4 * k * MP_DD + 8]);
            }
          } else if (TAIL == 1) {
            // two sums over alternate k-steps: the products of one would wait on each other
#pragma unroll
            for (int k = 0; k < KS; ++k)
              rr_dmma16(acc[k & 1], k < KR ? a0[k < KR ? k : 0] : as[(k - KR) * NRT * 64],
                        k < KR ? a1[k < KR ? k : 0] : as[(k - KR) * NRT * 64 + 32], Db[4 * k * MP_DD]);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[0][i] += acc[1][i];
          } else {
#pragma unroll
            for (int k = 0; k < KS; ++k)
              ws_dmma(acc[k & 1][0], acc[k & 1][1], k < KR ? a0[k < KR ? k : 0] : as[(k - KR) * NRT * 64], Db[4 * k * MP_DD]);
            acc[0][0] += acc[1][0];
            acc[0][1] += acc[1][1];
          }
          __syncwarp();
          if (lane == 0) mp_arrive(&S.bar[2 + s]);  // this warp has read D
          if (it >= 2 && ok) ok = mp_wait(&S.bar[6 + s], ph ^ 1);  // V of tile it-2 is scattered
          double* const V = S.V + s * L::VSZ + c0 + 2 * tq;
          *reinterpret_cast<double2*>(&V[r0 * MP_DV]) = make_double2(acc[0][0], acc[0][1]);
          if (pair || TAIL == 1) *reinterpret_cast<double2*>(&V[r1 * MP_DV]) = make_double2(acc[0][2], acc[0][3]);
          if (pair) {
            *reinterpret_cast<double2*>(&V[r0 * MP_DV + 8]) = make_double2(acc[1][0], acc[1][1]);
            *reinterpret_cast<double2*>(&V[r1 * MP_DV + 8]) = make_double2(acc[1][2], acc[1][3]);
          }
          __syncwarp();
          if (lane == 0) mp_arrive(&S.bar[4 + s]);  // this warp's part of V is there
        }
      }
    }
    if (!ok) bad_s = 1;
  } else {
    if constexpr (L::SPLIT) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(L::REG_MOV));
    const int mw = warp - L::NMMA;
    bool ok = true;
    int it = 0;
    for (int r = 0; r < g.rounds; ++r) {
      const long long q = (long long)r * gridDim.x + blockIdx.x;
      long long t0 = total * q / shares;
      const int n = it + (int)(total * (q + 1) / shares - t0);
      if (it == n) continue;
      for (int jb = mp_find<BATCH>(g, lane, &t0); it < n; ++jb) {
        const csffci_sigma_job_t& Q = BATCH ? g.jobs[jb] : g.job0;
        const int end = BATCH ? it + (int)min((long long)(n - it), mp_job_tiles(Q) - t0) : n;
        if (it == end) continue;
        int ct = mp_column(Q, &t0);
        for (; it < end; ++ct) {
          const int m = min(end - it, (int)(Q.Na - t0));
          mp_movers<NORB, PT, TAIL, BATCH>(g, S, Q, ct, (int)t0, it, m, mw * 32 + lane, lane, mw, ok);
          it += m;
          t0 = Q.sym ? (long long)(ct + 1) * MP_NB : 0;
        }
        t0 = 0;
      }
    }
    if (!ok) bad_s = 1;
  }
  __syncthreads();
  if (bad_s && warp == 0) mp_poison<BATCH>(g, total, lane);
}

long long sigma_mp_tiles(const csffci_sigma_job_t& J) {
  const long long m = J.Na / MP_NB, r = J.Na - m * MP_NB;
  return J.sym ? (MP_NB / 2) * m * (m + 1) + r * (m + 1) : J.Na * ((J.Nb + MP_NB - 1) / MP_NB);
}

bool sigma_mp_supported(int norb) { return norb >= 4 && norb <= 13; }

template <int NORB, int PT, int TAIL, bool BATCH>
static int mp_launch_as(int norb, MPArgs& g, long long max_nb, long long max_tiles,
                     long long nelem, cudaStream_t stream) {
  using L = MPLayout<NORB, PT, TAIL, BATCH>;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += (bytes + 15) & ~(size_t)15;
    return (unsigned)o;
  };
  take((size_t)2 * L::DSZ * sizeof(double));
  g.off_v = take((size_t)2 * L::VSZ * sizeof(double));
  g.off_a = take((size_t)L::AT * sizeof(double));
  g.off_t = take((size_t)L::TSZ * sizeof(unsigned));
  g.crow_ld = (int)((max_nb + 2) & ~1ll);  // and a zero behind the row
  g.off_crow = take((size_t)2 * g.crow_ld * sizeof(double));
  g.off_al = take((size_t)MP_AL * L::NP * sizeof(uint2));
  g.off_job = take(sizeof(MPJob));
  g.off_bar = take(8 * sizeof(unsigned long long));
  if (off > MAX_SMEM) {
    set_error("sigma: row-pair tiles exceed shared memory (%zu)", off);
    return CSFFCI_ERR_INVALID;
  }
  auto kern = k_sigma_mp<NORB, PT, TAIL, BATCH>;
  if (L::SPLIT) {
    // setmaxnreg re-splits the registers of the launch; with fewer the raise
    // would wait forever
    cudaFuncAttributes fa;
    CSF_CUDA(cudaFuncGetAttributes(&fa, kern));
    if (fa.numRegs != L::REG_LAUNCH) {
      set_error("sigma: row-pair kernel compiled to %d registers per thread, not %d", fa.numRegs, L::REG_LAUNCH);
      return CSFFCI_ERR_INVALID;
    }
  }
  CSF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM));
  const int grid = (int)(max_tiles < 148 ? (max_tiles > 0 ? max_tiles : 1) : 148);  // one CTA per SM
  g.rounds = (int)(nelem * 16 / MP_ROUND + 1);
  if (g.rounds > 256) g.rounds = 256;
  static const char* names[10] = {"k_sigma_mp_n4", "k_sigma_mp_n5", "k_sigma_mp_n6",  "k_sigma_mp_n7",  "k_sigma_mp_n8",
                                  "k_sigma_mp_n9", "k_sigma_mp_n10", "k_sigma_mp_n11", "k_sigma_mp_n12", "k_sigma_mp_n13"};
  ProfScope ps(BATCH ? names[norb - 4] : "k_sigma_mp", stream);
  kern<<<grid, L::NTH, off, stream>>>(g);
  return check_launch("sigma (pair rows)");
}

template <int NORB, int PT, int TAIL>
static int mp_launch(int norb, MPArgs& g, long long max_nb, long long max_tiles, long long nelem,
                     cudaStream_t stream) {
  return g.jobs ? mp_launch_as<NORB, PT, TAIL, true>(norb, g, max_nb, max_tiles, nelem, stream)
                : mp_launch_as<NORB, PT, TAIL, false>(norb, g, max_nb, max_tiles, nelem, stream);
}

// max_tiles: tiles of all jobs when every one is live
int sigma_mp_launch(int norb, int njobs, const csffci_sigma_job_t* jobs_dev, const csffci_sigma_job_t& job0,
                    long long max_nb, long long max_tiles,
                     long long nelem, cudaStream_t stream) {
  MPArgs g;
  memset(&g, 0, sizeof(g));
  g.jobs = jobs_dev;
  g.job0 = job0;
  g.njobs = jobs_dev ? njobs : 1;
  switch (norb) {  // 10, 15, 21, 28, 36, 45, 55, 66, 78, 91 pair rows
    case 4: return mp_launch<4, 0, 1>(norb, g, max_nb, max_tiles, nelem, stream);
    case 5: return mp_launch<5, 0, 1>(norb, g, max_nb, max_tiles, nelem, stream);
    case 6: return mp_launch<6, 2, 0>(norb, g, max_nb, max_tiles, nelem, stream);
    case 7: return mp_launch<7, 2, 0>(norb, g, max_nb, max_tiles, nelem, stream);
    case 8: return mp_launch<8, 2, 2>(norb, g, max_nb, max_tiles, nelem, stream);
    case 9: return mp_launch<9, 2, 1>(norb, g, max_nb, max_tiles, nelem, stream);
    case 10: return mp_launch<10, 4, 0>(norb, g, max_nb, max_tiles, nelem, stream);
    case 11: return mp_launch<11, 4, 2>(norb, g, max_nb, max_tiles, nelem, stream);
    case 12: return mp_launch<12, 4, 1>(norb, g, max_nb, max_tiles, nelem, stream);
    case 13: return mp_launch<13, 6, 0>(norb, g, max_nb, max_tiles, nelem, stream);
    default: break;
  }
  set_error("sigma: no row-pair kernel for norb %d", norb);
  return CSFFCI_ERR_INVALID;
}

}  // namespace csffci
