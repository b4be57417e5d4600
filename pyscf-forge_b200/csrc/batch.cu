// Batched kernels for many independent CI problems solved in lockstep: one
// launch per operation covers every problem of the batch (descriptor
// tables in device memory), so the launch count of a Davidson iteration does
// not grow with the number of problems.
//
//   csffci_transform_batch  det <-> CSF block GEMMs of many (problem, block)
//   csffci_dots_batch       dot products x.y or x.(P y), P = 1/(hdiag-(e-shift))
//   csffci_combine_batch    y = beta y + scale * coef . X   (subspace algebra)
//   csffci_precond_batch    t = (r - e1 x) P with e1 = ab[0]/ab[1] read on device
// Every reduction runs in a fixed order (one block per dot product).
#include "common.cuh"
#include "profile.cuh"
#include "batch_internal.cuh"
#include "transform_tile.cuh"

namespace csffci {

// ---------------------------------------------------------------------------
// transforms
// ---------------------------------------------------------------------------
// the last job whose tile_begin is at most u: 32 probes a round, so that a
// table of hundreds of jobs costs two dependent loads (walking from the first
// job took most of a launch over 120 jobs)
__device__ __forceinline__ int find_job(const csffci_transform_job_t* jobs, int njobs, int64_t u, int lane) {
  int lo = 0, hi = njobs;  // the answer is in [lo, hi)
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) / 32;
    const int at = lo + lane * step;
    const bool le = at < hi && jobs[at].tile_begin <= u;
    const int last = 31 - __clz((int)__ballot_sync(0xffffffffu, le));  // lane 0's job is always at or before u
    lo += last * step;
    hi = min(hi, lo + step);
  }
  return lo;
}

// One task = the CTA task of transform_tile.cuh of one job (one npair block of
// one problem); pad holds the tile class, the column chunks and the vectors of
// a tile.
__global__ void __launch_bounds__(XF_W * 32, 2) k_transform_batch(const csffci_transform_job_t* jobs, int njobs,
                                                                  int64_t total_tiles, int reverse) {
  __shared__ double red[XF_RED];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
    const csffci_transform_job_t& J = jobs[find_job(jobs, njobs, tile, lane)];
    XfTile B;
    B.nvec = J.live ? min(J.nvec, *J.live) : J.nvec;
    if (B.nvec <= 0) continue;  // uniform over the CTA
    B.x = J.x;
    B.y = J.y;
    B.mask = J.mask + J.csd_offset;
    B.u = J.umat;
    B.z = nullptr;
    B.sel = nullptr;
    B.ldx = J.ldx;
    B.ldy = J.ldy;
    B.csf_off = J.csf_offset;
    B.nconf = J.nconf;
    B.ndet = J.ndet;
    B.ncsf = J.ncsf;
    B.sign = J.sign;
    const int cls = J.pad & 7, nchunk = (J.pad >> 3) & 0x3fff, vper = J.pad >> 17;
    const int64_t t = tile - J.tile_begin;
    if (reverse) xf_run<XF_CSF2DET, true>(B, nullptr, cls, t, nchunk, vper, lane, warp, red);
    else xf_run<XF_DET2CSF, true>(B, nullptr, cls, t, nchunk, vper, lane, warp, red);
  }
}

// zero the determinant vectors of reverse jobs (blocks without CSFs must
// read as zero); one entry per (vector, det) of each zero job
__global__ void k_zero_batch(const csffci_zero_job_t* jobs, int njobs, int64_t total) {
  int j = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    while (j + 1 < njobs && jobs[j + 1].elem_begin <= i) ++j;
    const csffci_zero_job_t& J = jobs[j];
    const int64_t li = i - J.elem_begin;
    const int64_t v = li / J.n;
    J.y[v * J.ld + (li - v * J.n)] = 0.0;
  }
}

// ---------------------------------------------------------------------------
// dots: one block per dot product, fixed-order tree reduction
// ---------------------------------------------------------------------------
__device__ __forceinline__ double pinv(double h, double es) {
  double v = 1.0 / (h - es);
  if (fabs(v) > 1e8) v = 1e8;
  return v;
}

__global__ void __launch_bounds__(256) k_dots_batch(const csffci_dot_t* dots, int ndots, double* out) {
  __shared__ double red[256];
  for (int d = blockIdx.x; d < ndots; d += gridDim.x) {
    const csffci_dot_t D = dots[d];
    double acc = 0.0;
    if (D.hdiag) {
      for (int64_t k = threadIdx.x; k < D.n; k += blockDim.x)
        acc = fma(D.x[k] * pinv(D.hdiag[k], D.e_shift), D.y[k], acc);
    } else {
      for (int64_t k = threadIdx.x; k < D.n; k += blockDim.x) acc = fma(D.x[k], D.y[k], acc);
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
      if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
      __syncthreads();
    }
    if (threadIdx.x == 0) out[D.out_index] = red[0];
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// combine: y[r][k] = beta*y[r][k] + scale * sum_i coef[r*ldc + i] * x[i][k]
// ---------------------------------------------------------------------------
__global__ void k_combine_batch(const csffci_combine_t* ops, int nops, int64_t total_units) {
  int j = 0;
  for (int64_t u = blockIdx.x; u < total_units; u += gridDim.x) {
    while (j + 1 < nops && ops[j + 1].unit_begin <= u) ++j;
    const csffci_combine_t& O = ops[j];
    const int64_t k = (u - O.unit_begin) * blockDim.x + threadIdx.x;
    if (k >= O.n) continue;
    for (int r = 0; r < O.ny; ++r) {
      double acc = 0.0;
      for (int i = 0; i < O.nx; ++i) acc = fma(O.coef[r * O.ldc + i], O.x[i * O.ldx + k], acc);
      double* yp = O.y + r * O.ldy + k;
      *yp = (O.beta == 0.0 ? 0.0 : O.beta * *yp) + O.scale * acc;
    }
  }
}

// ---------------------------------------------------------------------------
// precond: t = (r - e1 x) P, e1 = ab[0] / ab[1] (0 when ab is NULL)
// ---------------------------------------------------------------------------
__global__ void k_precond_batch(const csffci_precond_t* ops, int nops, int64_t total_units) {
  int j = 0;
  for (int64_t u = blockIdx.x; u < total_units; u += gridDim.x) {
    while (j + 1 < nops && ops[j + 1].unit_begin <= u) ++j;
    const csffci_precond_t& O = ops[j];
    const int64_t k = (u - O.unit_begin) * blockDim.x + threadIdx.x;
    if (k >= O.n) continue;
    double e1 = 0.0;
    if (O.ab) {
      const double b = O.ab[1];
      e1 = b != 0.0 ? O.ab[0] / b : 0.0;
    }
    O.t[k] = (O.r[k] - e1 * O.x[k]) * pinv(O.hdiag[k], O.e_shift);
  }
}

int transform_batch_prepare(int reverse, int njobs, csffci_transform_job_t* jobs, int64_t* total_tiles) {
  int64_t tiles = 0;
  for (int i = 0; i < njobs; ++i) {
    csffci_transform_job_t& J = jobs[i];
    CSF_REQUIRE(J.x && J.y && J.mask && J.umat && J.ncsf > 0 && J.ndet > 0, "transform_batch: job %d incomplete", i);
    J.tile_begin = tiles;
    const XfShape sh = xf_shape(J.nconf, J.nvec, reverse ? J.ndet : J.ncsf, reverse ? J.ncsf : J.ndet);
    J.pad = sh.cls | sh.nchunk << 3 | sh.vper << 17;
    tiles += sh.ntask;
  }
  *total_tiles = tiles;
  return CSFFCI_OK;
}

int transform_batch_launch(int reverse, const csffci_transform_job_t* jobs_dev, int njobs, int64_t tiles,
                           cudaStream_t stream) {
  if (tiles == 0 || njobs == 0) return CSFFCI_OK;
  ProfScope ps("k_transform_batch", stream);
  k_transform_batch<<<grid_for(tiles, 1, 148 * 2), XF_W * 32, 0, stream>>>(jobs_dev, njobs, tiles, reverse);
  return check_launch("transform_batch");
}

}  // namespace csffci

using namespace csffci;

extern "C" {

int csffci_transform_batch(int reverse, int njobs, csffci_transform_job_t* jobs, int nzero,
                           csffci_zero_job_t* zjobs, void* work, size_t work_bytes,
                           cudaStream_t stream) {
  CSF_REQUIRE(njobs >= 0 && nzero >= 0, "transform_batch: bad counts");
  const size_t need = (size_t)njobs * sizeof(csffci_transform_job_t) + (size_t)nzero * sizeof(csffci_zero_job_t);
  if (need == 0) return CSFFCI_OK;
  if (work == nullptr || work_bytes < need) {
    set_error("transform_batch: workspace of %zu bytes < %zu required", work_bytes, need);
    return CSFFCI_ERR_MEMORY;
  }
  int64_t tiles = 0;
  int st = transform_batch_prepare(reverse, njobs, jobs, &tiles);
  if (st) return st;
  int64_t zelem = 0;
  for (int i = 0; i < nzero; ++i) {
    zjobs[i].elem_begin = zelem;
    zelem += zjobs[i].nvec * zjobs[i].n;
  }
  char* w = (char*)work;
  csffci_transform_job_t* dj = (csffci_transform_job_t*)w;
  csffci_zero_job_t* dz = (csffci_zero_job_t*)(w + (size_t)njobs * sizeof(csffci_transform_job_t));
  if (njobs) CSF_CUDA(cudaMemcpyAsync(dj, jobs, njobs * sizeof(*jobs), cudaMemcpyHostToDevice, stream));
  if (nzero) {
    CSF_CUDA(cudaMemcpyAsync(dz, zjobs, nzero * sizeof(*zjobs), cudaMemcpyHostToDevice, stream));
    k_zero_batch<<<grid_for(zelem, 256, 148 * 16), 256, 0, stream>>>(dz, nzero, zelem);
    st = check_launch("transform_batch zero");
    if (st) return st;
  }
  return transform_batch_launch(reverse, dj, njobs, tiles, stream);
}

int csffci_dots_batch(int ndots, const csffci_dot_t* dots, double* out, void* work, size_t work_bytes,
                      cudaStream_t stream) {
  CSF_REQUIRE(ndots >= 0, "dots_batch: bad count");
  if (ndots == 0) return CSFFCI_OK;
  const size_t need = (size_t)ndots * sizeof(csffci_dot_t);
  if (work == nullptr || work_bytes < need) {
    set_error("dots_batch: workspace of %zu bytes < %zu required", work_bytes, need);
    return CSFFCI_ERR_MEMORY;
  }
  CSF_CUDA(cudaMemcpyAsync(work, dots, need, cudaMemcpyHostToDevice, stream));
  k_dots_batch<<<grid_for(ndots, 1, 148 * 16), 256, 0, stream>>>((const csffci_dot_t*)work, ndots, out);
  return check_launch("dots_batch");
}

int csffci_combine_batch(int nops, csffci_combine_t* ops, void* work, size_t work_bytes,
                         cudaStream_t stream) {
  CSF_REQUIRE(nops >= 0, "combine_batch: bad count");
  if (nops == 0) return CSFFCI_OK;
  const size_t need = (size_t)nops * sizeof(csffci_combine_t);
  if (work == nullptr || work_bytes < need) {
    set_error("combine_batch: workspace of %zu bytes < %zu required", work_bytes, need);
    return CSFFCI_ERR_MEMORY;
  }
  int64_t units = 0;
  for (int i = 0; i < nops; ++i) {
    ops[i].unit_begin = units;
    units += (ops[i].n + 255) / 256;
  }
  CSF_CUDA(cudaMemcpyAsync(work, ops, need, cudaMemcpyHostToDevice, stream));
  if (units == 0) return CSFFCI_OK;
  k_combine_batch<<<grid_for(units, 1, 148 * 32), 256, 0, stream>>>((const csffci_combine_t*)work, nops, units);
  return check_launch("combine_batch");
}

int csffci_precond_batch(int nops, csffci_precond_t* ops, void* work, size_t work_bytes,
                         cudaStream_t stream) {
  CSF_REQUIRE(nops >= 0, "precond_batch: bad count");
  if (nops == 0) return CSFFCI_OK;
  const size_t need = (size_t)nops * sizeof(csffci_precond_t);
  if (work == nullptr || work_bytes < need) {
    set_error("precond_batch: workspace of %zu bytes < %zu required", work_bytes, need);
    return CSFFCI_ERR_MEMORY;
  }
  int64_t units = 0;
  for (int i = 0; i < nops; ++i) {
    ops[i].unit_begin = units;
    units += (ops[i].n + 255) / 256;
  }
  CSF_CUDA(cudaMemcpyAsync(work, ops, need, cudaMemcpyHostToDevice, stream));
  if (units == 0) return CSFFCI_OK;
  k_precond_batch<<<grid_for(units, 1, 148 * 32), 256, 0, stream>>>((const csffci_precond_t*)work, nops, units);
  return check_launch("precond_batch");
}

}  // extern "C"
