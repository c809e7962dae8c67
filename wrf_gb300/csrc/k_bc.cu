// On-device halo fill: the single-GPU replacement of the reference's
// set_physical_bc3d / set_physical_bc2d (share/module_bc.F:202-1107) at each
// sync site of solve_em, for periodic or open lateral boundaries in x and
// periodic, symmetric or open boundaries in y.
//
// The reference fills the x halo first and then copies whole rows into the
// y halo, so every halo point ends up holding the value of one other point:
// its periodic image, its mirror image (with a sign change for the normal
// velocity v), or, next to an open boundary, the edge value copied into
// three halo points (module_bc.F:864-1107, for the variables of
// open_bc_copy).  This kernel computes that source point directly, so all
// points of a field are written in one pass with no ordering between them.
// The points written and the values they receive are the reference's,
// except the never-read column ime of fields that are not x-staggered,
// which the reference fills with whatever its x pass left there and this
// kernel leaves untouched.
// Roofline: pure copy, 2 x 4 B per halo point; a few percent of a step.
#include "common.cuh"
#include "kernels.h"

namespace wrfgpu {

// Source index along one direction of halo index t (1-based domain extent
// n, nper = n - 1 interior mass points).  Periodic: the image one period
// away (|halo| <= 5 < nper, so one conditional add replaces the modulo).
__device__ __forceinline__ int bc_src(int t, int n, bool stag, bool periodic, bool normal_flip, bool* neg) {
  const int nper = n - 1;
  if (periodic) return t < 1 ? t + nper : (t > nper ? t - nper : t);
  if (!stag) {
    if (t < 1) return 1 - t;                  // dat(ids-i) = dat(ids+i-1)
    if (t > nper) return 2 * nper + 1 - t;    // dat(ide+i-1) = dat(ide-i)
    return t;
  }
  if (t < 1) { if (normal_flip) *neg = !*neg; return 2 - t; }      // dat(ids-i) = -dat(ids+i)
  if (t > n) { if (normal_flip) *neg = !*neg; return 2 * n - t; }  // dat(ide+i) = -dat(ide-i)
  return t;
}

// Open boundaries (module_bc.F:864-925 in x, :1059-1107 in y): the source of
// halo index t, or t itself where the open copy writes nothing (the fourth
// halo point, and t = ide+3 / ide+4 beyond the three copies).
__device__ __forceinline__ int open_src(int t, int n, bool stag) {
  if (t >= -2 && t <= 0) return 1;
  if (stag) return (t >= n + 1 && t <= n + 3) ? n : t;
  return (t >= n && t <= n + 2) ? n - 1 : t;
}
// open_bc_copy of set_physical_bc3d (module_bc.F:699-704) and
// set_physical_bc2d (:248-251)
__device__ __forceinline__ bool open_copy(char v, bool f3d) {
  if (v == 'u' || v == 'v' || v == 'w' || v == 't' || v == 'x' || v == 'y' || v == 'r' || v == 'p') return true;
  return f3d && (v == 'd' || v == 'e' || v == 'f');
}

// grid: (blocks per job, jobs, members).  Work units: for the x halo
// (periodic x) one (level, row) segment of nxw <= 9 points per thread, for
// the y halo one (level, halo row, 128 points of i) piece per warp, four
// points per lane.  The loads of a thread's x unit and its warp's y unit are all
// issued before the stores of either (a store may alias a later load as far as
// the compiler knows, so copying point by point would wait out one memory
// latency per point).  The points written by
// the two kinds of unit are disjoint and every source point is an interior
// point (or, without periodic x, a point no unit writes), so the units need
// no ordering.
__global__ void k_fill_halo(const Mem* __restrict__ mems, HaloJobs jobs) {
  const Mem& m = block_member(mems, blockIdx.z);
  const HaloJob& J = jobs.job[blockIdx.y];
  float* base = J.species >= 0 ? (J.species < m.nsp ? (J.old ? m.qo[J.species] : m.q[J.species]) : nullptr)
                               : (J.kind == 3 ? m.f3[J.id] : m.f2[J.id - WRFGPU_F2D_BASE]);
  if (!base) return;
  const char var = J.var;
  const bool us = (var == 'u' || var == 'x'), vs = (var == 'v' || var == 'y');
  const int istag = us ? 0 : -1, jstag = vs ? 0 : -1;
  int k_end = 1;
  if (J.kind == 3) {
    k_end = max(1, min(m.kde - 1, m.kte));
    if (var == 'w') k_end = min(m.kde, m.kte);
  }
  const int nk = (J.kind == 3) ? (k_end - m.kts + 1) : 1;
  const bool f3d = J.kind == 3;
  const bool px = m.cf.periodic_x, py = m.cf.periodic_y;
  const bool sy = m.cf.symmetric_ys && m.cf.symmetric_ye;
  const bool copy = open_copy(var, f3d);
  const bool ox = m.cf.open_xs && copy, oy = m.cf.open_ys && copy;  // open on both sides
  constexpr int NXW_MAX = 2 * WRFGPU_HALO + 1;
  // x halo columns written: periodic, ids-4..ids-1 and ide..ide+4+istag;
  // open, ids-3..ids-1 and three past the edge point
  const int nxl = ox ? 3 : WRFGPU_HALO;
  const int xr0 = ox ? (us ? m.ide + 1 : m.ide) : m.ide;
  const int xr1 = ox ? xr0 + 2 : m.ide + 4 + istag;
  const int nxw = nxl + (xr1 - xr0 + 1);  // <= NXW_MAX
  // y halo rows written
  const int ynl = oy ? 3 : WRFGPU_HALO;
  const int yr0 = oy ? (vs ? m.jde + 1 : m.jde) : (py ? m.jde : (vs ? m.jde + 1 : m.jde));
  const int yr1 = oy ? yr0 + 2 : (py ? m.jde + 4 + jstag : (vs ? m.jde + 4 : m.jde + 3));
  const int nyrows = ynl + (yr1 - yr0 + 1);
  // rows of the x units: the domain rows, and with open x and open y the two
  // 3-D rows of the x pass (jts-bdyzone .. jde+jstag+bdyzone, module_bc.F:870)
  // that the y pass does not overwrite
  const bool xextra = ox && oy && f3d;
  const int xj0 = m.jds, xj1 = m.jde + jstag;
  const int nxj = xj1 - xj0 + 1 + (xextra ? 2 : 0);
  const int yi0 = m.ims, yi1 = us ? m.ime : m.ide + 3;
  const int nyi = yi1 - yi0 + 1;
  // source column of x index ti as the x pass leaves it
  auto xsrc = [&](int ti, bool* neg) -> int {
    if (px) return bc_src(ti, m.ide, us, true, false, neg);
    if (ox) return open_src(ti, m.ide, us);
    return ti;
  };
  // 32-bit offsets of (i, k, j) / (i, j) in the field
  const int sk = (int)m.sk, sj = f3d ? (int)m.sj : (int)m.s2;
  auto off = [&](int i, int k, int j) { return (i - m.ims) + (f3d ? (k - m.kms) * sk : 0) + (j - m.jms) * sj; };
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthr = gridDim.x * blockDim.x;
  constexpr int PER = 4;  // points per lane of a y unit
  const int lane = threadIdx.x & 31, warp = tid >> 5, nwarps = nthr >> 5;
  const int npiece = (nyi + 32 * PER - 1) / (32 * PER);
  const int nux = (px || ox) ? nk * nxj : 0, nuy = (py || sy || oy) ? nk * nyrows * npiece : 0;
  // one x and one y unit at a time, the loads of both before the stores of either
  for (int u = tid, w = warp; u < nux || w < nuy; u += nthr, w += nwarps) {
    const bool ux = u < nux, uy = w < nuy;
    float val[NXW_MAX], vy[PER];
    bool neg[PER], negj = false;
    int k = 0, tj = 0, ky = 0, tjy = 0, pc = 0;
    if (ux) {
      const int kk = u / nxj, r = u - kk * nxj;
      k = kk + m.kts;
      tj = r <= xj1 - xj0 ? xj0 + r : (r == xj1 - xj0 + 1 ? m.jds - WRFGPU_HALO : m.jde + jstag + WRFGPU_HALO);
      const int sjj = (py || sy) ? bc_src(tj, m.jde, vs, py, var == 'v', &negj) : tj;
      const int row = off(0, k, sjj);
#pragma unroll
      for (int c = 0; c < NXW_MAX; ++c) {
        if (c < nxw) {
          const int ti = c < nxl ? m.ids - nxl + c : xr0 + (c - nxl);
          bool n = false;
          val[c] = base[row + xsrc(ti, &n)];
        }
      }
    }
    if (uy) {
      const int row = w / npiece, kk = row / nyrows, r = row - kk * nyrows;
      pc = w - row * npiece;
      ky = kk + m.kts;
      tjy = r < ynl ? m.jds - ynl + r : yr0 + (r - ynl);
      bool nj = false;
      const int sjj = oy ? open_src(tjy, m.jde, vs) : bc_src(tjy, m.jde, vs, py, var == 'v', &nj);
      const int from = off(0, ky, sjj);
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const int ii = pc * 32 * PER + q * 32 + lane;
        neg[q] = nj;
        if (ii < nyi) vy[q] = base[from + xsrc(yi0 + ii, &neg[q])];
      }
    }
    if (ux) {
      const int row = off(0, k, tj);
#pragma unroll
      for (int c = 0; c < NXW_MAX; ++c) {
        if (c < nxw) {
          const int ti = c < nxl ? m.ids - nxl + c : xr0 + (c - nxl);
          base[row + ti] = negj ? -val[c] : val[c];
        }
      }
    }
    if (uy) {
      const int row = off(yi0, ky, tjy);
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const int ii = pc * 32 * PER + q * 32 + lane;
        if (ii < nyi) base[row + ii] = neg[q] ? -vy[q] : vy[q];
      }
    }
  }
}

// Row copies between a contiguous buffer (rows of `cols` values, the
// caller's Fortran layout) and a field's padded device rows (`pitch` apart);
// `dst2`, when given, receives the same rows (a species' spare buffer).  One
// warp per row, the rows grid-strided over a grid of a few blocks per SM:
// coalesced loads and stores, and no launch of one tiny block per row
// fragment.
__device__ __forceinline__ void copy_rows(const float* __restrict__ src, size_t src_pitch, float* __restrict__ dst,
                                          float* __restrict__ dst2, size_t dst_pitch, int cols, int rows) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarp = (gridDim.x * blockDim.x) >> 5;
  for (int r = warp; r < rows; r += nwarp) {
    const float* sr = src + (size_t)r * src_pitch;
    float* dr = dst + (size_t)r * dst_pitch;
    float* dr2 = dst2 ? dst2 + (size_t)r * dst_pitch : nullptr;
    for (int c = lane; c < cols; c += 32) {
      const float v = sr[c];
      dr[c] = v;
      if (dr2) dr2[c] = v;
    }
  }
}
__global__ void k_unpack_rows(const float* __restrict__ src, float* __restrict__ dst, float* __restrict__ dst2,
                              int cols, int rows, int pitch) {
  copy_rows(src, cols, dst, dst2, pitch, cols, rows);
}
// The same for species s of member `member`, whose current and spare buffers
// are read from the device member table when the copy runs (the buffers
// exchange roles at every scalar update, so a captured copy must not hold
// their addresses).  Unpacking writes both buffers.
__global__ void k_unpack_species(const Mem* __restrict__ mems, int member, int s, const float* __restrict__ src,
                                 int cols, int rows, int pitch) {
  copy_rows(src, cols, mems[member].q[s], mems[member].qa[s], pitch, cols, rows);
}
// Several fields into their contiguous buffers, one per blockIdx.y.  A buffer
// may be page-locked host memory: the rows then cross the link as stores, with
// no staging copy and no copy of its own.
__global__ void k_pack_fields(const Mem* __restrict__ mems, const __grid_constant__ PackJobs jobs) {
  const PackJob& J = jobs.job[blockIdx.y];
  const float* src = J.species < 0 ? J.src : mems[J.member].q[J.species];
  copy_rows(src, J.pitch, J.dst, nullptr, J.cols, J.cols, J.rows);
}
static int rows_grid(int rows) {  // 256-thread blocks of 8 row-warps, at most 8 blocks per SM of 152
  return rows / 8 + 1 < 8 * 152 ? rows / 8 + 1 : 8 * 152;
}
void launch_unpack_rows(const float* src, float* dst, float* dst2, int cols, int rows, int pitch, cudaStream_t s) {
  if (cols > 0 && rows > 0) k_unpack_rows<<<rows_grid(rows), 256, 0, s>>>(src, dst, dst2, cols, rows, pitch);
}
void launch_unpack_species(const Mem* mems, int member, int s, const float* src, int cols, int rows, int pitch,
                           cudaStream_t st) {
  if (cols > 0 && rows > 0) k_unpack_species<<<rows_grid(rows), 256, 0, st>>>(mems, member, s, src, cols, rows, pitch);
}
void launch_pack_fields(const Mem* mems, const PackJobs& jobs, cudaStream_t st) {
  if (jobs.n <= 0) return;
  int rows = 0;
  for (int q = 0; q < jobs.n; ++q) rows = jobs.job[q].rows > rows ? jobs.job[q].rows : rows;
  const int per = 8 * 152 / jobs.n;
  const int g = rows / 8 + 1 < per ? rows / 8 + 1 : per;
  k_pack_fields<<<dim3(g, jobs.n), 256, 0, st>>>(mems, jobs);
}

void launch_fill_halo(const Mem* d_mems, int nmem, const HaloJobs& jobs, int blocks_per_job, cudaStream_t s) {
  if (jobs.n <= 0 || nmem <= 0) return;
  k_fill_halo<<<dim3(blocks_per_job, jobs.n, nmem), 256, 0, s>>>(d_mems, jobs);
}

}  // namespace wrfgpu
