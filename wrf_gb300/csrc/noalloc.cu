// advect_scalar_pd on the caller's device arrays, with no device allocation.
//
// Who needs it: a caller whose arrays already live on the GPU (a driver that
// keeps its state device-resident, e.g. a CUDA Fortran or OpenACC port of
// solve_em) and that cannot allocate at this point — its device memory is
// budgeted up front for the resident state, and cudaMalloc / cudaFree would
// also synchronize the device under its other streams.  The routine-level
// entry point wrfgpu_advect_scalar_pd copies host arrays into a cached device
// domain, which it allocates on first use; this variant runs the same kernel
// (pd_tile, k_scalar.cu) on the caller's pointers, which reach it in the
// member descriptor, a kernel parameter; the limiter factors stay in shared
// memory.  One launch, no device state between calls, no host memory read
// after the call returns.
//
// Limits and rules:
//   * the memory shape (ime-ims+1)(kme-kms+1)(jme-jms+1) may hold at most
//     NOALLOC_MAX_POINTS points (8 Mi: a 256 x 256 x 120 patch); larger
//     requests return WRFGPU_E_SIZE and launch nothing;
//   * the options are those a device domain accepts (periodic x, periodic or
//     symmetric y, 5th/3rd-order advection, ...): anything else returns
//     WRFGPU_E_ARG before any device work;
//   * the kernel has no device-side failure (no bounded wait, no health
//     check): the return code reports argument and launch errors, and there
//     is no device status word to read back.
#include <cstring>
#include "common.cuh"
#include "kernels.h"
#include "fcall.h"
#include "../../include/wrfgpu_fortran.h"

namespace wrfgpu {
constexpr long long NOALLOC_MAX_POINTS = 8ll * 1024 * 1024;
}  // namespace wrfgpu

using namespace wrfgpu;

extern "C" int wrfgpu_advect_scalar_pd_noalloc(
    const float* field, const float* field_old, float* tendency, const float* ru, const float* rv, const float* rom,
    const float* c1, const float* c2, const float* mut, const float* mub, const float* mu_old,
    const WrfDynConfig* config_flags, const float* msftx, const float* msfty, const float* fzm, const float* fzp,
    const float* rdx, const float* rdy, const float* rdzw, const float* dt, WRFGPU_DIMS_ARGS, void* stream) {
  const int* d[18] = {ids, ide, jds, jde, kds, kde, ims, ime, jms, jme, kms, kme, its, ite, jts, jte, kts, kte};
  for (int q = 0; q < 18; ++q)
    if (!d[q]) return WRFGPU_E_ARG;
  if (!field || !field_old || !tendency || !ru || !rv || !rom || !c1 || !c2 || !mut || !mub || !mu_old ||
      !config_flags || !msftx || !msfty || !fzm || !fzp || !rdx || !rdy || !rdzw || !dt)
    return WRFGPU_E_ARG;
  // the serial build's index space, one tile covering the patch (as the
  // routine-level entry points require)
  if (*ids != 1 || *jds != 1 || *kds != 1) return WRFGPU_E_ARG;
  if (*ims != 1 - WRFGPU_HALO || *ime != *ide + WRFGPU_HALO || *jms != 1 - WRFGPU_HALO ||
      *jme != *jde + WRFGPU_HALO || *kms != 1 || *kme != *kde)
    return WRFGPU_E_ARG;
  if (*its != 1 || *ite != *ide || *jts != 1 || *jte != *jde || *kts != 1 || *kte != *kde) return WRFGPU_E_ARG;
  if (*ide < 8 || *jde < 8 || *kde < 6 || *kde > KDE_MAX) return WRFGPU_E_ARG;  // the limits of a member
  const long long ni = *ime - *ims + 1, nk = *kme - *kms + 1, nj = *jme - *jms + 1;
  if (ni * nk * nj > NOALLOC_MAX_POINTS) return WRFGPU_E_SIZE;
  if (!(*dt > 0.f) || !(*rdx > 0.f) || !(*rdy > 0.f)) return WRFGPU_E_ARG;
  {  // the options a device domain accepts
    WrfGpuDomainDesc d{};
    d.ide = *ide; d.jde = *jde; d.kde = *kde; d.n_moist = 1; d.n_scalar = 0;
    d.config = *config_flags;
    d.scalars.dt = *dt; d.scalars.dx = 1.0 / *rdx; d.scalars.dy = 1.0 / *rdy;
    d.scalars.rdx = *rdx; d.scalars.rdy = *rdy;
    if (check_desc(d)) return WRFGPU_E_ARG;
  }

  Mem M;
  std::memset(&M, 0, sizeof(Mem));
  M.ids = *ids; M.ide = *ide; M.jds = *jds; M.jde = *jde; M.kds = *kds; M.kde = *kde;
  M.ims = *ims; M.ime = *ime; M.jms = *jms; M.jme = *jme; M.kms = *kms; M.kme = *kme;
  M.its = *its; M.ite = *ite; M.jts = *jts; M.jte = *jte; M.kts = *kts; M.kte = *kte;
  M.sk = ni; M.sj = ni * nk; M.s2 = ni;
  M.f3[WRFGPU_RU_M] = const_cast<float*>(ru);
  M.f3[WRFGPU_RV_M] = const_cast<float*>(rv);
  M.f3[WRFGPU_WW_M] = const_cast<float*>(rom);
  M.f3[WRFGPU_ADVECT_TEND] = tendency;
  M.f2[WRFGPU_MUTS - WRFGPU_F2D_BASE] = const_cast<float*>(mut);
  M.f2[WRFGPU_MUB - WRFGPU_F2D_BASE] = const_cast<float*>(mub);
  M.f2[WRFGPU_MU_1 - WRFGPU_F2D_BASE] = const_cast<float*>(mu_old);
  M.f2[WRFGPU_MSFTX - WRFGPU_F2D_BASE] = const_cast<float*>(msftx);
  M.f2[WRFGPU_MSFTY - WRFGPU_F2D_BASE] = const_cast<float*>(msfty);
  M.f1[WRFGPU_C1H - WRFGPU_F1D_BASE] = const_cast<float*>(c1);
  M.f1[WRFGPU_C2H - WRFGPU_F1D_BASE] = const_cast<float*>(c2);
  M.f1[WRFGPU_FNM - WRFGPU_F1D_BASE] = const_cast<float*>(fzm);
  M.f1[WRFGPU_FNP - WRFGPU_F1D_BASE] = const_cast<float*>(fzp);
  M.f1[WRFGPU_RDNW - WRFGPU_F1D_BASE] = const_cast<float*>(rdzw);
  M.q[0] = const_cast<float*>(field);
  M.qo[0] = const_cast<float*>(field_old);
  M.nsp = 1; M.n_moist = 1;
  M.ns_total = 1;
  M.dt = *dt; M.dtrk_fix = *dt;
  M.rdx = *rdx; M.rdy = *rdy;
  M.cf = *config_flags;
  M.err = nullptr;  // the PD kernel raises no device status

  // rk_step 3: the last stage, where the reference applies the PD scheme; the
  // tendency accumulates into the caller's array, as advect_scalar_pd does
  launch_advect_scalar_pd_member(M, 3, true, (cudaStream_t)stream);
  if (cudaGetLastError() != cudaSuccess) return WRFGPU_E_CUDA;
  return WRFGPU_OK;
}
