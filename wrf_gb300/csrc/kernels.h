// Host-side launch wrappers of the device kernels (one translation unit per
// kernel family; no relocatable device code needed).
#pragma once
#include <cuda_runtime.h>
#include "common.cuh"

namespace wrfgpu {

struct HaloJob {
  int id;        // field id (3-D or 2-D), ignored for species
  int kind;      // 3 or 2
  int species;   // >= 0: species index (uses q / qo), -1 otherwise
  int old;       // species: 1 = old (_1) copy
  char var;      // reference stagger code: 'u','v','w','p','t'
  char pad[3];
};
constexpr int MAX_HALO_JOBS = 24;
struct HaloJobs {
  int n;
  HaloJob job[MAX_HALO_JOBS];
};

// Fields copied from their padded device rows into contiguous buffers by one
// launch (k_pack_fields): a fixed device buffer, or the current buffer of
// species `species` of member `member`.
struct PackJob {
  const float* src;
  float* dst;
  int member, species;
  int cols, rows, pitch;
};
constexpr int MAX_PACK_JOBS = 32;
struct PackJobs {
  int n;
  PackJob job[MAX_PACK_JOBS];
};

// Stage / iteration arguments shared by the step kernels.
struct StepArgs {
  int rk_step;     // 1..3
  int iteration;   // acoustic iteration (1-based) or 0
  int species;     // species index for scalar kernels
  int flags;       // kernel-specific variant bits
};

// Variant bits of the tendency kernels (rk_tendency pieces).
enum : int {
  TF_ZERO = 1,      // start from zero (zero_tend) instead of accumulating
  TF_ADV = 2,       // advect_u / advect_v / advect_w / advect_scalar / rhs_ph
  TF_PG = 4,        // horizontal_pressure_gradient / pg_buoy_w
  TF_COR = 8,       // coriolis
  TF_CURV = 16,     // curvature
  TF_ALL = 31
};

// Run-time tuned launch variants (the autotuner in driver.cu times them on
// the real step and keeps the fastest).  Every variant of a family computes
// the same bits: they differ only in launch bounds (registers per thread,
// so blocks per SM) or in how many level chunks a column kernel is split into.
enum Tune { TU_PD = 0, TU_ADV, TU_AW, TU_AUV, TU_SUMF, TU_PREP, TU_SSF, TU_SSP, TU_CFL, TU_TENDW, TU_TENDU, TU_TENDV,
            TU_CPRP, TU_AMUT, NTUNE };
constexpr int TUNE_MAXVAR = 4;
constexpr int TUNE_NVAR[NTUNE] = {2, 3, 3, 4, 4, 2, 2, 4, 4, 3, 4, 4, 4, 4};
// (defaults measured on 512x512x80 and up: advance_mu_t 278 us with four blocks
// per SM against 393 with two, advance_w 340 against 388; the FP64 form of
// advance_mu_t is best with three, 524 against 571 us on the 16-member ensemble)
constexpr int TUNE_DEFAULT[NTUNE] = {1, 1, 2, 0, 2, 1, 0, 2, 2, 1, 3, 2, 2, 2};
// the parameter each variant stands for: blocks per SM, level chunks
// (sumflux: of calc_p_rho), or (advance_uv, rk_tend_u, rk_tend_v) 10 b + level
// chunks, b = 3: four 128-thread blocks per SM, b = 4: five.  Level chunks are the
// fewest: level_chunks adds to them.
constexpr int TUNE_PARAM[NTUNE][TUNE_MAXVAR] = {{1, 2, 0, 0}, {2, 3, 4, 0}, {2, 3, 4, 0}, {32, 42, 34, 44}, {1, 2, 4, 8},
                                                {3, 8, 0, 0}, {4, 8, 0, 0}, {1, 2, 4, 8}, {2, 4, 8, 16}, {2, 3, 4, 0},
                                                {32, 42, 34, 44}, {32, 42, 34, 44}, {1, 2, 4, 8}, {2, 3, 4, 5}};

void launch_rk_step_prep(const Launch& L, int nblocks, cudaStream_t s, int var = TUNE_DEFAULT[TU_PREP]);
// one block per row segment of 32 columns (rows jts-1 .. jte), levels over its
// warps; taken up to PREP_ROW_MAX segments.  ms per step, this form against the
// column march: 41x41x41 (84 segments) 0.038 / 0.147, 190x161x60 (972) 0.17 / 0.28,
// 256x256x80 (2322) 0.39 / 0.45, 24 small members (about 3000) 0.49 / 0.44.
constexpr int PREP_ROW_MAX = 2500;
void launch_rk_step_prep_row(const TileLaunch& L, int nblocks, cudaStream_t s);
void launch_fill_halo(const Mem* d_mems, int nmem, const HaloJobs& jobs, int blocks_per_job, cudaStream_t s);

// rk_tendency
void launch_tend_u(const Launch& L3, int nblocks, int flags, cudaStream_t s);
void launch_tend_v(const Launch& L3, int nblocks, int flags, cudaStream_t s);
void launch_tend_w(const Launch& L2, int nblocks, int flags, cudaStream_t s);
void launch_tend_w_col(const TileLaunch& L, int nblocks, int var, cudaStream_t s);  // TF_ALL, staggered tiles, tuned
void launch_tend_t(const Launch& L3, int nblocks, int flags, cudaStream_t s);
void launch_tend_ph(const Launch& L3, int nblocks, int flags, cudaStream_t s);
// column forms over tiles of the staggered extents
void launch_tend_u_col(const TileLaunch& L, int nblocks, cudaStream_t s, int var = 0);
void launch_tend_v_col(const TileLaunch& L, int nblocks, cudaStream_t s, int var = 0);
void launch_tend_t_col(const TileLaunch& L, int nblocks, int flags, cudaStream_t s);
void launch_tend_ph_col(const TileLaunch& L, int nblocks, int flags, cudaStream_t s);
// sixth-order diffusion of the dry state at stage 1, and rk_addtend_dry (k_diff.cu)
// mode 0: u, v, w, theta into ru_tendf .. t_tendf; 1: nsp species into sc_tend
void launch_forward_diff(const TileLaunch& L, int nblocks, int mode, cudaStream_t s, int nsp = 0);
void launch_species_diff_routine(const Launch& L, int nblocks, int qv, cudaStream_t s);
void launch_addtend_dry_routine(const Launch& L, int nblocks, int rk_step, cudaStream_t s);
void launch_rayleigh_damp(const Launch& L2, int nblocks, cudaStream_t s, bool acc_all = false);
void launch_addtend_dry(const TileLaunch& L, int nblocks, cudaStream_t s);  // staggered tiles

// acoustic steps
// 2-D part over column blocks, then the 3-D part over staggered tiles x level chunks
void launch_small_step_prep(const Launch& L2, int nb2, const TileLaunch& LST, int nb_st, StepArgs a, cudaStream_t s,
                            int var = TUNE_DEFAULT[TU_SSP]);
void launch_calc_p_rho(const Launch& L3, int nblocks, StepArgs a, cudaStream_t s);
void launch_calc_coef_w(const Launch& L2, int nblocks, StepArgs a, bool fp64, cudaStream_t s);
void launch_calc_coef_w_col(const TileLaunch& L, int nblocks, StepArgs a, bool fp64, cudaStream_t s);  // mass tiles
// mass row segments, FP32, up to COEF_ROW_MAX of them (its recursion runs in one
// warp of a block): ms per step, this form / the column march, 41x41x41 (82 segments)
// 0.037 / 0.083, 160x144x64 (720) 0.099 / 0.139, 190x161x60 (966) 0.129 / 0.136,
// 224x192x64 (1344) 0.141 / 0.151, 256x210x80 (1680) 0.221 / 0.184, 256x256x80 (2048)
// 0.270 / 0.196; FP64 75x90x128 (270) 0.43 / 0.40.  Timed alone the forms are level near
// 1500 segments, but in the step, beside the halo fill, this one's blocks cost more than
// it gains from 966 on (whole step 2.578 / 2.515, at 1344 3.536 / 3.448): the line is
// below that
constexpr int COEF_ROW_MAX = 900;
void launch_calc_coef_w_row(const TileLaunch& L, int nblocks, StepArgs a, cudaStream_t s);
void launch_advance_uv(const Launch& L3, int nblocks, StepArgs a, cudaStream_t s);
void launch_advance_mu_t(const Launch& L2, int nblocks, StepArgs a, bool fp64, cudaStream_t s);
void launch_advance_w(const Launch& L2, int nblocks, StepArgs a, bool fp64, cudaStream_t s);
void launch_sumflux_p_rho(const Launch& L3, int nblocks, StepArgs a, bool do_p_rho, cudaStream_t s);
void launch_sumflux(const Launch& L3, int nblocks, StepArgs a, cudaStream_t s);
// calc_mus: calc_mu_uv_1 fused in (the step); false: the caller's muus, muvs
void launch_small_step_finish(const Launch& L2, int nblocks, StepArgs a, cudaStream_t s, int var = TUNE_DEFAULT[TU_SSF],
                              bool calc_mus = true);

// scalars and diagnosis
void launch_update_scalar_pd(const Launch& L3, int nblocks, StepArgs a, cudaStream_t s);
void launch_advect_scalar(const Launch& L3, int nblocks, StepArgs a, cudaStream_t s);
// advect_scalar_pd of one species into advect_tend (accum: added to it), mass
// tiles; and of species 0 of one member given by value
void launch_advect_scalar_pd(const TileLaunch& L, int nblocks, int species, int rk_step, bool accum, cudaStream_t s);
void launch_advect_scalar_pd_member(const Mem& m, int rk_step, bool accum, cudaStream_t s);
void launch_update_scalar(const Launch& L3, int nblocks, StepArgs a, cudaStream_t s);
void launch_update_scalar_routine(const Launch& L3, int nblocks, int rk_step, int pd, cudaStream_t s);
void launch_calc_p_rho_phi(const Launch& L3, int nblocks, cudaStream_t s);
// host <-> device field copies through a contiguous staging buffer
void launch_unpack_rows(const float* src, float* dst, float* dst2, int cols, int rows, int pitch, cudaStream_t s);
void launch_unpack_species(const Mem* mems, int member, int s, const float* src, int cols, int rows, int pitch,
                           cudaStream_t st);
void launch_pack_fields(const Mem* mems, const PackJobs& jobs, cudaStream_t st);
// mass tiles x level chunks; iteration 0: step 0 of the stage, else the acoustic step (img: halo images stored; the
// acoustic step always does)
void launch_calc_p_rho_col(const TileLaunch& L, int nblocks, StepArgs a, cudaStream_t s, int chunks = 4,
                           bool img = false);
// sct: some member stores the species' sixth-order diffusion tendency sc_tend
void launch_update_scalar_pd_col(const TileLaunch& L, int nblocks, StepArgs a, cudaStream_t s, bool sct = false);  // mass tiles
void launch_calc_p_rho_phi_col(const TileLaunch& L, int nblocks, cudaStream_t s, int var = TUNE_DEFAULT[TU_CPRP]);  // mass tiles
void launch_set_w_surface(const Launch& L2, int nblocks, cudaStream_t s);
void launch_cfl_check_col(const TileLaunch& L, int nblocks, cudaStream_t s, int var = TUNE_DEFAULT[TU_CFL]);  // mass tiles

// fused scalar transport (k_scalar_fused.cu): one block per (tile, pair of
// species); `pairs` selects the pairs this launch transports (bit p: pair p)
void launch_scalar_adv_update(const TileLaunch& L, int nblocks, int rk_step, cudaStream_t s, int var = TUNE_DEFAULT[TU_ADV],
                              bool sct = false, unsigned pairs = ~0u);
// the face Courant numbers of the PD transport, once per step before it (column layout)
void launch_pd_courant(const Launch& L2, int nblocks, int rk_step, cudaStream_t s);
// nlev_max: the largest kme - kms + 1 of the members (sizes a per-level table in shared memory)
void launch_scalar_pd_update(const TileLaunch& L, int nblocks, int nlev_max, int rk_step, cudaStream_t s,
                             int var = TUNE_DEFAULT[TU_PD], unsigned pairs = ~0u);
// pairs: as for the transport
void launch_swap_species(Mem* d_mems, int nmem, cudaStream_t s, unsigned pairs = ~0u);

// the acoustic step (k_acoustic_col.cu): one block per tile of the staggered
// extents, then either one block per row segment of 32 mass columns
// (advance_mu_t, advance_w, sumflux's ww_m, calc_p_rho) or one thread per
// mass column (advance_mu_t and ww_m, then advance_w), then calc_p_rho
void launch_advance_uv_col(const TileLaunch& L, int nblocks, int rk_step, int iteration, cudaStream_t s,
                           int var = TUNE_DEFAULT[TU_AUV]);
// The largest number of row segments (all members) that k_advance_col takes.
// Its time grows with the number of blocks from the start; the three marching
// kernels take about 1.5 us per level until their 256-column tiles fill the
// GPU.  Measured on GB300, ms per large step, column kernel against marches:
// FP32  41x41x41 (82 segments) 0.15 / 0.80, 100x70x30 (280) 0.13 / 0.64,
// 190x161x60 (966) 0.77 / 1.33, 256x256x80 (2048) 1.70 / 1.99, 24 small members
// (about 2900) 2.23 / 2.30, 512x512x80 (8192) 6.30 / 5.67, 1024x1024x96 (32768)
// 29.0 / 24.9; FP64 columns (whose chains wait about 110 cycles per operation)
// 75x90x128 (270) 0.81 / 3.11, 200x170x80 (1190) 1.75 / 2.21, 256x256x80 (2048)
// 3.01 / 2.48, 384x320x80 (3840) 5.46 / 4.12, 512x384x80 (6144) 8.62 / 6.10, 16 members
// of up to 256x256x80 (about 14000) 17.5 / 9.3; with damp_opt = 3 160x144x64 (720)
// 0.76 / 1.39.  The FP64 forms cross between 1190 and 2048 segments; 1000 is on the
// column kernel's side, short of the crossing.
constexpr int col_max_segments(bool fp64) { return fp64 ? 1000 : 3000; }
// damp: some member uses damp_opt = 3 (compiles the damping into the kernel)
void launch_advance_col(const TileLaunch& L, int nblocks, int nlev_max, int rk_step, int iteration, bool fp64,
                        cudaStream_t s, bool damp = false);
void launch_advance_mu_t_col(const TileLaunch& L, int nblocks, int rk_step, int iteration, bool fp64, cudaStream_t s,
                             int var = TUNE_DEFAULT[TU_AMUT]);
void launch_advance_w_col(const TileLaunch& L, int nblocks, int rk_step, int iteration, bool fp64, cudaStream_t s,
                          int var = TUNE_DEFAULT[TU_AW], bool damp = false);

// edge strips of members with open lateral boundaries (open_adv.cuh): the
// tendencies of u, v, theta and ph after their tile kernels (k_tend.cu), rw_tend
// before its tile kernel (per column), and the scalar transport after its
// tile kernels (k_scalar.cu)
void launch_strip_tend(const StripLaunch& L, int nblocks, cudaStream_t s);
void launch_strip_tend_w(const StripLaunch& L, int nblocks, cudaStream_t s);
void launch_strip_scalar(const StripLaunch& L, int nblocks, int rk_step, int nsp_max, cudaStream_t s);
// the positive-definite species at the last stage, through the member's
// scratch (strip_cols of `wide` x levels x species floats): limiter factors over
// `wide`, then the limited divergence and update over L
void launch_strip_pd(const StripLaunch& wide, int nb_wide, const StripLaunch& L, int nb, int rk_step, int nsp_max,
                     float* const* d_scratch, cudaStream_t s);

}  // namespace wrfgpu
