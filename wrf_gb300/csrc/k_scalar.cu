// Scalar transport and diagnosis kernels:
//   rk_update_scalar_pd  dyn_em/module_em.F:1803-1916 (physics tendency 0)
//   advect_scalar        dyn_em/module_advect_em.F:3394-3650, :4306-4333
//   advect_scalar_pd     dyn_em/module_advect_em.F:6505-6779, :7595-7645, limiter :7681-7781,
//                        divergence :7783-7883 — routine-level calls: pd_tile, one launch, the
//                        face fluxes and limiter factors of a tile in shared memory; edge
//                        strips of the large step: the factors into a scratch, then the
//                        divergence of the limited fluxes (a face is only ever modified by its
//                        upwind cell, so the result does not depend on the reference's loop order)
//   rk_update_scalar     dyn_em/module_em.F:1587-1799
//   calc_p_rho_phi       dyn_em/module_big_step_utilities_em.F:953-1226 (non-hydrostatic)
//   set_w_surface        dyn_em/module_bc_em.F:1196-1295
// Roofline: calc_p_rho_phi and rk_update_scalar are HBM-bound; pd_tile and the
// strips are bound by instructions and latency (measured beside each).
#include "common.cuh"
#include "kernels.h"
#include "ffmath.h"
#include "open_adv.cuh"

namespace wrfgpu {

__device__ __forceinline__ bool mass_pt(const Mem& m, int i, int j) {
  return i >= m.its && i <= min(m.ite, m.ide - 1) && j >= m.jts && j <= min(m.jte, m.jde - 1);
}

// ------------------------------------------------------------ rk_update_scalar_pd
__global__ void __launch_bounds__(BX* BY) k_update_scalar_pd(Launch L, int rk_step) {
  BlockPos bp = block_pos(L);
  const Mem& m = block_member(L.mem, bp.m);
  if (!bp.valid) return;
  const int i = bp.i, j = bp.j, k = bp.k;
  if (!mass_pt(m, i, j) || k < m.kts || k > min(m.kte, m.kde - 1)) return;
  const Stage st = stage_of(m, rk_step);
  F1 c1 = f1(m, WRFGPU_C1H), c2 = f1(m, WRFGPU_C2H);
  F2 mu1 = f2(m, WRFGPU_MU_1), mub = f2(m, WRFGPU_MUB);
  const float muold = mu1(i, j) + mub(i, j);
  const float munew = mu1(i, j) + mub(i, j);
  const float tendency = 0.f;
  for (int s = 0; s < m.nsp; ++s) {
    int adv = s < m.n_moist ? m.cf.moist_adv_opt : m.cf.scalar_adv_opt;
    if (adv != 1) continue;
    F3 q = f3p(m, m.qo[s]);
    q(i, k, j) = ((c1(k) * muold + c2(k)) * q(i, k, j) + st.dt_rk * tendency) / (c1(k) * munew + c2(k));
  }
}

// Column form over mass tiles x level chunks (gridDim.y), species outermost,
// eight levels of loads in flight.
template <bool SCT>
__global__ void __launch_bounds__(TX* TY) k_update_scalar_pd_col(TileLaunch L, int rk_step) {
  const TilePos tp = tile_pos(L, false, false);
  const Mem& m = block_member(L.mem, tp.m);
  const int i = tp.i0 + threadIdx.x, j = tp.j0 + threadIdx.y;
  if (!mass_pt(m, i, j)) return;
  const int kts = m.kts, ktf = min(m.kte, m.kde - 1);
  const int per = (ktf - kts + 1 + (int)gridDim.y - 1) / (int)gridDim.y;
  const int k0 = kts + (int)blockIdx.y * per, k1 = min(ktf, k0 + per - 1);
  const Stage st = stage_of(m, rk_step);
  F1 c1 = f1(m, WRFGPU_C1H), c2 = f1(m, WRFGPU_C2H);
  const float muold = f2(m, WRFGPU_MU_1)(i, j) + f2(m, WRFGPU_MUB)(i, j);
  const float munew = f2(m, WRFGPU_MU_1)(i, j) + f2(m, WRFGPU_MUB)(i, j);
  for (int s = 0; s < m.nsp; ++s) {
    int adv = s < m.n_moist ? m.cf.moist_adv_opt : m.cf.scalar_adv_opt;
    if (adv != 1) continue;
    F3 q = f3p(m, m.qo[s]);
    // tendency = 0 + sc_tend (the stage-1 sixth-order diffusion, if any);
    // the reference zeroes sc_tend here (:1893), so no later stage adds it
    float* sc = SCT ? sc_tend_of(m, s) : nullptr;
    if (sc == nullptr) {
      const float tendency = 0.f;
      chunked_levels<8, float>(
          k0, k1, [&](int k, float& v) { v = q(i, k, j); },
          [&](int k, const float& v) {
            q(i, k, j) = ((c1(k) * muold + c2(k)) * v + st.dt_rk * tendency) / (c1(k) * munew + c2(k));
          });
    } else {
      F3 sct = f3p(m, sc);
      for (int k = k0; k <= k1; ++k) {
        float tendency = 0.f;
        tendency = tendency + sct(i, k, j);
        q(i, k, j) = ((c1(k) * muold + c2(k)) * q(i, k, j) + st.dt_rk * tendency) / (c1(k) * munew + c2(k));
      }
    }
  }
}

// ------------------------------------------------------------ advect_scalar (+ zero_tend)
__device__ __forceinline__ bool pd_applies(const Mem& m, int species, int rk_step) {
  int adv = species < m.n_moist ? m.cf.moist_adv_opt : m.cf.scalar_adv_opt;
  return rk_step == m.cf.rk_ord && adv == 1;
}

// mode 0: always; mode 1: skip members whose species is advected by the
// positive-definite scheme at this stage (module_em.F:1265-1280).
__global__ void __launch_bounds__(BX* BY) k_advect_scalar(Launch L, int species, int rk_step, int mode) {
  BlockPos bp = block_pos(L);
  const Mem& m = block_member(L.mem, bp.m);
  if (!bp.valid) return;
  if (species >= m.nsp) return;
  const bool accum = (mode & 4) != 0;  // tendency += (routine-level callers)
  if ((mode & 3) == 1 && pd_applies(m, species, rk_step)) return;
  const int i = bp.i, j = bp.j, k = bp.k;
  F3 tend = f3(m, WRFGPU_ADVECT_TEND);
  const bool in_zero = i >= m.its && i <= m.ite && j >= m.jts && j <= m.jte && k >= m.kts && k <= m.kte;
  const int ktf = min(m.kte, m.kde - 1);
  if (!(mass_pt(m, i, j) && k >= m.kts && k <= ktf)) {
    if (in_zero && !accum) tend(i, k, j) = 0.f;
    return;
  }
  const F3 fld = f3p(m, m.q[species]);
  const ScalarAdv a{fld, fld, f3(m, WRFGPU_RU_M), f3(m, WRFGPU_RV_M), f3(m, WRFGPU_WW_M), f2(m, WRFGPU_MSFTX),
                    f1(m, WRFGPU_FNM), f1(m, WRFGPU_FNP), f1(m, WRFGPU_RDNW)};
  tend(i, k, j) = adv_scalar_point(m, a, accum ? tend(i, k, j) : 0.f, i, j, k);
}

// ------------------------------------------------------------ advect_scalar_pd
// One species' limited transport into advect_tend, for the routine-level
// entry points: one block per (32 x 8 tile of mass columns, chunk of levels),
// marching up k.  The four input planes of a level (scalar, old scalar, ru, rv:
// the tile and a 4-point halo) arrive by cp.async, three levels ahead — the
// caller's arrays have any pitch and alignment, which a tensor map does not
// take.  Every face flux of the limiter region (tile + 1) is formed once, by
// one thread, into shared memory; the vertical ones stay in registers; one
// barrier per level (the face slots and factor slots are those of
// k_scalar_pd_update, k_scalar_fused.cu, which documents their reuse).  Two
// passes over points formed each flux two (limiter, divergence) times two
// (the face's two cells) times, with its two divisions, from global memory:
// a call on 231 x 180 x 64 took 384 us, with this form 130 us.  Issue-bound.
//
// The arithmetic is that of open_adv.cuh's point functions, term for term, with each
// face's Courant number and low-order factor formed here as k_pd_courant forms them.
struct PdrPlanes {
  static constexpr int HW = TX + 8, HH = TY + 8, HN = HW * HH;  // staged plane, origin (i0 - 4, j0 - 4)
  static constexpr int SW = TX + 2, SH = TY + 2, SN = SW * SH;  // limiter region
  static constexpr int XW = TX + 3, YW = TX + 2;                // x faces [SH][XW], y faces [SH + 1][YW]
  static constexpr int XN = XW * SH, YN = YW * (SH + 1);
  static constexpr int THREADS = SN + SH + YW;  // one per cell, one per face the cells leave out: 384
  static constexpr int RING = 4, FSLOT = 3;
  static constexpr int FLOATS = RING * 4 * HN + FSLOT * 2 * (XN + YN) + 2 * SN;
};
// Constants of level k: a = {c1, c2, rdzw, dz / dt}, b = {fzm, fzp, dz, 0} (dz of the z face k).
struct PdrLevel { float4 a, b; };

__device__ __forceinline__ void pd_tile(const Mem& m, int species, int rk_step, bool accum, int i0, int j0) {
  using P = PdrPlanes;
  extern __shared__ __align__(16) float pdr_smem[];
  const int tid = threadIdx.x;
  const int itf = min(m.ite, m.ide - 1), jtf = min(m.jte, m.jde - 1), ktf = min(m.kte, m.kde - 1);
  const int kts = m.kts, kde = m.kde, kme = m.kme;
  const Chunk ch = level_chunk_of(kts, ktf);
  const int k0 = ch.k0, k1 = ch.k1, L0 = max(kts, k0 - 1), L1 = min(ktf, k1 + 1);
  if (k0 > k1) return;  // block-uniform
  const float dt = stage_of(m, rk_step).dt_rk, rdx = m.rdx, rdy = m.rdy;
  float* ring = pdr_smem;
  float* sXH = ring + P::RING * 4 * P::HN;
  float* sXL = sXH + P::FSLOT * P::XN;
  float* sYH = sXL + P::FSLOT * P::XN;
  float* sYL = sYH + P::FSLOT * P::YN;
  float* sSC = sYL + P::FSLOT * P::YN;
  PdrLevel* sLV = reinterpret_cast<PdrLevel*>(sSC + 2 * P::SN);  // [k - kts]; SN and the rest are multiples of 4 floats
  static_assert((P::RING * 4 * P::HN + P::FSLOT * 2 * (P::XN + P::YN) + 2 * P::SN) % 4 == 0, "level table alignment");
  const F3 f = f3p(m, m.q[species]), fo = f3p(m, m.qo[species]), ru = f3(m, WRFGPU_RU_M), rv = f3(m, WRFGPU_RV_M),
           rom = f3(m, WRFGPU_WW_M), tend = f3(m, WRFGPU_ADVECT_TEND);
  const F2 mut2 = f2(m, WRFGPU_MUTS), msx = f2(m, WRFGPU_MSFTX), msy = f2(m, WRFGPU_MSFTY);
  const F1 c1 = f1(m, WRFGPU_C1H), c2 = f1(m, WRFGPU_C2H), fzm = f1(m, WRFGPU_FNM), fzp = f1(m, WRFGPU_FNP),
           rdzw = f1(m, WRFGPU_RDNW);

  // this thread's elements of a staged plane (indices clamped to the memory extent)
  constexpr int EL = (P::HN + P::THREADS - 1) / P::THREADS;
  int eoff[EL];
#pragma unroll
  for (int q = 0; q < EL; ++q) {
    const int e = min(tid + q * P::THREADS, P::HN - 1);
    const int ei = min(max(i0 - 4 + e % P::HW, m.ims), m.ime), ej = min(max(j0 - 4 + e / P::HW, m.jms), m.jme);
    eoff[q] = f.off(ei, m.kms, ej);
  }
  auto issue = [&](int k) {
    float* dst = ring + (k % P::RING) * 4 * P::HN;
    const int lk = (k - m.kms) * f.sk;
#pragma unroll
    for (int q = 0; q < EL; ++q) {
      const int e = tid + q * P::THREADS;
      if (e < P::HN) {
        cp_async4(dst + e, f.p + eoff[q] + lk);
        cp_async4(dst + P::HN + e, fo.p + eoff[q] + lk);
        cp_async4(dst + 2 * P::HN + e, ru.p + eoff[q] + lk);
        cp_async4(dst + 3 * P::HN + e, rv.p + eoff[q] + lk);
      }
    }
  };
  issue(L0);
  cp_async_commit();
  if (L0 + 1 <= L1) issue(L0 + 1);
  cp_async_commit();
  if (L0 + 2 <= L1) issue(L0 + 2);
  cp_async_commit();
  for (int k = kts + tid; k <= ktf; k += P::THREADS) {
    const float dz = k > kts ? 2.f / (rdzw(k) + rdzw(k - 1)) : 0.f;
    sLV[k - kts].a = make_float4(c1(k), c2(k), rdzw(k), dz / dt);
    sLV[k - kts].b = make_float4(fzm(k), fzp(k), dz, 0.f);
  }

  // this thread's limiter cell and its faces: cells 0..31 of each row on one
  // warp, the rows' last two cells on the next 20 threads, then the x faces
  // of column i0 + 33 and the y faces of row j0 + 9
  const bool has_cell = tid < P::SN;
  int sx, sy;
  bool fx = has_cell, fy = has_cell;
  if (tid < 32 * P::SH) { sy = tid >> 5; sx = tid & 31; }
  else if (has_cell) { const int q = tid - 32 * P::SH; sy = q >> 1; sx = 32 + (q & 1); }
  else if (tid < P::SN + P::SH) { sy = tid - P::SN; sx = P::SW; fx = true; }
  else { sy = P::SH; sx = tid - P::SN - P::SH; fy = true; }
  const int i = i0 - 1 + sx, j = j0 - 1 + sy;
  const int xq = sy * P::XW + sx, yq = sy * P::YW + sx;  // left and bottom face
  const int so = sy * P::SW + sx, o = (sy + 3) * P::HW + sx + 3;  // own point in the factor and staged planes
  const bool xok = fx && i >= m.its - 1 && i <= itf + 2 && j >= m.jts - 1 && j <= jtf + 1;
  const bool yok = fy && i >= m.its - 1 && i <= itf + 1 && j >= m.jts - 1 && j <= jtf + 2;
  const bool cell = has_cell && i >= m.its - 1 && i <= itf + 1 && j >= m.jts - 1 && j <= jtf + 1;
  const bool own = has_cell && sx >= 1 && sx <= TX && sy >= 1 && sy <= TY && i <= itf && j <= jtf;
  float mt = 0.f, mt_x = 0.f, mt_y = 0.f, dx = 1.f, dxdt = 1.f, dy = 1.f, dydt = 1.f, mx = 1.f, my = 1.f, mub = 0.f,
        mu_old = 0.f;
  int ox = 5, oy = 5;
  bool quirk = false, limited = false, xdiv = false, ydiv = false;
  if (xok || yok) { mt = mut2(i, j); mx = msx(i, j); my = msy(i, j); }
  if (xok) {
    ox = open_order_mass(i, m.cf.open_xs, m.cf.open_xe, m.ids, m.ide);
    quirk = ox == 2 && m.cf.open_xs && i == m.ids + 1;
    mt_x = mut2(i - 1, j);
    dx = 2.f / (my + msy(i - 1, j)) / rdx;
    dxdt = dx / dt;
  }
  if (yok) {
    oy = open_order_mass(j, m.cf.open_ys, m.cf.open_ye, m.jds, m.jde);
    mt_y = mut2(i, j - 1);
    dy = 2.f / (mx + msx(i, j - 1)) / rdy;
    dydt = dy / dt;
  }
  if (cell) {
    mub = f2(m, WRFGPU_MUB)(i, j); mu_old = f2(m, WRFGPU_MU_1)(i, j);
    limited = pd_limited(m, i, j);
    xdiv = pd_xdiv(m, i); ydiv = pd_ydiv(m, j);
  }
  // the column's vertical window: scalar at L-1 .. L+2, old scalar at L, L+1, omega of face L+1
  float fm1 = 0.f, f0 = 0.f, fp1 = 0.f, fp2 = 0.f, fo0 = 0.f, fop1 = 0.f, romp1 = 0.f;
  float hz0 = 0.f, lz0 = 0.f, hz1 = 0.f, lz1 = 0.f, hzm = 0.f, lzm = 0.f;  // z faces L, L+1, L-1
  __syncthreads();  // the level table
  // z face kk (pd_fz) from the scalars around it and the old scalars on its two sides
  auto zface = [&](int kk, float q_2, float q_1, float q0, float q1, float o_1, float o0, float vel, float* hi, float* lo) {
    if (kk == 1 || kk == kde) { *hi = 0.f; *lo = 0.f; return; }
    const float4 a = sLV[kk - kts].a, b = sLV[kk - kts].b;
    const float mu = 0.5f * ((a.x * mt + a.y) + (a.x * mt + a.y));
    const float cr = vel * dt / b.z / mu, lf = mu * a.w;
    const float l = lf * flux_upwind(o_1, o0, cr);
    float h;
    if (kk == kts + 1 || kk == ktf) h = vel * (b.x * q0 + b.y * q_1);
    else h = vel * pflux3(q_2, q_1, q0, q1, -vel);
    *lo = l; *hi = h - l;
  };
  if (cell) {
    f0 = f(i, L0, j); fp1 = f(i, L0 + 1, j);
    fp2 = L0 + 2 <= kme ? f(i, L0 + 2, j) : 0.f;
    fo0 = fo(i, L0, j); fop1 = fo(i, L0 + 1, j);
    romp1 = rom(i, L0 + 1, j);
    if (L0 > kts) {
      fm1 = f(i, L0 - 1, j);
      zface(L0, L0 - 2 >= kts ? f(i, L0 - 2, j) : 0.f, fm1, f0, fp1, fo(i, L0 - 1, j), fo0, rom(i, L0, j), &hz0, &lz0);
    }
  }
  float sc_m1 = -1.f, sc_0 = -1.f, sc_p1 = -1.f;  // own column's factors at levels L-2, L-1, L
  // (selections, no branches: a warp's faces have either sign)
  auto lim = [](float h, float sc) { return sc >= 0.f && h != 0.f ? sc * h : h; };
  cp_async_wait<2>();
  __syncthreads();  // level L0 staged
  for (int L = L0; L <= k1 + 1; ++L) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    const int fs = (L % P::FSLOT);
    float *XH = sXH + fs * P::XN, *XL = sXL + fs * P::XN, *YH = sYH + fs * P::YN, *YL = sYL + fs * P::YN;
    if (L <= ktf) {
      a = sLV[L - kts].a;
      const float* Q = ring + (L % P::RING) * 4 * P::HN;
      const float *FO = Q + P::HN, *RU = FO + P::HN, *RV = RU + P::HN;
      const float mk = a.x * mt + a.y;
      if (xok) {  // pd_fx
        const float mu = 0.5f * (mk + (a.x * mt_x + a.y));
        const float r = RU[o];
        float vel = r, cr;
        if (quirk) { vel = r / mu; cr = vel * dt / dx; }
        else cr = vel * dt / dx / mu;
        const float l = (mu * dxdt) * flux_upwind(FO[o - 1], FO[o], cr);
        float h;
        if (ox == 5) h = vel * pflux5(Q[o - 3], Q[o - 2], Q[o - 1], Q[o], Q[o + 1], Q[o + 2], vel);
        else if (ox == 3) h = vel * pflux3(Q[o - 2], Q[o - 1], Q[o], Q[o + 1], vel);
        else h = 0.5f * r * (Q[o] + Q[o - 1]);
        XH[xq] = h - l; XL[xq] = l;
      }
      if (yok) {  // pd_fy
        constexpr int W = P::HW;
        const float mu = 0.5f * (mk + (a.x * mt_y + a.y));
        const float vel = RV[o], cr = vel * dt / dy / mu;
        const float l = (mu * dydt) * flux_upwind(FO[o - W], FO[o], cr);
        float h;
        if (oy == 5) h = vel * pflux5(Q[o - 3 * W], Q[o - 2 * W], Q[o - W], Q[o], Q[o + W], Q[o + 2 * W], vel);
        else if (oy == 3) h = vel * pflux3(Q[o - 2 * W], Q[o - W], Q[o], Q[o + W], vel);
        else h = 0.5f * vel * (Q[o] + Q[o - W]);
        YH[yq] = h - l; YL[yq] = l;
      }
      if (cell) zface(L + 1, fm1, f0, fp1, fp2, fo0, fop1, romp1, &hz1, &lz1);
    }
    cp_async_wait<1>();  // this thread's copies of level L + 1
    __syncthreads();
    if (L + 3 <= L1) issue(L + 3);  // into the slot of level L - 1, read before this barrier
    cp_async_commit();
    // own inputs of the next level, and of the divergence below
    float fp3 = 0.f, fop2 = 0.f, romp2 = 0.f, t = 0.f;
    const int k = L - 1;
    const bool div = own && k >= k0;
    if (cell) {
      fp3 = L + 3 <= kme ? f(i, L + 3, j) : 0.f;
      fop2 = L + 2 <= kme ? fo(i, L + 2, j) : 0.f;
      romp2 = L + 2 <= kme ? rom(i, L + 2, j) : 0.f;
    }
    if (div && accum) t = tend(i, k, j);
    if (L <= ktf && cell) {  // pd_scale_cell
      float sc = -1.f;
      if (limited) {
        const float hx0 = XH[xq], hx1 = XH[xq + 1], lx0 = XL[xq], lx1 = XL[xq + 1];
        const float hy0 = YH[yq], hy1 = YH[yq + P::YW], ly0 = YL[yq], ly1 = YL[yq + P::YW];
        const float ph_low = ((a.x * mub + a.y) + (a.x * mu_old)) * fo0 -
                             dt * (mx * my * (rdx * (lx1 - lx0) + rdy * (ly1 - ly0)) + my * a.z * (lz1 - lz0));
        const float flux_out = dt * ((mx * my) * (rdx * (fmaxf_f(0.f, hx1) - fminf_f(0.f, hx0)) +
                                                  rdy * (fmaxf_f(0.f, hy1) - fminf_f(0.f, hy0))) +
                                     my * a.z * (fminf_f(0.f, hz1) - fmaxf_f(0.f, hz0)));
        if (flux_out > ph_low) sc = fmaxf_f(0.f, ph_low / (flux_out + 1.e-20f));
      }
      sSC[(L & 1) * P::SN + so] = sc;
      sc_p1 = sc;
    }
    if (div) {  // pd_tend_cell of level k = L - 1
      const int ks = k % P::FSLOT;
      const float *kXH = sXH + ks * P::XN, *kXL = sXL + ks * P::XN, *kYH = sYH + ks * P::YN, *kYL = sYL + ks * P::YN;
      const float* SC = sSC + (k & 1) * P::SN;
      t = scalar_radiation(m, f, fo, ru, rv, t, i, j, k);
      float h0 = hzm, h1 = hz0;
      if (k > 1) h0 = lim(h0, h0 < 0.f ? sc_m1 : sc_0);
      if (k + 1 < kde) h1 = lim(h1, h1 < 0.f ? sc_0 : sc_p1);
      t = t - sLV[k - kts].a.z * (h1 - h0 + lz0 - lzm);
      if (xdiv) {
        float g0 = kXH[xq], g1 = kXH[xq + 1];
        const float sm = SC[so - 1], sp = SC[so + 1];
        g0 = lim(g0, g0 > 0.f ? sm : sc_0);
        g1 = lim(g1, g1 > 0.f ? sc_0 : sp);
        t = t - mx * (rdx * (g1 - g0 + kXL[xq + 1] - kXL[xq]));
      }
      if (ydiv) {
        float g0 = kYH[yq], g1 = kYH[yq + P::YW];
        const float sm = SC[so - P::SW], sp = SC[so + P::SW];
        g0 = lim(g0, g0 > 0.f ? sm : sc_0);
        g1 = lim(g1, g1 > 0.f ? sc_0 : sp);
        t = t - mx * (rdy * (g1 - g0 + kYL[yq + P::YW] - kYL[yq]));
      }
      tend(i, k, j) = t;
    }
    sc_m1 = sc_0; sc_0 = sc_p1;
    hzm = hz0; lzm = lz0; hz0 = hz1; lz0 = lz1;
    fm1 = f0; f0 = fp1; fp1 = fp2; fp2 = fp3;
    fo0 = fop1; fop1 = fop2; romp1 = romp2;
  }
  if (!accum && own) {  // zero_tend of the tile's points that hold no mass
    for (int k = k0; k <= (k1 == ktf ? m.kte : k1); ++k) {
      if (k > ktf) tend(i, k, j) = 0.f;
      if (i == itf && m.ite > itf) tend(i + 1, k, j) = 0.f;
      if (j == jtf && m.jte > jtf) tend(i, k, j + 1) = 0.f;
      if (i == itf && m.ite > itf && j == jtf && m.jte > jtf) tend(i + 1, k, j + 1) = 0.f;
    }
  }
}
// of one member given by value (the caller's arrays; no table on the device)
__global__ void __launch_bounds__(PdrPlanes::THREADS, 2) k_pd_tend_member(const __grid_constant__ Mem m, int rk_step, bool accum) {
  const int ntx = tiles_x(m);
  pd_tile(m, 0, rk_step, accum, m.its + ((int)blockIdx.x % ntx) * TX, m.jts + ((int)blockIdx.x / ntx) * TY);
}
__global__ void __launch_bounds__(PdrPlanes::THREADS, 2) k_pd_tend(TileLaunch L, int species, int rk_step, bool accum) {
  const TilePos tp = tile_pos(L, TILE_ONE);
  const Mem& m = block_member(L.mem, tp.m);
  if (species >= m.nsp) return;
  pd_tile(m, species, rk_step, accum, tp.i0, tp.j0);
}

// ------------------------------------------------------------ edge strips
// The large step's scalar transport at the points next to an open boundary
// (open_adv.cuh), recomputed after the tile kernels from the same inputs
// (the arithmetic of k_scalar_adv_update / k_scalar_pd_update, so the
// points the open branches leave alone get the same bits twice), then
// rk_update_scalar into the spare buffer.
__device__ __forceinline__ void strip_update(const Mem& m, int s, int rk_step, int i, int j, int k, float tendency) {
  const Stage st = stage_of(m, rk_step);
  const F2 mu_old = f2(m, WRFGPU_MU_1), mu_new = f2(m, WRFGPU_MU_2), mub = f2(m, WRFGPU_MUB);
  const F1 c1 = f1(m, WRFGPU_C1H), c2 = f1(m, WRFGPU_C2H);
  const float muold = mu_old(i, j) + mub(i, j), munew = mu_new(i, j) + mub(i, j);
  const F3 q = f3p(m, m.q[s]), qo = f3p(m, m.qo[s]), qa = f3p(m, m.qa[s]);
  float q1;
  if (rk_step == 1) { q1 = q(i, k, j); qo(i, k, j) = q1; }
  else q1 = qo(i, k, j);
  qa(i, k, j) = ((c1(k) * muold + c2(k)) * q1 + st.dt_rk * tendency) / (c1(k) * munew + c2(k));
}
// advect_scalar species (every species at stages 1 and 2, the others at the
// last): the tendency plus the stored sc_tend of the species' diffusion.  A
// strip is a few hundred blocks of dependent loads: one species per blockIdx.y
// keeps more loads in flight (190x161x60, 4 species: 33 -> 26 us).
__global__ void __launch_bounds__(STRIP_THREADS) k_strip_scalar(StripLaunch L, int rk_step) {
  const StripPos sp = strip_pos(L);
  const Mem& m = block_member(L.mem, sp.m);
  if (!sp.valid) return;
  const int i = sp.i, j = sp.j, k = sp.k;
  if (!mass_pt(m, i, j) || k < m.kts || k > min(m.kte, m.kde - 1)) return;
  const F2 msfty = f2(m, WRFGPU_MSFTY);
  const int s = blockIdx.y;
  if (s >= m.nsp || pd_applies(m, s, rk_step)) return;
  const F3 fld = f3p(m, m.q[s]);
  const ScalarAdv a{fld, fld, f3(m, WRFGPU_RU_M), f3(m, WRFGPU_RV_M), f3(m, WRFGPU_WW_M), f2(m, WRFGPU_MSFTX),
                    f1(m, WRFGPU_FNM), f1(m, WRFGPU_FNP), f1(m, WRFGPU_RDNW)};
  float tendency = msfty(i, j) * adv_scalar_point(m, a, 0.f, i, j, k);
  const F3 sct = f3p(m, sc_tend_of(m, s));
  if (sct.p) tendency = tendency + sct(i, k, j);
  strip_update(m, s, rk_step, i, j, k, tendency);
}
// advect_scalar_pd species at the last stage, in two passes over every species
// (blockIdx.y): the limiter factors of the strip cells and their neighbours (the
// strip one wider, halo row / column included) into the member's scratch,
// [species][level][strip column], then the limited divergence and the update at
// the strip cells.  190x161x60, 4 species: a pass per species 16 and 19 us each,
// all species at once 56 and 66.
__global__ void __launch_bounds__(STRIP_THREADS) k_strip_pd_scale(StripLaunch L, int rk_step, float* const* scratch) {
  const StripPos sp = strip_pos(L);
  const Mem& m = block_member(L.mem, sp.m);
  const int s = blockIdx.y;
  if (!sp.valid || s >= m.nsp || !pd_applies(m, s, rk_step)) return;
  const int i = sp.i, j = sp.j, k = sp.k;
  if (k < m.kts || k > min(m.kte, m.kde - 1)) return;
  const Stage st = stage_of(m, rk_step);
  const PDCtx c = pd_ctx(m, s, st.dt_rk);
  const long long plane = (long long)strip_cols(m.ide, m.jde, m.cf.open_xs, m.cf.open_ys, L.w, L.h) * (m.kme - m.kms + 1);
  scratch[sp.m][s * plane + sp.p] = pd_scale_cell(m, c, i, k, j);
}
// ww, wh: the strip width and halo rows the factors were stored for
__global__ void __launch_bounds__(STRIP_THREADS) k_strip_pd_tend(StripLaunch L, int rk_step, int ww, int wh,
                                                                float* const* scratch) {
  const StripPos sp = strip_pos(L);
  const Mem& m = block_member(L.mem, sp.m);
  const int s = blockIdx.y;
  if (!sp.valid || s >= m.nsp || !pd_applies(m, s, rk_step)) return;
  const int i = sp.i, j = sp.j, k = sp.k;
  if (!mass_pt(m, i, j) || k < m.kts || k > min(m.kte, m.kde - 1)) return;
  const Stage st = stage_of(m, rk_step);
  const PDCtx c = pd_ctx(m, s, st.dt_rk);
  const int nc = strip_cols(m.ide, m.jde, m.cf.open_xs, m.cf.open_ys, ww, wh);
  const float* sc = scratch[sp.m] + (long long)s * nc * (m.kme - m.kms + 1);
  const float t = pd_tend_cell(m, c, i, k, j, 0.f, [&](int ci, int ck, int cj) {
    return sc[(ck - m.kms) * nc + strip_index(m.ide, m.jde, m.cf.open_xs, ci, cj, ww, wh)];
  });
  strip_update(m, s, rk_step, i, j, k, f2(m, WRFGPU_MSFTY)(i, j) * t);
}
void launch_strip_scalar(const StripLaunch& L, int nb, int rk_step, int nsp_max, cudaStream_t s) {
  if (nb > 0 && nsp_max > 0) k_strip_scalar<<<dim3(nb, nsp_max), STRIP_THREADS, 0, s>>>(L, rk_step);
}
void launch_strip_pd(const StripLaunch& wide, int nb_wide, const StripLaunch& L, int nb, int rk_step, int nsp_max,
                     float* const* d_scratch, cudaStream_t s) {
  if (nb <= 0 || nsp_max <= 0) return;
  k_strip_pd_scale<<<dim3(nb_wide, nsp_max), STRIP_THREADS, 0, s>>>(wide, rk_step, d_scratch);
  k_strip_pd_tend<<<dim3(nb, nsp_max), STRIP_THREADS, 0, s>>>(L, rk_step, wide.w, wide.h, d_scratch);
}

// ------------------------------------------------------------ rk_update_scalar
__global__ void __launch_bounds__(BX* BY) k_update_scalar(Launch L, int species, int rk_step) {
  BlockPos bp = block_pos(L);
  const Mem& m = block_member(L.mem, bp.m);
  if (!bp.valid) return;
  if (species >= m.nsp) return;
  const int i = bp.i, j = bp.j, k = bp.k;
  if (!mass_pt(m, i, j) || k < m.kts || k > min(m.kte, m.kde - 1)) return;
  const Stage st = stage_of(m, rk_step);
  F3 s1 = f3p(m, m.qo[species]), s2 = f3p(m, m.q[species]), at = f3(m, WRFGPU_ADVECT_TEND);
  F2 msfty = f2(m, WRFGPU_MSFTY), mu_old = f2(m, WRFGPU_MU_1), mu_new = f2(m, WRFGPU_MU_2), mub = f2(m, WRFGPU_MUB);
  F1 c1 = f1(m, WRFGPU_C1H), c2 = f1(m, WRFGPU_C2H);
  const float muold = mu_old(i, j) + mub(i, j), munew = mu_new(i, j) + mub(i, j);
  const float tendency = at(i, k, j) * msfty(i, j);
  float q1;
  if (rk_step == 1) { q1 = s2(i, k, j); s1(i, k, j) = q1; }
  else q1 = s1(i, k, j);
  s2(i, k, j) = ((c1(k) * muold + c2(k)) * q1 + st.dt_rk * tendency) / (c1(k) * munew + c2(k));
}

// ------------------------------------------------------------ routine-level scalar updates
// The routine-level C entry points' form of rk_update_scalar
// (module_em.F:1587-1799, pd = 0) and rk_update_scalar_pd (:1803-1916, pd =
// 1) for species 0 of a scratch domain, with the caller's sc_tend carried in
// the H_DIABATIC buffer: tendency = advect_tend msfty (rk_update_scalar only)
// + sc_tend, in the reference's order; rk_update_scalar_pd zeroes sc_tend
// after use and updates the old scalar with mu_old (MU_1) and mu_new (MU_2).
// The loop limits are the periodic / symmetric ones (the spec_zone limits of
// specified boundaries do not apply).
__global__ void __launch_bounds__(BX* BY) k_update_scalar_routine(Launch L, int rk_step, int pd) {
  BlockPos bp = block_pos(L);
  const Mem& m = block_member(L.mem, bp.m);
  if (!bp.valid) return;
  const int i = bp.i, j = bp.j, k = bp.k;
  if (!mass_pt(m, i, j) || k < m.kts || k > min(m.kte, m.kde - 1)) return;
  const Stage st = stage_of(m, rk_step);
  F3 s1 = f3p(m, m.qo[0]), s2 = f3p(m, m.q[0]), at = f3(m, WRFGPU_ADVECT_TEND), sct = f3(m, WRFGPU_H_DIABATIC);
  F2 msfty = f2(m, WRFGPU_MSFTY), mu_old = f2(m, WRFGPU_MU_1), mu_new = f2(m, WRFGPU_MU_2), mub = f2(m, WRFGPU_MUB);
  F1 c1 = f1(m, WRFGPU_C1H), c2 = f1(m, WRFGPU_C2H);
  const float muold = mu_old(i, j) + mub(i, j), munew = mu_new(i, j) + mub(i, j);
  if (pd) {
    float tendency = 0.f;
    tendency = tendency + sct(i, k, j);
    sct(i, k, j) = 0.f;
    s1(i, k, j) = ((c1(k) * muold + c2(k)) * s1(i, k, j) + st.dt_rk * tendency) / (c1(k) * munew + c2(k));
    return;
  }
  float tendency = at(i, k, j) * msfty(i, j);
  tendency = tendency + sct(i, k, j);
  float q1;
  if (rk_step == 1) { q1 = s2(i, k, j); s1(i, k, j) = q1; }
  else q1 = s1(i, k, j);
  s2(i, k, j) = ((c1(k) * muold + c2(k)) * q1 + st.dt_rk * tendency) / (c1(k) * munew + c2(k));
}

// ------------------------------------------------------------ calc_p_rho_phi
__global__ void __launch_bounds__(BX* BY) k_calc_p_rho_phi(Launch L) {
  BlockPos bp = block_pos(L);
  const Mem& m = block_member(L.mem, bp.m);
  if (!bp.valid) return;
  const int i = bp.i, j = bp.j, k = bp.k;
  if (!mass_pt(m, i, j) || k < m.kts || k > min(m.kte, m.kde - 1)) return;
  F3 al = f3(m, WRFGPU_AL), alb = f3(m, WRFGPU_ALB), ph = f3(m, WRFGPU_PH_2), phb = f3(m, WRFGPU_PHB),
     p = f3(m, WRFGPU_P), pb = f3(m, WRFGPU_PB), t = f3(m, WRFGPU_T_2);
  F2 mu = f2(m, WRFGPU_MU_2), muts = f2(m, WRFGPU_MUTS);
  F1 c1 = f1(m, WRFGPU_C1H), c2 = f1(m, WRFGPU_C2H), c3h = f1(m, WRFGPU_C3H), c4h = f1(m, WRFGPU_C4H),
     c3f = f1(m, WRFGPU_C3F), c4f = f1(m, WRFGPU_C4F), rdnw = f1(m, WRFGPU_RDNW);
  const float ptop = m.p_top;
  float alv;
  if (m.cf.hypsometric_opt == 1) {
    alv = -1.f / (c1(k) * muts(i, j) + c2(k)) * (alb(i, k, j) * (c1(k) * mu(i, j)) + rdnw(k) * (ph(i, k + 1, j) - ph(i, k, j)));
  } else {
    float pfu = c3f(k + 1) * muts(i, j) + c4f(k + 1) + ptop;
    float pfd = c3f(k) * muts(i, j) + c4f(k) + ptop;
    float phm = c3h(k) * muts(i, j) + c4h(k) + ptop;
    alv = (ph(i, k + 1, j) - ph(i, k, j) + phb(i, k + 1, j) - phb(i, k, j)) / phm / wrfgpu_ff::logf_cr(pfd / pfu) - alb(i, k, j);
  }
  al(i, k, j) = alv;
  float temp;
  if (m.cf.use_theta_m == 1) {
    temp = (R_D * (T0 + t(i, k, j))) / (P0 * (alv + alb(i, k, j)));
  } else {
    float qvf = 1.f + (461.6f / 287.f) * f3p(m, m.q[0])(i, k, j);
    temp = (R_D * (T0 + t(i, k, j)) * qvf) / (P0 * (alv + alb(i, k, j)));
  }
  float pv = wrfgpu_ff::powf_cr(temp, CPOVCV);
  p(i, k, j) = pv * P0 - pb(i, k, j);
}

// Column form over mass tiles x level chunks (gridDim.y chunks of
// kts..ktf): ph and phb of level k+1 carry down as level k of the next level,
// and so does the full-level pressure above (pfu(k) is pfd(k+1), the same
// expression), so each level reads ph and phb once.
__global__ void __launch_bounds__(TX* TY) k_calc_p_rho_phi_col(TileLaunch L) {
  const TilePos tp = tile_pos(L, false, false);
  const Mem& m = block_member(L.mem, tp.m);
  const int i = tp.i0 + threadIdx.x, j = tp.j0 + threadIdx.y;
  if (!mass_pt(m, i, j)) return;
  const int kts = m.kts, ktf = min(m.kte, m.kde - 1), kme = m.kme;
  const int per = (ktf - kts + 1 + (int)gridDim.y - 1) / (int)gridDim.y;
  const int k0 = kts + (int)blockIdx.y * per, k1 = min(ktf, k0 + per - 1);
  if (k0 > k1) return;
  const F3 al = f3(m, WRFGPU_AL), alb = f3(m, WRFGPU_ALB), ph = f3(m, WRFGPU_PH_2), phb = f3(m, WRFGPU_PHB),
           p = f3(m, WRFGPU_P), pb = f3(m, WRFGPU_PB), t = f3(m, WRFGPU_T_2), qv = f3p(m, m.q[0]);
  const F1 c1 = f1(m, WRFGPU_C1H), c2 = f1(m, WRFGPU_C2H), c3h = f1(m, WRFGPU_C3H), c4h = f1(m, WRFGPU_C4H),
           c3f = f1(m, WRFGPU_C3F), c4f = f1(m, WRFGPU_C4F), rdnw = f1(m, WRFGPU_RDNW);
  const float ptop = m.p_top;
  const float muts_c = f2(m, WRFGPU_MUTS)(i, j), mu_c = f2(m, WRFGPU_MU_2)(i, j);
  const bool hyps1 = m.cf.hypsometric_opt == 1, theta_m = m.cf.use_theta_m == 1;
  float ph_lo = ph(i, k0, j), phb_lo = hyps1 ? 0.f : phb(i, k0, j);
  float pfd = hyps1 ? 0.f : c3f(k0) * muts_c + c4f(k0) + ptop;
  for (int k = k0; k <= k1; ++k) {
    if (k + 3 <= kme) {
      prefetch_l2(&ph(i, k + 3, j)); prefetch_l2(&phb(i, k + 3, j)); prefetch_l2(&alb(i, k + 2, j));
      prefetch_l2(&t(i, k + 2, j)); prefetch_l2(&pb(i, k + 2, j));
      if (!theta_m) prefetch_l2(&qv(i, k + 2, j));
    }
    const float ph_hi = ph(i, k + 1, j);
    const float albk = alb(i, k, j);
    float alv;
    if (hyps1) {
      alv = -1.f / (c1(k) * muts_c + c2(k)) * (albk * (c1(k) * mu_c) + rdnw(k) * (ph_hi - ph_lo));
    } else {
      const float phb_hi = phb(i, k + 1, j);
      const float pfu = c3f(k + 1) * muts_c + c4f(k + 1) + ptop;
      const float phm = c3h(k) * muts_c + c4h(k) + ptop;
      alv = (ph_hi - ph_lo + phb_hi - phb_lo) / phm / wrfgpu_ff::logf_cr(pfd / pfu) - albk;
      pfd = pfu;
      phb_lo = phb_hi;
    }
    al(i, k, j) = alv;
    float temp;
    if (theta_m) {
      temp = (R_D * (T0 + t(i, k, j))) / (P0 * (alv + albk));
    } else {
      float qvf = 1.f + (461.6f / 287.f) * qv(i, k, j);
      temp = (R_D * (T0 + t(i, k, j)) * qvf) / (P0 * (alv + albk));
    }
    const float pv = wrfgpu_ff::powf_cr(temp, CPOVCV);
    p(i, k, j) = pv * P0 - pb(i, k, j);
    ph_lo = ph_hi;
  }
}

// ------------------------------------------------------------ set_w_surface
__global__ void __launch_bounds__(BX* BY) k_set_w_surface(Launch L) {
  BlockPos bp = block_pos(L);
  const Mem& m = block_member(L.mem, bp.m);
  if (!bp.valid) return;
  const int i = bp.i, j = bp.j;
  if (!mass_pt(m, i, j)) return;
  const bool px = m.cf.periodic_x, py = m.cf.periodic_y;
  int jm1_limit = px || py ? m.jds : m.jds, jp1_limit = m.jde - 1, im1_limit = m.ids, ip1_limit = m.ide - 1;
  if (px) { im1_limit = m.ids - 1; ip1_limit = m.ide; }
  if (py) { jm1_limit = m.jds - 1; jp1_limit = m.jde; }
  const int jm1 = max(j - 1, jm1_limit), jp1 = min(j + 1, jp1_limit), im1 = max(i - 1, im1_limit), ip1 = min(i + 1, ip1_limit);
  F3 w = f3(m, WRFGPU_W_2), u = f3(m, WRFGPU_U_2), v = f3(m, WRFGPU_V_2);
  F2 ht = f2(m, WRFGPU_HT), msftx = f2(m, WRFGPU_MSFTX), msfty = f2(m, WRFGPU_MSFTY);
  const float cf1 = m.cf1, cf2 = m.cf2, cf3 = m.cf3;
  w(i, 1, j) = msfty(i, j) * .5f * m.rdy *
                   ((ht(i, jp1) - ht(i, j)) * (cf1 * v(i, 1, j + 1) + cf2 * v(i, 2, j + 1) + cf3 * v(i, 3, j + 1)) +
                    (ht(i, j) - ht(i, jm1)) * (cf1 * v(i, 1, j) + cf2 * v(i, 2, j) + cf3 * v(i, 3, j))) +
               msftx(i, j) * .5f * m.rdx *
                   ((ht(ip1, j) - ht(i, j)) * (cf1 * u(i + 1, 1, j) + cf2 * u(i + 1, 2, j) + cf3 * u(i + 1, 3, j)) +
                    (ht(i, j) - ht(im1, j)) * (cf1 * u(i, 1, j) + cf2 * u(i, 2, j) + cf3 * u(i, 3, j)));
}

// ------------------------------------------------------------ w_damp CFL diagnostics + health
// module_big_step_utilities_em.F:2503-2712 (the diagnostics; the w_damping = 1
// term of rw_tend is applied by the w-tendency kernels, in rk_tendency's order).
// One thread per mass column of a 32x8 tile and one block per (tile, chunk
// of levels 2..kde-1: gridDim.y chunks), the maxima kept in registers and
// reduced once per block (warp shuffles, then shared memory).  A maximum does
// not depend on the order it is taken in, so the result equals the
// reference's loop order's.  Also the health check: any non-finite u, v, w,
// theta or Courant number raises ERR_NONFINITE.
__global__ void __launch_bounds__(TX* TY, 4) k_cfl_check_col(TileLaunch L) {
  const TilePos tp = tile_pos(L, false, false);
  const Mem& m = block_member(L.mem, tp.m);
  const int i = tp.i0 + threadIdx.x, j = tp.j0 + threadIdx.y;
  const int per = (m.kde - 2 + gridDim.y - 1) / gridDim.y;
  const int k0 = 2 + blockIdx.y * per, k1 = min(m.kde - 1, k0 + per - 1);
  float vmax = 0.f, hmax = 0.f;
  bool bad = false;
  if (mass_pt(m, i, j) && k0 <= k1) {
    F3 ww = f3(m, WRFGPU_WW), u = f3(m, WRFGPU_U_2), v = f3(m, WRFGPU_V_2), w = f3(m, WRFGPU_W_2), t = f3(m, WRFGPU_T_2);
    F1 c1f = f1(m, WRFGPU_C1F), c2f = f1(m, WRFGPU_C2F), rdnw = f1(m, WRFGPU_RDNW);
    const float mutc = f2(m, WRFGPU_MUT)(i, j), mux = f2(m, WRFGPU_MSFUX)(i, j), mvy = f2(m, WRFGPU_MSFVY)(i, j);
    const float dt = m.dt, rdx = m.rdx, rdy = m.rdy;
#pragma unroll 4
    for (int k = k0; k <= k1; ++k) {
      const float vc = fabsf(ww.ro(i, k, j) / (c1f(k) * mutc + c2f(k)) * rdnw(k) * dt);
      const float hc = fmaxf_f(fabsf(u.ro(i, k, j) * rdx * mux * dt), fabsf(v.ro(i, k, j) * rdy * mvy * dt));
      // every load unconditional: a short-circuit || would hold the w and t
      // loads back until the other checks are known
      const float wv = w.ro(i, k, j), tv = t.ro(i, k, j);
      bad = bad | !isfinite(vc) | !isfinite(hc) | !isfinite(wv) | !isfinite(tv);
      vmax = fmaxf_f(vmax, isfinite(vc) ? vc : 0.f);
      hmax = fmaxf_f(hmax, isfinite(hc) ? hc : 0.f);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    vmax = fmaxf_f(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    hmax = fmaxf_f(hmax, __shfl_xor_sync(0xffffffffu, hmax, o));
  }
  const bool wbad = __any_sync(0xffffffffu, bad);
  __shared__ float sv[TY], sh[TY];
  __shared__ int sb[TY];
  if (threadIdx.x == 0) { sv[threadIdx.y] = vmax; sh[threadIdx.y] = hmax; sb[threadIdx.y] = wbad ? 1 : 0; }
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y == 0) {
    float bv = 0.f, bh = 0.f;
    int bb = 0;
    for (int q = 0; q < TY; ++q) { bv = fmaxf_f(bv, sv[q]); bh = fmaxf_f(bh, sh[q]); bb |= sb[q]; }
    if (m.cfl_out) {
      atomicMax((unsigned*)&m.cfl_out[0], __float_as_uint(bv));
      atomicMax((unsigned*)&m.cfl_out[1], __float_as_uint(bh));
    }
    unsigned bits = 0;
    if (bb) bits |= ERR_NONFINITE;
    if (m.cfl_limit > 0.f && bv > m.cfl_limit) bits |= ERR_CFL;
    if (bits) raise_err(m, bits);
  }
}

// ------------------------------------------------------------ launchers
void launch_cfl_check_col(const TileLaunch& L, int nb, cudaStream_t s, int var) {
  k_cfl_check_col<<<dim3(nb, level_chunks(nb, L.nlev, TUNE_PARAM[TU_CFL][var], 2)), dim3(TX, TY), 0, s>>>(L);
}
void launch_update_scalar_pd(const Launch& L, int nb, StepArgs a, cudaStream_t s) {
  k_update_scalar_pd<<<nb, dim3(BX, BY), 0, s>>>(L, a.rk_step);
}
void launch_update_scalar_pd_col(const TileLaunch& L, int nb, StepArgs a, cudaStream_t s, bool sct) {
  const dim3 grid(nb, level_chunks(nb, L.nlev, 4, 2));
  if (sct) k_update_scalar_pd_col<true><<<grid, dim3(TX, TY), 0, s>>>(L, a.rk_step);
  else k_update_scalar_pd_col<false><<<grid, dim3(TX, TY), 0, s>>>(L, a.rk_step);
}
void launch_advect_scalar(const Launch& L, int nb, StepArgs a, cudaStream_t s) {
  k_advect_scalar<<<nb, dim3(BX, BY), 0, s>>>(L, a.species, a.rk_step, a.flags);
}
// Shared memory of pd_tile for columns of nlev levels.
constexpr size_t pdr_bytes(int nlev) { return PdrPlanes::FLOATS * 4 + (size_t)nlev * sizeof(PdrLevel); }
// a chunk computes two levels more than it writes; two blocks per SM
void launch_advect_scalar_pd(const TileLaunch& L, int nb, int species, int rk_step, bool accum, cudaStream_t s) {
  const dim3 grid(nb, level_chunks(nb, L.nlev, 1, 6, 2 * 152));
  allow_smem(k_pd_tend, pdr_bytes(KDE_MAX));
  k_pd_tend<<<grid, PdrPlanes::THREADS, pdr_bytes(L.nlev), s>>>(L, species, rk_step, accum);
}
void launch_advect_scalar_pd_member(const Mem& m, int rk_step, bool accum, cudaStream_t s) {
  const int nb = tiles_x(m) * tiles_y(m), nlev = m.kme - m.kms + 1;
  const dim3 grid(nb, level_chunks(nb, nlev, 1, 6, 2 * 152));
  allow_smem(k_pd_tend_member, pdr_bytes(KDE_MAX));
  k_pd_tend_member<<<grid, PdrPlanes::THREADS, pdr_bytes(nlev), s>>>(m, rk_step, accum);
}
void launch_update_scalar_routine(const Launch& L, int nb, int rk_step, int pd, cudaStream_t s) {
  k_update_scalar_routine<<<nb, dim3(BX, BY), 0, s>>>(L, rk_step, pd);
}
void launch_update_scalar(const Launch& L, int nb, StepArgs a, cudaStream_t s) {
  k_update_scalar<<<nb, dim3(BX, BY), 0, s>>>(L, a.species, a.rk_step);
}
void launch_calc_p_rho_phi(const Launch& L, int nb, cudaStream_t s) { k_calc_p_rho_phi<<<nb, dim3(BX, BY), 0, s>>>(L); }
void launch_calc_p_rho_phi_col(const TileLaunch& L, int nb, cudaStream_t s, int var) {
  k_calc_p_rho_phi_col<<<dim3(nb, level_chunks(nb, L.nlev, TUNE_PARAM[TU_CPRP][var], 2)), dim3(TX, TY), 0, s>>>(L);
}
void launch_set_w_surface(const Launch& L, int nb, cudaStream_t s) { k_set_w_surface<<<nb, dim3(BX, BY), 0, s>>>(L); }

}  // namespace wrfgpu
