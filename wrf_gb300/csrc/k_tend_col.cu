// Column-marching forms of the u and v large-step tendencies (rk_tendency,
// module_em.F:129-560 with advect_u / advect_v, module_advect_em.F:205-1700
// for 5th/3rd order; horizontal_pressure_gradient, module_big_step_utilities_em.F:1585-1718;
// coriolis :3106-3215; curvature :3234-3363).
//
// One thread per (i, j) column (u and v: two columns) of a 32 x 8 tile of the staggered extents,
// levels kts..kte in order (or one chunk of them per block along y).  For u
// and v, the advected field and the mass fluxes ru, rv of each level arrive
// by TMA as halo planes, several levels ahead, and every horizontal face
// flux is formed once, in shared memory, instead of once by each of the two
// columns it separates.  The per-point arithmetic is that of the point
// kernels in k_tend.cu, term for term and in the same order, with three
// exact reuses across levels:
//   * the vertical flux of face k+1 is the lower face of level k+1,
//   * dpn(k+1) of the pressure-gradient correction is dpn(k) one level up,
//   * values at level k+1 (p, ph, rw of the two columns) carry down,
// and the column-invariant products of map factors, Coriolis parameters and
// grid constants are formed once per column, in the reference's order of
// operations (so every rounding is unchanged).  The next levels' own-column
// inputs are prefetched into L2 two levels ahead.
#include "common.cuh"
#include "kernels.h"
#include "open_adv.cuh"
#include "pair.cuh"

namespace wrfgpu {

// Staged planes of the advected field and the two mass fluxes: the tile plus
// a 4-point halo, (TX + 8) x (TY + 8) from (i0 - 4, j0 - 4), TEND_RING levels
// in flight; the x and y face fluxes of a level are formed once each into
// shared memory (double-buffered), so one block barrier per level suffices.
constexpr int HALO_W = TX + 2 * TMA_HALO, HALO_H = TY + 2 * TMA_HALO;
constexpr int TEND_RING = 4;
using HaloRing = LevelRing<3, TEND_RING, HALO_W, HALO_H>;
constexpr int FXN = TY * (TX + 1), FYN = (TY + 1) * TX;
constexpr size_t TEND_SMEM = HaloRing::SMEM + 2 * (FXN + FYN) * 4;

// The tile's x faces (columns i0 .. i0+TX of rows j0 .. j0+TY-1) and y faces
// (rows j0 .. j0+TY of columns i0 .. i0+TX-1) of one level: 5th-order fluxes
// of Q with the face velocity vx(o) / vy(o), o the face's upper point in the
// halo plane.  Each thread forms its cell's left and bottom faces; the last
// column's right faces go to warp TY-1, the last row's top faces to warp TY-2.
template <class VX, class VY>
__device__ __forceinline__ void tile_faces(const float* Q, float* FX, float* FY, VX vx, VY vy, int tx, int ty) {
  auto xface = [&](int r, int c) {
    const int o = (r + TMA_HALO) * HALO_W + c + TMA_HALO;
    const float vel = vx(o);
    FX[r * (TX + 1) + c] = vel * flux5(Q[o - 3], Q[o - 2], Q[o - 1], Q[o], Q[o + 1], Q[o + 2], vel);
  };
  auto yface = [&](int r, int c) {
    const int o = (r + TMA_HALO) * HALO_W + c + TMA_HALO;
    const float vel = vy(o);
    FY[r * TX + c] = vel * flux5(Q[o - 3 * HALO_W], Q[o - 2 * HALO_W], Q[o - HALO_W], Q[o], Q[o + HALO_W],
                                 Q[o + 2 * HALO_W], vel);
  };
  xface(ty, tx);
  yface(ty, tx);
  if (ty == TY - 1 && tx < TY) xface(tx, TX);
  if (ty == TY - 2) yface(TY, tx);
}

// ---------------------------------------------------------------- ru_tend, rv_tend
// The two are one computation with the directions exchanged: DIR 0 is u (the
// other column of every average is i - 1), DIR 1 v (row j - 1).
//
// Two adjacent columns per thread: the planes are read and the own-column
// fields loaded in 8-byte pairs, the additions of both columns are packed
// (pair.cuh), and a level's addresses, coefficients and loop cost one thread
// instead of two.  One column per thread issued 600 instructions per column
// and level, 67% of the issue slots at 30% of HBM; ms per large step against
// two columns: rk_tend_u 5.54 / 4.31 and rk_tend_v 5.45 / 4.69 on 1024x1024x96,
// 1.31 / 0.99 and 1.22 / 1.06 on 512x512x80.  Every face flux is still
// formed once; a thread keeps its own cells' and takes the right and top
// neighbours' from shared memory.
constexpr int FX2 = TX + 2, FXN2 = TY * FX2;  // x faces of a tile, rows padded to an even length
constexpr size_t TEND2_SMEM = HaloRing::SMEM + 2 * (FXN2 + FYN) * 4;
constexpr int TEND2_THREADS = TX * TY / 2;

template <int DIR, int MINB>
__global__ void __launch_bounds__(TEND2_THREADS, MINB) k_tend_uv_col(TileLaunch L) {
  extern __shared__ __align__(128) unsigned char smem[];
  const TilePos tp = tile_pos(L, false, true);
  const Mem& m = block_member(L.mem, tp.m);
  const int tid = threadIdx.x, c = (tid & 15) * 2, ty = tid >> 4;
  const int i = tp.i0 + c, j = tp.j0 + ty;
  const F3 tend = f3(m, DIR ? WRFGPU_RV_TEND : WRFGPU_RU_TEND);
  const int kts = m.kts, kte = m.kte, kde = m.kde, kme = m.kme, ktf = min(kte, kde - 1);
  // the points that take a tendency, and (of the staggered tile) those set to zero
  const int iacc = DIR ? min(m.ite, m.ide - 1) : m.ite, jacc = DIR ? m.jte : min(m.jte, m.jde - 1);
  const bool in0 = i <= m.ite && j <= m.jte, in1 = i + 1 <= m.ite && j <= m.jte;
  const bool acc = i <= iacc && j <= jacc, acc1 = i + 1 <= iacc && j <= jacc;
  auto zero = [&](int k) {
    if (in0 && !acc) tend(i, k, j) = 0.f;
    if (in1 && !acc1) tend(i + 1, k, j) = 0.f;
  };
  if (blockIdx.y == 0)
    for (int k = kts; k <= kte; ++k) zero(k);
  const Chunk ch = level_chunk_of(kts, ktf);
  const int k0 = ch.k0, k1 = ch.k1;
  if (blockIdx.y == gridDim.y - 1)
    for (int k = ktf + 1; k <= kte; ++k) {
      if (acc) tend(i, k, j) = 0.f;
      if (acc1) tend(i + 1, k, j) = 0.f;
    }
  if (tp.i0 > iacc || tp.j0 > jacc || k0 > k1) return;  // block-uniform
  const F3 fld = f3(m, DIR ? WRFGPU_V_2 : WRFGPU_U_2), crs = f3(m, DIR ? WRFGPU_U_2 : WRFGPU_V_2),
           rw = f3(m, WRFGPU_RW), rom = f3(m, WRFGPU_WW);
  const F3 ph = f3(m, WRFGPU_PH_2), alt = f3(m, WRFGPU_ALT), p = f3(m, WRFGPU_P), pb = f3(m, WRFGPU_PB),
           al = f3(m, WRFGPU_AL), php = f3(m, WRFGPU_PHP), cq = f3(m, DIR ? WRFGPU_CQV : WRFGPU_CQU);
  const F1 fzm = f1(m, WRFGPU_FNM), fzp = f1(m, WRFGPU_FNP), rdzw = f1(m, WRFGPU_RDNW), c1h = f1(m, WRFGPU_C1H),
           c2h = f1(m, WRFGPU_C2H);
  const float rdx = m.rdx, rdy = m.rdy, rd = DIR ? rdy : rdx;
  HaloRing ring;
  ring.init(smem, k0);
  float* FXb = (float*)(smem + HaloRing::SMEM);
  float* FYb = FXb + 2 * FXN2;
  const CUtensorMap* maps[3] = {tmap_of(m, DIR ? WRFGPU_V_2 : WRFGPU_U_2, BOX_HALO), tmap_of(m, WRFGPU_RU, BOX_HALO),
                                tmap_of(m, WRFGPU_RV, BOX_HALO)};
  const int x0 = tp.i0 - TMA_HALO - m.ims, z0 = tp.j0 - TMA_HALO - m.jms;
  if (tid == 0) {
    ring.init_barriers();
    mbar_fence_init();
  }
  __syncthreads();
  if (tid == 0)
    for (int d = 0; d < TEND_RING - 1 && k0 + d <= k1; ++d) ring.issue(k0 + d, maps, x0, z0, m.kms);
  auto mul = [](float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); };
  auto div = [](float2 a, float2 b) { return make_float2(a.x / b.x, a.y / b.y); };
  auto at2 = [](const float* q) { return *reinterpret_cast<const float2*>(q); };
  // the pair's own value, its first neighbours' (DIR) given the own one, and at another point
  auto own = [&](const F3& a, int k) { return at2(a.p + a.off(i, k, j)); };
  auto low = [&](const F3& a, int k, float2 o) {
    return DIR ? at2(a.p + a.off(i, k, j - 1)) : make_float2(a(i - 1, k, j), o.x);
  };
  auto sum = [&](const F3& a, int k) { const float2 o = own(a, k); return add2(o, low(a, k, o)); };
  auto dif = [&](const F3& a, int k) { const float2 o = own(a, k); return sub2(o, low(a, k, o)); };
  auto g2 = [&](int f, int ii, int jj) { const F2 a = f2(m, f); return make_float2(a(ii, jj), a(ii + 1, jj)); };
  // column constants, formed in the order of the per-level expressions
  float2 mrdy, mrdx, ratio, pgA, pgB, mu_c, mu_l, mu_r, corA, corB, dvx_l, dvx_r, duy_l, duy_r;
  // own-column window of the field (k-1 .. k+2), the vertical flux of face k,
  // and the pressure-gradient / rw carries (formed afresh at the chunk's first
  // level, with the same expressions as one level down)
  float2 fm1 = bc2(0.f), f0, fp1, fp2 = bc2(0.f), vf_lo = bc2(0.f), p_l, p_r, ph_l, ph_r, dpn_lo, rw_l, rw_r;
  if (acc) {
    constexpr int il = DIR ? 0 : 1, jl = DIR ? 1 : 0;
    const float2 ma = g2(DIR ? WRFGPU_MSFVY : WRFGPU_MSFUX, i, j);
    mrdy = muls(rdy, ma); mrdx = muls(rdx, ma);
    ratio = div(ma, g2(DIR ? WRFGPU_MSFVX : WRFGPU_MSFUY, i, j));
    pgA = muls(rd, muls(.5f, ratio)); pgB = muls(rd, ratio);
    mu_c = g2(DIR ? WRFGPU_MUV : WRFGPU_MUU, i, j);
    mu_l = g2(WRFGPU_MU_2, i - il, j - jl);
    mu_r = g2(WRFGPU_MU_2, i, j);
    corA = muls(0.25f, mul(muls(0.5f, ratio), add2(g2(WRFGPU_F, i, j), g2(WRFGPU_F, i - il, j - jl))));
    const float2 es = add2(g2(WRFGPU_E, i, j), g2(WRFGPU_E, i - il, j - jl));
    const int cs = DIR ? WRFGPU_SINA : WRFGPU_COSA;
    const float2 ca = add2(g2(cs, i, j), g2(cs, i - il, j - jl));
    corB = muls(0.25f, mul(muls(0.5f, DIR ? mul(muls(0.5f, ratio), es) : muls(0.5f, es)), ca));
    dvx_r = sub2(g2(WRFGPU_MSFVX, i, j + 1), g2(WRFGPU_MSFVX, i, j));
    dvx_l = sub2(g2(WRFGPU_MSFVX, i - il, j + 1 - jl), g2(WRFGPU_MSFVX, i - il, j - jl));
    duy_r = sub2(g2(WRFGPU_MSFUY, i + 1, j), g2(WRFGPU_MSFUY, i, j));
    duy_l = sub2(g2(WRFGPU_MSFUY, i + 1 - il, j - jl), g2(WRFGPU_MSFUY, i - il, j - jl));
    if (k0 - 1 >= kts) fm1 = own(fld, k0 - 1);
    f0 = own(fld, k0); fp1 = own(fld, k0 + 1);
    if (k0 + 2 <= kme) fp2 = own(fld, k0 + 2);
    if (k0 != kts && k0 != kte) {
      const float2 vel = muls(0.5f, sum(rom, k0));
      if (k0 == kts + 1 || k0 == ktf) vf_lo = mul(vel, add2(muls(fzm(k0), f0), muls(fzp(k0), fm1)));
      else vf_lo = mul(vel, flux3_c2(own(fld, k0 - 2), fm1, f0, fp1, make_float2(-vel.x, -vel.y)));
    }
    p_r = own(p, k0); p_l = low(p, k0, p_r);
    ph_r = own(ph, k0); ph_l = low(ph, k0, ph_r);
    if (k0 == 1) dpn_lo = muls(.5f, add2(add2(muls(m.cf1, sum(p, 1)), muls(m.cf2, sum(p, 2))), muls(m.cf3, sum(p, 3))));
    else dpn_lo = muls(.5f, add2(muls(fzm(k0), add2(p_l, p_r)), muls(fzp(k0), sum(p, k0 - 1))));
    rw_r = own(rw, k0); rw_l = low(rw, k0, rw_r);
  }
  const int o = (ty + TMA_HALO) * HALO_W + c + TMA_HALO;  // own first point in the halo planes
  constexpr int W = HALO_W, d = DIR ? W : 1;
  bool ok = true;
  for (int k = k0; k <= k1; ++k) {
    ok = ring.wait(k) && ok;
    const float* Q = ring.plane(k, 0);
    const float* RU = ring.plane(k, 1);
    const float* RV = ring.plane(k, 2);
    float* FX = FXb + (k & 1) * FXN2;
    float* FY = FYb + (k & 1) * FYN;
    // face velocities at the two columns from q on: 0.5 (r(q) + r(q - d))
    auto vel2 = [&](const float* R, int q) {
      const float2 a = at2(R + q);
      return muls(0.5f, add2(a, DIR ? at2(R + q - W) : make_float2(R[q - 1], a.x)));
    };
    auto yfaces = [&](int q) {
      const float2 vel = vel2(RV, q);
      return mul(vel, flux5_c2(at2(Q + q - 3 * W), at2(Q + q - 2 * W), at2(Q + q - W), at2(Q + q), at2(Q + q + W),
                               at2(Q + q + 2 * W), vel));
    };
    // own left faces (columns c, c + 1) and bottom faces
    const float2 q2 = at2(Q + o), qm = at2(Q + o - 2), qp = at2(Q + o + 2);
    float2 fx, fy;
    {
      const float2 vel = vel2(RU, o);
      fx = mul(vel, flux5_c2(make_float2(Q[o - 3], qm.x), qm, make_float2(qm.y, q2.x), q2, make_float2(q2.y, qp.x), qp,
                             vel));
      fy = yfaces(o);
    }
    *reinterpret_cast<float2*>(FX + ty * FX2 + c) = fx;
    *reinterpret_cast<float2*>(FY + ty * TX + c) = fy;
    if (tid >= 96 && tid < 96 + TY) {  // the last column's right faces
      const int r = tid - 96, q = (r + TMA_HALO) * W + TX + TMA_HALO;
      const float vel = 0.5f * (RU[q] + RU[q - d]);
      FX[r * FX2 + TX] = vel * flux5(Q[q - 3], Q[q - 2], Q[q - 1], Q[q], Q[q + 1], Q[q + 2], vel);
    }
    if (tid >= 64 && tid < 80)  // the last row's top faces
      *reinterpret_cast<float2*>(FY + TY * TX + c) = yfaces((TY + TMA_HALO) * W + c + TMA_HALO);
    __syncthreads();
    // the slot of level k-1, which every thread has finished with
    if (tid == 0 && k + TEND_RING - 1 <= k1) ring.issue(k + TEND_RING - 1, maps, x0, z0, m.kms);
    if (!acc) continue;
    if (k + 2 <= kme) {
      prefetch_l2(&rom(i, k + 2, j)); prefetch_l2(&p(i, k + 2, j)); prefetch_l2(&ph(i, k + 2, j));
      prefetch_l2(&alt(i, k + 2, j)); prefetch_l2(&al(i, k + 2, j)); prefetch_l2(&pb(i, k + 2, j));
      prefetch_l2(&php(i, k + 2, j)); prefetch_l2(&cq(i, k + 2, j)); prefetch_l2(&rw(i, k + 2, j));
      prefetch_l2(&crs(i, k + 2, j));
    }
    // the level's own-column inputs go out together
    const int kk = k + 1;
    const float2 fp3 = k + 3 <= kme ? own(fld, k + 3) : bc2(0.f);
    const float2 romsum = (kk == kts || kk == kte) ? bc2(0.f) : sum(rom, kk);
    const float2 rw_r1 = own(rw, kk), rw_l1 = low(rw, kk, rw_r1);
    float2 p_r1 = bc2(0.f), p_l1 = bc2(0.f);
    if (kk != kde) { p_r1 = own(p, kk); p_l1 = low(p, kk, p_r1); }
    const float2 ph_r1 = own(ph, kk), ph_l1 = low(ph, kk, ph_r1);
    const float2 altsum = sum(alt, k), alsum = sum(al, k), pbd = dif(pb, k), phpd = dif(php, k), cqk = own(cq, k);
    // the two sums of the cross velocity: of the point and of its lower neighbour
    float2 cs_r, cs_l;
    {
      const float2 a = own(crs, k);
      if (DIR) {
        const float2 b = at2(crs.p + crs.off(i, k, j - 1));
        cs_r = make_float2(a.x + a.y, a.y + crs(i + 2, k, j));
        cs_l = make_float2(b.x + b.y, b.y + crs(i + 2, k, j - 1));
      } else {
        cs_r = add2(a, at2(crs.p + crs.off(i, k, j + 1)));
        cs_l = make_float2(crs(i - 1, k, j) + crs(i - 1, k, j + 1), cs_r.x);
      }
    }
    float2 t = bc2(0.f);
    t = sub2(t, mul(mrdy, sub2(at2(FY + (ty + 1) * TX + c), fy)));
    t = sub2(t, mul(mrdx, sub2(make_float2(fx.y, FX[ty * FX2 + c + 2]), fx)));
    const float rz = rdzw(k);
    {  // vertical flux of face k+1
      float2 vf_hi = bc2(0.f);
      if (kk != kts && kk != kte) {
        const float2 vel = muls(0.5f, romsum);
        if (kk == kts + 1 || kk == ktf) vf_hi = mul(vel, add2(muls(fzm(kk), fp1), muls(fzp(kk), f0)));
        else vf_hi = mul(vel, flux3_c2(fm1, f0, fp1, fp2, make_float2(-vel.x, -vel.y)));
      }
      t = sub2(t, mul(DIR ? muls(rz, ratio) : bc2(rz), sub2(vf_hi, vf_lo)));
      vf_lo = vf_hi;
    }
    {  // horizontal_pressure_gradient
      float2 dpn_hi = bc2(0.f);
      if (kk == kde) {
        if (m.cf.top_lid) dpn_hi = muls(.5f, add2(muls(m.cfn, sum(p, kde - 1)), muls(m.cfn1, sum(p, kde - 2))));
      } else {
        dpn_hi = muls(.5f, add2(muls(fzm(kk), add2(p_l1, p_r1)), muls(fzp(kk), add2(p_l, p_r))));
      }
      const float h1 = c1h(k), h2 = c2h(k);
      float2 dp = mul(mul(pgA, add2(muls(h1, mu_c), bc2(h2))),
                      add2(add2(sub2(add2(sub2(ph_r1, ph_l1), ph_r), ph_l), mul(altsum, sub2(p_r, p_l))), mul(alsum, pbd)));
      dp = add2(dp, mul(mul(pgB, phpd),
                        sub2(muls(rz, sub2(dpn_hi, dpn_lo)), muls(.5f, add2(muls(h1, mu_l), muls(h1, mu_r))))));
      t = sub2(t, mul(cqk, dp));
      dpn_lo = dpn_hi;
      p_l = p_l1; p_r = p_r1; ph_l = ph_l1; ph_r = ph_r1;
    }
    {  // coriolis, curvature
      const float2 rwsum = add2(add2(add2(rw_l1, rw_l), rw_r1), rw_r);
      float2 rsum, vx_r, vx_l;
      if (DIR) {
        const float2 a = at2(RU + o), b = at2(RU + o - W);
        rsum = add2(add2(add2(a, make_float2(a.y, RU[o + 2])), b), make_float2(b.y, RU[o - W + 2]));
        t = add2(sub2(t, mul(corA, rsum)), mul(corB, rwsum));
        vx_r = sub2(muls(rdy, mul(muls(0.5f, cs_r), dvx_r)), muls(rdx, mul(muls(0.5f, add2(f0, at2(Q + o + W))), duy_r)));
        vx_l = sub2(muls(rdy, mul(muls(0.5f, cs_l), dvx_l)), muls(rdx, mul(muls(0.5f, add2(at2(Q + o - W), f0)), duy_l)));
        t = sub2(sub2(t, mul(muls(0.25f, muls(0.5f, add2(vx_r, vx_l))), rsum)),
                 mul(muls(0.25f, muls(RERADIUS, mul(ratio, f0))), rwsum));
      } else {
        const float2 a = at2(RV + o), b = at2(RV + o + W);
        rsum = add2(add2(add2(make_float2(RV[o + W - 1], b.x), b), make_float2(RV[o - 1], a.x)), a);
        t = sub2(add2(t, mul(corA, rsum)), mul(corB, rwsum));
        vx_r = sub2(muls(rdy, mul(muls(0.5f, add2(f0, make_float2(q2.y, qp.x))), dvx_r)), muls(rdx, mul(muls(0.5f, cs_r), duy_r)));
        vx_l = sub2(muls(rdy, mul(muls(0.5f, add2(make_float2(qm.y, q2.x), f0)), dvx_l)), muls(rdx, mul(muls(0.5f, cs_l), duy_l)));
        t = sub2(add2(t, mul(muls(0.25f, muls(0.5f, add2(vx_r, vx_l))), rsum)), mul(muls(0.25f, muls(RERADIUS, f0)), rwsum));
      }
    }
    rw_l = rw_l1; rw_r = rw_r1;
    if (acc1) *reinterpret_cast<float2*>(tend.p + tend.off(i, k, j)) = t;
    else tend(i, k, j) = t.x;
    fm1 = f0; f0 = fp1; fp1 = fp2; fp2 = fp3;
  }
  if (!ok && tid == 0) raise_err(m, ERR_TIMEOUT);
}

// ---------------------------------------------------------------- rw_tend
// advect_w (module_advect_em.F:4364-6064), pg_buoy_w, coriolis and curvature
// (module_big_step_utilities_em.F) on the w levels.  pg_buoy_w overwrites
// cqw(k) with 1/(1+cqw(k)) after the k = kde point has read the original
// cqw(kde-1), so the last level chunk holds both.  The face velocities
// interpolate ru, rv between levels k and k-1 (k-1 and k-2 at the top), so
// the ring starts one level below the chunk and keeps the two levels below
// the current one: after the barrier of level k the slot of level k-3 is free.
constexpr int W_RING = 6;
using HaloRingW = LevelRing<3, W_RING, HALO_W, HALO_H>;
constexpr size_t TENDW_SMEM = HaloRingW::SMEM + 2 * (FXN + FYN) * 4;

template <int FL, int MINB>
__global__ void __launch_bounds__(TX* TY, MINB) k_tend_w_col(TileLaunch L) {
  static_assert(FL & TF_ADV, "the staged form includes advection");
  extern __shared__ __align__(128) unsigned char smem[];
  const TilePos tp = tile_pos(L, false, true);
  const Mem& m = block_member(L.mem, tp.m);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int i = tp.i0 + tx, j = tp.j0 + ty;
  const F3 tend = f3(m, WRFGPU_RW_TEND);
  const int kts = m.kts, kte = m.kte, kde = m.kde;
  const int itf = min(m.ite, m.ide - 1), jtf = min(m.jte, m.jde - 1), ktf = min(kte, kde - 1);
  const bool inside = i <= m.ite && j <= m.jte;
  const bool acc = inside && i <= itf && j <= jtf;
  if ((FL & TF_ZERO) && inside && !acc && blockIdx.y == 0)
    for (int k = kts; k <= kte; ++k) tend(i, k, j) = 0.f;
  Chunk ch = level_chunk_of(kts, ktf);
  if (ch.k0 <= ktf && ch.k1 == ktf) ch.k1 = kte;
  const int k0 = ch.k0, k1 = ch.k1, kf = max(kts, k0 - 1);  // this block's levels; first staged level
  if (!(tp.i0 <= itf && tp.j0 <= jtf) || k0 > k1) return;  // block-uniform
  // next to an open boundary rw_tend has been formed by the edge-strip
  // kernel (k_tend.cu) from the cqw this kernel overwrites: keep it
  const bool keep = !((m.cf.open_xs || m.cf.open_ys) && in_open_strip(m, i, j, STRIP_W_TEND));
  const F3 w = f3(m, WRFGPU_W_2), rom = f3(m, WRFGPU_WW), p = f3(m, WRFGPU_P), cqw = f3(m, WRFGPU_CQW);
  const F3 u = f3(m, WRFGPU_U_2), v = f3(m, WRFGPU_V_2);
  const F1 fzm = f1(m, WRFGPU_FNM), fzp = f1(m, WRFGPU_FNP), rdzu = f1(m, WRFGPU_RDN), rdnw = f1(m, WRFGPU_RDNW),
           c1f = f1(m, WRFGPU_C1F), c2f = f1(m, WRFGPU_C2F);
  const float rdx = m.rdx, rdy = m.rdy;
  HaloRingW ring;
  ring.init(smem, kf);
  float* FXb = (float*)(smem + HaloRingW::SMEM);
  float* FYb = FXb + 2 * FXN;
  const CUtensorMap* maps[3] = {tmap_of(m, WRFGPU_W_2, BOX_HALO), tmap_of(m, WRFGPU_RU, BOX_HALO),
                                tmap_of(m, WRFGPU_RV, BOX_HALO)};
  const int x0 = tp.i0 - TMA_HALO - m.ims, z0 = tp.j0 - TMA_HALO - m.jms;
  if (tid == 0) {
    ring.init_barriers();
    mbar_fence_init();
  }
  __syncthreads();
  if (tid == 0)
    for (int k = kf; k <= min(k0 + W_RING - 4, k1); ++k) ring.issue(k, maps, x0, z0, m.kms);
  auto vf = [&](int kk) -> float {
    if (kk == kts + 1 || kk == ktf + 1) return 0.25f * (rom(i, kk, j) + rom(i, kk - 1, j)) * (w(i, kk, j) + w(i, kk - 1, j));
    float vel = 0.5f * (rom(i, kk, j) + rom(i, kk - 1, j));
    return vel * flux3(w(i, kk - 2, j), w(i, kk - 1, j), w(i, kk, j), w(i, kk + 1, j), -vel);
  };
  // column constants, formed in the order of the per-level expressions
  float mrdy = 0.f, mrdx = 0.f, rmg = 0.f, ratio = 0.f, e_c = 0.f, cosa05 = 0.f, rsina05 = 0.f, ratio05 = 0.f;
  float muf_c = 0.f, mub_c = 0.f, cqw_top = 0.f, vf_lo = 0.f, mut_w = 0.f;
  const bool wdamp = m.cf.w_damping == 1;
  if (acc) {
    if (wdamp) mut_w = f2(m, WRFGPU_MUT)(i, j);
    const F2 msftx = f2(m, WRFGPU_MSFTX), msfty = f2(m, WRFGPU_MSFTY);
    mrdy = msftx(i, j) * rdy; mrdx = msftx(i, j) * rdx;
    rmg = (1.f / msfty(i, j)) * G;
    ratio = msftx(i, j) / msfty(i, j);
    if (FL & TF_COR) {
      e_c = f2(m, WRFGPU_E)(i, j);
      cosa05 = f2(m, WRFGPU_COSA)(i, j) * 0.5f;
      rsina05 = ratio * f2(m, WRFGPU_SINA)(i, j) * 0.5f;
    }
    ratio05 = ratio * 0.5f;
    if (FL & TF_PG) { muf_c = f2(m, WRFGPU_MU_2)(i, j); mub_c = f2(m, WRFGPU_MUB)(i, j); }
    if (k1 == kte) cqw_top = cqw(i, kde - 1, j);  // read before the k = kde-1 overwrite below
    // the vertical flux of face k+1 is the lower face of level k+1
    vf_lo = vf(max(k0, kts + 1));
  }
  // levels k-1 (and k-2) of the mass fluxes at the own point and its +i / +j
  // neighbours, and of u, v, p, carried down the column; w(k-1 .. k+1) and
  // omega(k) of the own column for the vertical flux of face k+1
  float ru0m = 0.f, ru1m = 0.f, rv0m = 0.f, rv1m = 0.f;
  float u0m = 0.f, u1m = 0.f, v0m = 0.f, v1m = 0.f, pkm = 0.f;
  float wkm1 = 0.f, wk0 = 0.f, wkp1 = 0.f, romk = 0.f;
  const int kme = m.kme;
  if (acc) {
    if (k0 > kts) wkm1 = w(i, k0 - 1, j);
    wk0 = w(i, k0, j);
    wkp1 = k0 + 1 <= kme ? w(i, k0 + 1, j) : 0.f;
    romk = rom(i, k0, j);
  }
  const int o = (ty + TMA_HALO) * HALO_W + tx + TMA_HALO;
  bool ok = true;
  if (k0 > kts) {  // what level k0 takes from the level below
    if (acc) {
      if (FL & TF_CURV) { u0m = u(i, k0 - 1, j); u1m = u(i + 1, k0 - 1, j); v0m = v(i, k0 - 1, j); v1m = v(i, k0 - 1, j + 1); }
      if (FL & TF_PG) pkm = p(i, k0 - 1, j);
    }
    ok = ring.wait(kf) && ok;
    const float* RU = ring.plane(kf, 1);
    const float* RV = ring.plane(kf, 2);
    ru0m = RU[o]; ru1m = RU[o + 1]; rv0m = RV[o]; rv1m = RV[o + HALO_W];
  }
  for (int k = k0; k <= k1; ++k) {
    // the level's global inputs, loaded together before the face work and
    // the level barrier so that their latency overlaps them
    float u0 = 0.f, u1 = 0.f, v0 = 0.f, v1 = 0.f, pk = 0.f, cqk = 0.f, romk1 = 0.f, wk2 = 0.f, t = 0.f;
    if (acc) {
      if (FL & TF_CURV) { u0 = u(i, k, j); u1 = u(i + 1, k, j); v0 = v(i, k, j); v1 = v(i, k, j + 1); }
      if (FL & TF_PG) {
        pk = p(i, k, j);
        if (k != kde && k >= 2) cqk = cqw(i, k, j);
      }
      romk1 = k + 1 <= kme ? rom(i, k + 1, j) : 0.f;
      wk2 = k + 2 <= kme ? w(i, k + 2, j) : 0.f;
      t = (FL & TF_ZERO) ? 0.f : tend(i, k, j);
    }
    ok = ring.wait(k) && ok;
    const float* Wk = ring.plane(k, 0);
    const float* RUk = ring.plane(k, 1);
    const float* RVk = ring.plane(k, 2);
    float* FX = FXb + (k & 1) * FXN;
    float* FY = FYb + (k & 1) * FYN;
    const bool adv = k >= kts + 1 && k <= ktf + 1;  // block-uniform
    if (adv) {
      const float* RUm = ring.plane(k - 1, 1);
      const float* RVm = ring.plane(k - 1, 2);
      if (k <= ktf) {
        const float a = fzm(k), b = fzp(k);
        tile_faces(Wk, FX, FY, [&](int q) { return a * RUk[q] + b * RUm[q]; },
                   [&](int q) { return a * RVk[q] + b * RVm[q]; }, tx, ty);
      } else {
        const float* RUmm = ring.plane(k - 2, 1);
        const float* RVmm = ring.plane(k - 2, 2);
        const float a = fzm(k - 1), b = fzp(k - 1);
        tile_faces(Wk, FX, FY, [&](int q) { return (2.f - a) * RUm[q] - b * RUmm[q]; },
                   [&](int q) { return (2.f - a) * RVm[q] - b * RVmm[q]; }, tx, ty);
      }
    }
    __syncthreads();
    if (tid == 0 && k - 3 + W_RING <= k1) ring.issue(k - 3 + W_RING, maps, x0, z0, m.kms);
    if (!acc) continue;
    const float ru0 = RUk[o], ru1 = RUk[o + 1], rv0 = RVk[o], rv1 = RVk[o + HALO_W];
    if (adv) {
      t = t - mrdy * (FY[(ty + 1) * TX + tx] - FY[ty * TX + tx]);
      t = t - mrdx * (FX[ty * (TX + 1) + tx + 1] - FX[ty * (TX + 1) + tx]);
      if (k <= ktf) {
        // vf(k + 1) from the carried window (the same operands and order)
        float vf_hi;
        if (k + 1 == kts + 1 || k + 1 == ktf + 1) vf_hi = 0.25f * (romk1 + romk) * (wkp1 + wk0);
        else {
          const float vel = 0.5f * (romk1 + romk);
          vf_hi = vel * flux3(wkm1, wk0, wkp1, wk2, -vel);
        }
        t = t - rdzu(k) * (vf_hi - vf_lo);
        vf_lo = vf_hi;
      } else {
        t = t + 2.f * rdzu(k - 1) * (vf_lo);
      }
    }
    if (FL & TF_PG) {
      if (k == kde) {
        float cq1 = 1.f / (1.f + cqw_top);
        float cq2 = cqw_top * cq1;
        t = t + rmg * (cq1 * 2.f * rdnw(k - 1) * (-pkm) - (c1f(k) * muf_c) - cq2 * (c1f(k) * mub_c + c2f(k)));
      } else if (k >= 2) {
        float cq1 = 1.f / (1.f + cqk);
        float cq2 = cqk * cq1;
        cqw(i, k, j) = cq1;
        t = t + rmg * (cq1 * rdzu(k) * (pk - pkm) - (c1f(k) * muf_c) - cq2 * (c1f(k) * mub_c + c2f(k)));
      }
    }
    // w_damp with w_damping = 1 (module_big_step_utilities_em.F:2687-2691),
    // after pg_buoy_w and before coriolis as rk_tendency calls them
    // (module_em.F:729-745); activation at w_beta (zadvect_implicit = 0)
    if (FL == TF_ALL && wdamp && k >= 2 && k <= kde - 1) {
      const float vert_cfl = fabsf(romk / (c1f(k) * mut_w + c2f(k)) * rdnw(k) * m.dt);
      if (vert_cfl > W_BETA)
        t = t - sgn1(Wk[o]) * W_ALPHA * (vert_cfl - m.cf.w_crit_cfl) * (c1f(k) * mut_w + c2f(k));
    }
    if (k >= kts + 1 && k <= ktf) {
      if (FL & TF_COR) {
        t = t + e_c * (cosa05 * (fzm(k) * (ru0 + ru1) + fzp(k) * (ru0m + ru1m)) -
                       rsina05 * (fzm(k) * (rv0 + rv1) + fzp(k) * (rv0m + rv1m)));
      }
    }
    if (k >= max(2, kts) && k <= ktf) {
      if (FL & TF_CURV) {
        t = t + RERADIUS * (0.5f * (fzm(k) * (ru0 + ru1) + fzp(k) * (ru0m + ru1m)) *
                                0.5f * (fzm(k) * (u0 + u1) + fzp(k) * (u0m + u1m)) +
                            ratio05 * (fzm(k) * (rv0 + rv1) + fzp(k) * (rv0m + rv1m)) *
                                0.5f * (fzm(k) * (v0 + v1) + fzp(k) * (v0m + v1m)));
      }
    }
    if (keep) tend(i, k, j) = t;
    ru0m = ru0; ru1m = ru1; rv0m = rv0; rv1m = rv1;
    u0m = u0; u1m = u1; v0m = v0; v1m = v1;
    pkm = pk;
    wkm1 = wk0; wk0 = wkp1; wkp1 = wk2; romk = romk1;
  }
  if (!ok && tid == 0) raise_err(m, ERR_TIMEOUT);
}

// ---------------------------------------------------------------- t_tend
// advect_scalar of theta (module_advect_em.F:3394-3650, :4306-4333) plus the
// zero_tend of the *_save arrays at the points small_step_prep leaves alone
// (module_em.F:395-428); the vertical flux and the own-column window of
// theta carry down the column.
template <int FL, int MINB>
__global__ void __launch_bounds__(TX* TY, MINB) k_tend_t_col(TileLaunch L) {
  static_assert(FL & TF_ADV, "the staged form includes advection");
  extern __shared__ __align__(128) unsigned char smem[];
  const TilePos tp = tile_pos(L, false, true);
  const Mem& m = block_member(L.mem, tp.m);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int i = tp.i0 + tx, j = tp.j0 + ty;
  const F3 tend = f3(m, WRFGPU_T_TEND);
  const int kts = m.kts, kte = m.kte, kme = m.kme;
  const int itf = min(m.ite, m.ide - 1), jtf = min(m.jte, m.jde - 1), ktf = min(kte, m.kde - 1);
  const bool inside = i <= m.ite && j <= m.jte;
  const Chunk ch = level_chunk_of(kts, ktf);
  const int k0 = ch.k0, k1 = ch.k1;
  if ((FL & TF_ZERO) && inside && blockIdx.y == 0) {
    const bool ie = i == m.ide, je = j == m.jde;
    const F3 us = f3(m, WRFGPU_U_SAVE), vs = f3(m, WRFGPU_V_SAVE), ts = f3(m, WRFGPU_T_SAVE),
             ws = f3(m, WRFGPU_W_SAVE), phs = f3(m, WRFGPU_PH_SAVE);
    for (int k = kts; k <= kte; ++k) {
      const bool kt = k == m.kde;
      if (kt || je) us(i, k, j) = 0.f;
      if (kt || ie) vs(i, k, j) = 0.f;
      if (kt || ie || je) ts(i, k, j) = 0.f;
      if (ie || je) { ws(i, k, j) = 0.f; phs(i, k, j) = 0.f; }
    }
    if (ie || je) f2(m, WRFGPU_MU_SAVE)(i, j) = 0.f;
  }
  const bool acc = inside && i <= itf && j <= jtf;
  if ((FL & TF_ZERO) && inside && !acc && blockIdx.y == 0)
    for (int k = kts; k <= kte; ++k) tend(i, k, j) = 0.f;
  if (tp.i0 <= itf && tp.j0 <= jtf && k0 <= k1) {  // block-uniform
    const F3 fld = f3(m, WRFGPU_T_2), rom = f3(m, WRFGPU_WW);
    const F1 fzm = f1(m, WRFGPU_FNM), fzp = f1(m, WRFGPU_FNP), rdzw = f1(m, WRFGPU_RDNW);
    HaloRing ring;
    ring.init(smem, k0);
    float* FXb = (float*)(smem + HaloRing::SMEM);
    float* FYb = FXb + 2 * FXN;
    const CUtensorMap* maps[3] = {tmap_of(m, WRFGPU_T_2, BOX_HALO), tmap_of(m, WRFGPU_RU, BOX_HALO),
                                  tmap_of(m, WRFGPU_RV, BOX_HALO)};
    const int x0 = tp.i0 - TMA_HALO - m.ims, z0 = tp.j0 - TMA_HALO - m.jms;
    if (tid == 0) {
      ring.init_barriers();
      mbar_fence_init();
    }
    __syncthreads();
    if (tid == 0)
      for (int d = 0; d < TEND_RING - 1 && k0 + d <= k1; ++d) ring.issue(k0 + d, maps, x0, z0, m.kms);
    float mrdy = 0.f, mrdx = 0.f, fm1 = 0.f, f0 = 0.f, fp1 = 0.f, fp2 = 0.f;
    if (acc) {
      const float msftx_c = f2(m, WRFGPU_MSFTX)(i, j);
      mrdy = msftx_c * m.rdy; mrdx = msftx_c * m.rdx;
      if (k0 > kts) fm1 = fld(i, k0 - 1, j);
      f0 = fld(i, k0, j); fp1 = fld(i, k0 + 1, j); fp2 = (k0 + 2 <= kme) ? fld(i, k0 + 2, j) : 0.f;
    }
    float vf_lo = 0.f;  // vf(k0), formed as level k0 - 1 forms its upper face; vf(kts) = 0
    if (acc && k0 > kts) {
      const float vel = rom(i, k0, j);
      if (k0 == kts + 1 || k0 == ktf) vf_lo = vel * (fzm(k0) * f0 + fzp(k0) * fm1);
      else vf_lo = vel * flux3(fld(i, k0 - 2, j), fm1, f0, fp1, -vel);
    }
    bool ok = true;
    for (int k = k0; k <= k1; ++k) {
      // the level's own-column loads, issued before the face work and the
      // barrier so that their latency overlaps them
      float fp3 = 0.f, romk1 = 0.f;
      if (acc) {
        fp3 = (k + 3 <= kme) ? fld(i, k + 3, j) : 0.f;
        romk1 = (k + 1 == kts || k + 1 == kte) ? 0.f : rom(i, k + 1, j);
      }
      ok = ring.wait(k) && ok;
      const float* T = ring.plane(k, 0);
      const float* RU = ring.plane(k, 1);
      const float* RV = ring.plane(k, 2);
      float* FX = FXb + (k & 1) * FXN;
      float* FY = FYb + (k & 1) * FYN;
      tile_faces(T, FX, FY, [&](int q) { return RU[q]; }, [&](int q) { return RV[q]; }, tx, ty);
      __syncthreads();
      if (tid == 0 && k + TEND_RING - 1 <= k1) ring.issue(k + TEND_RING - 1, maps, x0, z0, m.kms);
      if (!acc) continue;
      if (k + 2 <= kme) { prefetch_l2(&rom(i, k + 2, j)); prefetch_l2(&tend(i, k + 2, j)); }
      float t = (FL & TF_ZERO) ? 0.f : tend(i, k, j);
      t = t - mrdy * (FY[(ty + 1) * TX + tx] - FY[ty * TX + tx]);
      t = t - mrdx * (FX[ty * (TX + 1) + tx + 1] - FX[ty * (TX + 1) + tx]);
      const int kk = k + 1;
      float vf_hi;
      if (kk == kts || kk == kte) vf_hi = 0.f;
      else if (kk == kts + 1 || kk == ktf) vf_hi = romk1 * (fzm(kk) * fp1 + fzp(kk) * f0);
      else {
        const float vel = romk1;
        vf_hi = vel * flux3(fm1, f0, fp1, fp2, -vel);
      }
      t = t - rdzw(k) * (vf_hi - vf_lo);
      vf_lo = vf_hi;
      tend(i, k, j) = t;
      fm1 = f0; f0 = fp1; fp1 = fp2; fp2 = fp3;
    }
    if (!ok && tid == 0) raise_err(m, ERR_TIMEOUT);
  }
  if ((FL & TF_ZERO) && acc && blockIdx.y == 0)
    for (int k = ktf + 1; k <= kte; ++k) tend(i, k, j) = 0.f;
}

// ---------------------------------------------------------------- ph_tend
// rhs_ph (module_big_step_utilities_em.F:1365-2178, 5th/6th order branch):
// the vertical term's wdwn(k+1) is wdwn(k) one level up, u and v of levels
// k, k-1 carry down, the column's map factors and mass terms are read once.
constexpr int PH_RING = 4;
using PhRing = LevelRing<2, PH_RING, HALO_W, HALO_H>;  // ph, phb halo planes

template <int FL>
__global__ void __launch_bounds__(TX* TY, 4) k_tend_ph_col(TileLaunch L) {
  static_assert((FL & TF_ADV) && (FL & TF_ZERO), "the staged form starts from zero and advects");
  extern __shared__ __align__(128) unsigned char smem[];
  const TilePos tp = tile_pos(L, false, true);
  const Mem& m = block_member(L.mem, tp.m);
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
  const int i = tp.i0 + tx, j = tp.j0 + ty;
  const F3 tend = f3(m, WRFGPU_PH_TEND);
  const int kts = m.kts, kte = m.kte, kde = m.kde;
  const int itf = min(m.ite, m.ide - 1), jtf = min(m.jte, m.jde - 1);
  const bool inside = i <= m.ite && j <= m.jte;
  const bool acc = inside && i <= itf && j <= jtf;
  if (inside && !acc && blockIdx.y == 0)
    for (int k = kts; k <= kte; ++k) tend(i, k, j) = 0.f;
  if (!(tp.i0 <= itf && tp.j0 <= jtf)) return;  // block-uniform
  if (acc && blockIdx.y == 0)
    for (int k = kts; k <= min(kte, 1); ++k) tend(i, k, j) = 0.f;
  const Chunk ch = level_chunk_of(max(kts, 2), kte);
  const int ks = ch.k0, ke = ch.k1;  // this block's levels
  if (ks > ke) return;
  const F3 u = f3(m, WRFGPU_U_2), v = f3(m, WRFGPU_V_2), ww = f3(m, WRFGPU_WW), ph = f3(m, WRFGPU_PH_2),
           phb = f3(m, WRFGPU_PHB), w = f3(m, WRFGPU_W_2);
  const F1 c1f = f1(m, WRFGPU_C1F), c2f = f1(m, WRFGPU_C2F), fnm = f1(m, WRFGPU_FNM), fnp = f1(m, WRFGPU_FNP),
           rdnw = f1(m, WRFGPU_RDNW);
  PhRing ring;
  ring.init(smem, ks);
  const CUtensorMap* maps[2] = {tmap_of(m, WRFGPU_PH_2, BOX_HALO), tmap_of(m, WRFGPU_PHB, BOX_HALO)};
  const int x0 = tp.i0 - TMA_HALO - m.ims, z0 = tp.j0 - TMA_HALO - m.jms;
  if (tid == 0) {
    ring.init_barriers();
    mbar_fence_init();
  }
  __syncthreads();
  if (tid == 0)
    for (int d = 0; d < PH_RING - 1 && ks + d <= ke; ++d) ring.issue(ks + d, maps, x0, z0, m.kms);
  // column constants
  float mut_c = 0.f, msfty_c = 0.f, muv1 = 0.f, muv0 = 0.f, muu1 = 0.f, muu0 = 0.f, mvy1 = 0.f, mvy0 = 0.f;
  float mux1 = 0.f, mux0 = 0.f, cy4 = 0.f, cx4 = 0.f, cy2 = 0.f, cx2 = 0.f;
  const float cfn = m.cfn, cfn1 = m.cfn1;
  const bool adv2 = m.cf.phi_adv_z == 2;
  auto wdwn = [&](int kk) {
    if (adv2) return rdnw(kk - 1) * (ph(i, kk, j) - ph(i, kk - 1, j) + phb(i, kk, j) - phb(i, kk - 1, j));
    return .5f * (ww(i, kk, j) + ww(i, kk - 1, j)) * rdnw(kk - 1) * (ph(i, kk, j) - ph(i, kk - 1, j) + phb(i, kk, j) - phb(i, kk - 1, j));
  };
  // carried: wdwn(k), ph, phb and ww of level k, and u, v of levels k-1,
  // k-2 at (i, i+1) / (j, j+1)
  float u0m = 0.f, u1m = 0.f, v0m = 0.f, v1m = 0.f, u0mm = 0.f, u1mm = 0.f, v0mm = 0.f, v1mm = 0.f, wd_lo = 0.f;
  float ph_c = 0.f, phb_c = 0.f, ww_c = 0.f;
  if (acc) {
    mut_c = f2(m, WRFGPU_MUT)(i, j); msfty_c = f2(m, WRFGPU_MSFTY)(i, j);
    muv1 = f2(m, WRFGPU_MUV)(i, j + 1); muv0 = f2(m, WRFGPU_MUV)(i, j);
    muu1 = f2(m, WRFGPU_MUU)(i + 1, j); muu0 = f2(m, WRFGPU_MUU)(i, j);
    mvy1 = f2(m, WRFGPU_MSFVY)(i, j + 1); mvy0 = f2(m, WRFGPU_MSFVY)(i, j);
    mux1 = f2(m, WRFGPU_MSFUX)(i + 1, j); mux0 = f2(m, WRFGPU_MSFUX)(i, j);
    cy4 = 0.25f * m.rdy / msfty_c; cx4 = 0.25f * m.rdx / msfty_c;
    cy2 = 0.5f * m.rdy / msfty_c; cx2 = 0.5f * m.rdx / msfty_c;
    u0m = u(i, ks - 1, j); u1m = u(i + 1, ks - 1, j); v0m = v(i, ks - 1, j); v1m = v(i, ks - 1, j + 1);
    if (ks == kte) {  // the top level extrapolates from the two below it
      u0mm = u(i, ks - 2, j); u1mm = u(i + 1, ks - 2, j); v0mm = v(i, ks - 2, j); v1mm = v(i, ks - 2, j + 1);
    }
    wd_lo = (ks <= kte - 1) ? wdwn(ks) : 0.f;  // wdwn(k) at k = ks
    ph_c = ph(i, ks, j); phb_c = phb(i, ks, j); ww_c = ww(i, ks, j);
  }
  const int o = (ty + TMA_HALO) * HALO_W + tx + TMA_HALO;
  bool ok = true;
  for (int k = ks; k <= ke; ++k) {
    // the level's global inputs, loaded together before the barrier so that
    // their latency overlaps it
    float ph_n = 0.f, phb_n = 0.f, ww_n = 0.f, u0 = 0.f, u1 = 0.f, v0 = 0.f, v1 = 0.f, wk = 0.f;
    if (acc) {
      if (k <= kte - 1) {
        ph_n = ph(i, k + 1, j); phb_n = phb(i, k + 1, j); ww_n = ww(i, k + 1, j);
        u0 = u(i, k, j); u1 = u(i + 1, k, j); v0 = v(i, k, j); v1 = v(i, k, j + 1);
      }
      if (m.cf.non_hydrostatic) wk = w(i, k, j);
    }
    __syncthreads();  // every thread is done with level k-1's slot
    if (tid == 0 && k + PH_RING - 1 <= ke) ring.issue(k + PH_RING - 1, maps, x0, z0, m.kms);
    ok = ring.wait(k) && ok;
    if (!acc) continue;
    const float* PH = ring.plane(k, 0);
    const float* PHB = ring.plane(k, 1);
    if (k + 2 <= kte) {
      prefetch_l2(&ph(i, k + 2, j)); prefetch_l2(&phb(i, k + 2, j)); prefetch_l2(&u(i, k + 2, j));
      prefetch_l2(&v(i, k + 2, j)); prefetch_l2(&ww(i, k + 2, j)); prefetch_l2(&w(i, k + 2, j));
    }
    float t = 0.f;
    // vertical advection of ph (:1396-1428): wdwn(k + 1) from the carried
    // level-k values (the same operands and order)
    if (k <= kte - 1) {
      const float wd_hi = adv2 ? rdnw(k) * (ph_n - ph_c + phb_n - phb_c)
                               : .5f * (ww_n + ww_c) * rdnw(k) * (ph_n - ph_c + phb_n - phb_c);
      if (adv2) t = t - ww_c * (fnm(k) * wd_hi + fnp(k) * wd_lo);
      else t = t - (fnm(k) * wd_hi + fnp(k) * wd_lo);
      wd_lo = wd_hi;
    }
    // "gw" term (:1432-1446)
    if (m.cf.non_hydrostatic) {
      if (k == kde) t = 0.f;
      t = t + (c1f(k) * mut_c + c2f(k)) * G * wk / msfty_c;
    }
    auto S = [&](int d) {  // 6th-order centred difference of ph + phb, stride d in the halo plane
      return 45.f * (PH[o + d] - PH[o - d]) - 9.f * (PH[o + 2 * d] - PH[o - 2 * d]) + (PH[o + 3 * d] - PH[o - 3 * d]) +
             45.f * (PHB[o + d] - PHB[o - d]) - 9.f * (PHB[o + 2 * d] - PHB[o - 2 * d]) +
             (PHB[o + 3 * d] - PHB[o - 3 * d]);
    };
    if (k <= kte - 1) {
      t = t - cy4 * (((c1f(k) * muv1 + c2f(k)) * (v1 + v1m) * mvy1 + (c1f(k) * muv0 + c2f(k)) * (v0 + v0m) * mvy0) *
                     (1.f / 60.f) * S(HALO_W));
      t = t - cx4 * (((c1f(k) * muu1 + c2f(k)) * (u1 + u1m) * mux1 + (c1f(k) * muu0 + c2f(k)) * (u0 + u0m) * mux0) *
                     (1.f / 60.f) * S(1));
    } else {
      t = t - cy2 * (((c1f(k) * muv1 + c2f(k)) * (cfn * v1m + cfn1 * v1mm) * mvy1 +
                      (c1f(k) * muv0 + c2f(k)) * (cfn * v0m + cfn1 * v0mm) * mvy0) *
                     (1.f / 60.f) * S(HALO_W));
      t = t - cx2 * (((c1f(k) * muu1 + c2f(k)) * (cfn * u1m + cfn1 * u1mm) * mux1 +
                      (c1f(k) * muu0 + c2f(k)) * (cfn * u0m + cfn1 * u0mm) * mux0) *
                     (1.f / 60.f) * S(1));
    }
    tend(i, k, j) = t;
    u0mm = u0m; u1mm = u1m; v0mm = v0m; v1mm = v1m;
    u0m = u0; u1m = u1; v0m = v0; v1m = v1;
    ph_c = ph_n; phb_c = phb_n; ww_c = ww_n;
  }
  if (!ok && tid == 0) raise_err(m, ERR_TIMEOUT);
}

// The shortest level chunk of the staged tendencies.
constexpr int TEND_MINLEV = 4;

// variant parameter: 10 x blocks per SM + level chunks (4: as many registers
// as 5 blocks of 128 threads leave, else 4)
template <int DIR>
static void launch_tend_uv(const TileLaunch& L, int nb, cudaStream_t s, int p) {
  const dim3 grid(nb, level_chunks(nb, L.nlev, p % 10, TEND_MINLEV));
  if (p / 10 == 4) k_tend_uv_col<DIR, 5><<<grid, TEND2_THREADS, TEND2_SMEM, s>>>(L);
  else k_tend_uv_col<DIR, 4><<<grid, TEND2_THREADS, TEND2_SMEM, s>>>(L);
}
void launch_tend_u_col(const TileLaunch& L, int nb, cudaStream_t s, int var) {
  launch_tend_uv<0>(L, nb, s, TUNE_PARAM[TU_TENDU][var]);
}
void launch_tend_v_col(const TileLaunch& L, int nb, cudaStream_t s, int var) {
  launch_tend_uv<1>(L, nb, s, TUNE_PARAM[TU_TENDV][var]);
}
void launch_tend_w_col(const TileLaunch& L, int nb, int var, cudaStream_t s) {
  const int minb = TUNE_PARAM[TU_TENDW][var];
  const dim3 grid(nb, level_chunks(nb, L.nlev, 1, TEND_MINLEV));
  auto run = [&](auto kernel) {
    allow_smem(kernel, TENDW_SMEM);
    kernel<<<grid, dim3(TX, TY), TENDW_SMEM, s>>>(L);
  };
  if (minb == 2) run(k_tend_w_col<TF_ALL, 2>);
  else if (minb == 3) run(k_tend_w_col<TF_ALL, 3>);
  else run(k_tend_w_col<TF_ALL, 4>);
}
void launch_tend_t_col(const TileLaunch& L, int nb, int flags, cudaStream_t s) {
  if (flags == (TF_ZERO | TF_ADV)) k_tend_t_col<TF_ZERO | TF_ADV, 4><<<dim3(nb, level_chunks(nb, L.nlev, 1, TEND_MINLEV)), dim3(TX, TY), TEND_SMEM, s>>>(L);
}
void launch_tend_ph_col(const TileLaunch& L, int nb, int flags, cudaStream_t s) {
  if (flags == (TF_ZERO | TF_ADV)) k_tend_ph_col<TF_ZERO | TF_ADV><<<dim3(nb, level_chunks(nb, L.nlev, 1, TEND_MINLEV)), dim3(TX, TY), PhRing::SMEM, s>>>(L);
}

}  // namespace wrfgpu
