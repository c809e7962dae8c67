// Column forms of the acoustic-step kernels used by the fused solver (the
// routine kernels of k_small.cu stay for routine-level calls):
//
//   k_advance_uv_col    advance_uv (module_small_step_em.F:654-967) and the
//                       ru_m, rv_m sums of sumflux (:1473-1633)
//   k_advance_mu_t_col  advance_mu_t (:969-1175) and the ww_m sum
//   k_advance_w_col     advance_w (:1178-1469)
//   k_advance_col       the last two and calc_p_rho (:438-568) in one pass, for
//                       domains whose columns alone do not fill the GPU
//
// The per-point arithmetic is the reference's, in its order: results are
// bit-identical to k_small.cu.
#include "common.cuh"
#include "kernels.h"
#include "ffmath.h"
#include "pair.cuh"

namespace wrfgpu {

// ---------------------------------------------------------------------------
// advance_uv (module_small_step_em.F:654-967) on the u and v points of the
// column, and sumflux's sums of ru_m and rv_m there: the new u and v are in
// registers, so the sums cost one read and one write of ru_m and rv_m (in a
// kernel of their own they read u and v again).
//
// A tile of 32 x 8 staggered columns per block, two columns per thread: every
// field of the pair is one 8-byte load, the pair's left neighbour one scalar
// load, and the additions are packed (pair.cuh).  With one column per thread
// each level cost 26 loads per column of which 12 re-read the neighbours.  ms per
// large step, one column per thread against two: 100x70x30 0.103 / 0.083,
// 256x256x80 0.72 / 0.67, 512x512x80 2.53 / 2.48, 1024x1024x96 10.95 / 10.81 (18
// arrays at 4.7 TB/s).  p, ph and dpn of level k are kept from the level below.
// ---------------------------------------------------------------------------
template <int MINB>
__global__ void __launch_bounds__(TX* TY / 2, MINB) k_advance_uv_col(TileLaunch L, int rk_step, int iteration) {
  const TilePos tp = tile_pos(L, false, true);
  const Mem& m = block_member(L.mem, tp.m);
  const Stage st = stage_of(m, rk_step);
  if (iteration > st.nsmall) return;
  const int i = tp.i0 + 2 * ((int)threadIdx.x & 15), j = tp.j0 + ((int)threadIdx.x >> 4);
  if (i > m.ite || j > m.jte) return;
  const float dts = st.dts_rk;
  const WrfDynConfig& cf = m.cf;
  const int i_start = m.its, i_end = min(m.ite, m.ide - 1), j_start = m.jts, i_endu = m.ite, j_endv = m.jte;
  int i_start_up = i_start, i_end_up = i_endu, j_start_vp = j_start, j_end_vp = j_endv;
  if ((cf.open_xs || cf.symmetric_xs) && m.its == m.ids) i_start_up = i_start_up + 1;
  if ((cf.open_xe || cf.symmetric_xe) && m.ite == m.ide) i_end_up = i_end_up - 1;
  if ((cf.open_ys || cf.symmetric_ys || cf.polar) && m.jts == m.jds) j_start_vp = j_start_vp + 1;
  if ((cf.open_ye || cf.symmetric_ye || cf.polar) && m.jte == m.jde) j_end_vp = j_end_vp - 1;
  int i_start_u_tend = i_start, i_end_u_tend = i_endu, j_start_v_tend = j_start, j_end_v_tend = j_endv;
  if (cf.symmetric_xs && m.its == m.ids) i_start_u_tend = i_start_u_tend + 1;
  if (cf.symmetric_xe && m.ite == m.ide) i_end_u_tend = i_end_u_tend - 1;
  if (cf.symmetric_ys && m.jts == m.jds) j_start_v_tend = j_start_v_tend + 1;
  if (cf.symmetric_ye && m.jte == m.jde) j_end_v_tend = j_end_v_tend - 1;
  // what each column of the pair takes part in: u's update, its tendency and
  // pressure gradient, v's, and the sums (whose points at the first iteration
  // start from zero over the whole staggered tile)
  struct Col { bool in, ut, up, u, v, vp, us, vs; };
  auto col_of = [&](int ii) {
    Col c;
    c.in = ii <= m.ite;
    const bool urow = c.in && j <= min(m.jte, m.jde - 1);
    c.ut = urow && ii >= i_start_u_tend && ii <= i_end_u_tend;
    c.up = urow && ii >= i_start_up && ii <= i_end_up;
    c.u = urow && ii >= min(i_start_u_tend, i_start_up) && ii <= max(i_end_u_tend, i_end_up);
    c.v = j >= j_start_v_tend && j <= j_end_v_tend && ii <= i_end;
    c.vp = c.v && j >= j_start_vp && j <= j_end_vp;
    c.us = urow;
    c.vs = ii <= i_end;
    return c;
  };
  const Col ca = col_of(i), cb = col_of(i + 1);
  const bool first = iteration == 1, last = iteration == st.nsmall;
  const float fns = float(st.nsmall);
  F3 ru_m = f3(m, WRFGPU_RU_M), rv_m = f3(m, WRFGPU_RV_M), ww_m = f3(m, WRFGPU_WW_M);
  F3 usv = f3(m, WRFGPU_U_SAVE), vsv = f3(m, WRFGPU_V_SAVE);
  F3 p = f3(m, WRFGPU_P), pb = f3(m, WRFGPU_PB), ph = f3(m, WRFGPU_PH_2), php = f3(m, WRFGPU_PHP),
     alt = f3(m, WRFGPU_ALT), al = f3(m, WRFGPU_AL);
  F3 u = f3(m, WRFGPU_U_2), ru_tend = f3(m, WRFGPU_RU_TEND), cqu = f3(m, WRFGPU_CQU);
  F3 v = f3(m, WRFGPU_V_2), rv_tend = f3(m, WRFGPU_RV_TEND), cqv = f3(m, WRFGPU_CQV);
  F1 c1h = f1(m, WRFGPU_C1H), c2h = f1(m, WRFGPU_C2H), fnm = f1(m, WRFGPU_FNM), fnp = f1(m, WRFGPU_FNP),
     rdnw = f1(m, WRFGPU_RDNW);
  const float rdx = m.rdx, rdy = m.rdy, emdiv = m.emdiv, cf1 = m.cf1, cf2 = m.cf2, cf3 = m.cf3;
  const int kde = m.kde, k_start = m.kts, k_end = m.kte - 1;
  auto mul = [](float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); };
  auto div = [](float2 a, float2 b) { return make_float2(a.x / b.x, a.y / b.y); };
  auto ro = [&](const F3& a, int k, int jj) { return __ldg(reinterpret_cast<const float2*>(a.p + a.off(i, k, jj))); };
  auto rw = [&](const F3& a, int k) { return *reinterpret_cast<const float2*>(a.p + a.off(i, k, j)); };
  // the pair (i - 1, i): its own first column is the pair's
  auto left = [&](const F3& a, int k, float2 own) { return make_float2(a.ro(i - 1, k, j), own.x); };
  auto put = [&](const F3& a, int k, float2 val, bool ea, bool eb) {
    if (ea && eb) *reinterpret_cast<float2*>(a.p + a.off(i, k, j)) = val;
    else if (ea) a.p[a.off(i, k, j)] = val.x;
    else if (eb) a.p[a.off(i, k, j) + 1] = val.y;
  };
  auto sel = [](bool ea, bool eb, float2 t, float2 f) { return make_float2(ea ? t.x : f.x, eb ? t.y : f.y); };
  auto g2 = [&](int f, int ii, int jj) { const F2 a = f2(m, f); return make_float2(a.ro(ii, jj), a.ro(ii + 1, jj)); };
  // per-column factors (the reference's left-to-right products, split where they start)
  const float2 mu_i = g2(WRFGPU_MU_2, i, j), mu_im = make_float2(f2(m, WRFGPU_MU_2).ro(i - 1, j), mu_i.x),
               mu_jm = g2(WRFGPU_MU_2, i, j - 1);
  const float2 msfuy = g2(WRFGPU_MSFUY, i, j), mxi = g2(WRFGPU_MSFVX_INV, i, j);
  const float2 muu = g2(WRFGPU_MUU, i, j), muv = g2(WRFGPU_MUV, i, j);
  float2 ua, uc, va, vc, mudf_u, mudf_v;
  {
    const float2 d = g2(WRFGPU_MUDF, i, j), dl = make_float2(f2(m, WRFGPU_MUDF).ro(i - 1, j), d.x),
                 dd = g2(WRFGPU_MUDF, i, j - 1);
    const float dx = 1.f / rdx, dy = 1.f / rdy;
    mudf_u = div(muls(-emdiv * dx, sub2(d, dl)), msfuy);
    mudf_v = mul(muls(-emdiv * dy, sub2(d, dd)), mxi);
    const float2 ru = div(g2(WRFGPU_MSFUX, i, j), msfuy), rv = div(g2(WRFGPU_MSFVY, i, j), g2(WRFGPU_MSFVX, i, j));
    ua = muls(rdx, muls(.5f, ru));
    uc = muls(rdx, ru);
    va = muls(rdy, muls(.5f, rv));
    vc = muls(rdy, rv);
  }
  const bool pg_u = ca.up || cb.up, pg_v = ca.vp || cb.vp;
  // this block's chunk of levels (gridDim.y chunks); the levels are
  // independent but for the carried p, ph and dpn of the level below
  const int per = (k_end - k_start + 1 + (int)gridDim.y - 1) / (int)gridDim.y;
  const int k0 = k_start + (int)blockIdx.y * per, k1 = min(k_end, k0 + per - 1);
  if (k0 > k1) return;
  // level k0 values of p and ph, and dpn(k0) (dpn(1) has its own formula);
  // dpn(kde) is zero unless the lid is rigid.  x: columns i - 1, y: row j - 1
  auto edge = [&](float a1, int ka, float a2, int kb, float a3, int kc, bool x) {
    auto both = [&](int k) {
      const float2 o = ro(p, k, j);
      return x ? add2(o, left(p, k, o)) : add2(o, ro(p, k, j - 1));
    };
    return muls(.5f, add2(add2(muls(a1, both(ka)), muls(a2, both(kb))), muls(a3, both(kc))));
  };
  float2 p0 = ro(p, k0, j), ph0 = ro(ph, k0, j), p0x = left(p, k0, p0), ph0x = left(ph, k0, ph0),
         p0y = ro(p, k0, j - 1), ph0y = ro(ph, k0, j - 1);
  float2 dpn_u, dpn_v, dpn_u_top = bc2(0.f), dpn_v_top = bc2(0.f);
  if (k0 == 1) {
    dpn_u = edge(cf1, 1, cf2, 2, cf3, 3, true);
    dpn_v = edge(cf1, 1, cf2, 2, cf3, 3, false);
  } else {
    const float2 pm = ro(p, k0 - 1, j);
    dpn_u = muls(.5f, add2(muls(fnm(k0), add2(p0, p0x)), muls(fnp(k0), add2(pm, left(p, k0 - 1, pm)))));
    dpn_v = muls(.5f, add2(muls(fnm(k0), add2(p0, p0y)), muls(fnp(k0), add2(pm, ro(p, k0 - 1, j - 1)))));
  }
  if (cf.top_lid) {
    dpn_u_top = edge(cf1, kde - 1, cf2, kde - 2, cf3, kde - 3, true);
    dpn_v_top = edge(cf1, kde - 1, cf2, kde - 2, cf3, kde - 3, false);
  }
  for (int k = k0; k <= k1; ++k) {
    const int kk = k + 1;
    // a level's inputs go out together
    const float2 c_u = rw(u, k), c_v = rw(v, k), rut = ro(ru_tend, k, j), rvt = ro(rv_tend, k, j);
    const float2 c_rum = first ? bc2(0.f) : rw(ru_m, k), c_rvm = first ? bc2(0.f) : rw(rv_m, k);
    const float2 c_us = last ? ro(usv, k, j) : bc2(0.f), c_vs = last ? ro(vsv, k, j) : bc2(0.f);
    const float2 c_cqu = ro(cqu, k, j), c_cqv = ro(cqv, k, j);
    const float2 p1 = ro(p, kk, j), ph1 = ro(ph, kk, j), c_pb = ro(pb, k, j), c_php = ro(php, k, j), c_alt = ro(alt, k, j),
                 c_al = ro(al, k, j);
    const float2 p1x = left(p, kk, p1), ph1x = left(ph, kk, ph1), pbx = left(pb, k, c_pb), phpx = left(php, k, c_php),
                 altx = left(alt, k, c_alt), alx = left(al, k, c_al);
    const float2 p1y = ro(p, kk, j - 1), ph1y = ro(ph, kk, j - 1), pby = ro(pb, k, j - 1), phpy = ro(php, k, j - 1),
                 alty = ro(alt, k, j - 1), aly = ro(al, k, j - 1);
    const float h1 = c1h(k), h2 = c2h(k), rz = rdnw(k);
    const float zm = kk < kde ? fnm(kk) : 0.f, zp = kk < kde ? fnp(kk) : 0.f;
    const float2 mh = muls(h1, mu_i);
    // u
    float2 uv = sel(ca.ut, cb.ut, add2(c_u, muls(dts, rut)), c_u);
    if (pg_u) {
      const float2 dpn_hi = kk == kde ? dpn_u_top : muls(.5f, add2(muls(zm, add2(p1, p1x)), muls(zp, add2(p0, p0x))));
      float2 dpxy = mul(mul(ua, add2(muls(h1, muu), bc2(h2))),
                        add2(add2(add2(sub2(ph1, ph1x), sub2(ph0, ph0x)), mul(add2(c_alt, altx), sub2(p0, p0x))),
                             mul(add2(c_al, alx), sub2(c_pb, pbx))));
      dpxy = add2(dpxy, mul(mul(uc, sub2(c_php, phpx)),
                            sub2(muls(rz, sub2(dpn_hi, dpn_u)), muls(.5f, add2(muls(h1, mu_im), mh)))));
      uv = sel(ca.up, cb.up, add2(sub2(uv, mul(muls(dts, c_cqu), dpxy)), muls(h1, mudf_u)), uv);
      dpn_u = dpn_hi;
    }
    put(u, k, uv, ca.u, cb.u);
    // v
    float2 vv = sel(ca.v, cb.v, add2(c_v, muls(dts, rvt)), c_v);
    if (pg_v) {
      const float2 dpn_hi = kk == kde ? dpn_v_top : muls(.5f, add2(muls(zm, add2(p1, p1y)), muls(zp, add2(p0, p0y))));
      float2 dpxy = mul(mul(va, add2(muls(h1, muv), bc2(h2))),
                        add2(add2(add2(sub2(ph1, ph1y), sub2(ph0, ph0y)), mul(add2(c_alt, alty), sub2(p0, p0y))),
                             mul(add2(c_al, aly), sub2(c_pb, pby))));
      dpxy = add2(dpxy, mul(mul(vc, sub2(c_php, phpy)),
                            sub2(muls(rz, sub2(dpn_hi, dpn_v)), muls(.5f, add2(muls(h1, mu_jm), mh)))));
      vv = sel(ca.vp, cb.vp, add2(sub2(vv, mul(muls(dts, c_cqv), dpxy)), muls(h1, mudf_v)), vv);
      dpn_v = dpn_hi;
    }
    put(v, k, vv, ca.v, cb.v);
    // sumflux
    float2 rum = add2(c_rum, uv), rvm = add2(c_rvm, vv);
    if (last) {
      rum = add2(div(rum, bc2(fns)), div(mul(add2(muls(h1, muu), bc2(h2)), c_us), msfuy));
      rvm = add2(div(rvm, bc2(fns)), mul(mul(add2(muls(h1, muv), bc2(h2)), c_vs), mxi));
    }
    if (first) {
      put(ru_m, k, sel(ca.us, cb.us, rum, bc2(0.f)), ca.in, cb.in);
      put(rv_m, k, sel(ca.vs, cb.vs, rvm, bc2(0.f)), ca.in, cb.in);
      put(ww_m, k, bc2(0.f), ca.in && !(ca.us && ca.vs), cb.in && !(cb.us && cb.vs));
    } else {
      put(ru_m, k, rum, ca.us, cb.us);
      put(rv_m, k, rvm, ca.vs, cb.vs);
    }
    p0 = p1; ph0 = ph1; p0x = p1x; ph0x = ph1x; p0y = p1y; ph0y = ph1y;
  }
  if (first && k1 == k_end) {  // level kde holds no mass flux but ww_m of the mass columns
    const int kt = k_end + 1;
    put(ru_m, kt, bc2(0.f), ca.in, cb.in);
    put(rv_m, kt, bc2(0.f), ca.in, cb.in);
    put(ww_m, kt, bc2(0.f), ca.in && !(ca.us && ca.vs), cb.in && !(cb.us && cb.vs));
  }
}

// variant parameter: 10 x blocks per SM (of the one-column form's 256 threads) + level chunks
void launch_advance_uv_col(const TileLaunch& L, int nblocks, int rk_step, int iteration, cudaStream_t s, int var) {
  const int p = TUNE_PARAM[TU_AUV][var], chunks = level_chunks(nblocks, L.nlev, p % 10, 2);
  const dim3 grid(nblocks, chunks), block(TX * TY / 2);
  if (p / 10 == 4) k_advance_uv_col<5><<<grid, block, 0, s>>>(L, rk_step, iteration);
  else k_advance_uv_col<4><<<grid, block, 0, s>>>(L, rk_step, iteration);
}

// ---------------------------------------------------------------------------
// advance_mu_t (module_small_step_em.F:969-1175), one thread per mass column:
// pass 1 the column divergence (kept per level) and its sum, then mu, and
// pass 2 omega by upward recursion, theta, sumflux's sum of ww_m (:1473-1633)
// and advance_w's t_2ave, whose inputs are at hand here (the old and new
// theta, the column masses): advance_w then reads one array instead of three
// and writes none of them back.
// RC: accumulation type of the column sum and the recursion (float: the
// reference; double: mixed form).
// ---------------------------------------------------------------------------
constexpr int KCOL = 129;  // column scratch (kde <= 128)

template <typename RC, int MINB>
__global__ void __launch_bounds__(TX* TY, MINB) k_advance_mu_t_col(TileLaunch L, int rk_step, int iteration) {
  const TilePos tp = tile_pos(L, false, false);
  const Mem& m = block_member(L.mem, tp.m);
  const Stage st = stage_of(m, rk_step);
  if (iteration > st.nsmall) return;
  const int i = tp.i0 + threadIdx.x, j = tp.j0 + threadIdx.y;
  const int i_end = min(m.ite, m.ide - 1), j_end = min(m.jte, m.jde - 1);
  if (i > i_end || j > j_end) return;
  const int k_start = m.kts, k_end = m.kte - 1, kde = m.kde;
  const float dts = st.dts_rk, epssm = m.epssm, rdx = m.rdx, rdy = m.rdy;
  F3 ww = f3(m, WRFGPU_WW), ww_1 = f3(m, WRFGPU_WW1), u = f3(m, WRFGPU_U_2), u_1 = f3(m, WRFGPU_U_SAVE),
     v = f3(m, WRFGPU_V_2), v_1 = f3(m, WRFGPU_V_SAVE), t = f3(m, WRFGPU_T_2), t_1 = f3(m, WRFGPU_T_SAVE),
     t_ave = f3(m, WRFGPU_T_2SAVE), ft = f3(m, WRFGPU_T_TEND);
  F2 MU = f2(m, WRFGPU_MU_2), MUT = f2(m, WRFGPU_MUT), MUAVE = f2(m, WRFGPU_MUAVE), MUTS = f2(m, WRFGPU_MUTS),
     muu = f2(m, WRFGPU_MUU), muv = f2(m, WRFGPU_MUV), MUDF = f2(m, WRFGPU_MUDF), MU_TEND = f2(m, WRFGPU_MU_TEND),
     msfuy = f2(m, WRFGPU_MSFUY), msfvx_inv = f2(m, WRFGPU_MSFVX_INV), msftx = f2(m, WRFGPU_MSFTX),
     msfty = f2(m, WRFGPU_MSFTY);
  F1 c1h = f1(m, WRFGPU_C1H), c2h = f1(m, WRFGPU_C2H), dnw = f1(m, WRFGPU_DNW), fnm = f1(m, WRFGPU_FNM),
     fnp = f1(m, WRFGPU_FNP), rdnw = f1(m, WRFGPU_RDNW);
  const float mxy = msftx.ro(i, j) * msfty.ro(i, j);
  const float muv0 = muv.ro(i, j), muv1 = muv.ro(i, j + 1), muu0 = muu.ro(i, j), muu1 = muu.ro(i + 1, j);
  const float vi0 = msfvx_inv.ro(i, j), vi1 = msfvx_inv.ro(i, j + 1), uy0 = msfuy.ro(i, j), uy1 = msfuy.ro(i + 1, j);
  // pass 1: dvdxi(k) and dmdt
  struct D1 { float v1, v0, vo1, vo0, u1, u0, uo1, uo0; };
  auto load1 = [&](int k, D1& d) {
    d.v1 = v.ro(i, k, j + 1); d.vo1 = v_1.ro(i, k, j + 1); d.v0 = v.ro(i, k, j); d.vo0 = v_1.ro(i, k, j);
    d.u1 = u.ro(i + 1, k, j); d.uo1 = u_1.ro(i + 1, k, j); d.u0 = u.ro(i, k, j); d.uo0 = u_1.ro(i, k, j);
  };
  float dv[KCOL];
  RC dmdt = RC(0.);
  // the levels' loads are independent: four levels in flight at a time; the
  // sum is still taken in k order
  chunked_levels<4, D1>(k_start, k_end, load1, [&](int k, const D1& cur) {
    const float d = mxy * (rdy * ((cur.v1 + (c1h(k) * muv1 + c2h(k)) * cur.vo1 * vi1) -
                                  (cur.v0 + (c1h(k) * muv0 + c2h(k)) * cur.vo0 * vi0)) +
                           rdx * ((cur.u1 + (c1h(k) * muu1 + c2h(k)) * cur.uo1 / uy1) -
                                  (cur.u0 + (c1h(k) * muu0 + c2h(k)) * cur.uo0 / uy0)));
    dv[k] = d;
    if constexpr (sizeof(RC) == 8) dmdt = fma((RC)dnw(k), (RC)d, dmdt);  // mixed form: one FP64 fma per level
    else dmdt = dmdt + (RC)dnw(k) * (RC)d;
  });
  const float mu_tend = MU_TEND.ro(i, j);
  const float muave = MU(i, j);
  const float mu = (float)((RC)muave + (RC)dts * (dmdt + (RC)mu_tend));
  const float mudf = (float)(dmdt + (RC)mu_tend), muts = MUT.ro(i, j) + mu;
  MassImages img;
  img.init(m, i, j);
  img.store([&](int ii, int jj) { MU(ii, jj) = mu; MUDF(ii, jj) = mudf; MUTS(ii, jj) = muts; });
  const float mua = .5f * ((1.f + epssm) * mu + (1.f - epssm) * muave);
  MUAVE(i, j) = mua;
  const float my = msfty.ro(i, j), mx = msftx.ro(i, j);
  const RC rmy = rcp_rc<RC>((RC)my);  // mixed form only
  // pass 2: omega (recursion one level ahead of theta) and theta
  F3 ww_m = f3(m, WRFGPU_WW_M);
  const bool first = iteration == 1, last = iteration == st.nsmall;
  const float fns = float(st.nsmall);
  struct D2 { float ww1, wwm, t, ft, t1, t1xm, t1xp, t1ym, t1yp, u0, u1, v0, v1; };
  auto load2 = [&](int k, D2& d) {
    d.ww1 = ww_1.ro(i, k, j); d.wwm = first ? 0.f : ww_m(i, k, j); d.t = t(i, k, j); d.ft = ft.ro(i, k, j);
    d.t1 = t_1.ro(i, k, j); d.t1xm = t_1.ro(i - 1, k, j); d.t1xp = t_1.ro(i + 1, k, j);
    d.t1ym = t_1.ro(i, k, j - 1); d.t1yp = t_1.ro(i, k, j + 1);
    d.u0 = u.ro(i, k, j); d.u1 = u.ro(i + 1, k, j); d.v0 = v.ro(i, k, j); d.v1 = v.ro(i, k, j + 1);
  };
  RC wwk = (RC)ww(i, 1, j);
  // mixed form: the recursion factored into fmas, c1h (dmdt + mu_tend) + dv
  // times dnw / my (FP64 runs at 1/64 of the FP32 rate on this part)
  const RC dm_mt = (RC)dmdt + (RC)mu_tend;
  // final omega of level 1 (the recursion starts from the unchanged ww(1))
  float wwf_k = ww(i, 1, j) - ww_1.ro(i, 1, j);
  float wdtn_lo = 0.f;  // wdtn(1) = 0
  D2 cur, nxt;
  load2(k_start, cur);
  for (int k = k_start; k <= k_end; ++k) {
    if (k + 1 <= k_end) load2(k + 1, nxt);
    // omega of level k+1 (recursion from level k), needed by wdtn(k+1)
    float wwf_kp1 = 0.f;
    if (k + 1 <= k_end) {
      const int kk = k + 1, kl = kk - 1;
      if constexpr (sizeof(RC) == 8)
        wwk = fma(-fma((RC)c1h(kl), dm_mt, (RC)dv[kk - 1]), (RC)dnw(kk - 1) * rmy, wwk);
      else
        wwk = wwk - (RC)dnw(kk - 1) * (((RC)c1h(kl) * dmdt) + (RC)dv[kk - 1] + ((RC)c1h(kl) * (RC)mu_tend)) / (RC)my;
      wwf_kp1 = (float)wwk - nxt.ww1;
    }
    ww(i, k, j) = wwf_k;
    {
      float wwm = cur.wwm + wwf_k;
      if (last) wwm = wwm / fns + cur.ww1;
      ww_m(i, k, j) = wwm;
    }
    // theta of level k
    const float tv = cur.t;
    float tt = tv + my * dts * cur.ft;
    const float wdtn_hi = (k + 1 == kde) ? 0.f : wwf_kp1 * (fnm(k + 1) * (k + 1 <= k_end ? nxt.t1 : 0.f) + fnp(k + 1) * cur.t1);
    tt = tt - dts * my *
                  (mx * (.5f * rdy * (cur.v1 * (cur.t1yp + cur.t1) - cur.v0 * (cur.t1 + cur.t1ym)) +
                         .5f * rdx * (cur.u1 * (cur.t1xp + cur.t1) - cur.u0 * (cur.t1 + cur.t1xm))) +
                   rdnw(k) * (wdtn_hi - wdtn_lo));
    t(i, k, j) = tt;
    float tav = .5f * ((1.f + epssm) * tt + (1.f - epssm) * tv);
    tav = (tav + (c1h(k) * mua) * T0) / ((c1h(k) * muts + c2h(k)) * (T0 + cur.t1));
    t_ave(i, k, j) = tav;
    wdtn_lo = wdtn_hi;
    wwf_k = wwf_kp1;
    cur = nxt;
  }
  {  // level kde, whose omega stays
    float wwm = (first ? 0.f : ww_m(i, kde, j)) + ww.ro(i, kde, j);
    if (last) wwm = wwm / fns + ww_1.ro(i, kde, j);
    ww_m(i, kde, j) = wwm;
  }
}

// ---------------------------------------------------------------------------
// advance_w (module_small_step_em.F:1178-1469), one thread per mass column.
// Upward pass: at level L, the raw right-hand side of L+1, the
// omega advection term that completes rhs(L), and the explicit w and forward
// elimination of level L-1 (which needs rhs(L)); everything the elimination
// reads from neighbouring levels sits in register windows.  Downward pass:
// back substitution and the geopotential update.  RC as above (the mixed
// form keeps a, alpha, gamma in FP64).
// ---------------------------------------------------------------------------
// Level inputs of advance_w staged by TMA: plane index of each field in a
// ring slot (the FP64 a / alpha of the mixed form are read from global
// memory instead, so that form stages the first 11).
enum AwPlane { AW_TA = 0, AW_PH, AW_W, AW_RWT, AW_CQW, AW_C2A, AW_ALT, AW_PHT, AW_WW, AW_PH1, AW_PHB,
               AW_A, AW_AL, AW_NPLANE };
// Ring depth: levels L, L+1 resident and L+2, L+3 in flight (52 KB: four
// blocks per SM fit).
constexpr int AW_RING = 4;
template <typename RC> struct AwCfg {
  static constexpr int NF = sizeof(RC) == 8 ? AW_A : AW_NPLANE;
  using Ring = TileRing<NF, AW_RING>;
};

template <typename RC, int MINB, bool DAMP>
__global__ void __launch_bounds__(TX* TY, MINB) k_advance_w_col(TileLaunch L, int rk_step, int iteration) {
  using Ring = typename AwCfg<RC>::Ring;
  constexpr int NF = AwCfg<RC>::NF;
  extern __shared__ __align__(128) unsigned char smem[];
  const TilePos tp = tile_pos(L, false, false);
  const Mem& m = block_member(L.mem, tp.m);
  const Stage st = stage_of(m, rk_step);
  if (iteration > st.nsmall) return;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx, po = ty * TX + tx;
  const int i = tp.i0 + tx, j = tp.j0 + ty;
  const int i_end = min(m.ite, m.ide - 1), j_end = min(m.jte, m.jde - 1);
  // every thread takes part in the ring's barriers; only columns of the
  // domain compute and store
  const bool act = i <= i_end && j <= j_end;
  const int ic = act ? i : tp.i0, jc = act ? j : tp.j0;  // in-range indices for the column loads
  const int k_end = m.kte - 1, kde = m.kde;
  const float dts = st.dts_rk, epssm = m.epssm, rdx = m.rdx, rdy = m.rdy;

  Ring ring;
  ring.init(smem, 1);
  {
    const int ids[AW_NPLANE] = {WRFGPU_T_2SAVE, WRFGPU_PH_2, WRFGPU_W_2, WRFGPU_RW_TEND,
                                WRFGPU_CQW, WRFGPU_C2A, WRFGPU_ALT, WRFGPU_PH_TEND, WRFGPU_WW, WRFGPU_PH_SAVE,
                                WRFGPU_PHB, WRFGPU_A, WRFGPU_ALPHA};
    const CUtensorMap* maps[NF];
    for (int f = 0; f < NF; ++f) maps[f] = tmap_of(m, ids[f], BOX_TILE);
    const int x0 = tp.i0 - m.ims, z0 = tp.j0 - m.jms;
    if (tid == 0) {
      ring.init_barriers();
      mbar_fence_init();
    }
    __syncthreads();
    if (tid == 0)
      for (int k = 1; k <= min(AW_RING - 1, kde); ++k) ring.issue(k, maps, x0, z0, m.kms);
    bool ok = true;

    F3 w = f3(m, WRFGPU_W_2), ph = f3(m, WRFGPU_PH_2), u = f3(m, WRFGPU_U_2),
       v = f3(m, WRFGPU_V_2);
    F2 ht = f2(m, WRFGPU_HT), msftx = f2(m, WRFGPU_MSFTX), msfty = f2(m, WRFGPU_MSFTY);
    F1 c1h = f1(m, WRFGPU_C1H), c2h = f1(m, WRFGPU_C2H), c1f = f1(m, WRFGPU_C1F), c2f = f1(m, WRFGPU_C2F),
       fnm = f1(m, WRFGPU_FNM), fnp = f1(m, WRFGPU_FNP), rdnw = f1(m, WRFGPU_RDNW), rdn = f1(m, WRFGPU_RDN);
    const bool fp64 = sizeof(RC) == 8;
    const bool adv2 = m.cf.phi_adv_z == 2;
    const float msft_inv = 1.f / msfty.ro(ic, jc);
    const float my = msfty.ro(ic, jc), mx = msftx.ro(ic, jc), mutij = f2(m, WRFGPU_MUT).ro(ic, jc),
                mua = f2(m, WRFGPU_MUAVE).ro(ic, jc), mts = f2(m, WRFGPU_MUTS).ro(ic, jc);
    auto P = [&](int k, int f) -> float { return ring.plane(k, f)[po]; };
    auto Acoef = [&](int k) -> RC {
      if (fp64) return (RC)__ldg(&d3(m, m.wd[0])(ic, k, jc));
      return (RC)P(k, AW_A < NF ? AW_A : 0);
    };
    auto ALcoef = [&](int k) -> RC {
      if (fp64) return (RC)__ldg(&d3(m, m.wd[1])(ic, k, jc));
      return (RC)P(k, AW_AL < NF ? AW_AL : 0);
    };
    auto GAcoef = [&](int k) -> RC {
      return fp64 ? (RC)__ldg(&d3(m, m.wd[2])(ic, k, jc)) : (RC)f3(m, WRFGPU_GAMMA).ro(ic, k, jc);
    };
    const float eps1 = 1.f + epssm, eps0 = 1.f - epssm;

    // surface w (needs only u, v of the lowest levels)
    const float cf1 = m.cf1, cf2 = m.cf2, cf3 = m.cf3;
    const int I = ic, J = jc;
    const float w1 = (my * .5f * rdy *
                          ((ht.ro(I, J + 1) - ht.ro(I, J)) * (cf1 * v.ro(I, 1, J + 1) + cf2 * v.ro(I, 2, J + 1) + cf3 * v.ro(I, 3, J + 1)) +
                           (ht.ro(I, J) - ht.ro(I, J - 1)) * (cf1 * v.ro(I, 1, J) + cf2 * v.ro(I, 2, J) + cf3 * v.ro(I, 3, J))) +
                      mx * .5f * rdx *
                          ((ht.ro(I + 1, J) - ht.ro(I, J)) * (cf1 * u.ro(I + 1, 1, J) + cf2 * u.ro(I + 1, 2, J) + cf3 * u.ro(I + 1, 3, J)) +
                           (ht.ro(I, J) - ht.ro(I - 1, J)) * (cf1 * u.ro(I, 1, J) + cf2 * u.ro(I, 2, J) + cf3 * u.ro(I, 3, J))));

    // explicit w of level k (FP32, the reference's expression) and forward
    // elimination (RC: FP64 in the mixed form)
    RC wprev = (RC)w1;
    RC wcol[KCOL];
    auto sweep = [&](int k, float wk_in, float rwt, float cqwk, float c2ak, float altk, RC ak, RC alk, float tak,
                     float c2am, float altm, float tam, float r_p1, float r_0, float r_m1, float ph_p1, float ph_0,
                     float ph_m1) {
      const float wkf = wk_in + dts * rwt +
                        msft_inv * cqwk *
                            (+.5f * dts * G * rdn(k) *
                             (c2ak * rdnw(k) / (c1h(k) * mutij + c2h(k)) * (eps1 * (r_p1 - r_0) + eps0 * (ph_p1 - ph_0)) -
                              c2am * rdnw(k - 1) / (c1h(k - 1) * mutij + c2h(k - 1)) *
                                  (eps1 * (r_0 - r_m1) + eps0 * (ph_0 - ph_m1)))) +
                        dts * G * msft_inv * (rdn(k) * (c2ak * altk * tak - c2am * altm * tam) - (c1f(k) * mua));
      RC wk;
      if constexpr (sizeof(RC) == 8) wk = fma(-ak, wprev, (RC)wkf) * alk;  // mixed form: one FP64 fma
      else wk = ((RC)wkf - ak * wprev) * alk;
      wcol[k] = wk;
      wprev = wk;
    };
    float rhs[KCOL];
    rhs[1] = 0.f;
    // windows: level L-1 and L-2 values of what the elimination reads
    float r_m1 = 0.f, r_m2 = 0.f;          // rhs(L-1), rhs(L-2)
    float ph_m1 = 0.f, ph_m2 = 0.f;        // ph(L-1), ph(L-2)
    float ta_m1 = 0.f, ta_m2 = 0.f;        // t_2ave(L-1), t_2ave(L-2)
    float c2a_m1 = 0.f, c2a_m2 = 0.f, alt_m1 = 0.f, alt_m2 = 0.f;
    float w_m1 = 0.f, rwt_m1 = 0.f, cqw_m1 = 0.f;
    RC a_m1 = RC(0.), al_m1 = RC(0.);
    float wd_k = 0.f;   // wdwn(L)
    float rr_k = 0.f;   // raw rhs(L)
    ok = ring.wait(1) && ok;
    float ww_k = P(1, AW_WW), ph1_k = P(1, AW_PH1), phb_k = P(1, AW_PHB);
    for (int Lk = 1; Lk <= k_end; ++Lk) {
      __syncthreads();  // level Lk-1's slot is free
      if (tid == 0 && Lk + AW_RING - 1 <= kde) ring.issue(Lk + AW_RING - 1, maps, x0, z0, m.kms);
      ok = ring.wait(Lk + 1) && ok;
      const float tav = P(Lk, AW_TA), c_ph = P(Lk, AW_PH);
      const float c_w = P(Lk, AW_W), c_rwt = P(Lk, AW_RWT), c_cqw = P(Lk, AW_CQW), c_c2a = P(Lk, AW_C2A),
                  c_alt = P(Lk, AW_ALT);
      const RC c_a = Acoef(Lk), c_al = ALcoef(Lk);
      const float c_pht1 = P(Lk + 1, AW_PHT), c_w1 = P(Lk + 1, AW_W), c_ww1 = P(Lk + 1, AW_WW),
                  c_ph11 = P(Lk + 1, AW_PH1), c_phb1 = P(Lk + 1, AW_PHB);
      // raw rhs(L+1), wdwn(L+1)
      const float rr_next = dts * (c_pht1 + .5f * G * (1.f - epssm) * c_w1);
      float wd_hi;
      if (adv2) wd_hi = rdnw(Lk) * (c_ph11 - ph1_k + c_phb1 - phb_k);
      else wd_hi = .5f * (c_ww1 + ww_k) * rdnw(Lk) * (c_ph11 - ph1_k + c_phb1 - phb_k);
      // rhs(L) complete
      float r_0 = 0.f;
      if (Lk >= 2) {
        float r = rr_k;
        if (adv2) r = r - (dts * ww_k * (fnm(Lk) * wd_hi + fnp(Lk) * wd_k));
        else r = r - (dts * (fnm(Lk) * wd_hi + fnp(Lk) * wd_k));
        r = c_ph + my * r / (c1f(Lk) * mutij + c2f(Lk));
        rhs[Lk] = r;
        r_0 = r;
      }
      // elimination of level L-1
      if (Lk >= 3)
        sweep(Lk - 1, w_m1, rwt_m1, cqw_m1, c2a_m1, alt_m1, a_m1, al_m1, ta_m1, c2a_m2, alt_m2, ta_m2, r_0, r_m1,
              r_m2, c_ph, ph_m1, ph_m2);
      // slide
      r_m2 = r_m1; r_m1 = r_0;
      ph_m2 = ph_m1; ph_m1 = c_ph;
      ta_m2 = ta_m1; ta_m1 = tav;
      c2a_m2 = c2a_m1; c2a_m1 = c_c2a; alt_m2 = alt_m1; alt_m1 = c_alt;
      w_m1 = c_w; rwt_m1 = c_rwt; cqw_m1 = c_cqw; a_m1 = c_a; al_m1 = c_al;
      ww_k = c_ww1; ph1_k = c_ph11; phb_k = c_phb1;
      wd_k = wd_hi; rr_k = rr_next;
    }
    // top: rhs(kde) has no omega term (level kde is resident: waited at Lk = k_end)
    const int kt = k_end + 1;
    const float ph_top = P(kt, AW_PH);
    float r_top = ph_top + my * rr_k / (c1f(kt) * mutij + c2f(kt));
    if (m.cf.top_lid) r_top = 0.f;
    rhs[kt] = r_top;
    // elimination of level k_end
    sweep(k_end, w_m1, rwt_m1, cqw_m1, c2a_m1, alt_m1, a_m1, al_m1, ta_m1, c2a_m2, alt_m2, ta_m2, r_top, r_m1, r_m2,
          ph_top, ph_m1, ph_m2);
    {  // level kde
      const int k = kt;
      const float r = rdnw(k - 1);
      float wkf = P(k, AW_W) + dts * P(k, AW_RWT) +
                  msft_inv * (-.5f * dts * G / (c1h(k - 1) * mutij + c2h(k - 1)) * (r * r) * 2.f * c2a_m1 *
                                  (eps1 * (r_top - r_m1) + eps0 * (ph_top - ph_m1)) -
                              dts * G * (2.f * rdnw(k - 1) * c2a_m1 * alt_m1 * ta_m1 + (c1f(k) * mua)));
      if (m.cf.top_lid) wkf = 0.f;
      RC wk;
      if constexpr (sizeof(RC) == 8) wk = fma(-Acoef(k), wprev, (RC)wkf) * ALcoef(k);
      else wk = ((RC)wkf - Acoef(k) * wprev) * ALcoef(k);
      wcol[k] = wk;
    }
    if (!ok && tid == 0) raise_err(m, ERR_TIMEOUT);
    if (!act) return;
    MassImages img;  // the halo images of ph
    img.init(m, i, j);
    w(i, 1, j) = w1;
    // ---- damp_opt = 3 (module_small_step_em.F:1445-1458): after the back
    // substitution, w relaxes toward w_save in the top zdamp metres with
    // weight dampmag sin^2(pi/2 (h - hbot) / zdamp); the geopotential then
    // takes the damped w.  The recursion itself runs on the undamped values.
    // DAMP: compiled in only when some member uses it (the launcher's choice)
    const bool damp3 = DAMP && m.cf.damp_opt == 3;
    const F3 w_save = f3(m, WRFGPU_W_SAVE), ph_1 = f3(m, WRFGPU_PH_SAVE), phb = f3(m, WRFGPU_PHB);
    const float hdepth = m.cf.zdamp, dampmag = dts * m.cf.dampcoef;
    const float htop = damp3 ? (ph_1.ro(i, kt, j) + phb.ro(i, kt, j)) / G : 0.f;
    auto damped = [&](int k, float wk, float ph1k, float phbk, float wsk) -> float {
      const float hk = (ph1k + phbk) / G;
      const float hbot = htop - hdepth;
      float dampwt = 0.f;
      if (hk >= hbot) {
        const float sn = wrfgpu_ff::sinf_cr(.5f * PI_F * (hk - hbot) / hdepth);
        dampwt = dampmag * sn * sn;
      }
      return (wk - dampwt * (c1f(k) * mutij + c2f(k)) * wsk) / (1.f + dampwt);
    };
    // ---- back substitution (RC) and geopotential (FP32, from the new w)
    RC wup = wcol[kt];
    {
      float wst = (float)wup;
      if (damp3) wst = damped(kt, wst, ph_1.ro(i, kt, j), phb.ro(i, kt, j), w_save.ro(i, kt, j));
      w(i, kt, j) = wst;
      const float phv = rhs[kt] + my * .5f * dts * G * eps1 * wst / (c1f(kt) * mts + c2f(kt));
      img.store([&](int ii, int jj) { ph(ii, kt, jj) = phv; });
    }
    // four levels at a time: their gamma, eliminated w and rhs (global and
    // local-memory loads, independent of the recursion) go out first
    for (int kb = k_end; kb >= 2; kb -= 4) {
      RC gv[4], wv[4];
      float rv[4], p1v[4], pbv[4], wsv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = kb - q;
        if (k >= 2) {
          gv[q] = GAcoef(k); wv[q] = wcol[k]; rv[q] = rhs[k];
          if (damp3) { p1v[q] = ph_1.ro(i, k, j); pbv[q] = phb.ro(i, k, j); wsv[q] = w_save.ro(i, k, j); }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = kb - q;
        if (k >= 2) {
          RC wk;
          if constexpr (sizeof(RC) == 8) wk = fma(-gv[q], wup, wv[q]);
          else wk = wv[q] - gv[q] * wup;
          float wst = (float)wk;
          if (damp3) wst = damped(k, wst, p1v[q], pbv[q], wsv[q]);
          w(i, k, j) = wst;
          const float phv = rv[q] + my * .5f * dts * G * eps1 * wst / (c1f(k) * mts + c2f(k));
          img.store([&](int ii, int jj) { ph(ii, k, jj) = phv; });
          wup = wk;
        }
      }
    }
  }
}

void launch_advance_mu_t_col(const TileLaunch& L, int nblocks, int rk_step, int iteration, bool fp64, cudaStream_t s,
                             int var) {
  const int minb = TUNE_PARAM[TU_AMUT][var];
  if (fp64) {
    if (minb == 2) k_advance_mu_t_col<double, 2><<<nblocks, dim3(TX, TY), 0, s>>>(L, rk_step, iteration);
    else if (minb == 3) k_advance_mu_t_col<double, 3><<<nblocks, dim3(TX, TY), 0, s>>>(L, rk_step, iteration);
    else if (minb == 4) k_advance_mu_t_col<double, 4><<<nblocks, dim3(TX, TY), 0, s>>>(L, rk_step, iteration);
    else k_advance_mu_t_col<double, 5><<<nblocks, dim3(TX, TY), 0, s>>>(L, rk_step, iteration);
  } else {
    if (minb == 2) k_advance_mu_t_col<float, 2><<<nblocks, dim3(TX, TY), 0, s>>>(L, rk_step, iteration);
    else if (minb == 3) k_advance_mu_t_col<float, 3><<<nblocks, dim3(TX, TY), 0, s>>>(L, rk_step, iteration);
    else if (minb == 4) k_advance_mu_t_col<float, 4><<<nblocks, dim3(TX, TY), 0, s>>>(L, rk_step, iteration);
    else k_advance_mu_t_col<float, 5><<<nblocks, dim3(TX, TY), 0, s>>>(L, rk_step, iteration);
  }
}
template <bool DAMP>
static void launch_advance_w_var(const TileLaunch& L, int nblocks, int rk_step, int iteration, bool fp64,
                                 cudaStream_t s, int minb) {
  constexpr size_t S32 = AwCfg<float>::Ring::SMEM, S64 = AwCfg<double>::Ring::SMEM;
  auto run = [&](auto kernel, size_t smem) {
    allow_smem(kernel, smem);
    kernel<<<nblocks, dim3(TX, TY), smem, s>>>(L, rk_step, iteration);
  };
  if (fp64) {
    if (minb == 2) run(k_advance_w_col<double, 2, DAMP>, S64);
    else if (minb == 3) run(k_advance_w_col<double, 3, DAMP>, S64);
    else run(k_advance_w_col<double, 4, DAMP>, S64);
  } else {
    if (minb == 2) run(k_advance_w_col<float, 2, DAMP>, S32);
    else if (minb == 3) run(k_advance_w_col<float, 3, DAMP>, S32);
    else run(k_advance_w_col<float, 4, DAMP>, S32);
  }
}
void launch_advance_w_col(const TileLaunch& L, int nblocks, int rk_step, int iteration, bool fp64, cudaStream_t s,
                          int var, bool damp) {
  const int minb = TUNE_PARAM[TU_AW][var];
  if (damp) launch_advance_w_var<true>(L, nblocks, rk_step, iteration, fp64, s, minb);
  else launch_advance_w_var<false>(L, nblocks, rk_step, iteration, fp64, s, minb);
}

// ---------------------------------------------------------------------------
// advance_mu_t, advance_w, the ww_m sum of sumflux and calc_p_rho on one row
// segment of 32 mass columns per block.  None of the four reads what another
// column's four write, so once u and v have advanced they are one pass over
// the column.
//
// Two columns per lane (8-byte accesses, packed adds), so 16 lanes hold the
// segment and every half warp takes its own contiguous chunk of levels; the
// column's intermediate values live in shared memory.  Only what the
// reference sums or recurs level after level stays serial: the divergence sum
// and the omega recursion are one add per level and are walked by every half
// warp for itself (FP64 form: by warp 0, one lane per column), the tridiagonal
// elimination and back substitution by warp 0.  Everything else — the
// divergence, theta, the right-hand sides, the geopotential, p and al — runs
// with all levels in flight.  A march of one thread per column took 1.1 to 2
// us per level (barrier, loads and divisions in one chain) whatever the
// domain's size, and left a narrow domain's other SMs idle.
//
// RC: type of the column sums and recursions (float: the reference; double:
// the mixed form).
// ---------------------------------------------------------------------------
constexpr int COL_MAXW = 16;  // warps per block

template <typename RC> struct alignas(2 * sizeof(RC)) Pair { RC x, y; };

// Shared memory: level tables, then columns [kde + 1][32] of type RC (sW: the
// sum's terms, then c2a alt t_2ave, then w; FP32 three more: a, alpha, gamma,
// before them the omega recursion's terms; FP64 one more: the omega recursion's
// terms, then omega, then gamma, a and alpha read from global memory by the
// elimination) and float (two: dv, then rhs; theta's part of p).  With all
// four in FP64, 128 levels took 170 KB, one block per SM, and 270 segments two
// waves; with two they take 106 KB and two blocks (75x90x128: 2.39 and 2.18 ms per step).
template <typename RC> constexpr size_t col_smem(int nlev) {
  return (size_t)(nlev + 2) * (2 * sizeof(float4) + 32 * (2 * sizeof(float) + (sizeof(RC) == 8 ? 2 : 4) * sizeof(RC))) +
         2 * COL_MAXW * 32 * sizeof(float);
}

template <typename RC, bool DAMP>
__global__ void __launch_bounds__(32 * COL_MAXW, 1) k_advance_col(TileLaunch L, int rk_step, int iteration) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr bool fp64 = sizeof(RC) == 8;
  using P = Pair<RC>;
  const int mi = find_member(L.block_start, L.nmem, blockIdx.x);
  const Mem& m = block_member(L.mem, mi);
  const Stage st = stage_of(m, rk_step);
  if (iteration > st.nsmall) return;  // members with fewer acoustic steps
  const int tid = threadIdx.x, hw = tid >> 4, c = (tid & 15) * 2;  // half warp, first column
  const int lb = (int)blockIdx.x - __ldg(L.block_start + mi), ntx = tiles_x(m);
  const int i0 = m.its + (lb % ntx) * 32, j = m.jts + lb / ntx;
  const int i_end = min(m.ite, m.ide - 1);
  // every lane takes part in the block's barriers; only columns of the domain
  // store (a lane past them works on the segment's first pair; a pair's
  // second column may be the first halo column)
  const bool act = i0 + c <= i_end, act2 = i0 + c + 1 <= i_end;
  const int i = act ? i0 + c : i0;
  const int k_end = m.kte - 1, kde = m.kde, nlev = m.kme - m.kms + 1;
  const bool first = iteration == 1, last = iteration == st.nsmall;
  const float dts = st.dts_rk, epssm = m.epssm, rdx = m.rdx, rdy = m.rdy;
  // this half warp's levels (a short column leaves the last half warps without)
  const int nh = min((int)blockDim.x >> 4, nlev);
  const int per = (k_end + nh - 1) / nh, ka = 1 + hw * per, kb = min(k_end, ka + per - 1);
  const bool some = ka <= kb, top = some && kb == k_end;  // top: this half warp also owns level kde

  const int NC = (nlev + 2) * 32;
  // level tables: {c1h, c2h, c1f, c2f}, {dnw, rdnw, fnm, fnp} (the column kernels'
  // 1-D coefficients, one 16-byte shared load instead of four global ones each)
  float4* tA = reinterpret_cast<float4*>(smem);
  float4* tB = tA + nlev + 2;
  RC* sW = reinterpret_cast<RC*>(tB + nlev + 2);
  RC* sA = sW + NC;
  RC* sAL = fp64 ? nullptr : sA + NC;
  RC* sGA = fp64 ? sA : sAL + NC;
  float* sR = reinterpret_cast<float*>(sGA + NC);
  float* sQ = sR + NC;
  RC* sS = reinterpret_cast<RC*>(sQ);  // FP64, before sQ is in use: the divergence sum, omega of level 1
  float* sX = sQ + NC;  // c2a alt t_2ave of each half warp's last level
  auto at = [&](int k) { return k * 32 + c; };
  auto rd = [&](const RC* s, int k) -> P { return *reinterpret_cast<const P*>(s + at(k)); };
  auto wr = [&](RC* s, int k, RC a, RC b) { *reinterpret_cast<P*>(s + at(k)) = P{a, b}; };
  auto rdf = [&](const float* s, int k) -> float2 { return *reinterpret_cast<const float2*>(s + at(k)); };
  auto wrf = [&](float* s, int k, float2 v) { *reinterpret_cast<float2*>(s + at(k)) = v; };
  auto gro = [&](const F3& a, int ii, int k, int jj) { return __ldg(reinterpret_cast<const float2*>(a.p + a.off(ii, k, jj))); };
  auto g = [&](const F3& a, int k) { return *reinterpret_cast<const float2*>(a.p + a.off(i, k, j)); };
  auto put = [&](const F3& a, int k, float2 v) {
    if (act2) *reinterpret_cast<float2*>(a.p + a.off(i, k, j)) = v;
    else if (act) a.p[a.off(i, k, j)] = v.x;
  };
  auto g2 = [&](int f, int ii, int jj) { const F2 a = f2(m, f); return make_float2(a.ro(ii, jj), a.ro(ii + 1, jj)); };
  auto mul = [](float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); };
  auto div = [](float2 a, float2 b) { return make_float2(a.x / b.x, a.y / b.y); };
  // s1 x + s2
  auto lin = [](float s1, float2 x, float s2) { return add2(muls(s1, x), bc2(s2)); };

  F3 ww = f3(m, WRFGPU_WW), ww_1 = f3(m, WRFGPU_WW1), u = f3(m, WRFGPU_U_2), v = f3(m, WRFGPU_V_2),
     t = f3(m, WRFGPU_T_2), t_1 = f3(m, WRFGPU_T_SAVE);
  const F1 rdn = f1(m, WRFGPU_RDN);
  {
    F1 c1h = f1(m, WRFGPU_C1H), c2h = f1(m, WRFGPU_C2H), c1f = f1(m, WRFGPU_C1F), c2f = f1(m, WRFGPU_C2F),
       dnw = f1(m, WRFGPU_DNW), fnm = f1(m, WRFGPU_FNM), fnp = f1(m, WRFGPU_FNP), rdnw = f1(m, WRFGPU_RDNW);
    for (int k = 1 + tid; k <= kde; k += blockDim.x) {
      tA[k] = make_float4(c1h(k), c2h(k), c1f(k), c2f(k));
      tB[k] = make_float4(dnw(k), rdnw(k), fnm(k), fnp(k));
    }
  }
  const float2 my = g2(WRFGPU_MSFTY, i, j), mx = g2(WRFGPU_MSFTX, i, j);
  const float2 mu_tend = g2(WRFGPU_MU_TEND, i, j), mutij = g2(WRFGPU_MUT, i, j);
  // read by every half warp before the first barrier, written by one after it
  const float2 mu_old = make_float2(f2(m, WRFGPU_MU_2)(i, j), f2(m, WRFGPU_MU_2)(i + 1, j)), ww_bot = g(ww, 1);
  __syncthreads();  // the level tables

  // ---- advance_mu_t: the column divergence
  const bool one_y = __all_sync(~0u, my.x == 1.f && my.y == 1.f);  // x / 1 = x: no map factor, no division
  {
    F3 u_1 = f3(m, WRFGPU_U_SAVE), v_1 = f3(m, WRFGPU_V_SAVE);
    const float2 mxy = mul(mx, my);
    const float2 muv0 = g2(WRFGPU_MUV, i, j), muv1 = g2(WRFGPU_MUV, i, j + 1), muu0 = g2(WRFGPU_MUU, i, j),
                 muu1 = g2(WRFGPU_MUU, i + 1, j);
    const float2 vi0 = g2(WRFGPU_MSFVX_INV, i, j), vi1 = g2(WRFGPU_MSFVX_INV, i, j + 1), uy0 = g2(WRFGPU_MSFUY, i, j),
                 uy1 = g2(WRFGPU_MSFUY, i + 1, j);
    const bool one_u = __all_sync(~0u, uy0.x == 1.f && uy0.y == 1.f && uy1.y == 1.f);
#pragma unroll 2
    for (int k = ka; k <= kb; ++k) {
      const float2 v0 = gro(v, i, k, j), v1 = gro(v, i, k, j + 1), vo0 = gro(v_1, i, k, j), vo1 = gro(v_1, i, k, j + 1);
      const float2 u0 = gro(u, i, k, j), uo0 = gro(u_1, i, k, j);
      const float2 u1 = make_float2(u0.y, u.ro(i + 2, k, j)), uo1 = make_float2(uo0.y, u_1.ro(i + 2, k, j));
      const float4 ta = tA[k];
      float2 q0 = mul(lin(ta.x, muu0, ta.y), uo0), q1 = mul(lin(ta.x, muu1, ta.y), uo1);
      if (!one_u) { q0 = div(q0, uy0); q1 = div(q1, uy1); }
      const float2 dv =
          mul(mxy, add2(muls(rdy, sub2(add2(v1, mul(mul(lin(ta.x, muv1, ta.y), vo1), vi1)),
                                       add2(v0, mul(mul(lin(ta.x, muv0, ta.y), vo0), vi0)))),
                        muls(rdx, sub2(add2(u1, q1), add2(u0, q0)))));
      wrf(sR, k, dv);
      const float dnw = tB[k].x;
      // FP64: the product is exact, so adding it is the fused multiply-add of the mixed form
      wr(sW, k, (RC)dnw * (RC)dv.x, (RC)dnw * (RC)dv.y);
    }
  }
  __syncthreads();
  // its sum in k order, and the omega recursion: the FP32 form leaves the
  // recursion's terms in sAL, the FP64 form omega itself
  P dmdt{RC(0.), RC(0.)};
  if constexpr (fp64) {
    // the conversions and products are formed by all warps, so that one FP64
    // operation per level is left in each chain (it waits about 110 cycles
    // for its predecessor)
    if (tid < 32) {
      RC s = RC(0.);
#pragma unroll 8
      for (int k = 1; k <= k_end; ++k) s = s + sW[k * 32 + tid];
      sS[tid] = s;
    }
    __syncthreads();
    dmdt = rd(sS, 0);
    const P rmy{rcp_rc<RC>((RC)my.x), rcp_rc<RC>((RC)my.y)};
    const P dm{dmdt.x + (RC)mu_tend.x, dmdt.y + (RC)mu_tend.y};
    for (int k = ka; k <= kb; ++k) {
      const RC c1 = (RC)tA[k].x, dn = (RC)tB[k].x;
      const float2 dv = rdf(sR, k);
      wr(sA, k, -fma(c1, dm.x, (RC)dv.x), -fma(c1, dm.y, (RC)dv.y));
      wr(sW, k, dn * rmy.x, dn * rmy.y);
    }
    if (hw == 0) wr(sS, 1, (RC)ww_bot.x, (RC)ww_bot.y);
    __syncthreads();
    if (tid < 32) {  // omega of level k + 1 over the term it took
      RC wwk = sS[32 + tid];
#pragma unroll 4
      for (int k = 1; k < k_end; ++k) {
        wwk = fma(sA[k * 32 + tid], sW[k * 32 + tid], wwk);
        sA[k * 32 + tid] = wwk;
      }
    }
  } else {
    float2 s = bc2(0.f);
#pragma unroll 8
    for (int k = 1; k <= k_end; ++k) s = add2(s, rdf(sW, k));
    dmdt = P{s.x, s.y};
    for (int k = ka; k <= kb; ++k) {
      const float c1 = tA[k].x;
      float2 tt = muls(tB[k].x, add2(add2(muls(c1, s), rdf(sR, k)), muls(c1, mu_tend)));
      if (!one_y) tt = div(tt, my);
      wrf(sAL, k, tt);
    }
  }
  __syncthreads();
  float2 mu, mudf;
  mu.x = (float)((RC)mu_old.x + (RC)dts * (dmdt.x + (RC)mu_tend.x));
  mu.y = (float)((RC)mu_old.y + (RC)dts * (dmdt.y + (RC)mu_tend.y));
  mudf.x = (float)(dmdt.x + (RC)mu_tend.x);
  mudf.y = (float)(dmdt.y + (RC)mu_tend.y);
  const float2 mts = add2(mutij, mu);
  const float2 mua = muls(.5f, add2(muls(1.f + epssm, mu), muls(1.f - epssm, mu_old)));
  MassImages im0, im1;  // the halo images of mu, mudf, muts, ph, p and al
  im0.init(m, i, j);
  im1.init(m, i + 1, j);
  const bool img = im0.any || im1.any || !act2;
  // v into field a at level k and its halo images
  auto put_img = [&](const F3& a, int k, float2 val) {
    if (!img) {
      *reinterpret_cast<float2*>(a.p + a.off(i, k, j)) = val;
      return;
    }
    if (act) im0.store([&](int ii, int jj) { a.p[a.off(ii, k, jj)] = val.x; });
    if (act2) im1.store([&](int ii, int jj) { a.p[a.off(ii, k, jj)] = val.y; });
  };
  if (hw == 0) {
    F2 MU = f2(m, WRFGPU_MU_2), MUDF = f2(m, WRFGPU_MUDF), MUTS = f2(m, WRFGPU_MUTS), MUAVE = f2(m, WRFGPU_MUAVE);
    if (act) {
      im0.store([&](int ii, int jj) { MU(ii, jj) = mu.x; MUDF(ii, jj) = mudf.x; MUTS(ii, jj) = mts.x; });
      MUAVE(i, j) = mua.x;
    }
    if (act2) {
      im1.store([&](int ii, int jj) { MU(ii, jj) = mu.y; MUDF(ii, jj) = mudf.y; MUTS(ii, jj) = mts.y; });
      MUAVE(i + 1, j) = mua.y;
    }
  }

  // ---- theta and ww_m; then per level what advance_w and calc_p_rho take
  // from theta, and advance_w's rhs
  F3 ph = f3(m, WRFGPU_PH_2), w = f3(m, WRFGPU_W_2), c2a = f3(m, WRFGPU_C2A), alt = f3(m, WRFGPU_ALT);
  const bool adv2 = m.cf.phi_adv_z == 2;
  float2 x_top = bc2(0.f);  // 2 rdnw c2a alt t_2ave of level k_end, for the lid's w
  if (some) {
    F3 ww_m = f3(m, WRFGPU_WW_M), ft = f3(m, WRFGPU_T_TEND), pht = f3(m, WRFGPU_PH_TEND), ph1 = f3(m, WRFGPU_PH_SAVE),
       phb = f3(m, WRFGPU_PHB), t_2ave = f3(m, WRFGPU_T_2SAVE);
    const float fns = float(st.nsmall);
    const bool keep_tave = last && rk_step == 3;  // t_2ave as the large step leaves it
    const float2 mydts = muls(dts, my);  // my dts = dts my
    // omega before the linear part is taken off, at levels ka - 1 and ka
    float2 wr_m = bc2(0.f), wrr = ww_bot;
    if constexpr (fp64) {
      auto om = [&](int k) {  // of level k
        if (k <= 1) return ww_bot;
        const P b = rd(sA, k - 1);
        return make_float2((float)b.x, (float)b.y);
      };
      wr_m = om(ka - 1);
      wrr = om(ka);
    } else {
#pragma unroll 8
      for (int k = 2; k <= ka; ++k) { wr_m = wrr; wrr = sub2(wrr, rdf(sAL, k - 1)); }
    }
    float2 ww1_k = gro(ww_1, i, ka, j), ww_k = sub2(wrr, ww1_k);
    float2 t1_k = gro(t_1, i, ka, j), ph1_k = gro(ph1, i, ka, j), phb_k = gro(phb, i, ka, j);
    float2 wdtn_lo = bc2(0.f), wd_k = bc2(0.f);
    if (ka > 1) {
      const float4 tb = tB[ka];
      const float2 ww_km = sub2(wr_m, gro(ww_1, i, ka - 1, j));
      wdtn_lo = mul(ww_k, add2(muls(tb.z, t1_k), muls(tb.w, gro(t_1, i, ka - 1, j))));
      const float2 dphi = sub2(add2(sub2(ph1_k, gro(ph1, i, ka - 1, j)), phb_k), gro(phb, i, ka - 1, j));
      const float rd_m = tB[ka - 1].y;
      if (adv2) wd_k = muls(rd_m, dphi);
      else wd_k = mul(muls(rd_m, muls(.5f, add2(ww_k, ww_km))), dphi);
    }
    const float2 ww_top = top ? gro(ww, i, kde, j) : bc2(0.f);
    float2 x = bc2(0.f);
    for (int k = ka; k <= kb; ++k) {
      const bool in = k < k_end;
      const float2 ww1_n = (in || last) ? gro(ww_1, i, k + 1, j) : bc2(0.f);
      const float2 c_t = g(t, k), c_ft = gro(ft, i, k, j), t1_n = in ? gro(t_1, i, k + 1, j) : bc2(0.f);
      const float2 ym = gro(t_1, i, k, j - 1), yp = gro(t_1, i, k, j + 1);
      const float2 xm = make_float2(t_1.ro(i - 1, k, j), t1_k.x), xp = make_float2(t1_k.y, t_1.ro(i + 2, k, j));
      const float2 u0 = gro(u, i, k, j), u1 = make_float2(u0.y, u.ro(i + 2, k, j));
      const float2 v0 = gro(v, i, k, j), v1 = gro(v, i, k, j + 1);
      const float2 c_alt = gro(alt, i, k, j), c_c2a = gro(c2a, i, k, j), c_ph = g(ph, k);
      const float2 ph1_n = gro(ph1, i, k + 1, j), phb_n = gro(phb, i, k + 1, j);
      const float2 c_pht = gro(pht, i, k, j), c_w = g(w, k);
      const float2 c_wwm = first ? bc2(0.f) : g(ww_m, k);
      const float4 ta = tA[k], tb = tB[k], tn = tB[k + 1];
      // omega of the level above: wwf for theta (zero at the lid), ww for phi
      float2 wwf_n = bc2(0.f), ww_n = ww_top;
      if (in) {
        if constexpr (fp64) {
          const P b = rd(sA, k);
          wrr = make_float2((float)b.x, (float)b.y);
        } else {
          wrr = sub2(wrr, rdf(sAL, k));
        }
        wwf_n = sub2(wrr, ww1_n);
        ww_n = wwf_n;
      }
      if (last || k == 1) put(ww, k, ww_k);
      {  // sumflux
        float2 wwm = add2(c_wwm, ww_k);
        if (last) wwm = add2(div(wwm, bc2(fns)), ww1_k);
        put(ww_m, k, wwm);
      }
      // theta
      const float2 wdtn_hi = in ? mul(wwf_n, add2(muls(tn.z, t1_n), muls(tn.w, t1_k))) : bc2(0.f);
      float2 tt = add2(c_t, mul(mydts, c_ft));
      tt = sub2(tt, mul(mydts,
                        add2(mul(mx, add2(muls(.5f * rdy, sub2(mul(v1, add2(yp, t1_k)), mul(v0, add2(t1_k, ym)))),
                                          muls(.5f * rdx, sub2(mul(u1, add2(xp, t1_k)), mul(u0, add2(t1_k, xm)))))),
                             muls(tb.y, sub2(wdtn_hi, wdtn_lo)))));
      put(t, k, tt);
      wdtn_lo = wdtn_hi;
      // t_2ave, and theta's part of p
      const float2 mth = mul(lin(ta.x, mts, ta.y), add2(bc2(T0), t1_k));
      float2 tav = muls(.5f, add2(muls(1.f + epssm, tt), muls(1.f - epssm, c_t)));
      tav = div(add2(tav, muls(T0, muls(ta.x, mua))), mth);
      if (keep_tave) put(t_2ave, k, tav);
      x = mul(mul(c_c2a, c_alt), tav);
      wr(sW, k, (RC)x.x, (RC)x.y);
      if (k == k_end) x_top = mul(mul(muls(2.f * tb.y, c_c2a), c_alt), tav);
      wrf(sQ, k, div(mul(c_alt, sub2(tt, mul(muls(ta.x, mu), t1_k))), mth));
      // rhs
      const float2 dphi = sub2(add2(sub2(ph1_n, ph1_k), phb_n), phb_k);
      float2 wd_hi;
      if (adv2) wd_hi = muls(tb.y, dphi);
      else wd_hi = mul(muls(tb.y, muls(.5f, add2(ww_n, ww_k))), dphi);
      float2 r = bc2(0.f);
      if (k >= 2) {
        r = muls(dts, add2(c_pht, muls(.5f * G * (1.f - epssm), c_w)));
        const float2 wdi = add2(muls(tb.z, wd_hi), muls(tb.w, wd_k));
        if (adv2) r = sub2(r, mul(muls(dts, ww_k), wdi));
        else r = sub2(r, muls(dts, wdi));
        r = add2(c_ph, div(mul(my, r), lin(ta.z, mutij, ta.w)));
      }
      wrf(sR, k, r);
      wd_k = wd_hi; ww_k = ww_n; ww1_k = ww1_n; t1_k = t1_n; ph1_k = ph1_n; phb_k = phb_n;
    }
    *reinterpret_cast<float2*>(sX + hw * 32 + c) = x;
    if (top) {  // level kde: rhs without omega; ww_m
      float2 wwm = add2(first ? bc2(0.f) : g(ww_m, kde), ww_top);
      if (last) wwm = add2(div(wwm, bc2(fns)), ww1_k);
      put(ww_m, kde, wwm);
      const float4 ta = tA[kde];
      const float2 rr = muls(dts, add2(gro(pht, i, kde, j), muls(.5f * G * (1.f - epssm), g(w, kde))));
      float2 r = add2(g(ph, kde), div(mul(my, rr), lin(ta.z, mutij, ta.w)));
      if (m.cf.top_lid) r = bc2(0.f);
      wrf(sR, kde, r);
    }
  }
  __syncthreads();

  // ---- advance_w: explicit w of every level, and the elimination's coefficients
  const float eps1 = 1.f + epssm, eps0 = 1.f - epssm;
  float2 w1 = bc2(0.f);
  if (hw == 0) {  // surface w
    F2 ht = f2(m, WRFGPU_HT);
    const float cf1 = m.cf1, cf2 = m.cf2, cf3 = m.cf3;
    auto surf = [&](int I, int J, float myc, float mxc) {
      return (myc * .5f * rdy *
                  ((ht.ro(I, J + 1) - ht.ro(I, J)) * (cf1 * v.ro(I, 1, J + 1) + cf2 * v.ro(I, 2, J + 1) + cf3 * v.ro(I, 3, J + 1)) +
                   (ht.ro(I, J) - ht.ro(I, J - 1)) * (cf1 * v.ro(I, 1, J) + cf2 * v.ro(I, 2, J) + cf3 * v.ro(I, 3, J))) +
              mxc * .5f * rdx *
                  ((ht.ro(I + 1, J) - ht.ro(I, J)) * (cf1 * u.ro(I + 1, 1, J) + cf2 * u.ro(I + 1, 2, J) + cf3 * u.ro(I + 1, 3, J)) +
                   (ht.ro(I, J) - ht.ro(I - 1, J)) * (cf1 * u.ro(I, 1, J) + cf2 * u.ro(I, 2, J) + cf3 * u.ro(I, 3, J))));
    };
    w1 = make_float2(surf(i, j, my.x, mx.x), surf(i + 1, j, my.y, mx.y));
    put(w, 1, w1);  // level 1 of w is not read in this kernel after the last barrier
  }
  if (some) {
    F3 rwt = f3(m, WRFGPU_RW_TEND), cqw = f3(m, WRFGPU_CQW);
    auto coef = [&](int q, int k) -> P {
      if constexpr (fp64) {
        const double2 d = __ldg(reinterpret_cast<const double2*>(&d3(m, m.wd[q])(i, k, j)));
        return P{d.x, d.y};
      } else {
        const float2 d = gro(f3(m, q == 0 ? WRFGPU_A : q == 1 ? WRFGPU_ALPHA : WRFGPU_GAMMA), i, k, j);
        return P{d.x, d.y};
      }
    };
    const float2 msft_inv = div(bc2(1.f), my);
    // level k's term of the vertical difference, from levels k and k+1
    auto dz = [&](int k, float2 c2ak, float2 r_0, float2 r_p, float2 ph_0, float2 ph_p) {
      const float4 ta = tA[k];
      return mul(div(muls(tB[k].y, c2ak), lin(ta.x, mutij, ta.y)),
                 add2(muls(eps1, sub2(r_p, r_0)), muls(eps0, sub2(ph_p, ph_0))));
    };
    float2 r_k = rdf(sR, ka), ph_k = g(ph, ka);
    float2 dz_m = bc2(0.f), x_m = bc2(0.f), c_c2a = bc2(0.f);
    if (ka > 1) {
      dz_m = dz(ka - 1, gro(c2a, i, ka - 1, j), rdf(sR, ka - 1), r_k, g(ph, ka - 1), ph_k);
      x_m = *reinterpret_cast<const float2*>(sX + (hw - 1) * 32 + c);
    }
    float2 r_m = bc2(0.f), ph_m = bc2(0.f);
    // (the loads of two levels go out together)
    struct L4 { float2 c2a, ph, w, rwt, cqw; P a, al, ga; };
    chunked_levels<2, L4>(
        ka, kb,
        [&](int k, L4& d) {
          d.c2a = gro(c2a, i, k, j); d.ph = g(ph, k + 1); d.w = g(w, k);
          d.rwt = gro(rwt, i, k, j); d.cqw = gro(cqw, i, k, j);
          if constexpr (!fp64) { d.a = coef(0, k); d.al = coef(1, k); }
          d.ga = coef(2, k);
        },
        [&](int k, const L4& d) {
          c_c2a = d.c2a;
          const float2 ph_p = d.ph, r_p = rdf(sR, k + 1);
          const P xr = rd(sW, k);
          const float2 x = make_float2((float)xr.x, (float)xr.y);
          const float2 dz_k = dz(k, c_c2a, r_k, r_p, ph_k, ph_p);
          if (k >= 2) {
            const float rdnk = rdn(k);
            const float2 wk = add2(add2(add2(d.w, muls(dts, d.rwt)),
                                        mul(mul(msft_inv, d.cqw), muls(+.5f * dts * G * rdnk, sub2(dz_k, dz_m)))),
                                   mul(muls(dts * G, msft_inv), sub2(muls(rdnk, sub2(x, x_m)), muls(tA[k].z, mua))));
            wr(sW, k, (RC)wk.x, (RC)wk.y);
            if constexpr (!fp64) {
              wr(sA, k, d.a.x, d.a.y);
              wr(sAL, k, d.al.x, d.al.y);
            }
            wr(sGA, k, d.ga.x, d.ga.y);
          }
          dz_m = dz_k; x_m = x; r_m = r_k; ph_m = ph_k; r_k = r_p; ph_k = ph_p;
        });
    if (hw == 0) wr(sW, 1, (RC)w1.x, (RC)w1.y);
    if (top) {
      const int k = kde;
      const float r = tB[k - 1].y;
      const float4 tm = tA[k - 1];
      const float2 q = muls(r * r, div(bc2(-.5f * dts * G), lin(tm.x, mutij, tm.y)));
      const float2 a = mul(mul(muls(2.f, q), c_c2a),
                           add2(muls(eps1, sub2(r_k, r_m)), muls(eps0, sub2(ph_k, ph_m))));
      float2 wk = add2(add2(g(w, k), muls(dts, gro(rwt, i, k, j))),
                       mul(msft_inv, sub2(a, muls(dts * G, add2(x_top, muls(tA[k].z, mua))))));
      if (m.cf.top_lid) wk = bc2(0.f);
      wr(sW, k, (RC)wk.x, (RC)wk.y);
      if constexpr (!fp64) {
        const P ca = coef(0, k), cal = coef(1, k);
        wr(sA, k, ca.x, ca.y);
        wr(sAL, k, cal.x, cal.y);
      }
    }
  }
  __syncthreads();
  // ---- the tridiagonal solve, one lane per column; a batch of levels is read
  // ahead of its recursion
  if (tid < 32) {
    constexpr int Q = 8;  // FP64, whose a and alpha come from global memory: 4 / 6 / 8 2.23 / 2.19 / 2.18 ms per step
    RC wk = sW[32 + tid], b[Q], a[Q], al[Q];
    const int ic = i0 + tid <= i_end ? i0 + tid : i0;  // a lane past the domain takes the first column
    auto up = [&](int kq) {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int k = min(kq + q, kde), o = k * 32 + tid;
        b[q] = sW[o];
        if constexpr (fp64) {
          a[q] = __ldg(&d3(m, m.wd[0])(ic, k, j)); al[q] = __ldg(&d3(m, m.wd[1])(ic, k, j));
        } else {
          a[q] = sA[o]; al[q] = sAL[o];
        }
      }
    };
    up(2);
    for (int kq = 2; kq <= kde; kq += Q) {
      RC r[Q], cb[Q], ca[Q], cal[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) { cb[q] = b[q]; ca[q] = a[q]; cal[q] = al[q]; }
      up(kq + Q);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if constexpr (fp64) wk = fma(-ca[q], wk, cb[q]) * cal[q];  // mixed form: one FP64 fma
        else wk = (cb[q] - ca[q] * wk) * cal[q];
        r[q] = wk;
      }
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (kq + q <= kde) sW[(kq + q) * 32 + tid] = r[q];
    }
    wk = sW[kde * 32 + tid];
    auto down = [&](int kq) {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int o = max(kq - q, 2) * 32 + tid;
        b[q] = sW[o]; a[q] = sGA[o];
      }
    };
    down(k_end);
    for (int kq = k_end; kq >= 2; kq -= Q) {
      RC r[Q], cb[Q], ca[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) { cb[q] = b[q]; ca[q] = a[q]; }
      down(kq - Q);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if constexpr (fp64) wk = fma(-ca[q], wk, cb[q]);
        else wk = cb[q] - ca[q] * wk;
        r[q] = wk;
      }
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (kq - q >= 2) sW[(kq - q) * 32 + tid] = r[q];
    }
  }
  __syncthreads();
  if (!some || !act) return;

  // ---- damp_opt = 3 (module_small_step_em.F:1445-1458): after the back
  // substitution, w relaxes toward w_save in the top zdamp metres with
  // weight dampmag sin^2(pi/2 (h - hbot) / zdamp); the geopotential then
  // takes the damped w.  The recursion itself ran on the undamped values.
  // DAMP: compiled in only when some member uses it (the launcher's choice)
  const bool damp3 = DAMP && m.cf.damp_opt == 3;
  const F3 w_save = f3(m, WRFGPU_W_SAVE), ph_1 = f3(m, WRFGPU_PH_SAVE), phb = f3(m, WRFGPU_PHB);
  const float hdepth = m.cf.zdamp, dampmag = dts * m.cf.dampcoef;
  float2 hbot = bc2(0.f);
  if (damp3) {
    const float2 h = add2(gro(ph_1, i, kde, j), gro(phb, i, kde, j));
    hbot = make_float2(h.x / G - hdepth, h.y / G - hdepth);
  }
  auto damped = [&](float wk, float h, float hb, float mass, float ws) -> float {
    const float hk = h / G;
    float dampwt = 0.f;
    if (hk >= hb) {
      const float sn = wrfgpu_ff::sinf_cr(.5f * PI_F * (hk - hb) / hdepth);
      dampwt = dampmag * sn * sn;
    }
    return (wk - dampwt * mass * ws) / (1.f + dampwt);
  };
  auto new_w = [&](int k) -> float2 {
    const P r = rd(sW, k);
    float2 wk = make_float2((float)r.x, (float)r.y);
    if (damp3) {
      const float2 h = add2(gro(ph_1, i, k, j), gro(phb, i, k, j)), ws = gro(w_save, i, k, j);
      const float2 mass = lin(tA[k].z, mutij, tA[k].w);
      wk = make_float2(damped(wk.x, h.x, hbot.x, mass.x, ws.x), damped(wk.y, h.y, hbot.y, mass.y, ws.y));
    }
    return wk;
  };
  const float2 pc = muls(eps1, muls(G, muls(dts, muls(.5f, my))));  // my .5 dts g (1 + epssm), left to right
  auto new_ph = [&](int k, float2 wst) {
    const float4 ta = tA[k];
    return add2(rdf(sR, k), div(mul(pc, wst), lin(ta.z, mts, ta.w)));
  };
  // ---- w, the geopotential, and calc_p_rho between two of its levels
  F3 al = f3(m, WRFGPU_AL), p = f3(m, WRFGPU_P), pm1 = f3(m, WRFGPU_PM1);
  const float smdiv = m.smdiv;
  float2 ph_k;
  if (ka == 1) {
    ph_k = g(ph, 1);
  } else {
    const float2 wst = new_w(ka);
    put(w, ka, wst);
    ph_k = new_ph(ka, wst);
    put_img(ph, ka, ph_k);
  }
  struct L6 { float2 a, c2a, pm1; };
  chunked_levels<2, L6>(
      ka, kb, [&](int k, L6& d) { d.a = gro(alt, i, k, j); d.c2a = gro(c2a, i, k, j); d.pm1 = g(pm1, k); },
      [&](int k, const L6& d) {
        const int kn = k + 1;
        const float2 wst = new_w(kn), ph_n = new_ph(kn, wst);
        if (kn <= kb || kn == kde) {  // else the next half warp's own level
          put(w, kn, wst);
          put_img(ph, kn, ph_n);
        }
        const float4 ta = tA[k];
        const float2 alv = mul(div(bc2(-1.f), lin(ta.x, mts, ta.y)),
                               add2(mul(d.a, muls(ta.x, mu)), muls(tB[k].y, sub2(ph_n, ph_k))));
        put_img(al, k, alv);
        const float2 pn = mul(d.c2a, sub2(rdf(sQ, k), alv));
        put(pm1, k, pn);
        put_img(p, k, add2(pn, muls(smdiv, sub2(pn, d.pm1))));
        ph_k = ph_n;
      });
}

void launch_advance_col(const TileLaunch& L, int nblocks, int nlev_max, int rk_step, int iteration, bool fp64,
                        cudaStream_t s, bool damp) {
  const size_t sm = fp64 ? col_smem<double>(nlev_max) : col_smem<float>(nlev_max);
  // two blocks of 8 warps per SM; 16 warps where shared memory or the domain
  // leaves an SM one block (41x41x41: 0.131 against 0.145 ms per step)
  const int threads = 32 * (sm > 113 * 1024 || nblocks <= 152 ? COL_MAXW : COL_MAXW / 2);
  auto run = [&](auto kernel, size_t largest) {
    allow_smem(kernel, largest);
    kernel<<<nblocks, threads, sm, s>>>(L, rk_step, iteration);
  };
  if (fp64 && damp) run(k_advance_col<double, true>, col_smem<double>(KDE_MAX));
  else if (fp64) run(k_advance_col<double, false>, col_smem<double>(KDE_MAX));
  else if (damp) run(k_advance_col<float, true>, col_smem<float>(KDE_MAX));
  else run(k_advance_col<float, false>, col_smem<float>(KDE_MAX));
}

}  // namespace wrfgpu
