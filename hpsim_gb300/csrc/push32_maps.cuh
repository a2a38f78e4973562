// push32_maps.cuh -- element transfer maps on FP32 particle state, as device
// functors.  A map's apply() takes one live particle (in registers) and
// returns the set of fields it changed, so one kernel template serves every
// element and the same map can run alone, followed by a reduction of the
// new state, or after the space-charge kick (push32.cu).
//
// Particle state: x, x', y, y' in FP32; phi and W as FP32 offsets from the
// synchronous particle, which the host advances in FP64.  Every phase and
// energy increment is formed as a difference from the synchronous
// particle's increment: 1/beta_i - 1/beta_ref from dinvb, cos(p + e) - cos(p)
// from half-angle products, transit-time factors re-expanded about the
// reference's beta.
//
// A map gives a particle the same bits in every sweep it runs in (alone, in a
// run, around a kick, in a batch): wherever a product meets a sum, fmaf,
// __fmul_rn or __fadd_rn says what is rounded, so that the choice is not the
// compiler's in each kernel.  The space-charge kick behind a map takes one of
// two fields by a comparison that particles on the mesh's edge decide either
// way by their last bit.
#pragma once

#include "common.cuh"

namespace hps {

struct Part {
  uint32_t lo;                  // loss flag
  float x, xp, y, yp, ph, w;    // ph, w: offsets from the synchronous particle
};

enum : uint32_t { WR_X = 1, WR_XP = 2, WR_Y = 4, WR_YP = 8, WR_PH = 16, WR_W = 32, WR_LOSS = 64 };

__device__ inline Part load_part(const DevBeam &b, uint32_t i) {
  return {b.loss[i], b.fx[i], b.fxp[i], b.fy[i], b.fyp[i], b.fphi[i], b.fw[i]};
}
__device__ inline void store_part(const DevBeam &b, uint32_t i, const Part &p, uint32_t m) {
  if (m & WR_X) b.fx[i] = p.x;
  if (m & WR_XP) b.fxp[i] = p.xp;
  if (m & WR_Y) b.fy[i] = p.y;
  if (m & WR_YP) b.fyp[i] = p.yp;
  if (m & WR_PH) b.fphi[i] = p.ph;
  if (m & WR_W) b.fw[i] = p.w;
  if (m & WR_LOSS) b.loss[i] = p.lo;
}

constexpr float F_TWOPI = 6.28318530717958647692f;

// SimulatePartialDriftKernel, simulation_kernel.cu:86-118
struct DriftMap {
  RefK r;
  float hf, aper2, c;  // c = 2 pi hf / lambda
  uint32_t eid;
  __device__ uint32_t apply(Part &p) const { return apply(p, [&] { return dinvb(p.w, r); }); }
  // D(): 1/beta of the particle minus the synchronous particle's
  template <class F>
  __device__ uint32_t apply(Part &p, const F &D) const {
    const float x = fmaf(p.xp, hf, p.x), y = fmaf(p.yp, hf, p.y);
    if (aper2 != 0.0f && fmaf(x, x, y * y) > aper2) { p.lo = eid; return WR_LOSS; }
    p.x = x;
    p.y = y;
    p.ph = fmaf(c, D(), p.ph);
    return WR_X | WR_Y | WR_PH;
  }
  // on a live particle, without an aperture
  __device__ void open(Part &p, float D) const {
    p.x = fmaf(p.xp, hf, p.x);
    p.y = fmaf(p.yp, hf, p.y);
    p.ph = fmaf(c, D, p.ph);
  }
};

// SimulateHalfQuadKernel, simulation_kernel.cu:142-218 (coordinates are
// written before the aperture test, the phase only for particles kept).
// k = sqrt(|qG| c / (m beta gamma)) differs from the synchronous particle's
// k_r by a small fraction, so sin, cos, sinh, cosh of k ds/4 are Taylor
// steps of order 4 from their FP64 values at k_r ds/4 (truncation below
// e^5/120 for the step e).
struct QuadMap {
  RefK r;
  float len, aper2, qg, c;         // c = 2 pi len / (2 lambda)
  float sk0, isk0;                 // sqrt(|qG| c / m) and its inverse
  float kds_r, s_r, c_r, sh_r, ch_r;
  uint32_t eid;
  __device__ uint32_t apply(Part &p) const { return apply(p, [&] { return dinvb(p.w, r); }); }
  template <class F>
  __device__ uint32_t apply(Part &p, const F &D) const {
    float x = p.x, y = p.y, xp = p.xp, yp = p.yp;
    uint32_t m;
    if (qg == 0.0f) {
      // the drifted coordinates are stored, but the aperture test below sees
      // the ones before the half (the reference writes memory and tests its
      // unchanged locals)
      p.x = fmaf(xp * len, 0.5f, x);
      p.y = fmaf(yp * len, 0.5f, y);
      m = WR_X | WR_Y;
      if (aper2 != 0.0f && fmaf(x, x, y * y) > aper2) { p.lo = eid; return m | WR_LOSS; }
      p.ph = fmaf(c, D(), p.ph);
      return m | WR_PH;
    } else {
      const float sl = fmaf(yp, yp, fmaf(xp, xp, 1.0f));
      if (qg > 0.0f) focus(x, xp, y, yp, p.w, sl);
      else focus(y, yp, x, xp, p.w, sl);
      m = WR_X | WR_Y | WR_XP | WR_YP;
    }
    p.x = x; p.y = y; p.xp = xp; p.yp = yp;
    if (aper2 != 0.0f && fmaf(y, y, x * x) > aper2) { p.lo = eid; return m | WR_LOSS; }
    p.ph = fmaf(c, D(), p.ph);
    return m | WR_PH;
  }
  // the half's two steps: u is the focusing plane, v the other; sl = 1 + x'^2 + y'^2
  __device__ void focus(float &u, float &up, float &v, float &vp, float w, float sl) const {
    const float g = fmaf(w, r.minv, r.g);
    const float bg = sqrt_norm(g * (g + 2.0f) * sl);
    const float rb = rsqrt_fast(bg);
    const float k = sk0 * rb;              // sqrt(kcoef / bg)
    const float inv_k = bg * rb * isk0;    // sqrt(bg / kcoef)
    const float e = fmaf(len * 0.25f, k, -kds_r);
    const float e2 = e * e;
    const float t1 = e * fmaf(e2, 1.0f / 6.0f, 1.0f), t01 = fmaf(e2, fmaf(e2, 1.0f / 24.0f, 0.5f), 1.0f);
    // sin(a + e) = s_r (1 - e^2/2 + e^4/24) + c_r (e - e^3/6); sinh, cosh alike
    const float so = fmaf(-(e * e2), 1.0f / 6.0f, e), co = fmaf(-e2, fmaf(-e2, 1.0f / 24.0f, 0.5f), 1.0f);
    const float s = fmaf(c_r, so, s_r * co);
    const float cc = fmaf(-s_r, so, c_r * co);
    const float sh = fmaf(ch_r, t1, sh_r * t01);
    const float ch = fmaf(sh_r, t1, ch_r * t01);
    const float sovk = s * inv_k, shovk = sh * inv_k, sk = s * k, shk = sh * k;
#pragma unroll
    for (int rep = 0; rep < 2; ++rep) {
      const float un = fmaf(cc, u, sovk * up), vn = fmaf(ch, v, shovk * vp);
      up = fmaf(cc, up, -sk * u);
      vp = fmaf(shk, v, ch * vp);
      u = un;
      v = vn;
    }
  }
  // on a live particle, without an aperture; SIGN of qg
  template <int SIGN>
  __device__ void open(Part &p, float D) const {
    const float sl = fmaf(p.yp, p.yp, fmaf(p.xp, p.xp, 1.0f));
    if constexpr (SIGN > 0) focus(p.x, p.xp, p.y, p.yp, p.w, sl);
    else if constexpr (SIGN < 0) focus(p.y, p.yp, p.x, p.xp, p.w, sl);
    else {
      p.x = fmaf(p.xp * len, 0.5f, p.x);
      p.y = fmaf(p.yp * len, 0.5f, p.y);
    }
    p.ph = fmaf(c, D, p.ph);
  }
};

// SimulateSteererKernel, simulation_kernel.cu:120-140
struct SteerMap {
  RefK r;
  float kh, kv;  // B L q c / m of each plane, 0 when off
  __device__ uint32_t apply(Part &p) const {
    const float g = fmaf(p.w, r.minv, r.g);
    const float btgm = sqrtf(g * (g + 2.0f));
    uint32_t m = 0;
    if (kh != 0.0f) { p.xp += kh / btgm; m |= WR_XP; }
    if (kv != 0.0f) { p.yp += kv / btgm; m |= WR_YP; }
    return m;
  }
};

// RF gap first half (simulation_kernel.cu:226-288): every branch advances
// phi by K / beta: DTL K = beta_in (pi clbl + dps) + pi dcell/lambda -
// pi q1/lambda, CCL K = betag (pi clbl + dps) (+ const), zero amplitude
// K = 2 pi dd1 / lambda.
struct Gap1Map {
  RefK r;
  float dd1, K;
  __device__ uint32_t apply(Part &p) const { return apply(p, [&] { return dinvb(p.w, r); }); }
  template <class F>
  __device__ uint32_t apply(Part &p, const F &D) const {
    p.x = fmaf(dd1, p.xp, p.x);
    p.y = fmaf(dd1, p.yp, p.y);
    p.ph = fmaf(K, D(), p.ph);
    return WR_X | WR_Y | WR_PH;
  }
};

// sin and cos of a phase: reduced to [-pi, pi] by whole turns, then the
// hardware approximation (absolute error about 2^-21 there, below the FP32
// rounding of the phase offsets it is applied to)
__device__ __forceinline__ void fast_sincos(float a, float *s, float *c) {
  const float r = fmaf(-6.28318530717958647692f, rintf(a * 0.15915494309189533577f), a);
  __sincosf(r, s, c);
}

// Bessi0c / Bessi1c (simulation_kernel.cu:15-73) in FP32; bessi0c also
// returns I0 - 1 without cancellation
__device__ inline float fbessi0c(float x, float *m1) {
  const float ax = fabsf(x);
  if (ax < 3.75f) {
    float cy = x * (1.0f / 3.75f);
    cy = cy * cy;
    float s = fmaf(cy, 0.45813e-2f, 0.360768e-1f);
    s = fmaf(cy, s, 0.2659732f);
    s = fmaf(cy, s, 1.2067492f);
    s = fmaf(cy, s, 3.0899424f);
    s = fmaf(cy, s, 3.5156229f);
    s = __fmul_rn(cy, s);
    *m1 = s;
    return __fadd_rn(1.0f, s);
  }
  const float cy = div_fast(3.75f, ax);
  float ans = fmaf(cy, 0.392377e-2f, -0.1647633e-1f);
  ans = fmaf(cy, ans, 0.2635537e-1f);
  ans = fmaf(cy, ans, -0.2057706e-1f);
  ans = fmaf(cy, ans, 0.916281e-2f);
  ans = fmaf(cy, ans, -0.157565e-2f);
  ans = fmaf(cy, ans, 0.225319e-2f);
  ans = fmaf(cy, ans, 0.1328592e-1f);
  ans = fmaf(cy, ans, 0.39894228f);
  ans = __fmul_rn(expf(ax) * rsqrt_fast(ax), ans);
  *m1 = __fadd_rn(ans, -1.0f);
  return ans;
}
__device__ inline float fbessi1c(float x) {
  const float ax = fabsf(x);
  float ans;
  if (ax < 3.75f) {
    float cy = x * (1.0f / 3.75f);
    cy = cy * cy;
    ans = fmaf(cy, 0.32411e-3f, 0.301532e-2f);
    ans = fmaf(cy, ans, 0.2658733e-1f);
    ans = fmaf(cy, ans, 0.15084934f);
    ans = fmaf(cy, ans, 0.51498869f);
    ans = fmaf(cy, ans, 0.87890594f);
    ans = fmaf(cy, ans, 0.5f);
    ans = __fmul_rn(ax, ans);
  } else {
    const float cy = div_fast(3.75f, ax);
    ans = fmaf(-cy, 0.420059e-2f, 0.1787654e-1f);
    ans = fmaf(cy, ans, -0.2895312e-1f);
    ans = fmaf(cy, ans, 0.2282967e-1f);
    ans = fmaf(cy, ans, -0.1031555e-1f);
    ans = fmaf(cy, ans, 0.163801e-2f);
    ans = fmaf(cy, ans, -0.362018e-2f);
    ans = fmaf(cy, ans, -0.3988024e-1f);
    ans = fmaf(cy, ans, 0.39894228f);
    ans = __fmul_rn(ans, expf(ax) * rsqrt_fast(ax));
  }
  return x < 0.0f ? -ans : ans;
}

// RF gap second half (simulation_kernel.cu:310-497).  The synchronous
// particle's kick is formed on the host; a particle's is taken as the
// difference from it.  When the synchronous particle drifts through the
// gap (zero amplitude, or a CCL gap below the fit range) a kicked particle
// is measured from a hypothetical kicked synchronous particle (rh) and moved
// to the actual one by corr_phi / corr_w.
struct Gap2Map {
  RefK rin, rh;          // reference before the gap, reference after its (hypothetical) kick
  float dd2, drift_c;    // drift branch: phi += drift_c / beta
  float fbc, fbm, b0, tc[6], sc[6], inv2pifbc;  // T(beta), S(beta) as Taylor series about b0
  float beta_in, inv_beta_in, betag_ccl, gmg, inv_gmg, q, efl, efl_m, concomm, concomm1, con1, con2nex, inv_gmg2,
      inv_gmgcl, inv_fkis, fkr, sinps, cosps, X, ccl_dg;
  float sinF, cosF, prome1_r, sinP, cosP, tw_r, prome_r, K2;
  float dphi_ref, dw_ref;  // actual reference change
  float corr_phi, corr_w;  // hypothetical minus actual reference after the gap
  int ccl, amp0, ref_drift;
  __device__ uint32_t apply(Part &p) const {
    const Gap2Map &G = *this;
    float x = p.x, y = p.y, xp = p.xp, yp = p.yp;
    const float dphi = p.ph, dw = p.w;
    float beta, bg1;
    const float D = dinvb<false>(dw, G.rin, beta, bg1);
    // GetTransitTimeFactors (simulation_kernel.cu:290-308) about the reference's beta
    float bcl = beta;
    if (beta > 1.1f * G.fbc) bcl = G.fbc;
    else if (beta < G.fbm) bcl = G.fbm;
    const float u = __fadd_rn(bcl, -G.b0);
    const float dT = __fmul_rn(u, fmaf(u, fmaf(u, fmaf(u, fmaf(u, tc[5], tc[4]), tc[3]), tc[2]), tc[1]));
    const float t = __fadd_rn(tc[0], dT);
    // the derivatives: c1 + u (2 c2 + u (3 c3 + u (4 c4 + 5 u c5)))
    const float u5 = 5.0f * u;
    float dTd = fmaf(4.0f, tc[4], __fmul_rn(u5, tc[5]));
    dTd = fmaf(3.0f, tc[3], __fmul_rn(u, dTd));
    dTd = fmaf(u, fmaf(2.0f, tc[2], __fmul_rn(u, dTd)), tc[1]);
    float dSd = fmaf(u5, sc[5], __fmul_rn(4.0f, sc[4]));
    dSd = fmaf(u, dSd, __fmul_rn(3.0f, sc[3]));
    dSd = fmaf(u, fmaf(u, dSd, __fmul_rn(2.0f, sc[2])), sc[1]);
    const float coef = bcl * bcl * G.inv2pifbc;
    const float tp = __fmul_rn(coef, dTd), sp = __fmul_rn(-coef, dSd);
    if (G.amp0 || (G.ccl && beta < G.fbm)) {
      p.x = fmaf(G.dd2, xp, x);
      p.y = fmaf(G.dd2, yp, y);
      if (G.ref_drift) {
        p.ph = fmaf(G.drift_c, D, dphi);
        return WR_X | WR_Y | WR_PH;
      }
      p.ph = dphi + G.drift_c / beta - G.dphi_ref;
      p.w = dw - G.dw_ref;
      return WR_X | WR_Y | WR_PH | WR_W;
    }
    float tw, dtw;
    if (G.ccl) {
      tw = fmaf(-(F_TWOPI * tp * fmaf(G.beta_in, rcp_fast(beta), -1.0f) * G.betag_ccl), G.inv_beta_in, t);
      dtw = tw - G.tw_r;
    } else {
      tw = t;
      dtw = dT;
    }
    const float con5nex = __fmul_rn(G.concomm, fmaf(t, G.inv_fkis, -(G.X * tp * G.inv_gmg2)));
    const float con5nex1 = __fmul_rn(G.concomm1, t);
    const float con5nex2 = -G.con2nex * t * G.inv_fkis;
    const float delta = G.ccl ? fmaf(-G.ccl_dg, D, dphi) : dphi;
    float sd, cd;
    fast_sincos(delta, &sd, &cd);
    const float sinp1 = fmaf(G.sinF, cd, G.cosF * sd), cosp1 = fmaf(G.cosF, cd, -(G.sinF * sd));
    // the difference of the phase modulation from the reference's
    const float dprome1 = fmaf(-G.con1, fmaf(tp, sinp1 - G.sinps, sp * (cosp1 - G.cosps)), -G.prome1_r);
    const float eps = delta + dprome1;
    // sin and cos of eps from those of eps/2 (one evaluation instead of two;
    // 2 sin^2(eps/2) = 1 - cos(eps) is the form dcos needs anyway)
    float sh, ch;
    fast_sincos(0.5f * eps, &sh, &ch);
    const float se = __fmul_rn(2.0f * sh, ch), omc = __fmul_rn(2.0f * sh, sh), ce = __fadd_rn(1.0f, -omc);
    const float sinp = fmaf(G.sinP, ce, G.cosP * se), cosp = fmaf(G.cosP, ce, -(G.sinP * se));
    const float dcos = fmaf(-G.cosP, omc, -(G.sinP * se));
    const float rs_p = fmaf(x, x, y * y), rrp = fmaf(x, xp, y * yp);
    const float ris = sqrt_fast(rs_p), fkrris = G.fkr * ris;
    float b0m1;
    const float b0c = fbessi0c(fkrris, &b0m1);
    const float b1c = fbessi1c(fkrris);
    const float b1p = fkrris != 0.0f ? fmaf(-b1c, rcp_fast(fkrris), b0c) : 0.5f;
    const float bes1covr = ris != 0.0f ? div_fast(b1c, ris) : G.fkr * 0.5f;
    const float rest = fmaf(-(tw * G.gmg), bes1covr,
                            fmaf(fmaf(-F_TWOPI, tp, tw) * G.inv_gmg, bes1covr, tw * G.inv_gmg * G.fkr * b1p));
    const float gain = fmaf(rest * rrp, sinp,
                            fmaf(tw * b0c, dcos, fmaf(dtw, b0c, G.tw_r * b0m1) * G.cosP));
    const float dwh = fmaf(G.q * G.efl, gain, dw);
    float betah, bg;
    const float Dh = dinvb(dwh, G.rh, betah, bg);
    const float bgr = div_fast(bg1, bg);
    const float onema = fmaf(-fmaf(con5nex2, bes1covr, fmaf(con5nex1, b1p, con5nex * bes1covr)), cosp, 1.0f);
    const float dovbl = G.con2nex * bes1covr * tw * sinp;
    const float bgrovonema = div_fast(bgr, onema);
    xp = fmaf(bgrovonema, xp, -dovbl * x);
    x = fmaf(x, onema, G.dd2 * xp);
    yp = fmaf(bgrovonema, yp, -dovbl * y);
    y = fmaf(y, onema, G.dd2 * yp);
    const float rpris = rs_p > 0.0f ? div_fast(rrp, ris) : 0.0f;
    const float mod = fmaf(ris * tw * b1c, G.inv_gmgcl, -tp * b0c);
    const float prome = fmaf(2.0f * G.con1 * mod, sinp - G.sinps, -(G.efl_m * tw * b1c * rpris * (cosp - G.cosps)));
    const float dphih = fmaf(G.K2, Dh, dphi) + (prome - G.prome_r);
    const float wabs = G.rh.w + dwh;
    if (wabs <= 0.0f || x != x || y != y || xp != xp || yp != yp || dwh != dwh || dphih != dphih) {
      p.lo = 33333333u;
      return WR_LOSS;
    }
    p.x = x; p.y = y; p.xp = xp; p.yp = yp;
    p.ph = dphih + G.corr_phi;
    p.w = dwh + G.corr_w;
    return WR_X | WR_Y | WR_XP | WR_YP | WR_PH | WR_W;
  }
};

// SimulateBuncherKernel, simulation_kernel.cu:807-871
struct BunchMap {
  RefK r;
  float hr, sinB, cosB, k2q, qV, con1, beta_w, aper2;
  uint32_t eid;
  __device__ uint32_t apply(Part &p) const {
    const float x = p.x, y = p.y, dw = p.w;
    const float r2 = fmaf(x, x, y * y);
    if (aper2 != 0.0f && r2 > aper2) { p.lo = eid; return WR_LOSS; }
    const float delta = hr * p.ph;
    float sd, cd;
    sincosf(delta, &sd, &cd);
    const float cosph = fmaf(cosB, cd, -(sinB * sd)), sinph = fmaf(sinB, cd, cosB * sd);
    const float sh = sinf(0.5f * delta);
    const float dcos = fmaf(-cosB * 2.0f * sh, sh, -(sinB * sd));
    const float arg = k2q * r2;
    const float poly = __fmul_rn(arg, fmaf(arg, 0.25f + arg / 36.0f, 1.0f));
    const float dwi = qV * cosph * __fadd_rn(1.0f, poly);
    const float w = r.w + dw;
    const float wb_par = fmaf(0.5f, dwi, w), wf = __fadd_rn(w, dwi);
    if (wb_par <= 0.0f || wf <= 0.0f) { p.lo = eid; return WR_LOSS; }
    float gt = wb_par * r.minv;
    const float bav = sqrtf(gt * (gt + 2.0f)) / (gt + 1.0f);
    gt = fmaf(dw, r.minv, r.g);
    const float bg = sqrtf(gt * (gt + 2.0f));
    gt = wf * r.minv;
    const float rbgf = rsqrtf(gt * (gt + 2.0f));
    const float del = -con1 * sinph * fmaf(-bav, beta_w, 1.0f) * fmaf(arg, 0.25f + arg / 24.0f, 0.5f) / bav;
    p.xp = fmaf(p.xp, bg, del * x) * rbgf;
    p.yp = fmaf(p.yp, bg, del * y) * rbgf;
    p.w = fmaf(qV, fmaf(cosph, poly, dcos), dw);
    return WR_XP | WR_YP | WR_W;
  }
};

// SimulateRotationKernel, simulation_kernel.cu:511-529
struct RotMap {
  float cosa, sina;
  __device__ uint32_t apply(Part &p) const {
    const float x = p.x, y = p.y, xp = p.xp, yp = p.yp;
    p.x = fmaf(x, cosa, y * sina);
    p.y = fmaf(y, cosa, -(x * sina));
    p.xp = fmaf(xp, cosa, yp * sina);
    p.yp = fmaf(yp, cosa, -(xp * sina));
    return WR_X | WR_Y | WR_XP | WR_YP;
  }
};

// Simulate{First,Second}HalfDipoleKernel, simulation_kernel.cu:603-805
struct DipMap {
  float r11, r12, r16, r21, r22, r26, r33, r34, r43, r44, r51, r52, r56, e21, e43;
  float cdp, dpop_ref, cph;  // dpop_i = dpop_ref + cdp * dw; phase offset = cph * (...)
  int second;
  __device__ uint32_t apply(Part &p) const {
    float x = p.x, xp = p.xp, y = p.y, yp = p.yp;
    const float ddp = __fmul_rn(cdp, p.w);
    const float dpop = __fadd_rn(dpop_ref, ddp);
    // a u + b v, and a u + b v + c w
    auto two = [](float a, float u, float b, float v) { return fmaf(a, u, b * v); };
    auto three = [](float a, float u, float b, float v, float c, float w) { return fmaf(c, w, fmaf(a, u, b * v)); };
    if (!second) {
      xp = fmaf(e21, x, xp);
      yp = fmaf(-e43, y, yp);
      p.x = three(r11, x, r12, xp, r16, dpop);
      p.xp = three(r21, x, r22, xp, r26, dpop);
      p.y = two(r33, y, r34, yp);
      p.yp = two(r43, y, r44, yp);
      p.ph = fmaf(-cph, three(r51, x, r52, xp, r56, ddp), p.ph);
    } else {
      p.ph = fmaf(-cph, three(r51, x, r52, xp, r56, ddp), p.ph);
      p.x = three(r11, x, r12, xp, r16, dpop);
      p.y = two(r33, y, r34, yp);
      p.xp = fmaf(e21, p.x, three(r21, x, r22, xp, r26, dpop));
      p.yp = fmaf(-e43, p.y, two(r43, y, r44, yp));
    }
    return WR_X | WR_Y | WR_XP | WR_YP | WR_PH;
  }
};

}  // namespace hps
