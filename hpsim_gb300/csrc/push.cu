// push.cu -- element transfer maps on FP64 particle state.
//
// Each kernel restates one kernel of src/simulation/inc/simulation_kernel.cu;
// FP64 beams follow the reference to rounding.  The sweeps are bound by the
// FP64 pipe (a quotient or root is a dozen of its instructions, and it takes
// two a cycle and SM), so what all particles share is formed on the host,
// quotients by a particle's beta, radius or momentum share one reciprocal
// root, and increments whose terms all divide by beta are one product with
// 1 / beta.  65,536 particles: half quad 23.4 -> 13.5 us, drift 7.6 -> 4.1; 150,001:
// gap second half 149 -> 63, first half 33.6 -> 5.7.  Launches use a grid-stride loop sized from the
// particle count (not the reference's NextPow2 geometry); where the
// reference's geometry changes what is computed, the host reproduces it
// (invalid zero-thread launches are not issued).
#include <cmath>

#include "internal.h"
#include "reduce.cuh"

namespace hps {

void load_gap_args(const double *p, GapArgs *g) {
  g->length = p[HPS_P_LENGTH];
  g->frequency = p[HPS_P_RF_FREQ];
  g->clbl = p[HPS_P_RF_CLBL];
  g->amplitude = p[HPS_P_RF_AMP];
  g->phase_ref = p[HPS_P_RF_PHASE_REF];
  g->phase_shift = p[HPS_P_RF_PHASE_SHIFT];
  g->energy_out = p[HPS_P_RF_ENERGY_OUT];
  g->beta_center = p[HPS_P_RF_BETA_CENTER];
  g->dg = p[HPS_P_RF_DG];
  g->t = p[HPS_P_RF_T];
  g->tp = p[HPS_P_RF_TP];
  g->sp = p[HPS_P_RF_SP];
  g->fbc = p[HPS_P_RF_FIT_BETA_CENTER];
  g->fbm = p[HPS_P_RF_FIT_BETA_MIN];
  for (int k = 0; k < 6; ++k) g->ta[k] = p[HPS_P_RF_FIT_T0 + k];
  for (int k = 0; k < 5; ++k) g->sa[k] = p[HPS_P_RF_FIT_S1 + k];
}

namespace {

#define PARTICLES(b) for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (b).n; i += gridDim.x * blockDim.x)

// 1 / beta of kinetic energy w
__device__ __forceinline__ double inv_beta(double w, double inv_mass) {
  const double g = w * inv_mass;
  return (g + 1.0) * rsqrt(g * (g + 2.0));
}

// SimulatePartialDriftKernel, simulation_kernel.cu:86-118; cph = 2 pi hf / lambda
__global__ void k_partial_drift(DevBeam b, double hf, double aper, double cph, double inv_mass, uint32_t eid) {
  PARTICLES(b) {
    if (b.loss[i] != 0u) continue;
    double aper2 = aper * aper;
    double x = b.x[i], y = b.y[i];
    x += b.xp[i] * hf;
    y += b.yp[i] * hf;
    if (aper2 != 0.0 && x * x + y * y > aper2) b.loss[i] = eid;
    else {
      b.x[i] = x;
      b.y[i] = y;
      b.phi[i] += cph * inv_beta(b.w[i], inv_mass);
    }
  }
}

// SimulateSteererKernel, simulation_kernel.cu:120-140
__global__ void k_steerer(DevBeam b, double blh, double blv) {
  PARTICLES(b) {
    if (b.loss[i] != 0u) continue;
    double gm1 = b.w[i] / b.mass;
    double btgm = sqrt(gm1 * (gm1 + 2.0));
    double p = btgm * b.mass / CLIGHT;
    if (blh > 1e-10) b.xp[i] += blh * b.charge / p;
    if (blv > 1e-10) b.yp[i] += blv * b.charge / p;
  }
}

// sin, cos, sinh and cosh of x by their Taylor series about zero, |x| < 0.75:
// the first terms left out are below x^19 / 19! = 4e-20 and x^18 / 18! = 9e-19
__device__ __forceinline__ void trig_small(double x, double *s, double *c, double *sh, double *ch) {
  const double z = x * x;
  const double o3 = 1.0 / 6.0, o5 = 1.0 / 120.0, o7 = 1.0 / 5040.0, o9 = 1.0 / 362880.0, o11 = 1.0 / 39916800.0,
               o13 = 1.0 / 6227020800.0, o15 = 1.0 / 1307674368000.0, o17 = 1.0 / 355687428096000.0;
  const double e4 = 1.0 / 24.0, e6 = 1.0 / 720.0, e8 = 1.0 / 40320.0, e10 = 1.0 / 3628800.0, e12 = 1.0 / 479001600.0,
               e14 = 1.0 / 87178291200.0, e16 = 1.0 / 20922789888000.0;
  // even and odd terms of sinh(x) / x - 1 and cosh(x) - 1 in z^2: their sums
  // are the hyperbolic functions, their differences the circular ones
  const double v = z * z;
  const double sa = fma(v, fma(v, fma(v, o15, o11), o7), o3) * z, sb = v * fma(v, fma(v, fma(v, o17, o13), o9), o5);
  const double ca = fma(v, fma(v, fma(v, e14, e10), e6), 0.5) * z, cb = v * fma(v, fma(v, fma(v, e16, e12), e8), e4);
  *sh = fma(x, sb + sa, x);
  *s = fma(x, sb - sa, x);
  *ch = 1.0 + (cb + ca);
  *c = 1.0 + (cb - ca);
}

// SimulateHalfQuadKernel, simulation_kernel.cu:142-218; sk0 = sqrt(|qG| c / m),
// cph = pi len / lambda
__global__ void k_half_quad(DevBeam b, double len, double aper, double qg, double sk0, double isk0, double cph,
                            double inv_mass, uint32_t eid) {
  double aper2 = aper * aper;
  PARTICLES(b) {
    if (b.loss[i] != 0u) continue;
    double x = b.x[i], y = b.y[i], xp = b.xp[i], yp = b.yp[i];
    const double g = b.w[i] * inv_mass, g2 = g * (g + 2.0);
    if (qg == 0) {
      b.x[i] = x + xp * len * 0.5;
      b.y[i] = y + yp * len * 0.5;
    } else {
      const double bg = sqrt(g2 * (1.0 + xp * xp + yp * yp)), rb = rsqrt(bg);
      const double k = sk0 * rb, inv_k = isk0 * (bg * rb), kds = len * 0.25 * k;
      double s, c, sh, ch;
      if (fabs(kds) < 0.75) trig_small(kds, &s, &c, &sh, &ch);
      else {
        sincos(kds, &s, &c);
        sh = sinh(kds);
        ch = cosh(kds);
      }
      double xx, yy, sovk = s * inv_k, shovk = sh * inv_k, sk = s * k, shk = sh * k;
#pragma unroll
      for (int rep = 0; rep < 2; ++rep) {
        if (qg > 0.0) {
          xx = c * x + sovk * xp; xp = -sk * x + c * xp; x = xx;
          yy = ch * y + shovk * yp; yp = shk * y + ch * yp; y = yy;
        } else {
          xx = ch * x + shovk * xp; xp = shk * x + ch * xp; x = xx;
          yy = c * y + sovk * yp; yp = -sk * y + c * yp; y = yy;
        }
      }
      b.x[i] = x; b.y[i] = y; b.xp[i] = xp; b.yp[i] = yp;
    }
    if (aper2 != 0 && x * x + y * y > aper2) b.loss[i] = eid;
    else b.phi[i] += cph * ((g + 1.0) * rsqrt(g2));
  }
}

// SimulateRFGapFirstHalfKernel, simulation_kernel.cu:226-288: every branch
// advances the phase by k0 + k1 / beta (push_gap_first)
__global__ void k_gap_first(DevBeam b, double dd1, double k0, double k1, double inv_mass) {
  PARTICLES(b) {
    if (b.loss[i] != 0u) continue;
    const double x = b.x[i], y = b.y[i], xp = b.xp[i], yp = b.yp[i], phi = b.phi[i], w = b.w[i];
    b.x[i] = x + dd1 * xp;
    b.y[i] = y + dd1 * yp;
    b.phi[i] = phi + fma(k1, inv_beta(w, inv_mass), k0);
  }
}

// Bessi0c / Bessi1c, simulation_kernel.cu:15-73
__device__ inline double bessi0c(double r_x) {
  double ans, cy, ax = fabs(r_x);
  if (ax < 3.75) {
    cy = r_x * (1.0 / 3.75);
    cy = cy * cy;
    ans = 1.0 + cy * (3.5156229 + cy * (3.0899424 + cy * (1.2067492 + cy * (0.2659732 +
          cy * (0.360768e-1 + cy * 0.45813e-2)))));
  } else {
    cy = 3.75 / ax;
    ans = (exp(ax) * rsqrt(ax)) * (0.39894228 + cy * (0.1328592e-1 + cy * (0.225319e-2 +
          cy * (-0.157565e-2 + cy * (0.916281e-2 + cy * (-0.2057706e-1 + cy * (0.2635537e-1 +
          cy * (-0.1647633e-1 + cy * 0.392377e-2))))))));
  }
  return ans;
}
__device__ inline double bessi1c(double r_x) {
  double cy, ans, ax = fabs(r_x);
  if (ax < 3.75) {
    cy = r_x * (1.0 / 3.75);
    cy = cy * cy;
    ans = ax * (0.5 + cy * (0.87890594 + cy * (0.51498869 + cy * (0.15084934 + cy * (0.2658733e-1 +
          cy * (0.301532e-2 + cy * 0.32411e-3))))));
  } else {
    cy = 3.75 / ax;
    ans = 0.2282967e-1 + cy * (-0.2895312e-1 + cy * (0.1787654e-1 - cy * 0.420059e-2));
    ans = 0.39894228 + cy * (-0.3988024e-1 + cy * (-0.362018e-2 + cy * (0.163801e-2 + cy *
          (-0.1031555e-1 + cy * ans))));
    ans = ans * (exp(ax) * rsqrt(ax));
  }
  return r_x < 0.0 ? -ans : ans;
}

// what all particles share of a gap's second half
struct Gap2C {
  double dd2, inv_mass, drift_c;                 // drift_c = 2 pi dd2 / lambda
  double fbc, fbm, ttf_c, ta[6], sa[5];          // ttf_c = 1 / (2 pi fbc)
  double beta_in, tw_c;                          // tw_c: CCL 2 pi betag / beta_in
  double gmg, inv_gmg, fkr, inv_fkr, inv_fkis, inv_gmgcl, x_tp;
  double qefl, efl_m, concomm, concomm1, con1, con2nex, sinps, cosps, shift, dg_c;
  double k0, k2;                                 // phase: k0 + k2 / beta after the kick
  int ccl, amp0;
};

Gap2C gap2_consts(const DevBeam &b, const GapArgs &g) {
  Gap2C c{};
  const double mass = b.mass, inv_mass = 1.0 / mass;
  const double cell_len = g.length + g.q1 * 0.5 + g.q2 * 0.5;
  c.dd2 = 0.5 * cell_len + g.dg - g.q2 * 0.5;
  c.inv_mass = inv_mass;
  c.drift_c = TWOPI * c.dd2 / g.wl;
  c.fbc = g.fbc;
  c.fbm = g.fbm;
  c.ttf_c = 1.0 / (TWOPI * g.fbc);
  for (int k = 0; k < 6; ++k) c.ta[k] = g.ta[k];
  for (int k = 0; k < 5; ++k) c.sa[k] = g.sa[k];
  c.ccl = g.ccl;
  c.amp0 = g.amplitude == 0.0;
  if (c.amp0) return c;
  const double gm_in = g.design_w_in * inv_mass + 1.0;
  c.beta_in = sqrt(1.0 - 1.0 / (gm_in * gm_in));
  const double wave_len = CLIGHT / g.frequency, cl = cell_len / g.clbl, betag_ccl = cl / wave_len;
  const double betag = g.ccl ? g.beta_center : betag_ccl, betag2 = betag * betag;
  c.gmg = 1.0 / sqrt(1.0 - betag2);
  c.inv_gmg = 1.0 / c.gmg;
  const double inv_gmg2 = 1.0 / (c.gmg * c.gmg);
  const double q = fabs(b.charge);
  const double gm_out = g.energy_out * inv_mass + 1.0, beta_out = sqrt(1.0 - 1.0 / (gm_out * gm_out));
  const double efl = g.amplitude * cell_len;
  c.qefl = q * efl;
  c.efl_m = efl * inv_mass;
  c.concomm = q * efl / (mass * betag2);
  c.concomm1 = c.concomm * inv_gmg2 / c.gmg;
  c.con1 = PI * c.concomm1;
  c.con2nex = c.concomm * inv_gmg2;
  if (g.ccl) {
    c.inv_gmgcl = 1.0 / (c.gmg * betag * wave_len);
    c.inv_fkis = betag * wave_len / TWOPI;
    c.x_tp = betag_ccl * wave_len * inv_gmg2;
    c.tw_c = TWOPI * betag_ccl / c.beta_in;
    c.shift = g.phase_shift + g.ccl_cell_num * PI;
    c.dg_c = TWOPI * g.dg / wave_len;
    const double A = PI * g.clbl + (g.phi_in - g.phase_ref);
    c.k0 = A * (1.0 - betag_ccl / beta_out);
    c.k2 = A * betag_ccl;
  } else {
    c.inv_gmgcl = 1.0 / (c.gmg * cl);
    c.inv_fkis = cl / TWOPI;
    c.x_tp = c.beta_in * wave_len * inv_gmg2;
    c.shift = g.phase_shift;
    const double d_cell_len = cell_len - g.beta_center * wave_len;
    const bool dc = d_cell_len > 1e-15 || d_cell_len < -1e-15;
    c.k2 = beta_out * (PI * g.clbl + (g.phase_ref - g.phi_in)) + (dc ? PI * d_cell_len / wave_len : 0.0) -
           PI * g.q2 / wave_len;
  }
  c.fkr = TWOPI * c.inv_gmgcl;
  c.inv_fkr = 1.0 / c.fkr;
  c.sinps = sin(g.phase_ref);
  c.cosps = cos(g.phase_ref);
  return c;
}

// SimulateRFGapSecondHalfKernel, simulation_kernel.cu:310-497
__global__ void k_gap_second(DevBeam b, const __grid_constant__ Gap2C G) {
  PARTICLES(b) {
    if (b.loss[i] != 0u) continue;
    double x = b.x[i], y = b.y[i], xp = b.xp[i], yp = b.yp[i];
    const double phi = b.phi[i];
    double w = b.w[i];
    const double gam = w * G.inv_mass, s1 = gam * (gam + 2.0), r1 = rsqrt(s1), bg1 = s1 * r1;
    const double ib1 = (gam + 1.0) * r1, beta = 1.0 / ib1;
    if (G.amp0 || (G.ccl && beta < G.fbm)) {
      b.x[i] = x + G.dd2 * xp;
      b.y[i] = y + G.dd2 * yp;
      b.phi[i] = phi + G.drift_c * ib1;
      continue;
    }
    // GetTransitTimeFactors, simulation_kernel.cu:290-308
    double bt = beta;
    if (beta > 1.1 * G.fbc) bt = G.fbc;
    else if (beta < G.fbm) bt = G.fbm;
    const double *ta = G.ta, *sa = G.sa;
    const double t = ta[0] + bt * (ta[1] + bt * (ta[2] + bt * (ta[3] + bt * (ta[4] + bt * ta[5]))));
    const double coef = bt * bt * G.ttf_c;
    const double tp = coef * (ta[1] + bt * (2 * ta[2] + bt * (3 * ta[3] + bt * (4 * ta[4] + 5 * bt * ta[5]))));
    const double sp = -coef * (sa[0] + bt * (2 * sa[1] + bt * (3 * sa[2] + bt * (4 * sa[3] + 5 * bt * sa[4]))));
    const double con5nex = G.concomm * (t * G.inv_fkis - G.x_tp * tp);
    const double tw = G.ccl ? t - tp * (G.beta_in * ib1 - 1.0) * G.tw_c : t;
    const double con5nex1 = G.concomm1 * t, con5nex2 = -G.con2nex * t * G.inv_fkis;
    double phi1 = phi + G.shift, sinp1, cosp1;
    if (G.ccl) phi1 -= G.dg_c * ib1;
    sincos(phi1, &sinp1, &cosp1);
    const double prome1 = -G.con1 * (tp * (sinp1 - G.sinps) + sp * (cosp1 - G.cosps));
    sincos(phi1 + prome1, &sinp1, &cosp1);
    const double rs_p = x * x + y * y, rrp = x * xp + y * yp;
    const bool off = rs_p > 0.0;
    const double ir = off ? rsqrt(rs_p) : 0.0, ris = rs_p * ir, fkrris = G.fkr * ris;
    const double b0c = bessi0c(fkrris), b1c = bessi1c(fkrris);
    const double bes1covr = off ? b1c * ir : G.fkr * 0.5;
    const double b1p = off ? b0c - bes1covr * G.inv_fkr : 0.5;
    const double delte = G.qefl * (tw * b0c * cosp1 + ((tw - TWOPI * tp) * G.inv_gmg * bes1covr +
                         tw * G.inv_gmg * G.fkr * b1p - tw * G.gmg * bes1covr) * rrp * sinp1);
    w += delte;
    const double gf = w * G.inv_mass, r2 = rsqrt(gf * (gf + 2.0));
    const double onema = 1.0 - (con5nex * bes1covr + con5nex1 * b1p + con5nex2 * bes1covr) * cosp1;
    const double dovbl = G.con2nex * bes1covr * tw * sinp1;
    const double bgrovonema = bg1 * r2 / onema;
    xp = -dovbl * x + bgrovonema * xp;
    x = x * onema + G.dd2 * xp;
    yp = -dovbl * y + bgrovonema * yp;
    y = y * onema + G.dd2 * yp;
    const double prome = 2.0 * G.con1 * (-tp * b0c + ris * tw * b1c * G.inv_gmgcl) * (sinp1 - G.sinps) -
                         G.efl_m * tw * b1c * (rrp * ir) * (cosp1 - G.cosps);
    const double phi_new = phi + (fma(G.k2, (gf + 1.0) * r2, G.k0) + prome);
    if (w <= 0.0 || x != x || y != y || xp != xp || yp != yp || w != w || phi_new != phi_new) {
      b.loss[i] = 33333333u;
    } else {
      b.x[i] = x; b.y[i] = y; b.xp[i] = xp; b.yp[i] = yp; b.w[i] = w; b.phi[i] = phi_new;
    }
  }
}

// SimulateBuncherKernel, simulation_kernel.cu:807-871
__global__ void k_buncher(DevBeam b, double wl, double w_ref, double freq, double voltage, double phase,
                          double aper, double freq_ratio, uint32_t eid) {
  const double mass = b.mass;
  PARTICLES(b) {
    if (b.loss[i] != 0u) continue;
    double x = b.x[i], y = b.y[i], xp = b.xp[i], yp = b.yp[i];
    double phi = b.phi[i] * freq_ratio;
    double w = b.w[i];
    double r2 = x * x + y * y;
    double aper2 = aper * aper;
    if (aper2 != 0.0 && r2 > aper2) { b.loss[i] = eid; continue; }
    double h = freq * wl / CLIGHT;
    double gm1 = w_ref / mass;
    double gm = gm1 + 1.0;
    double btgm = sqrt(gm1 * (gm1 + 2.0));
    double beta = btgm / gm;
    double k = h * TWOPI / (btgm * wl);
    double k2 = k * k;
    double q = b.charge;
    q = q > 0.0 ? q : -q;
    double con1 = TWOPI * h * voltage * q / (beta * wl * mass);
    double arg = k2 * r2 * 0.25;
    double ph = h * phi + phase;
    double dw = q * voltage * cos(ph) * (1.0 + arg * (1.0 + arg * (0.25 + arg / 36.0)));
    double wb_par = w + 0.5 * dw;
    double wf = w + dw;
    if (wb_par <= 0.0 || wf <= 0.0) { b.loss[i] = eid; continue; }
    double gmtmp = wb_par / mass;
    double bav = sqrt(gmtmp * (gmtmp + 2.0)) / (gmtmp + 1.0);
    gmtmp = w / mass;
    double bg = sqrt(gmtmp * (gmtmp + 2.0));
    gmtmp = wf / mass;
    double rbgf = rsqrt(gmtmp * (gmtmp + 2.0));
    double del = -con1 * sin(ph) * (1.0 - bav * beta) * (0.5 + arg * (0.25 + arg / 24.0)) / bav;
    b.xp[i] = (xp * bg + del * x) * rbgf;
    b.yp[i] = (yp * bg + del * y) * rbgf;
    b.w[i] = wf;
  }
}

// SimulateRotationKernel, simulation_kernel.cu:511-529
__global__ void k_rotation(DevBeam b, double cosa, double sina) {
  PARTICLES(b) {
    if (b.loss[i] != 0u) continue;
    double x = b.x[i], y = b.y[i], xp = b.xp[i], yp = b.yp[i];
    b.x[i] = x * cosa + y * sina;
    b.y[i] = y * cosa - x * sina;
    b.xp[i] = xp * cosa + yp * sina;
    b.yp[i] = yp * cosa - xp * sina;
  }
}

// Simulate{Circular,Rectangular}ApertureKernel, simulation_kernel.cu:543-575;
// the centroid is the x_avg / y_avg left by UpdateAvgXY (index 0 skipped)
__global__ void k_aperture(DevBeam b, int rect, double aper, double xl, double xr, double yt, double yb,
                           uint32_t eid) {
  double cx = b.st->st[X_AVG], cy = b.st->st[Y_AVG];
  PARTICLES(b) {
    if (i == 0 || b.loss[i] != 0u) continue;
    if (!rect) {
      double aper2 = aper * aper;
      double x = b.x[i] - cx, y = b.y[i] - cy;
      if (x * x + y * y > aper2) b.loss[i] = eid;
    } else {
      double xmin = cx - xl, xmax = cx + xr, ymin = cy - yb, ymax = cy + yt;
      double x = b.x[i], y = b.y[i];
      if (x < xmin || x > xmax || y < ymin || y > ymax) b.loss[i] = eid;
    }
  }
}

// Simulate{First,Second}HalfDipoleKernel, simulation_kernel.cu:603-805
struct DipoleMap {
  double r11, r12, r16, r21, r22, r26, r33, r34, r43, r44, r51, r52, r56, beta, dl, design_w, gamma,
      e21, e43;
};

__global__ void k_dipole(DevBeam b, DipoleMap d, double wl, int second) {
  PARTICLES(b) {
    if (b.loss[i] != 0u) continue;
    double x = b.x[i], xp = b.xp[i], y = b.y[i], yp = b.yp[i];
    double dpop = d.gamma / (d.design_w * (d.gamma + 1.0)) * (b.w[i] - d.design_w);
    if (!second) {
      xp += d.e21 * x;
      yp -= d.e43 * y;
      b.x[i] = d.r11 * x + d.r12 * xp + d.r16 * dpop;
      b.xp[i] = d.r21 * x + d.r22 * xp + d.r26 * dpop;
      b.y[i] = d.r33 * y + d.r34 * yp;
      b.yp[i] = d.r43 * y + d.r44 * yp;
      b.phi[i] += TWOPI * (-(d.r51 * x + d.r52 * xp + d.r56 * dpop) + d.dl) / (d.beta * wl);
    } else {
      b.phi[i] += TWOPI * (-(d.r51 * x + d.r52 * xp + d.r56 * dpop) + d.dl) / (d.beta * wl);
      double x_new = d.r11 * x + d.r12 * xp + d.r16 * dpop;
      xp = d.r21 * x + d.r22 * xp + d.r26 * dpop;
      double y_new = d.r33 * y + d.r34 * yp;
      yp = d.r43 * y + d.r44 * yp;
      b.x[i] = x_new;
      b.y[i] = y_new;
      b.xp[i] = xp + d.e21 * x_new;
      b.yp[i] = yp - d.e43 * y_new;
    }
  }
}

// The particle-independent part of the dipole kernels, evaluated once on the
// host with the same operations (simulation_kernel.cu:620-693, 722-783).
DipoleMap dipole_map(const double *p, double mass, int second) {
  DipoleMap m;
  double h = 1.0 / p[HPS_P_DIP_RADIUS];
  double findx = p[HPS_P_DIP_FIELD_INDEX];
  m.design_w = p[HPS_P_DIP_KINETIC_ENERGY];
  double h2 = h * h;
  m.dl = 0.5 * p[HPS_P_DIP_RADIUS] * p[HPS_P_DIP_ANGLE];
  double yk2 = findx * h2;
  double yk = sqrt(fabs(yk2));
  double inv_yk = 1.0 / yk;
  double ykl = yk * m.dl;
  double xk2 = h2 - yk2;
  double inv_xk2 = 1.0 / xk2;
  double xk = sqrt(fabs(xk2));
  double inv_xk = 1.0 / xk;
  double xkl = xk * m.dl;
  double cxkl = 1.0, sxokx = m.dl;
  if (xk2 > 0.0) { cxkl = cos(xkl); sxokx = sin(xkl) * inv_xk; }
  else if (xk2 < 0.0) { cxkl = cosh(xkl); sxokx = sinh(xkl) * inv_xk; }
  double cykl = 1.0, syoky = m.dl;
  if (yk2 > 0.0) { cykl = cos(ykl); syoky = sin(ykl) * inv_yk; }
  else if (yk2 < 0.0) { cykl = cosh(ykl); syoky = sinh(ykl) * inv_yk; }
  m.r11 = cxkl; m.r12 = sxokx; m.r21 = -xk2 * sxokx; m.r22 = cxkl;
  m.r33 = cykl; m.r34 = syoky; m.r43 = -yk2 * syoky; m.r44 = cykl;
  m.r26 = h * sxokx;
  m.r16 = h * (1.0 - cxkl) * inv_xk2;
  m.r51 = -m.r26;
  m.r52 = -m.r16;
  m.gamma = m.design_w / mass + 1.0;
  double beta2 = 1.0 - 1.0 / (m.gamma * m.gamma);
  m.beta = sqrt(beta2);
  m.r56 = -h2 * (m.dl * beta2 - sxokx) * inv_xk2 + m.dl * (1.0 - h2 * inv_xk2) / (m.gamma * m.gamma);
  double bedge = second ? p[HPS_P_DIP_EDGE_OUT] : p[HPS_P_DIP_EDGE_IN];
  double c1 = 2.0 * p[HPS_P_DIP_HALF_GAP] * p[HPS_P_DIP_K1] * h;
  double sinb = sin(bedge), inv_cosb = 1.0 / cos(bedge);
  double psi = c1 * (1.0 + sinb * sinb) * inv_cosb * (1.0 - c1 * p[HPS_P_DIP_K2] * sinb * inv_cosb);
  m.e21 = tan(bedge) * h;
  m.e43 = tan(bedge - psi) * h;
  return m;
}

}  // namespace

void push_partial_drift(const DevBeam &b, double wl, double hf, double aper, uint32_t eid, cudaStream_t st) {
  k_partial_drift<<<grid_for(b.n), kBlock, 0, st>>>(b, hf, aper, TWOPI * hf / wl, 1.0 / b.mass, eid);
  note_launch();
}
void push_half_quad(const DevBeam &b, double wl, double len, double aper, double grad, uint32_t eid,
                    cudaStream_t st) {
  const double qg = grad * b.charge, sk0 = sqrt(fabs(qg) * CLIGHT / b.mass);
  k_half_quad<<<grid_for(b.n), kBlock, 0, st>>>(b, len, aper, qg, sk0, 1.0 / sk0, TWOPI * len * 0.5 / wl, 1.0 / b.mass,
                                                eid);
  note_launch();
}
void push_steerer(const DevBeam &b, double blh, double blv, cudaStream_t st) {
  k_steerer<<<grid_for(b.n), kBlock, 0, st>>>(b, blh, blv); note_launch();
}
void push_gap_first(const DevBeam &b, const GapArgs &g, cudaStream_t st) {
  const double wave_len = CLIGHT / g.frequency, cell_len = g.length + g.q1 * 0.5 + g.q2 * 0.5;
  const double dd1 = 0.5 * cell_len - g.dg - 0.5 * g.q1;
  double k0 = 0.0, k1;
  if (g.amplitude == 0.0) {
    k1 = TWOPI * dd1 / wave_len;
  } else {
    // phi += (1 - (beta - beta_in) / beta) A + ... (DTL),
    //        (1 - (beta - beta_in) betag / (beta beta_in)) A (CCL)
    const double gam = g.design_w_in / b.mass, beta_in = sqrt((gam + 2.0) * gam) / (gam + 1.0);
    const double A = PI * g.clbl + (g.phase_ref - g.phi_in);
    if (!g.ccl) {
      const double d_cell_len = cell_len - g.beta_center * wave_len;
      const bool dc = d_cell_len > 1e-15 || d_cell_len < -1e-15;
      k1 = beta_in * A + (dc ? PI * d_cell_len / wave_len : 0.0) - PI * g.q1 / wave_len;
    } else {
      const double betag = cell_len / (g.clbl * wave_len);
      k0 = A * (1.0 - betag / beta_in);
      k1 = A * betag;
    }
  }
  k_gap_first<<<grid_for(b.n), kBlock, 0, st>>>(b, dd1, k0, k1, 1.0 / b.mass);
  note_launch();
}
void push_gap_second(const DevBeam &b, const GapArgs &g, cudaStream_t st) {
  k_gap_second<<<grid_for(b.n), kBlock, 0, st>>>(b, gap2_consts(b, g));
  note_launch();
}
void push_buncher(const DevBeam &b, double wl, double w_ref, double freq, double voltage, double phase,
                  double aper, double freq_ratio, uint32_t eid, cudaStream_t st) {
  k_buncher<<<grid_for(b.n), kBlock, 0, st>>>(b, wl, w_ref, freq, voltage, phase, aper, freq_ratio, eid);
  note_launch();
}
void push_rotation(const DevBeam &b, double angle, cudaStream_t st) {
  k_rotation<<<grid_for(b.n), kBlock, 0, st>>>(b, cos(angle), sin(angle)); note_launch();
}
void push_aperture(const DevBeam &b, int rect, const double *p, uint32_t eid, cudaStream_t st) {
  k_aperture<<<grid_for(b.n), kBlock, 0, st>>>(b, rect, p[HPS_P_APERTURE], p[HPS_P_APT_XL], p[HPS_P_APT_XR],
                                                p[HPS_P_APT_YT], p[HPS_P_APT_YB], eid);
  note_launch();
}
void push_dipole(const DevBeam &b, const double *p, double wl, int second, cudaStream_t st) {
  k_dipole<<<grid_for(b.n), kBlock, 0, st>>>(b, dipole_map(p, b.mass, second), wl, second); note_launch();
}

}  // namespace hps
