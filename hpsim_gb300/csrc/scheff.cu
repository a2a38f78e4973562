// scheff.cu -- the SCHEFF 2D r-z space-charge kick on FP64 particle state.
//
// Reference: Scheff::Start (src/simulation/src/space_charge.cpp:82-139), the
// launcher glue of src/simulation/src/space_charge.cu and the kernels of
// src/simulation/inc/space_charge_kernel.cu.  The reference reads five
// moments back to the host per kick and decides there whether to rebuild the
// mesh; here the statistics, the decision and the mesh sizing all stay on
// the device, so a whole lattice pass is a fixed launch sequence that can be
// captured in a CUDA graph.  Launch sequence per kick:
//   3 statistics sweeps (the last one also decides) -> [max-r sweep when
//   adjacent bunches are on] -> Green's table -> deposit -> contraction ->
//   kick, where the mesh kernels return at once unless the decision was
//   "remesh".
#include <mutex>

#include "../../include/hpsim_gb300.h"
#include "internal.h"
#include "contract.cuh"
#include "contract64.cuh"
#include "reduce.cuh"
#include "scheff_common.cuh"

namespace hps {

namespace {

__device__ inline bool good(const DevBeam &b, uint32_t i) { return (uint32_t)(b.loss[i] + b.lloss[i]) == 0u; }
__device__ inline double surv(const DevBeam &b) { return (double)(uint32_t)(b.n - b.st->num_loss); }


// Beam::UpdateLongitudinalLoss first half: UpdateGoodParticleCount,
// UpdateAvgPhi(true)  (beam.cpp:776-782, 788-791, 846-852)
struct OpGoodPhi {
  static constexpr int K = 2;
  using Comb = SumComb;
  DevBeam b;
  __device__ bool enabled() const { return true; }
  __device__ void particle(uint32_t i, double (&a)[K]) const {
    if (!good(b, i)) return;
    a[0] += 1.0;
    a[1] += b.phi[i];
  }
  __device__ void finalize(const double *t, int tid, int) const {
    if (tid) return;
    uint32_t ng = (uint32_t)t[0];
    b.st->num_good = ng;
    b.st->st[PHI_AVG_GOOD] = ng > 0 ? t[1] / ng : -99999;
  }
};

// UpdateLongitudinalLossCoordinateKernel + UpdateLossCountKernelCall(lloss)
// + UpdateGoodParticleCount + UpdateAvgPhi(true)  (beam.cpp:780-781, 1008-1009)
struct OpLlossGoodPhi {
  static constexpr int K = 3;
  using Comb = SumComb;
  DevBeam b;
  __device__ bool enabled() const { return true; }
  __device__ void particle(uint32_t i, double (&a)[K]) const {
    double lim = b.st->st[PHI_AVG_GOOD];
    uint32_t ll = b.lloss[i];
    if (b.phi[i] > lim + TWOPI + PI) {
      ll = 1u;
      b.lloss[i] = 1u;
    }
    a[0] += ll != 0u;
    if ((uint32_t)(b.loss[i] + ll) == 0u) {
      a[1] += 1.0;
      a[2] += b.phi[i];
    }
  }
  __device__ void finalize(const double *t, int tid, int) const {
    if (tid) return;
    uint32_t ng = (uint32_t)t[1];
    b.st->num_lloss = (uint32_t)t[0];
    b.st->num_good = ng;
    b.st->st[PHI_AVG_GOOD] = ng > 0 ? t[2] / ng : -99999;
  }
};

// The rest of UpdateStatForSpaceCharge (beam.cpp:1010-1014): relative phase
// about <phi>_good for every particle, <phi_r> over loss == 0 divided by
// num - num_loss, sigma(phi_r) over good particles, <x>, sigma_x, <y>,
// sigma_y over good particles divided by num - num_loss
// (UpdateHorizontalAvgSigKernel), <w> over good particles; then, when a
// solver is attached, the Scheff::Start decision.
struct OpScStats {
  static constexpr int K = 8;
  using Comb = SumComb;
  DevBeam b;
  ScState *sc;
  ScTables t;
  double freq, frac;
  __device__ bool enabled() const { return true; }
  __device__ void particle(uint32_t i, double (&a)[K]) const {
    double pr = rel_phase(b.phi[i], b.st->st[PHI_AVG_GOOD]);
    b.phi_r[i] = pr;
    if (b.loss[i] != 0u) return;
    a[0] += pr;
    if (b.lloss[i] != 0u) return;
    double x = b.x[i], y = b.y[i];
    a[1] += pr; a[2] += pr * pr;
    a[3] += x; a[4] += x * x; a[5] += y; a[6] += y * y;
    a[7] += b.w[i];
  }
  __device__ void finalize(const double *s, int tid, int nth) const {
    // independent quotients and roots on a thread each (a dependent FP64
    // quotient costs about a third of a microsecond)
    __shared__ double q[8], sig[3];
    __shared__ ScheffKin kin;
    if (tid < 8) {
      const double sv = surv(b), ng = b.st->num_good;
      q[tid] = s[tid] / (tid == 1 || tid == 2 || tid == 7 ? ng : sv);
    }
    __syncthreads();
    if (tid < 3) {  // sigma of phi, x, y
      const double a = q[1 + 2 * tid];
      sig[tid] = sqrt(q[2 + 2 * tid] - a * a);
    } else if (tid == 32) {
      q[7] = b.st->num_good > 0 ? q[7] : -99999;
      const ScheffKin k = scheff_kin(q[7], b.mass);
      kin.gamma = k.gamma;
      kin.beta = k.beta;
    } else if (tid == 64) {
      kin.lmbd = 299.792458 / freq;
    }
    __syncthreads();
    if (tid == 0) {
      BeamStats &st = *b.st;
      st.st[PHI_AVG_R] = q[0];
      st.st[PHI_SIG_GOOD] = sig[0];
      st.st[X_AVG_GOOD] = q[3];
      st.st[X_SIG_GOOD] = sig[1];
      st.st[Y_AVG_GOOD] = q[5];
      st.st[Y_SIG_GOOD] = sig[2];
      st.st[W_AVG_GOOD] = q[7];
      if (sc) scheff_decide(b, sc, freq, frac, kin);
    }
    if (!sc) return;
    __syncthreads();
    zero_mesh_tables(sc, t, tid, nth);
  }
};

// UpdateMaxRPhi + UpdateScheffMeshSizeKernel(r_max, coef = 1) when adjacent
// bunches are on (space_charge.cu:124-128)
struct OpAdjMesh {
  static constexpr int K = 2;
  using Comb = MaxComb;
  DevBeam b;
  ScState *sc;
  __device__ bool enabled() const { return sc->remesh && sc->adj != 0u; }
  __device__ void particle(uint32_t i, double (&a)[K]) const {
    if (b.loss[i] != 0u) return;
    double tx = b.x[i] - b.st->st[X_AVG], ty = b.y[i] - b.st->st[Y_AVG];
    double r2 = tx * tx + ty * ty;
    double tp = b.phi_r[i] - b.st->st[PHI_AVG_R];
    tp = tp > 0.0 ? tp : -tp;
    a[0] = a[0] < r2 ? r2 : a[0];
    a[1] = a[1] < tp ? tp : a[1];
  }
  __device__ void finalize(const double *t, int tid, int) const {
    if (tid) return;
    b.st->st[R_MAX] = sqrt(t[0]);
    b.st->st[ABS_PHI_MAX] = t[1];
    mesh_size(sc, b.st->st[R_MAX], 0.0, 1.0);
  }
};

// Scheff::Start with num_particle <= 2: statistics are not refreshed, the
// decision still runs on whatever they hold.
__global__ void k_decide_only(DevBeam b, ScState *sc, ScTables t, double freq, double frac) {
  if (threadIdx.x == 0) {
    ScheffKin kin = scheff_kin(b.st->st[W_AVG_GOOD], b.mass);
    kin.lmbd = 299.792458 / freq;
    scheff_decide(b, sc, freq, frac, kin);
  }
  __syncthreads();
  zero_mesh_tables(sc, t, threadIdx.x, blockDim.x);
}

// UpdateFldTbl1Kernel, space_charge_kernel.cu:39-100 (rows rs >= (nr/by)*by
// are not written, as in the reference's grid); not needed when a field
// surrogate's field was accepted.  Bound by the FP64 pipe: an entry costs one
// quotient, one reciprocal root and one logarithm; the source radii's root and
// 1 / (2 rp) are taken once a block.  1 - m with m = 4 rs rp / (b + d^2) is
// formed as (c + d^2) / (b + d^2) where it is small, which does not cancel.
// A block of 16 warps an SM takes consecutive entries, so that no SM waits
// for another's last round (two blocks of 8 warps with a grid stride left
// 13% of the rounds empty at 32 x 128).  32 x 128: 38.5 -> 26.5 us, with one adjacent
// bunch 88 -> 57.5.
struct Green64 {
  double er, ez;
};
__device__ __forceinline__ void green64_add(Green64 &s, double rs2mrp2, double b, double c, double rsrp4, double hrp,
                                            double d) {
  const double d2 = d * d, cd = c + d2;
  const double r = rsqrt(b + d2), r2 = r * r, m = rsrp4 * r2;
  const double g = m < 0.5 ? 1.0 - m : cd * r2;
  const double h = log(g);
  const double ee = 1.0 + g * (0.4630106 - 0.2452740 * h + g * (0.1077857 - 0.04125321 * h));
  const double ek = 1.38629436 - 0.5 * h + g * (0.1119697 - 0.1213486 * h + g * (0.07253230 - 0.02887472 * h));
  const double q = ee / cd;
  s.er += (ek - (rs2mrp2 + d2) * q) * r * hrp;
  s.ez += d * q * r;
}
constexpr int kGreenThreads = 512;
constexpr int kGreenBlocks = 152;
__global__ void __launch_bounds__(kGreenThreads, 1) k_green(const ScState *sc, ScTables t, uint32_t num_part,
                                                            double cur_ov_mc2) {
  if (!sc->remesh || sc->sur_accepted) return;
  extern __shared__ double green_r[];  // rs of each source radius, then 1 / (2 rp) of each field radius (0 on axis)
  const uint32_t nr = sc->nx, nz = sc->nz;
  const uint32_t by = (512 / nz < nr) ? 512 / nz : nr;
  const uint32_t nrs = by ? (nr / by) * by : 0;
  const uint32_t total = (nr + 1) * nrs * nz;
  const double r_beta = sc->beta, r_freq = sc->freq;
  const uint32_t adj = sc->adj;
  const double gm = rsqrt(1.0 - r_beta * r_beta);
  const double dr = sc->dr, dzg = sc->dz * gm;
  const double wave_len = CLIGHT / r_freq;
  const double pl = r_beta * gm * wave_len;
  const double c1 = 5721.67 * cur_ov_mc2 / (r_freq * 1e6 * (double)num_part);
  for (uint32_t k = threadIdx.x; k < nr; k += blockDim.x) {
    green_r[k] = sqrt(0.5 * (k * k + (k + 1) * (k + 1))) * dr;
    green_r[nr + k + 1] = 0.5 / ((k + 1) * dr);
    if (k == 0) green_r[nr] = 0.0;
  }
  __syncthreads();
  const uint32_t share = ((total + gridDim.x - 1) / gridDim.x + 31) / 32 * 32;
  const uint32_t e0 = blockIdx.x * share, e1 = min(total, e0 + share);
  for (uint32_t e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
    const uint32_t k = e % nrs, tz = (e / nrs) % nz, rpi = e / (nz * nrs);
    const double rs = green_r[k], hrp = green_r[nr + rpi];
    const double zs = 0.5 * dzg, zp = (tz + 1) * dzg, rp = rpi * dr, d = zp - zs;
    const double c = (rp - rs) * (rp - rs), b = (rp + rs) * (rp + rs), rsrp4 = 4.0 * (rs * rp);
    const double rs2mrp2 = rs * rs - rp * rp;
    Green64 s{0.0, 0.0};
    green64_add(s, rs2mrp2, b, c, rsrp4, hrp, d);
    for (uint32_t i = 1; i <= adj; ++i) {
      const double sft = i * pl;
      green64_add(s, rs2mrp2, b, c, rsrp4, hrp, d - sft);
      green64_add(s, rs2mrp2, b, c, rsrp4, hrp, d + sft);
    }
    // stored [rp][dz][rs], rs fastest, for the contraction's lanes
    ((double2 *)t.fld1)[((size_t)rpi * nz + tz) * nr + k] = make_double2(c1 * s.er, c1 * s.ez);
  }
}
void green64_launch(const ScState *sc, const ScTables &t, uint32_t nr_max, uint32_t num_part, double cur_ov_mc2,
                    cudaStream_t st) {
  k_green<<<kGreenBlocks, kGreenThreads, (2 * (size_t)nr_max + 1) * sizeof(double), st>>>(sc, t, num_part, cur_ov_mc2);
}

__device__ inline void dep_add(unsigned long long *h, int k, double v) {
  long long q = __double2ll_rn(v * kBinScale);
  if (q) atomicAdd(h + k, (unsigned long long)q);
}

// What all particles of a kick share, formed once a block by one warp: the
// independent quotients on a lane each (one FP64 quotient's latency for all of
// them), where every thread used to form them for its one or two particles,
// a third of these kernels' FP64 instructions.
struct Kick64 {
  double gmg, epsq, inv_epsq, xfac, yfac, xbar, ybar, phimc, c2, pl;
  double dr, inv_dr, dzg, inv_dzg, hl;
  double beta, inv_mass, c3, cbg, er_c3, ez_c3;  // the kick's alone
  uint32_t nx, nz, adj;
};
// KICK: the mesh as the kick sees it (ratio-scaled); else as the deposit does
template <bool KICK>
__device__ __forceinline__ void kick64_consts(Kick64 &K, const DevBeam &bm, const ScState *sc, double length,
                                              double current) {
  __shared__ double q[10];
  const int lane = threadIdx.x;
  if (lane < 32) {
    const BeamStats &st = *bm.st;
    const double beta = sc->beta, gmg = rsqrt(1.0 - beta * beta), xs = st.st[X_SIG_GOOD], ys = st.st[Y_SIG_GOOD];
    const double rr = KICK ? sc->ratio_r : 1.0, rz = KICK ? sc->ratio_z : 1.0;
    const double dr = sc->dr * rr, dzg = sc->dz * gmg * rz;
    double num = 1.0, den = 1.0;
    switch (lane) {
      case 0: num = xs; den = ys; break;
      case 1: num = ys; den = xs; break;
      case 2: num = CLIGHT; den = sc->freq; break;
      case 3: den = dr; break;
      case 4: den = dzg; break;
      case 5: num = length; den = beta * gmg; break;
      case 6: den = bm.mass; break;
      case 7: num = 5721.67 * (current * sc->frac); den = sc->freq * 1e6 * (double)bm.n * bm.mass; break;
      case 8: num = sc->ratio_q; den = sc->ratio_r * sc->ratio_z * sc->ratio_g * sc->ratio_g; break;
      case 9: num = sc->ratio_q; den = sc->ratio_z * sc->ratio_z; break;
      default: break;
    }
    const double v = num / den;
    if (lane < 10) q[lane] = v;
    __syncwarp();
    if (lane == 0) {
      K.gmg = gmg;
      K.epsq = q[0];
      K.inv_epsq = q[1];
      K.xbar = st.st[X_AVG_GOOD];
      K.ybar = st.st[Y_AVG_GOOD];
      K.phimc = st.st[PHI_AVG_R];
      K.pl = beta * gmg * q[2];
      K.c2 = K.pl * (1.0 / TWOPI);
      K.dr = dr;
      K.inv_dr = q[3];
      K.dzg = dzg;
      K.inv_dzg = q[4];
      K.nx = sc->nx;
      K.nz = sc->nz;
      K.adj = sc->adj;
      K.hl = K.nz * 0.5 * dzg;
      if (KICK) {
        K.xfac = 2.0 / (q[0] + 1.0);
        K.yfac = q[0] * K.xfac;
        K.beta = beta;
        K.inv_mass = q[6];
        K.c3 = q[5];
        K.cbg = q[7] * q[5] * PI * 0.5 * sc->num_on_mesh;
        K.er_c3 = q[8] * q[5];
        K.ez_c3 = q[9] * q[5];
      }
    }
  }
  __syncthreads();
}

__device__ __forceinline__ double wrap_turns64(double d) {
  for (int guard = 0; (d > PI || d < -PI) && guard < 1000000; ++guard) {
    if (d > 0.0) d -= TWOPI;
    else d += TWOPI;
  }
  return d;
}

// DistributeParticleKernel, space_charge_kernel.cu:123-224: each block
// deposits into its own histogram in shared memory (integer weights), then
// adds it to the global table; integer sums make the table independent of
// the order in which particles arrive.
__global__ void k_deposit(DevBeam bm, ScState *sc, ScTables t) {
  if (!sc->remesh) return;
  extern __shared__ unsigned long long hist[];
  __shared__ Kick64 K;
  const uint32_t nx = sc->nx, nz = sc->nz, nb = nx * nz;
  for (uint32_t k = threadIdx.x; k < nb; k += blockDim.x) hist[k] = 0ull;
  kick64_consts<false>(K, bm, sc, 0.0, 0.0);
  const double dr = K.dr, drdr = dr * dr, inv_drdr = K.inv_dr * K.inv_dr;
  uint32_t cnt = 0;
  for (uint32_t np = blockIdx.x * blockDim.x + threadIdx.x; np < bm.n; np += gridDim.x * blockDim.x) {
    if (!(bm.loss[np] == 0u && bm.lloss[np] == 0u)) continue;
    const double dx = bm.x[np] - K.xbar, dy = bm.y[np] - K.ybar;
    const double rsq_sh = dx * dx * K.inv_epsq + dy * dy * K.epsq;
    const int i = (int)(sqrt(rsq_sh) * K.inv_dr + 1);
    if (!(i >= 1 && (uint32_t)i <= nx)) continue;
    const double z = -K.c2 * wrap_turns64(bm.phi_r[np] - K.phimc);
    if (!(fabs(z) < K.hl)) continue;
    const double zz = z + K.hl;
    const int jm1 = (int)(zz * K.inv_dzg + 1);
    int i1 = i + 1;
    if (rsq_sh < 0.5 * drdr * (double)(i * i + (i - 1) * (i - 1))) i1 = i - 1;
    if (i1 < 1) i1 = 1;
    if (i1 > (int)nx) i1 = nx;
    int j1 = jm1 + 1;
    if (zz < (jm1 - 1 + 0.5) * K.dzg) j1 = jm1 - 1;
    if (j1 < 1) j1 = 1;
    if (j1 > (int)nz) j1 = nz;
    if (jm1 < 1 || jm1 > (int)nz) continue;  // cannot happen for |z| < hl
    double a;
    if (i1 == i) a = 1.0;
    else {
      // radii in units of dr: rmax^2 - rmin^2 = q = sqrt(4 r^2 - 1)
      const double q2 = 4.0 * rsq_sh * inv_drdr - 1.0, iq = rsqrt(q2), q = q2 * iq;
      const double rmin2 = 0.25 * (q - 1.0) * (q - 1.0);
      if (i1 < i) a = (rmin2 + q - (double)((i - 1) * (i - 1))) * iq;
      else a = ((double)((i1 - 1) * (i1 - 1)) - rmin2) * iq;
    }
    double cc = 1.0;
    if (j1 != jm1) cc = (zz - (j1 - 1 + 0.5) * K.dzg) * (j1 < jm1 ? K.inv_dzg : -K.inv_dzg);
    const double bb = 1.0 - a, d = 1.0 - cc;
    int k = (jm1 - 1) * nx + i;
    dep_add(hist, k - 1, a * cc);
    k += i1 - i;
    dep_add(hist, k - 1, bb * cc);
    k = (j1 - 1) * nx + i;
    dep_add(hist, k - 1, a * d);
    k += i1 - i;
    dep_add(hist, k - 1, bb * d);
    ++cnt;
  }
  for (int off = 16; off > 0; off >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, off);
  if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(&sc->num_on_mesh, cnt);
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < nb; k += blockDim.x) {
    unsigned long long v = hist[k];
    if (v) atomicAdd(t.bin_fx + k, v);
  }
}


// ApplySpchKickKernel, space_charge_kernel.cu:573-706.  The reference's
// grid-stride loop `while (indx > 0 && ...)` ends thread 0 before its first
// particle, so particles whose index is a multiple of its launch's thread
// count (skip_stride) are never kicked; the same set is skipped here.
// Per particle: three roots, two reciprocals (nine quotients and three roots
// before).  65,536 particles: kick 38 -> 20.6 us, deposit 26.7 -> 16.9.
__global__ void k_kick(DevBeam bm, const ScState *sc, ScTables t, double length, double current,
                       uint64_t skip_stride) {
  __shared__ Kick64 K;
  kick64_consts<true>(K, bm, sc, length, current);
  const uint32_t nx = K.nx, nz = K.nz, tbl_sz = (nx + 1) * (nz + 1);
  const double *fld = t.fld2;
  for (uint32_t indx = blockIdx.x * blockDim.x + threadIdx.x; indx < bm.n; indx += gridDim.x * blockDim.x) {
    if (indx % skip_stride == 0) continue;
    if (!(bm.loss[indx] == 0u && bm.lloss[indx] == 0u)) continue;
    const double x = bm.x[indx], y = bm.y[indx], phi = bm.phi_r[indx], w = bm.w[indx];
    const double g = w * K.inv_mass, gm = g + 1.0, bgz = sqrt(g * (g + 2.0));
    double bgx = bgz * bm.xp[indx], bgy = bgz * bm.yp[indx];
    double bgzstar = K.gmg * (bgz - K.beta * gm);
    const double xxbar = x - K.xbar, yybar = y - K.ybar;
    const double r2 = xxbar * xxbar * K.inv_epsq + yybar * yybar * K.epsq;
    const double inv_r = r2 == 0.0 ? 1.0e8 : rsqrt(r2), r = r2 == 0.0 ? 1.0e-8 : r2 * inv_r;
    const double xovr = xxbar * K.xfac * inv_r, yovr = yybar * K.yfac * inv_r;
    double z = -K.c2 * wrap_turns64(phi - K.phimc);
    double cbgr, cbgzs;
    if (r > nx * K.dr || fabs(z) > K.hl) {
      z = -K.c2 * (phi - K.phimc);
      double d = sqrt(z * z + r * r);
      double invd3 = 1.0 / (d * d * d);
      double rod3 = r * invd3;
      double zod3 = z * invd3;
      for (uint32_t nb = 1; nb <= K.adj; ++nb) {
        int xi = (int)nb;
        for (int lr = 1; lr <= 2; ++lr) {
          double sft = z + xi * K.pl;
          d = sqrt(sft * sft + r * r);
          invd3 = 1.0 / (d * d * d);
          rod3 += r * invd3;
          zod3 += sft * invd3;
          xi = -xi;
        }
      }
      cbgr = K.cbg * rod3;
      cbgzs = K.cbg * zod3;
    } else {
      const double ri = r * K.inv_dr, zi = (z + K.hl) * K.inv_dzg;
      const uint32_t i = 1 + (int)ri;
      const double a = ri - (i - 1.0), bb = 1.0 - a;
      const uint32_t j = 1 + (int)zi;
      const double c = zi - (j - 1.0), d = 1.0 - c;
      uint32_t l = (j - 1) * (nx + 1) + i;
      uint32_t m = l + (nx + 1);
      if (m >= tbl_sz) m = tbl_sz - 1;
      // l leaves the table only for r == nx*dr with z == hl, or NaN input
      if (l >= tbl_sz || l < 1) l = tbl_sz - 1;
      if (m < 1) m = 1;
      cbgr = K.er_c3 * (d * (a * fld[2 * l] + bb * fld[2 * (l - 1)]) + c * (a * fld[2 * m] + bb * fld[2 * (m - 1)]));
      cbgzs = K.ez_c3 * (d * (a * fld[2 * l + 1] + bb * fld[2 * (l - 1) + 1]) +
                         c * (a * fld[2 * m + 1] + bb * fld[2 * (m - 1) + 1]));
    }
    bgx += cbgr * xovr;
    bgy += cbgr * yovr;
    bgzstar += cbgzs;
    const double gstar = 1.0 + 0.5 * bgzstar * bgzstar;
    const double bgzf = K.gmg * (bgzstar + K.beta * gstar);
    if (bgzf <= 0.0) bm.loss[indx] = 9999u;
    else {
      const double inv_f = 1.0 / bgzf;
      bm.xp[indx] = bgx * inv_f;
      bm.yp[indx] = bgy * inv_f;
      bm.w[indx] = w * (1.0 + (gm + 1.0) * (bgzf - bgz) / (gm * bgz));
    }
  }
}

}  // namespace

void beam_update_stat_for_sc(const DevBeam &b, PassScratch s, cudaStream_t st) {
  if (b.n <= 2) return;
  launch_pass(OpGoodPhi{b}, b.n, s, st);
  launch_pass(OpLlossGoodPhi{b}, b.n, s, st);
  launch_pass(OpScStats{b, nullptr, ScTables{}, 0.0, 0.0}, b.n, s, st);
  note_launch(3);
}

void sc_stats(const DevBeam &b, ScState *sc, const ScTables &t, const ScKickArgs &a, PassScratch s,
              cudaStream_t st) {
  if (a.stats_ok) {
    launch_pass(OpGoodPhi{b}, b.n, s, st);
    launch_pass(OpLlossGoodPhi{b}, b.n, s, st);
    launch_pass(OpScStats{b, sc, t, a.freq, a.frac}, b.n, s, st);
    note_launch(3);
  } else {
    k_decide_only<<<1, kBlock, 0, st>>>(b, sc, t, a.freq, a.frac);
    note_launch();
  }
}

// UpdateFldTbl2KernelDouble (space_charge_kernel.cu:472-568) on the FP64
// tables: contract64.cuh's kernel where the kick's mesh is known on the host
// and one it takes, contract.cuh's general one, sized for the largest mesh
// the solver takes, otherwise
void contract64(const ScState *sc, const ScTables &t, uint32_t nx_max, uint32_t nz_max, bool mesh_fixed,
                cudaStream_t st) {
  static PerDevice configured;
  configured.once([] {
    contract_configure<double>();
    contract64_configure();
  });
  if (mesh_fixed && contract64_ok(nx_max, nz_max)) contract64_launch(sc, t, nx_max, nz_max, st);
  else contract_launch<double>(sc, t, nx_max, nz_max, st);
}

void sc_mesh(const DevBeam &b, ScState *sc, const ScTables &t, const ScKickArgs &a, PassScratch s,
             cudaStream_t st, const SurNet *sur, const Fork *fork) {
  launch_pass(OpAdjMesh{b, sc}, b.n, s, st);
  note_launch();
  // mesh kernels are sized for the largest mesh this solver can take; with a
  // field surrogate the deposit comes first, and an accepted surrogate field
  // makes the Green's table and the contraction return at once
  if (!sur) {
    green64_launch(sc, t, a.nx_max, b.n, a.current * a.frac / b.mass, st);
    note_launch();
  }
  if (a.deposit_ok) {
    k_deposit<<<grid_for(b.n), kBlock, a.deposit_smem, st>>>(b, sc, t);
    note_launch();
  }
  if (sur) {
    sur_solve(b, sc, t, a, *sur, st, 0, fork);
    green64_launch(sc, t, a.nx_max, b.n, a.current * a.frac / b.mass, st);
    note_launch();
  }
  contract64(sc, t, a.nx_max, a.nz_max, a.mesh_fixed, st);
  note_launch();
}

void sc_kick(const DevBeam &b, ScState *sc, const ScTables &t, const ScKickArgs &a, cudaStream_t st) {
  if (a.skip_stride) {
    k_kick<<<grid_for(b.n), kBlock, 0, st>>>(b, sc, t, a.length, a.current, a.skip_stride);
    note_launch();
  }
}

// the limit only grows, per device (the attribute is per device)
void sc_configure(size_t max_deposit_smem) {
  static std::mutex m;
  static size_t configured[kMaxDevices] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaFuncSetAttribute(k_deposit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_deposit_smem);
    return;
  }
  std::lock_guard<std::mutex> lock(m);
  if (max_deposit_smem <= configured[dev]) return;
  configured[dev] = max_deposit_smem;
  cudaFuncSetAttribute(k_deposit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_deposit_smem);
}

// ---- standalone field solve: charge table -> field table ------------------

namespace {

// Mesh description of a standalone solve (what Scheff::Start would have
// settled on before UpdateTblsKernelCall / UpdateFinalFldTblKernelCall).
__global__ void k_field_setup(ScState *sc, uint32_t nr, uint32_t nz, double dr, double dz, double beta,
                              double freq, uint32_t adj) {
  sc->nx = nr; sc->nz = nz; sc->nx_init = nr; sc->nz_init = nz; sc->nx_max = nr; sc->nz_max = nz;
  sc->dr = dr; sc->dz = dz; sc->beta = beta; sc->freq = freq; sc->adj = adj;
  sc->remesh = 1;
}

// charge table in FP64 -> the deposit's fixed-point table
__global__ void k_bins_to_fixed(const double *bins, unsigned long long *fx, uint32_t nb) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nb; k += gridDim.x * blockDim.x)
    fx[k] = (unsigned long long)__double2ll_rn(bins[k] * kBinScale);
}

bool mesh_ok(uint32_t nr, uint32_t nz) {
  return nr && nz && !(nr & (nr - 1)) && !(nz & (nz - 1)) && nz <= 512 && nr <= 256;
}

}  // namespace

// Green's table + contraction for a given charge table (UpdateFldTbl1Kernel
// and UpdateFldTbl2KernelDouble).  sc, fx, fld1 and fld2 are device buffers
// sized for (nr, nz); fld2 is overwritten.
// Returns the status of the field table's clearing or of the launches.
cudaError_t sc_field_solve(ScState *sc, unsigned long long *fx, double *fld1, double *fld2, uint32_t nr, uint32_t nz,
                           const double *bins_dev, const double *mesh, cudaStream_t st) {
  k_field_setup<<<1, 1, 0, st>>>(sc, nr, nz, mesh[0], mesh[1], mesh[2], mesh[3], (uint32_t)mesh[6]);
  k_bins_to_fixed<<<64, kBlock, 0, st>>>(bins_dev, fx, nr * nz);
  const cudaError_t me = cudaMemsetAsync(fld2, 0, (size_t)(nz + 1) * (nr + 1) * 2 * sizeof(double), st);
  if (me != cudaSuccess) return me;
  ScTables t{};
  t.bin_fx = fx;
  t.fld1 = fld1;
  t.fld2 = fld2;
  green64_launch(sc, t, nr, (uint32_t)mesh[4], mesh[5], st);
  contract64(sc, t, nr, nz, true, st);
  note_launch(4);
  return cudaGetLastError();
}

}  // namespace hps

extern "C" {

// UpdateTblsKernelCall (Green's table part) + UpdateFinalFldTblKernelCall,
// src/simulation/src/space_charge.cu:148-218, on a caller-given charge table.
hps_status hps_scheff_field(uint32_t nr, uint32_t nz, const double *bins, const double *mesh, double *field) {
  using namespace hps;
  if (!bins || !mesh || !field) return (hps_status)set_error(HPS_ERR_INVALID, "scheff_field: null pointer");
  if (!mesh_ok(nr, nz))
    return (hps_status)set_error(HPS_ERR_INVALID, "scheff_field: nr and nz must be powers of two, nz <= 512, nr <= 256");
  size_t nb = (size_t)nr * nz, n1 = (size_t)(nr + 1) * nr * nz * 2, n2 = (size_t)(nz + 1) * (nr + 1) * 2;
  ScState *sc = nullptr;
  unsigned long long *fx = nullptr;
  double *b = nullptr, *f1 = nullptr, *f2 = nullptr;
  cudaError_t e = cudaMalloc((void **)&sc, sizeof(ScState));
  if (e == cudaSuccess) e = cudaMalloc((void **)&fx, nb * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc((void **)&b, nb * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc((void **)&f1, n1 * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc((void **)&f2, n2 * sizeof(double));
  if (e == cudaSuccess) e = cudaMemset(sc, 0, sizeof(ScState));
  if (e == cudaSuccess) e = cudaMemcpy(b, bins, nb * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = sc_field_solve(sc, fx, f1, f2, nr, nz, b, mesh, 0);
  if (e == cudaSuccess) e = cudaMemcpy(field, f2, n2 * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(sc); cudaFree(fx); cudaFree(b); cudaFree(f1); cudaFree(f2);
  if (e != cudaSuccess) return (hps_status)set_error(HPS_ERR_CUDA, cudaGetErrorString(e));
  return HPS_OK;
}

}  // extern "C"

// ---- field solve without allocation --------------------------------------
//
// Some callers cannot allocate device memory while they run: an online model
// that re-solves the space-charge field inside a control-system cycle and
// must not wait on the CUDA allocator, or a host application that owns the
// whole device through its own memory pool and hands its plugins finished
// buffers.  hps_scheff_field_noalloc serves them: the caller supplies the
// charge table and the field table in device memory, and the intermediate
// tables live in one statically sized device array of this library (held
// by every GPU that loads the library until the process exits).
namespace hps {
namespace {

constexpr uint32_t kNoAllocMaxBins = 4096;                // nr * nz
constexpr uint32_t kNoAllocMaxGreen = 33u * 32u * 128u;   // (nr + 1) * nr * nz
constexpr size_t kNoAllocStateBytes = 256;
constexpr size_t kNoAllocBytes =
    kNoAllocStateBytes + kNoAllocMaxBins * sizeof(unsigned long long) + (size_t)kNoAllocMaxGreen * 2 * sizeof(double);
static_assert(sizeof(ScState) <= kNoAllocStateBytes, "ScState outgrew its slot in the static scratch");

// state block | fixed-point charge table | Green's table
static __device__ __align__(256) unsigned char g_field_scratch[kNoAllocBytes];

std::mutex g_scratch_mutex;
void *g_scratch_addr[kMaxDevices];  // device address of g_field_scratch, per device

// Device address of the scratch array on the current device.  The symbol's
// name is only a host-side handle: the address has to be asked for once per
// device, with that device current.  The cached address belongs to the
// device's current context: after cudaDeviceReset the library has to be
// reloaded before this entry point is used on that device again.
int scratch_address(void **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return set_error(HPS_ERR_CUDA, cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return set_error(HPS_ERR_UNSUPPORTED, "scheff_field_noalloc: device index too large");
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (!g_scratch_addr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_field_scratch);
    if (e != cudaSuccess) return set_error(HPS_ERR_CUDA, cudaGetErrorString(e));
    g_scratch_addr[dev] = p;
  }
  *out = g_scratch_addr[dev];
  return HPS_OK;
}

}  // namespace
}  // namespace hps

extern "C" {

// Same computation as hps_scheff_field on device buffers, allocating nothing.
// The first call on a device looks up the scratch array's device address;
// make that first call before any stream capture.  Meshes are limited to
// nr*nz <= 4096 and (nr+1)*nr*nz <= 135168 (32 x 128 at most for nr = 32);
// larger ones are rejected.  All calls share the scratch, so calls whose
// work overlaps on the GPU (different streams, or other threads) race; the
// scratch keeps the previous call's tables, and every entry this call reads
// is rewritten first.  The field table is cleared before it is summed into.
hps_status hps_scheff_field_noalloc(uint32_t nr, uint32_t nz, const double *bins_dev, const double *mesh,
                                    double *field_dev, void *stream) {
  using namespace hps;
  if (!bins_dev || !mesh || !field_dev) return (hps_status)set_error(HPS_ERR_INVALID, "scheff_field_noalloc: null pointer");
  if (!mesh_ok(nr, nz))
    return (hps_status)set_error(HPS_ERR_INVALID, "scheff_field_noalloc: nr and nz must be powers of two");
  if ((size_t)nr * nz > kNoAllocMaxBins || (size_t)(nr + 1) * nr * nz > kNoAllocMaxGreen)
    return (hps_status)set_error(HPS_ERR_INVALID,
                                 "scheff_field_noalloc: mesh too large for the static scratch "
                                 "(limit nr*nz <= 4096 and (nr+1)*nr*nz <= 135168, e.g. 32 x 128)");
  // an error left pending by earlier work is the caller's, not this call's
  const cudaError_t pending = cudaPeekAtLastError();
  if (pending != cudaSuccess)
    return (hps_status)set_error(HPS_ERR_CUDA, (std::string("scheff_field_noalloc: an earlier CUDA error is "
                                                            "pending: ") + cudaGetErrorString(pending)).c_str());
  void *base = nullptr;
  int st = scratch_address(&base);
  if (st != HPS_OK) return (hps_status)st;
  unsigned char *p = (unsigned char *)base;
  ScState *sc = (ScState *)p;
  unsigned long long *fx = (unsigned long long *)(p + kNoAllocStateBytes);
  double *fld1 = (double *)(p + kNoAllocStateBytes + kNoAllocMaxBins * sizeof(unsigned long long));
  const cudaError_t e = sc_field_solve(sc, fx, fld1, field_dev, nr, nz, bins_dev, mesh, (cudaStream_t)stream);
  if (e != cudaSuccess) return (hps_status)set_error(HPS_ERR_CUDA, cudaGetErrorString(e));
  return HPS_OK;
}

}  // extern "C"
