// contract64.cuh -- the SCHEFF ring-to-mesh field sum of FP64 beams
// (UpdateFldTbl2KernelDouble, src/simulation/inc/space_charge_kernel.cu:
// 472-568) on meshes whose charges and one field radius's table fit an SM.
//
// The sum is contract.cuh's: for each source radius a convolution along z,
// the lanes over the source radii, a ring of table values in registers that
// takes one load a row.  What bounds it is the FP64 pipe (two multiply-adds a
// cycle and SM: 59 us for the 2 x 129 x 33 x 4096 of a 32 x 128 mesh), so
// this form spends FP64 instructions on nothing else and gives every SM the
// same number of them:
//  * the field points go to one block an SM in groups of four rows of a field
//    radius, numbered radius after radius; a block takes consecutive groups
//    (1,056 on 152 SMs: seven each but the last), so it stages one or two
//    radii's tables.  Blocks of 16 rows, two an SM, left SMs with one and
//    SMs with two of them (97 us);
//  * the last group of a radius carries the row zp = nz as a fifth point;
//  * the sign of E_z at and above the point is an exclusive-or;
//  * the charges stay whole numbers, converted once a block, and 2^-36 (a
//    power of two) multiplies the finished sums;
//  * a warp's eight sums are folded over the lanes with nine additions.
// A group's source rows are shared by four warps (by 32 / nr lane groups too
// where a mesh has fewer than 32 radii), whose sums are added in order.
// 32 x 128: 97 -> 69 us, against 64 bits exact to 1.6e-16 (2.7e-16 before).
#pragma once

#include "common.cuh"
#include "reduce.cuh"

namespace hps {
namespace {

constexpr int kC64Threads = 512;
constexpr int kC64Blocks = 152;   // one an SM
constexpr int kC64Groups = 16;    // groups of a block at most
constexpr int kC64Parts = 4;      // warps sharing a group's source rows
constexpr size_t kC64Smem = 196608;

// Meshes it takes: powers of two whose table fits, from 1024 bins on (below,
// the reference's partition of the table leaves bins out, see contract.cuh).
inline bool contract64_ok(uint32_t nr, uint32_t nz) {
  return (nr & (nr - 1)) == 0 && (nz & (nz - 1)) == 0 && nz <= 512 && nr <= 256 && nr * nz >= 1024 &&
         (size_t)nr * nz * 24 <= kC64Smem && nz / kC64Parts * (nr < 32 ? nr : 32) >= 32;  // rows for every lane group
}

// g(k) of radius r from the staged rows: row k - 1 for k >= 1, row -k with
// E_z negated for k <= 0
__device__ __forceinline__ double2 g64(const double2 *tab, int k, int nr) {
  const bool below = k >= 1;
  double2 v = tab[(below ? k - 1 : -k) * nr];
  v.y = __hiloint2double(__double2hiint(v.y) ^ (below ? 0 : (int)0x80000000), __double2loint(v.y));
  return v;
}

// the sums of P points zp0 .. zp0 + P - 1 over rows [za, za + span) of radius
// r (tab, qs: the radius's columns), a[j] += E_r, a[P + j] += E_z of point j
template <int P>
__device__ __forceinline__ void walk64(const double2 *tab, const double *qs, int zp0, int za, int span, int nr,
                                       double (&a)[2 * P]) {
  constexpr int R = P + 1;
  // slot (j - u) mod R holds g(zp0 + j - zs) at row zs = za + s + u
  double2 ring[R];
#pragma unroll
  for (int j = 0; j < P; ++j) ring[j] = g64(tab, zp0 + j - za, nr);
  for (int s = 0; s < span; s += R) {
#pragma unroll
    for (int u = 0; u < R; ++u) {
      if (s + u >= span) break;
      const int zs = za + s + u;
      if (s + u + 1 < span) ring[(R - 1 - u) % R] = g64(tab, zp0 - zs - 1, nr);
      const double q = qs[zs * nr];
#pragma unroll
      for (int j = 0; j < P; ++j) {
        const double2 g = ring[(j - u + R) % R];
        a[j] = fma(q, g.x, a[j]);
        a[P + j] = fma(q, g.y, a[P + j]);
      }
    }
  }
}

template <int P>
__device__ __forceinline__ void task64(const double2 *tab, const double *qs, int zp0, int part, int nr, int nz,
                                       double *out) {
  const int lane = threadIdx.x & 31, width = nr < 32 ? nr : 32, nseg = 32 / width;
  const int span = nz / (kC64Parts * nseg), za = (part * nseg + lane / width) * span;
  double a[2 * P];
#pragma unroll
  for (int k = 0; k < 2 * P; ++k) a[k] = 0.0;
  for (int r = lane % width; r < nr; r += 32) walk64<P>(tab + r, qs + r, zp0, za, span, nr, a);
  int slot;
  double v;
  if (warp_fold<SumComb>(a, lane, slot, v)) out[slot] = v;
}

__global__ void __launch_bounds__(kC64Threads, 1) k_contract64(const ScState *sc, ScTables t) {
  if (!sc->remesh || sc->sur_accepted) return;
  extern __shared__ __align__(16) unsigned char c64_raw[];
  __shared__ double part[kC64Groups][kC64Parts][10];
  const int nr = (int)sc->nx, nz = (int)sc->nz, nb = nr * nz, per_rp = nz / 4, groups = (nr + 1) * per_rp;
  const int per = (groups + gridDim.x - 1) / gridDim.x, g0 = blockIdx.x * per, g1 = min(groups, g0 + per);
  if (g0 >= g1) return;
  double2 *tab = (double2 *)c64_raw;      // [dz][rs] of one field radius
  double *qs = (double *)(tab + nb);      // [zs][rs]
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int e = tid; e < nb; e += kC64Threads) qs[e] = (double)(long long)__ldg(t.bin_fx + e);
  for (int ga = g0; ga < g1;) {
    const int rp = ga / per_rp, gb = min(g1, (rp + 1) * per_rp);
    __syncthreads();  // the last radius's table has been read
    const double2 *src = (const double2 *)t.fld1 + (size_t)rp * nb;
    for (int e = tid; e < nb; e += 8 * kC64Threads) {
      double2 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (e + u * kC64Threads < nb) v[u] = __ldg(src + e + u * kC64Threads);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (e + u * kC64Threads < nb) tab[e + u * kC64Threads] = v[u];
    }
    __syncthreads();
    for (int k = warp; k < (gb - ga) * kC64Parts; k += kC64Threads / 32) {
      const int g = ga + k / kC64Parts, p = k % kC64Parts, zp0 = 4 * (g % per_rp);
      if (zp0 + 4 < nz) task64<4>(tab, qs, zp0, p, nr, nz, part[g - g0][p]);
      else task64<5>(tab, qs, zp0, p, nr, nz, part[g - g0][p]);
    }
    ga = gb;
  }
  __syncthreads();
  for (int k = tid; k < (g1 - g0) * 10; k += kC64Threads) {
    const int g = g0 + k / 10, slot = k % 10, rp = g / per_rp, zp0 = 4 * (g % per_rp), P = zp0 + 4 < nz ? 4 : 5;
    if (slot >= 2 * P) continue;
    const double *v = &part[g - g0][0][slot];
    const size_t pt = (size_t)(zp0 + slot % P) * (nr + 1) + rp;
    t.fld2[2 * pt + slot / P] = (((v[0] + v[10]) + v[20]) + v[30]) * kBinInvScale;
  }
}

inline void contract64_configure() {
  cudaFuncSetAttribute(k_contract64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kC64Smem);
}
inline void contract64_launch(const ScState *sc, const ScTables &t, uint32_t nr, uint32_t nz, cudaStream_t st) {
  const uint32_t groups = (nr + 1) * (nz / 4);
  k_contract64<<<groups < (uint32_t)kC64Blocks ? groups : (uint32_t)kC64Blocks, kC64Threads, (size_t)nr * nz * 24, st>>>(
      sc, t);
}

}  // namespace
}  // namespace hps
