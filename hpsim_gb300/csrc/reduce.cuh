// reduce.cuh -- one-launch deterministic reductions over the particles.
//
// The reference reduces every moment with a Harris two-level tree: a first
// pass capped at 64 blocks, a second pass, then a <<<1,1>>> finaliser kernel
// (src/beam/src/beam.cu:411-436, 651-678); about 30 launches and 5 blocking
// scalar reads per space-charge kick.  Here one launch does all of it: every
// block reduces its grid-stride share of the particles (each thread in index
// order, warps by a fixed shuffle order, warps in index order), writes one
// partial per block, and the last block to finish (threadfence + counter)
// sums the partials in a fixed order and runs the finaliser.  The result is
// bitwise reproducible for a given particle count, and the per-particle
// callback may also write per-particle outputs (relative phase, loss flags)
// in the same sweep.
#pragma once

#include <algorithm>

#include <type_traits>

#include "common.cuh"
#include "lockstep.cuh"

namespace hps {

// comb() is overloaded for float so that FP32 warp trees stay on the FP32
// pipes (a float argument promoted to the double overload would run every
// shuffle step through FP64 arithmetic).
struct SumComb {
  __device__ static double ident() { return 0.0; }
  __device__ static double comb(double a, double b) { return a + b; }
  __device__ static float comb(float a, float b) { return a + b; }
};
struct MaxComb {  // MaxR2PhiReduceKernel starts from 0 (beam_kernel.cu:809-810)
  __device__ static double ident() { return 0.0; }
  __device__ static double comb(double a, double b) { return a < b ? b : a; }
  __device__ static float comb(float a, float b) { return a < b ? b : a; }
};

// Totals over a warp of K accumulators a lane, K <= 32, by folding: a step
// halves the lanes' distance and the accumulators a lane still carries (it
// sends one half to its partner and keeps the other), so K sums cost about
// K + log2(32 / K) combinations a lane where a shuffle tree for each costs
// 5 K.  The lanes whose low bits are zero hold the totals: true with the slot
// number, in an order fixed by the lane numbers.
template <class C, int K, class T>
__device__ __forceinline__ bool warp_fold(const T (&a)[K], int lane, int &slot, T &total) {
  constexpr int P = K > 16 ? 32 : K > 8 ? 16 : K > 4 ? 8 : K > 2 ? 4 : K > 1 ? 2 : 1;
  T v[P];
#pragma unroll
  for (int k = 0; k < P; ++k) v[k] = k < K ? a[k] : (T)C::ident();
  int base = 0, off = 16;
#pragma unroll
  for (int cnt = P / 2; cnt >= 1; cnt /= 2, off /= 2) {
    const bool hi = lane & off;
#pragma unroll
    for (int k = 0; k < cnt; ++k) {
      const T keep = hi ? v[k + cnt] : v[k], send = hi ? v[k] : v[k + cnt];
      v[k] = C::comb(keep, __shfl_xor_sync(0xffffffffu, send, off));
    }
    if (hi) base += cnt;
  }
  T x = v[0];
#pragma unroll
  for (int o = 16 / P; o > 0; o /= 2) x = C::comb(x, __shfl_xor_sync(0xffffffffu, x, o));
  slot = base;
  total = x;
  return (lane & (32 / P - 1)) == 0 && base < K;
}

// Rows per slot that the FP64 combine's first step leaves: as many as the
// block has threads for, within a short second step.
template <int K>
constexpr int combine_rows() {
  return K <= 4 ? 64 : kBlock / K < 16 ? (kBlock / K > 8 ? kBlock / K : 8) : 16;
}

// Total of the per-block partials, taken by the last block: thread t sums
// slot t mod K over rows t / K, t / K + G, ... (eight loads in flight, so the
// sweep costs a memory round trip or two), then K threads the G rows left.
// FP64 additions run at two a cycle on an SM, and a warp's instruction takes
// its 64 cycles whatever lanes it has: a shuffle tree per slot (5 K additions
// by every warp) was 5 us of a beam statistics record's 17 slots, this order
// does one addition per partial.
template <class C, int K>
__device__ inline void combine_partials(const double *part, uint32_t nb, double (*sm)[K], double *tot) {
  constexpr int G = combine_rows<K>();
  static_assert(G * K <= kBlock, "a thread per row and slot");
  const int t = threadIdx.x;
  if (t < G * K) {
    double x = C::ident();
    for (uint32_t r = t / K; r < nb; r += 8 * G) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = r + u * G < nb ? __ldcg(part + (size_t)(r + u * G) * K + t % K) : C::ident();
      x = C::comb(x, C::comb(C::comb(C::comb(v[0], v[1]), C::comb(v[2], v[3])),
                             C::comb(C::comb(v[4], v[5]), C::comb(v[6], v[7]))));
    }
    sm[t / K][t % K] = x;
  }
  __syncthreads();
  if (t < K) {
    double v[4] = {C::ident(), C::ident(), C::ident(), C::ident()};
#pragma unroll
    for (int g = 0; g < G; ++g) v[g & 3] = C::comb(v[g & 3], sm[g][t]);
    tot[t] = C::comb(C::comb(v[0], v[1]), C::comb(v[2], v[3]));
  }
  __syncthreads();
}

// From the totals q of three coordinate pairs (a, a^2, b, b^2, a b of the
// horizontal, vertical and longitudinal plane) over m particles: o[plane][0..4]
// = <a>, sigma_a, <b>, sigma_b, emittance, the transverse emittances times
// beta gamma of kinetic energy w0.  Every thread of the block calls it.  A
// dependent FP64 quotient or root costs about a third of a microsecond on one
// thread, so the 15 quotients are taken by 15 threads and the 9 roots by 9.
__device__ inline void plane_moments(const double *q, double m, double w0, double mass, double (*o)[5]) {
  __shared__ double mean[15], bg;
  const int t = threadIdx.x;
  if (t < 15) mean[t] = q[t] / m;
  if (t == 32) {
    const double g1 = w0 / mass;
    bg = sqrt(g1 * (g1 + 2.0));
  }
  __syncthreads();
  if (t < 9) {
    const int pl = t / 3, kind = t % 3;
    const double *c = mean + 5 * pl;
    const double a = c[0], a2 = c[1], b = c[2], b2 = c[3], ab = c[4];
    const double va = a2 - a * a, vb = b2 - b * b, cv = ab - a * b;
    const double r = sqrt(kind == 0 ? va : kind == 1 ? vb : va * vb - cv * cv);
    if (kind == 0) { o[pl][0] = a; o[pl][1] = r; }
    else if (kind == 1) { o[pl][2] = b; o[pl][3] = r; }
    else o[pl][4] = pl < 2 ? r * bg : r;
  }
  __syncthreads();
}

// Op must provide:
//   static constexpr int K;            number of accumulators (<= 32)
//   using Comb = SumComb | MaxComb;
//   __device__ bool enabled() const;   device-side predicate (false: no work)
//   __device__ void particle(uint32_t i, double (&acc)[K]) const;
//   __device__ void finalize(const double* tot, int tid, int nthreads) const;
template <class Op>
__global__ void __launch_bounds__(kBlock) pass_kernel(Op op, uint32_t n, PassScratch scr) {
  constexpr int K = Op::K;
  using C = typename Op::Comb;
  if (!op.enabled()) return;
  double acc[K];
#pragma unroll
  for (int k = 0; k < K; ++k) acc[k] = C::ident();
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) op.particle(i, acc);

  __shared__ double sm[combine_rows<K>()][K];
  __shared__ double tot[K];
  __shared__ int is_last;
  {
    int slot;
    double v;
    if (warp_fold<C>(acc, threadIdx.x & 31, slot, v)) sm[threadIdx.x >> 5][slot] = v;
  }
  __syncthreads();
  if (threadIdx.x < K) {
    double v = C::ident();
#pragma unroll
    for (int w = 0; w < kBlock / 32; ++w) v = C::comb(v, sm[w][threadIdx.x]);
    scr.part[blockIdx.x * K + threadIdx.x] = v;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = (atomicAdd(scr.counter, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  combine_partials<C, K>(scr.part, gridDim.x, sm, tot);
  op.finalize(tot, threadIdx.x, blockDim.x);
  __syncthreads();
  if (threadIdx.x == 0) *scr.counter = 0u;
}

template <class Op>
inline void launch_pass(const Op &op, uint32_t n, PassScratch scr, cudaStream_t s) {
  pass_kernel<Op><<<pass_blocks(n), kBlock, 0, s>>>(op, n, scr);
}

// Same scheme for FP32 particle state: each thread accumulates its particles
// in FP32 and the warp tree runs in FP32 (FP64 arithmetic on GB300 runs at
// 1/64 of the FP32 rate, so per-particle FP64 sums would dominate); warps,
// blocks and the finaliser combine in FP64.  Op::setup() returns constants
// (offsets of device-side averages from the synchronous particle), computed
// once per block.  A thread takes its particles kPassBatch at a time (2 for
// ops with many accumulators, to stay within registers): Op::load(i) reads
// particle i into an Op::P, and Op::use(i, p, acc, ctx)
// accumulates it (and may write per-particle outputs), so every load of a
// batch is in flight before the first store.
constexpr int kPassBatch = 4;
template <int K> constexpr int pass_batch() { return K > 10 ? 2 : kPassBatch; }

// An Op with `static constexpr bool kFast = true` has its block and grid
// partials combined in FP32 (counts stay exact below 2^24 particles); the
// space-charge statistics that only size the mesh and scale the kick use
// it, reported beam statistics do not.
template <class Op, class = void>
struct op_fast : std::false_type {};
template <class Op>
struct op_fast<Op, std::void_t<decltype(Op::kFast)>> : std::integral_constant<bool, Op::kFast> {};

// An Op with kFast fixes its blocks per SM (`static constexpr int kGridPerSm`):
// the order of its sums follows from the number of blocks, and must not change
// with the registers that a compiler gives the kernel.
template <class Op, class = void>
struct op_grid_per_sm : std::integral_constant<int, 2> {};
template <class Op>
struct op_grid_per_sm<Op, std::void_t<decltype(Op::kGridPerSm)>> : std::integral_constant<int, Op::kGridPerSm> {};

// Slot k's total over the FP32 partials of nblk blocks, taken by a warp: lane l
// sums blocks l, l + 32, ... (eight loads in flight), then a fixed shuffle tree
// (lane 0 has the result).  Slots from MF on hold maxima of any sign.  Partials
// lie slot by slot, kMaxPassBlocks apart.
template <class C, int MF>
__device__ __forceinline__ float combine_slot_f(const float *part, int k, uint32_t nblk) {
  const int lane = threadIdx.x & 31;
  const float *p = part + (size_t)k * kMaxPassBlocks;
  float v = k >= MF ? -INFINITY : 0.0f;
  auto comb = [k](float a, float b) { return k >= MF ? fmaxf(a, b) : (float)C::comb(a, b); };
  for (uint32_t b = lane; b < nblk; b += 8 * 32) {
    float r[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (b + 32 * u < nblk) r[u] = __ldcg(p + b + 32 * u);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (b + 32 * u < nblk) v = comb(v, r[u]);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = comb(v, __shfl_down_sync(0xffffffffu, v, off));
  return v;
}

// block bid of nblk blocks of the pass over particles 0..n-1
template <class Op>
__device__ __forceinline__ void pass_body_f(const Op &op, uint32_t n, PassScratch scr, uint32_t bid, uint32_t nblk) {
  constexpr int K = Op::K;
  constexpr int B = pass_batch<K>();
  using C = typename Op::Comb;
  if (!op.enabled()) return;
  __shared__ double tot[K];
  __shared__ int is_last;
  __shared__ typename Op::Ctx sctx;
  if (threadIdx.x == 0) sctx = op.setup();
  __syncthreads();
  const typename Op::Ctx ctx = sctx;
  float acc[K];
#pragma unroll
  for (int k = 0; k < K; ++k) acc[k] = 0.0f;
  const uint32_t stride = nblk * blockDim.x;
  for (uint32_t base = bid * blockDim.x + threadIdx.x; base < n; base += B * stride) {
    typename Op::P p[B];
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const uint32_t i = base + u * stride;
      if (i < n) p[u] = op.load(i);
    }
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const uint32_t i = base + u * stride;
      if (i < n) op.use(i, p[u], acc, ctx);
    }
  }

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if constexpr (op_fast<Op>::value) {
    // FP32 partials: warps summed in order per block, blocks by the warps of
    // the last block (slot k by warp k mod 8).  No FP64 arithmetic on the
    // reduction's critical path.
    __shared__ float smf[kBlock / 32][K];
    float *partf = (float *)scr.part;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      float v = acc[k];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v = C::comb(v, __shfl_down_sync(0xffffffffu, v, off));
      if (lane == 0) smf[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < K) {
      const int k = threadIdx.x;
      float v = 0.0f;
      for (int w = 0; w < kBlock / 32; ++w) v = C::comb(v, smf[w][k]);
      partf[(size_t)k * kMaxPassBlocks + bid] = v;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = (atomicAdd(scr.counter, 1u) == nblk - 1);
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int k = warp; k < K; k += kBlock / 32) {
      const float v = combine_slot_f<C, K>(partf, k, nblk);
      if (lane == 0) tot[k] = (double)v;
    }
    __syncthreads();
  } else {
    __shared__ double sm[combine_rows<K>()][K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      float v = acc[k];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v = C::comb(v, __shfl_down_sync(0xffffffffu, v, off));
      if (lane == 0) sm[warp][k] = (double)v;
    }
    __syncthreads();
    if (threadIdx.x < K) {
      double v = C::ident();
#pragma unroll
      for (int w = 0; w < kBlock / 32; ++w) v = C::comb(v, sm[w][threadIdx.x]);
      scr.part[bid * K + threadIdx.x] = v;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = (atomicAdd(scr.counter, 1u) == nblk - 1);
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    combine_partials<C, K>(scr.part, nblk, sm, tot);
  }
  op.finalize(tot, threadIdx.x, blockDim.x);
  __syncthreads();
  if (threadIdx.x == 0) *scr.counter = 0u;
}

template <class Op>
__global__ void __launch_bounds__(kBlock) pass_kernel_f(Op op, uint32_t n, PassScratch scr) {
  pdl_enter();
  pass_body_f(op, n, scr, blockIdx.x, gridDim.x);
}

// one beam's share of a lockstep launch of pass_kernel_f
template <class Op>
struct PassSeg {
  Op op;
  uint32_t n;
  PassScratch scr;
};
template <class Op, int B>
__global__ void __launch_bounds__(kBlock) pass_kernel_f_seg(const __grid_constant__ SegArgs<PassSeg<Op>, B> a) {
  uint32_t bid, nblk;
  const PassSeg<Op> &p = a.p[seg_find(a, blockIdx.x, bid, nblk)];
  pass_body_f(p.op, p.n, p.scr, bid, nblk);
}
template <class Op>
inline void pass_merge(const std::vector<const Rec *> &recs, SegFork &, cudaStream_t st, cudaStream_t) {
  seg_chunks<PassSeg<Op>>(recs, [&](const auto &a, uint32_t blocks) {
    pass_kernel_f_seg<Op, std::decay_t<decltype(a)>::kB><<<blocks, kBlock, 0, st>>>(a);
  });
}
// a pass_kernel_f launch of `blocks` blocks, or its record under a lockstep recorder
template <class Op>
inline void launch_pass_f_grid(const Op &op, uint32_t n, PassScratch scr, cudaStream_t s, uint32_t blocks,
                               const char *site) {
  if (recorder()) {
    record(site, &pass_merge<Op>, blocks, PassSeg<Op>{op, n, scr});
    return;
  }
  launch_after(n, pass_kernel_f<Op>, dim3(blocks), dim3(kBlock), 0, s, op, n, scr);
}

// Blocks of a pass: four particles a thread until there are per_sm blocks on
// every SM, then more a thread.  With the FP64 combine that is two: the last
// block sums every block's partials in FP64 on one SM (1/64-rate FP64 on
// GB300), so fewer, fuller blocks keep that tail short.
inline int pass_blocks_f(uint32_t n, int per_sm = 2) {
  uint32_t b = (uint32_t)(((uint64_t)n + kPassBatch * kBlock - 1) / (kPassBatch * kBlock));
  if (b < 1) b = 1;
  const uint32_t cap = std::min<uint32_t>((uint32_t)per_sm * 152u, (uint32_t)kMaxPassBlocks);
  if (b > cap) b = cap;
  return (int)b;
}

template <class Op>
inline void launch_pass_f(const Op &op, uint32_t n, PassScratch scr, cudaStream_t s) {
  launch_pass_f_grid(op, n, scr, s, (uint32_t)pass_blocks_f(n, op_grid_per_sm<Op>::value), "pass");
}

// FP32 version of rel_phase for offsets that are already small
__device__ inline float rel_phase_f(float d) {
  const float pi = 3.14159265358979323846f, twopi = 6.28318530717958647692f;
  float tmp = d + pi;
  float sign = 1.0f;
  if (tmp < 0.0f) { sign = -1.0f; tmp = -tmp; }
  if (tmp < twopi) return sign * (tmp - pi);
  return sign * (fmodf(tmp, twopi) - pi);
}

// wrap(phi - ref) as UpdateRelativePhiKernel, beam_kernel.cu:1507-1525
__device__ inline double rel_phase(double phi, double ref) {
  double tmp = phi - ref + PI;
  double sign = 1.0;
  if (tmp < 0) { sign = -1.0; tmp = -tmp; }
  if (tmp < TWOPI) return sign * (tmp - PI);  // fmod returns it as it is
  return sign * (fmod(tmp, TWOPI) - PI);
}

}  // namespace hps
