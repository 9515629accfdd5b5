// Per-cell LBM update shared by the dense, batched and served kernels, plus
// the storage codecs and the deterministic FP64 block reduction.
//
// A "domain" is a box of cells stored in an arena of Q planes with plane
// stride p.n; its cells start at arena index p.base and run
// (z*NY + y)*NX + x. The dense solver is one domain at base 0; the batched
// and served forms place many domains in one arena. Whatever the launch
// shape, every cell goes through cell3()/cell2() below, so the arithmetic of
// all forms is the same instruction stream.
//
// Reference arithmetic:
//   cell3   common_d3_step.wgsl:224-400 (step) + common_d3_force.wgsl:171-283
//   cell2   lbm_step.wgsl:137-270 (step) + lbm_force.wgsl main
#pragma once

#include <type_traits>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "dense.cuh"
#include "geometry.cuh"
#include "lattice.cuh"

namespace lbm {

// 1 / c_s^2. The moving-wall term 2 w_i rho_w (e_i . u_w) / c_s^2 multiplies
// by it: a division there is an IEEE-rounded divide with a slow-path branch
// per link, which in the 3D AMR substep (most tile cells near the body) cost
// a third of the kernel's instructions.
constexpr float kInvCS2 = 3.0f;

// ---- storage codecs --------------------------------------------------------
// FP32 planes hold f itself; the 16-bit planes hold (f - off_i) * scale (see
// Pack), rounded to nearest even. Arithmetic is f32 throughout.
#ifndef LBM_STREAMING_STORES
#define LBM_STREAMING_STORES 0
#endif
template <typename S> struct Codec;
template <> struct Codec<float> {
  static __device__ __forceinline__ float ld(const float *p, int, const Pack &) { return __ldg(p); }
  static __device__ __forceinline__ void st(float *p, float v, int, const Pack &) {
    if (LBM_STREAMING_STORES) __stcs(p, v); else *p = v;
  }
};
// FP32 populations that other blocks of the same launch write (a persistent
// kernel): read from L2.
struct CgFloat {
  float v;
};
template <> struct Codec<CgFloat> {
  static __device__ __forceinline__ float ld(const CgFloat *p, int, const Pack &) { return __ldcg(&p->v); }
  static __device__ __forceinline__ void st(CgFloat *p, float v, int, const Pack &) { p->v = v; }
};
template <> struct Codec<__half> {
  static __device__ __forceinline__ float dec(__half v, int i, const Pack &k) {
    return fmaf(__half2float(v), k.inv, k.off[i]);
  }
  static __device__ __forceinline__ float ld(const __half *p, int i, const Pack &k) { return dec(__ldg(p), i, k); }
  static __device__ __forceinline__ void st(__half *p, float v, int i, const Pack &k) {
    *p = __float2half_rn(fmaf(v, k.scale, k.noff[i]));
  }
};
template <> struct Codec<__nv_bfloat16> {
  static __device__ __forceinline__ float dec(__nv_bfloat16 v, int i, const Pack &k) {
    return fmaf(__bfloat162float(v), k.inv, k.off[i]);
  }
  static __device__ __forceinline__ float ld(const __nv_bfloat16 *p, int i, const Pack &k) { return dec(__ldg(p), i, k); }
  static __device__ __forceinline__ void st(__nv_bfloat16 *p, float v, int i, const Pack &k) {
    *p = __float2bfloat16_rn(fmaf(v, k.scale, k.noff[i]));
  }
};

// ---- deterministic block reduction + last-block finish -------------------

// The warp's sums of 8 values per lane: v8[lane % 8] of lane k holds value k's
// sum, k = 0..7. Each of the first three rounds halves the values a lane
// carries (it keeps one half and adds its partner's copy of it), so 9
// exchanges do what 8 trees of 5 do, in a fixed order.
__device__ __forceinline__ double warp_sum8(const double (&v)[8]) {
  const int lane = threadIdx.x & 31;
  double a[4], b[2], c;
  const bool h4 = lane & 4, h2 = lane & 2, h1 = lane & 1;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double keep = h4 ? v[k + 4] : v[k], give = h4 ? v[k] : v[k + 4];
    a[k] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double keep = h2 ? a[k + 2] : a[k], give = h2 ? a[k] : a[k + 2];
    b[k] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
  }
  {
    const double keep = h1 ? b[1] : b[0], give = h1 ? b[0] : b[1];
    c = keep + __shfl_xor_sync(0xffffffffu, give, 1);
  }
  c += __shfl_xor_sync(0xffffffffu, c, 8);
  c += __shfl_xor_sync(0xffffffffu, c, 16);
  return c;
}

template <int NV, int THREADS>
__device__ __forceinline__ void block_sum(double (&v)[NV], double *sm) {
  constexpr int NW = THREADS / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if constexpr (NV == 8) {
    const double c = warp_sum8(v);
    __syncthreads();
    if (lane < 8) sm[lane * NW + warp] = c;
  } else {
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    __syncthreads();
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < NV; ++k) sm[k * NW + warp] = v[k];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double t = lane < NW ? sm[k * NW + lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (o < NW) t += __shfl_down_sync(0xffffffffu, t, o);
      v[k] = t;
    }
  }
}

// The fixed-order sum of nparts partials by one warp (lane = threadIdx.x):
// lane l adds partials l, l + 32, ... in order, then the warp's fixed tree.
// Every caller that sums the same partials this way gets the same bits.
template <int NV>
__device__ __forceinline__ void sum_partials_warp(const double *partials, int nparts, double *out) {
  const int lane = threadIdx.x & 31;
  double acc[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) acc[k] = 0.0;
  for (int j = lane; j < nparts; j += 32)
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] += __ldcg(&partials[(int64_t)j * NV + k]);
  if constexpr (NV == 8) {
    const double c = warp_sum8(acc);
    if (lane < 8) out[lane] = c;
    __syncwarp();  // lane 0 may read the whole sum next
  } else {
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_down_sync(0xffffffffu, acc[k], o);
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < NV; ++k) out[k] = acc[k];
  }
}

// Writes this block's partial (thread 0 holds it), and if this block is the
// last of `nparts` to do so, sums all partials in a fixed order into `out`
// and re-arms the ticket counter for the next step. Only warp 0 takes part:
// the other warps leave as soon as their share is in `sm`, so they do not
// hold the SM while thread 0 waits on its fence and ticket. Returns true in
// warp 0 of the last block.
template <int NV, int THREADS>
__device__ bool finish_sum(const double (&v)[NV], double *partials, unsigned int *counter,
                           int nparts, int part, double *out, double *) {
  if (threadIdx.x >= 32) return false;
  const int lane = threadIdx.x;
  unsigned int last = 0u;
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) partials[(int64_t)part * NV + k] = v[k];
    __threadfence();
    const unsigned int ticket = atomicAdd(counter, 1u);
    last = ticket == (unsigned int)(nparts - 1) ? 1u : 0u;
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return false;
  __threadfence();
  sum_partials_warp<NV>(partials, nparts, out);
  if (lane == 0) *counter = 0u;
  return true;
}

__device__ __forceinline__ float sponge_weight(float d, float sw) {
  if (sw <= 0.0f) return 0.0f;
  float w = fminf(fmaxf(1.0f - d / sw, 0.0f), 1.0f);
  return w * w * (3.0f - 2.0f * w);
}

__device__ __forceinline__ double finite_or_zero(float v, double &bad) {
  if (isfinite(v)) return (double)v;
  bad += 1.0;
  return 0.0;
}

// Force/torque contribution of one cell to the body (f32, as the reference
// forms it per cell).
struct CellForce {
  float fx = 0.f, fy = 0.f, fz = 0.f, tx = 0.f, ty = 0.f, tz = 0.f;
};

// A thread's FP64 running sum of cell contributions; a non-finite cell
// component is counted and contributes 0 (the reference's safeFixed).
struct ForceAcc {
  double v[6] = {0, 0, 0, 0, 0, 0};
  double bad = 0.0;
  __device__ __forceinline__ void add(const CellForce &c) {
    v[0] += finite_or_zero(c.fx, bad);
    v[1] += finite_or_zero(c.fy, bad);
    v[2] += finite_or_zero(c.fz, bad);
    v[3] += finite_or_zero(c.tx, bad);
    v[4] += finite_or_zero(c.ty, bad);
    v[5] += finite_or_zero(c.tz, bad);
  }
};

// The block's FP64 partial of the force of its cells, one per thread, written
// to partials[part]; the caller's stream sums the partials after the launch.
// Most blocks of a force region hold no cell with a contribution (the region
// is the body's box; only its shell touches the body): when every thread's
// components are 0 the block writes its zero partial directly.
// The other blocks are a small domain's critical path. They add groups of
// eight lanes out of shared memory, one thread per group and component (three
// levels of independent adds), and only then exchange between lanes: in the
// association of block_sum (lanes 4, 2, 1, 8, 16 apart, then warps), so with
// its bits, in 6 instead of 14 dependent steps and one barrier instead of
// three. us per step with block_sum and with this: D3Q19 FP32 sphere in 32^3
// 6.94 -> 5.17, 64^3 9.89 -> 8.29, D3Q27 box in 100^3 47.7 -> 45.7, 256x128x128
// 104.2 -> 103.7; D2Q9 512^2 6.7 -> 5.0, 200x150 5.7 -> 4.0. (With no sum at
// all the first takes 5.1.)
template <int THREADS>
__device__ __forceinline__ void publish_force(const CellForce &c, double *partials, int part) {
  constexpr int kGroups = THREADS / 8;  // of a component; 4 per warp
  static_assert(THREADS >= 64 && THREADS <= 256 && 7 * kGroups <= THREADS, "one thread per group and component");
  __shared__ float4 sm[7 * THREADS / 4];
  const float x[6] = {c.fx, c.fy, c.fz, c.tx, c.ty, c.tz};
  float *row = reinterpret_cast<float *>(sm) + threadIdx.x;
  float bad = 0.f;
  bool mine = false;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const bool ok = isfinite(x[k]);
    row[k * THREADS] = ok ? __fadd_rn(x[k], 0.f) : 0.f;  // -0 counts as 0
    if (!ok) bad += 1.f;
    mine = mine || x[k] != 0.f;
  }
  row[6 * THREADS] = bad;
  double *out = partials + (int64_t)part * kForceSlots;
  if (!__syncthreads_or(mine)) {
    if (threadIdx.x < kForceSlots) out[threadIdx.x] = 0.0;
    return;
  }
  if (threadIdx.x >= 7 * kGroups) return;
  const int k = threadIdx.x / kGroups, g = threadIdx.x % kGroups;
  const float4 lo = sm[2 * threadIdx.x], hi = sm[2 * threadIdx.x + 1];  // lanes 8g .. 8g + 7 of component k
  double v = (((double)lo.x + (double)hi.x) + ((double)lo.z + (double)hi.z)) +
             (((double)lo.y + (double)hi.y) + ((double)lo.w + (double)hi.w));
  const int in_warp = 7 * kGroups - (int)(threadIdx.x & ~31u);  // threads of this warp still here
  const unsigned mask = in_warp >= 32 ? 0xffffffffu : (1u << in_warp) - 1u;
  v += __shfl_xor_sync(mask, v, 1);
  v += __shfl_xor_sync(mask, v, 2);
#pragma unroll
  for (int o = kGroups / 2; o >= 4; o >>= 1) v += __shfl_xor_sync(mask, v, o);
  if (g == 0) out[k] = v;
  if (threadIdx.x == 0) out[7] = 0.0;
}

// The sum of a launch's force partials, spread over the first blocks of a
// later launch so that no block waits on more than a round or two of loads:
// up to kSumOne of them are one block's (one to four per thread, then the
// block tree). More are cut into groups of kSumGroup: block b adds those of
// group b, one per thread, into groups[b]; the last group to finish (a
// ticket behind one fence per group, not per partial) sums the groups in
// order into out. The order depends only on nparts (threads past kSumGroup
// add zeros), so every launch that sums the same partials gets the same bits.
template <int THREADS>
__device__ __forceinline__ void sum_partials_grouped(const double *partials, int nparts, double *groups,
                                                     unsigned int *counter, double *out, int b) {
  static_assert(THREADS >= kSumGroup, "one partial per thread");
  __shared__ double sm[kForceSlots * (THREADS / 32)];
  double acc[kForceSlots];
  const int j = b * kSumGroup + (int)threadIdx.x;
  const bool mine = threadIdx.x < kSumGroup && j < nparts;
#pragma unroll
  for (int k = 0; k < kForceSlots; ++k) acc[k] = mine ? partials[(int64_t)j * kForceSlots + k] : 0.0;
  if (nparts <= kSumOne) {
    // no second level: no fence and no ticket
    if (threadIdx.x < kSumGroup)
#pragma unroll 1
      for (int m = j + kSumGroup; m < nparts; m += kSumGroup)
#pragma unroll
        for (int k = 0; k < kForceSlots; ++k) acc[k] += partials[(int64_t)m * kForceSlots + k];
    block_sum<kForceSlots, THREADS>(acc, sm);
    if (threadIdx.x == 0)
#pragma unroll
      for (int k = 0; k < kForceSlots; ++k) out[k] = acc[k];
    return;
  }
  block_sum<kForceSlots, THREADS>(acc, sm);
  finish_sum<kForceSlots, THREADS>(acc, groups, counter, sum_groups(nparts), b, out, sm);
}

// Returns true in the block that summed the partials (the last to finish).
template <int THREADS>
__device__ __forceinline__ bool reduce_force(const ForceAcc &a, double *partials, unsigned int *counter,
                                             int nparts, int part, double *out) {
  __shared__ double sm[kForceSlots * (THREADS / 32)];
  double v[kForceSlots];
#pragma unroll
  for (int k = 0; k < 6; ++k) v[k] = a.v[k];
  v[6] = a.bad;
  v[7] = 0.0;
  block_sum<kForceSlots, THREADS>(v, sm);
  return finish_sum<kForceSlots, THREADS>(v, partials, counter, nparts, part, out, sm);
}

// Cell `cell` of a plane. 16-bit storage addresses it by a 32-bit byte offset
// from the plane's base, which is the same for the whole block (a plane of
// fewer than 2^31 cells has fewer than 2^32 bytes): its step is bound by
// instruction issue, and a 64-bit address per population was a fifth of it
// (256x128x128 sphere, 104.6 -> 99.2 us per step; D3Q27 150.9 -> 137.3). FP32
// planes can be larger, and their step is bound by memory (103.6 against
// 104.4 us with the offsets).
template <typename S> __device__ __forceinline__ S *plane_cell(S *plane, int cell) {
  if constexpr (sizeof(S) == 2) {
    using B = std::conditional_t<std::is_const_v<S>, const char, char>;
    return reinterpret_cast<S *>(reinterpret_cast<B *>(plane) + (size_t)((unsigned)cell * 2u));
  } else {
    return plane + cell;
  }
}

// The BGK collision with Guo forcing and the sponge blend, written over
// opposite pairs (e, -e). With a = (1-s) omega rho, b = (1-s)(1 - omega/2)
// (s the sponge weight) and per direction eu = e.u, eF = e.F:
//   (1-s)[omega feq + S](+-e) = w (A +- B),
//     A = c0 + eu (4.5 a eu + 9 b eF),   c0 = a (1 - 1.5 u.u) - 3 b u.F
//     B = 3 a eu + 3 b eF
//   f_out(+-e) = (1-s)(1-omega) f(+-e) + s f_far(+-e) + w (A +- B).
// The products of w with a, b and c0 are formed once per weight class, so
// a pair costs about a dozen FP32 instructions. Outside the sponge (s = 0)
// this is the plain BGK + Guo update. The reference's per-direction form
// (common_d3_step.wgsl:331-357) and mix() blend (common_sponge.wgsl:7-11),
// reassociated.
// Where a cell's post-collision populations go: MemSink stores them (the
// step); NullSink drops them (a force-only pass, whose collision the
// compiler then removes as dead code).
template <typename S> struct MemSink {
  S *fo;
  int64_t n;
  int cell;
  const Pack &pk;
  __device__ __forceinline__ void put(int i, float v) { Codec<S>::st(plane_cell(fo + (int64_t)i * n, cell), v, i, pk); }
};
// The D2Q9 update's: with plane_cell's offsets its kernels, two cells a thread
// in a batch, spilled more (a 16-bit batch's step: 200 bytes of stores instead
// of 128).
template <typename S> struct MemSink2 {
  S *fo;
  int64_t n;
  int cell;
  const Pack &pk;
  __device__ __forceinline__ void put(int i, float v) { Codec<S>::st(fo + (int64_t)i * n + cell, v, i, pk); }
};
struct NullSink {
  __device__ __forceinline__ void put(int, float) {}
};

// TRT (dw = omega_- - omega != 0): the odd part of each pair relaxes at
// omega_- instead, in the reference's delta form (plans/TRT.md sec 8.0(1)):
//   f_i += -dw (f_i^- - feq_i^-) - dw/2 S_i^-,
//   f_i^- = (f_i - f_j)/2, feq_i^- = 3 w rho e.u, S_i^- = 3 w e.F,
// the odd forcing prefactor becoming (1 - omega_-/2); the sponge blend
// scales it by (1 - s) like the rest of the collided value, and f_j takes
// the negative. TRT = false is the BGK loop alone (dw ignored); the kernels
// pick the instantiation from dw != 0 per launch, so the BGK code keeps its
// register allocation.
//
// Every operation is explicit (no contraction left to the compiler), so that
// a cell's bits do not depend on the kernel it is updated in. Only the
// nonzero components of e enter e.u and e.F (edot): written as ex*ux + ey*uy
// + ez*uz the products with 0 stay in the code (0 * NaN is not 0), two of
// them per direction pair and dot product.
__device__ __forceinline__ float edot(int ex, int ey, int ez, float x, float y, float z) {
  float v = x;
  bool have = ex != 0, neg = ex < 0;
  if (ey) {
    if (!have) { v = y; neg = ey < 0; }
    else if ((ey < 0) == neg) v = __fadd_rn(v, y);
    else if (neg) { v = __fsub_rn(y, v); neg = false; }
    else v = __fsub_rn(v, y);
    have = true;
  }
  if (ez) {
    if (!have) { v = z; neg = ez < 0; }
    else if ((ez < 0) == neg) v = __fadd_rn(v, z);
    else if (neg) { v = __fsub_rn(z, v); neg = false; }
    else v = __fsub_rn(v, z);
  }
  return neg ? -v : v;
}

template <class L, int Q, class Sink, bool TRT = false>
__device__ __forceinline__ void collide_store(const float (&f)[Q], float rho, float ux, float uy, float uz, float Fx,
                                              float Fy, float Fz, float omg, float spw, const float *ftarget,
                                              Sink &sink, float dw = 0.f) {
  float usq = __fmaf_rn(ux, ux, __fmul_rn(uy, uy));
  float uF = __fmaf_rn(ux, Fx, __fmul_rn(uy, Fy));
  if (L::D == 3) {
    usq = __fmaf_rn(uz, uz, usq);
    uF = __fmaf_rn(uz, Fz, uF);
  }
  const float ks = __fsub_rn(1.0f, spw);
  const float a = __fmul_rn(__fmul_rn(omg, ks), rho);
  const float b = __fmul_rn(__fmaf_rn(-0.5f, omg, 1.0f), ks);
  const float keep = __fmul_rn(__fsub_rn(1.0f, omg), ks);
  const float c0 = __fmaf_rn(a, __fmaf_rn(-1.5f, usq, 1.0f), __fmul_rn(__fmul_rn(-3.0f, b), uF));
  auto blend = [&](int i, float v) { return __fmaf_rn(spw, ftarget[i], v); };
  sink.put(0, __fmaf_rn(keep, f[0], blend(0, __fmul_rn(L::w(0), c0))));
  const float kd = TRT ? __fmul_rn(ks, -dw) : 0.f, nrho3 = TRT ? __fmul_rn(-3.0f, rho) : 0.f;
  float a45, b9, a3, b3, wc0;  // per weight class, the classes in direction order
#pragma unroll
  for (int i = 1; i < Q; ++i) {
    const int j = L::opp(i);
    const float w = L::w(i);
    if (i == 1 || L::w(i) != L::w(i - 1)) {
      a45 = __fmul_rn(4.5f * w, a);
      b9 = __fmul_rn(9.0f * w, b);
      a3 = __fmul_rn(3.0f * w, a);
      b3 = __fmul_rn(3.0f * w, b);
      wc0 = __fmul_rn(w, c0);
    }
    if (j < i) continue;
    const float eu = edot(L::ex(i), L::ey(i), L::ez(i), ux, uy, uz);
    const float eF = edot(L::ex(i), L::ey(i), L::ez(i), Fx, Fy, Fz);
    const float t = __fmaf_rn(b9, eF, __fmul_rn(a45, eu));
    const float A = __fmaf_rn(eu, t, wc0);
    const float B = __fmaf_rn(a3, eu, __fmul_rn(b3, eF));
    float oi = __fmaf_rn(keep, f[i], blend(i, __fadd_rn(A, B)));
    float oj = __fmaf_rn(keep, f[j], blend(j, __fsub_rn(A, B)));
    if (TRT) {
      const float odd = __fmul_rn(w, __fmaf_rn(1.5f, eF, __fmul_rn(nrho3, eu)));
      const float D = __fmaf_rn(0.5f, __fsub_rn(f[i], f[j]), odd);
      oi = __fmaf_rn(kd, D, oi);
      oj = __fmaf_rn(-kd, D, oj);
    }
    sink.put(i, oi);
    sink.put(j, oj);
  }
}

// rho and rho u* from the gathered populations, summed over opposite pairs.
template <class L, int Q>
__device__ __forceinline__ void moments(const float (&f)[Q], float &rho, float &mx, float &my, float &mz) {
  rho = f[0];
  mx = my = mz = 0.f;
  bool hx = false, hy = false, hz = false;  // whether a sum has begun (compile-time)
#pragma unroll
  for (int i = 1; i < Q; ++i) {
    const int j = L::opp(i);
    if (j < i) continue;
    const float s = f[i] + f[j], d = f[i] - f[j];
    rho += s;
    if (L::ex(i)) { mx = L::ex(i) > 0 ? (hx ? mx + d : d) : mx - d; hx = true; }
    if (L::ey(i)) { my = L::ey(i) > 0 ? (hy ? my + d : d) : my - d; hy = true; }
    if (L::ez(i)) { mz = L::ez(i) > 0 ? (hz ? mz + d : d) : mz - d; hz = true; }
  }
}

__device__ __forceinline__ float sponge_weight_inv(float d, float inv_sw) {
  const float w = fminf(fmaxf(__fmaf_rn(-d, inv_sw, 1.0f), 0.0f), 1.0f);
  return __fmul_rn(__fmul_rn(w, w), __fmaf_rn(-2.0f, w, 3.0f));
}

// ---- row-major walks without divisions --------------------------------------
// A thread of a multi-domain launch visits cells c0, c0 + step, c0 + 2 step,
// ... of one domain. Its first cell takes the divisions; every later one
// adds the step's own decomposition (dx, dy, dz) with one carry per axis
// (x + dx < 2 nx and y + dy + 1 < 2 ny, so a single subtraction suffices).
struct CellWalk {
  int x, y, z;
  int dx, dy, dz;
  int nx, ny;
  __device__ __forceinline__ CellWalk(int c0, int step, int nx_, int ny_) : nx(nx_), ny(ny_) {
    const int r = c0 / nx;
    x = c0 - r * nx;
    y = r % ny;
    z = r / ny;
    const int rs = step / nx;
    dx = step - rs * nx;
    dy = rs % ny;
    dz = rs / ny;
  }
  __device__ __forceinline__ void advance() {
    x += dx;
    y += dy;
    z += dz;
    if (x >= nx) { x -= nx; ++y; }
    if (y >= ny) { y -= ny; ++z; }
  }
};

// The D3Q27 directions (D3Q19 their first 19), as a table in constant
// memory for loops over a runtime direction index.
struct DirTable {
  signed char ex[27], ey[27], ez[27];
};
constexpr DirTable make_dirs() {
  DirTable t{};
  for (int i = 0; i < 27; ++i) {
    t.ex[i] = (signed char)detail::ex27(i);
    t.ey[i] = (signed char)detail::ey27(i);
    t.ez[i] = (signed char)detail::ez27(i);
  }
  return t;
}
static __constant__ DirTable c_dirs = make_dirs();

// The directions of a cell at pos whose pull source lies inside the body, as
// phi3 < 0 decides.
//  * Sphere: phi3 < 0 is sqrt(d^2) < a, and as the square root rounds
//    monotonically that is d^2 < a2, the smallest number whose root reaches
//    a (p.ball2). With the squares of the three offsets per axis shared, a
//    link costs two additions and a comparison instead of a square root of
//    its own: 18 roots were most of a near cell's time.
//  * Box and spheroid: from the source's position in the body's frame, the
//    cell's less a combination of the frame's columns, so a link costs no
//    rotation: the spheroid's side of its equation rr = 1 needs no Newton
//    step, the box's distance no call. That position is rounded differently
//    from phi3's, so where the outcome is within a margin far above the
//    rounding (1e-3), phi3 itself decides.
//  * Under a moving window a link may lead to another image of the body than
//    the cell's; then phi3 decides too. WIN: instantiated for windowed domains,
//    where the other links (and a sphere's) are tested in the body's frame as
//    well. (With phi3 for every windowed link, D3Q19 FP32 sphere in 128^3 67.2 us
//    per step against 62.9; D3Q27 FP16 rounded box in 246x60x19, window on all
//    axes, 42.0 against 25.3. It is a copy of its own because its registers
//    would make every kernel that calls the other one spill.)
template <int Q, bool WIN>
static __device__ __noinline__ unsigned solid_links_call(float x, float y, float z, const lbm_body *b, const Win *w) {
  const Q4 q = {b->qw, b->qx, b->qy, b->qz};
  const V3 dl = body_delta({x, y, z}, *b, *w);
  // whether every link sees the cell's image of the body
  bool one = !w->on;
  if (WIN)
    one = (w->n[0] <= 0.f || fabsf(dl.x) < 0.5f * w->n[0] - 1.5f) &&
          (w->n[1] <= 0.f || fabsf(dl.y) < 0.5f * w->n[1] - 1.5f) &&
          (w->n[2] <= 0.f || fabsf(dl.z) < 0.5f * w->n[2] - 1.5f);
  const V3 l0 = q_rot_inv(q, dl);
  const V3 cx = q_rot_inv(q, {1.f, 0.f, 0.f}), cy = q_rot_inv(q, {0.f, 1.f, 0.f}), cz = q_rot_inv(q, {0.f, 0.f, 1.f});
  const bool spheroid = b->shape == LBM_SHAPE_SPHEROID, box = b->shape == LBM_SHAPE_ROUNDBOX;
  const float ia2 = 1.f / (b->a * b->a), ic2 = 1.f / (b->c * b->c);
  unsigned solid = 0u;
#pragma unroll 1
  for (int i = 1; i < Q; ++i) {
    const float ex = (float)c_dirs.ex[i], ey = (float)c_dirs.ey[i], ez = (float)c_dirs.ez[i];
    const V3 l = {l0.x - (ex * cx.x + ey * cy.x + ez * cz.x), l0.y - (ex * cx.y + ey * cy.y + ez * cz.y),
                  l0.z - (ex * cx.z + ey * cy.z + ez * cz.z)};
    float d = 0.f;  // its sign, where |d| is above the margin
    if (spheroid) {
      d = (l.x * l.x + l.y * l.y) * ia2 + l.z * l.z * ic2 - 1.f;
    } else if (box) {
      const float hx = fabsf(l.x) - (b->a - b->r), hy = fabsf(l.y) - (b->b - b->r), hz = fabsf(l.z) - (b->c - b->r);
      const float mx = fmaxf(hx, 0.f), my = fmaxf(hy, 0.f), mz = fmaxf(hz, 0.f);
      d = sqrtf(mx * mx + my * my + mz * mz) + fminf(fmaxf(hx, fmaxf(hy, hz)), 0.f) - b->r;
    } else if (WIN) {
      d = sqrtf(l.x * l.x + l.y * l.y + l.z * l.z) - b->a;
    }
    const bool cut = fabsf(d) > 1e-3f && one ? d < 0.f : phi3_call(x - ex, y - ey, z - ez, b, w) < 0.f;
    solid |= cut ? 1u << i : 0u;
  }
  return solid;
}

template <int Q, bool WIN>
__device__ __forceinline__ unsigned solid_links(const StepParams &p, const V3 &pos) {
  using L = Lattice<Q>;
  if (WIN || p.body.shape != LBM_SHAPE_SPHERE || p.win.on)
    return solid_links_call<Q, WIN>(pos.x, pos.y, pos.z, &p.body, &p.win);
  unsigned solid = 0u;
  float xx[3], yy[3], zz[3];  // of the sources at e = -1, 0, +1
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const float o = (float)(e - 1);
    const float dx = (pos.x - o) - p.body.cx, dy = (pos.y - o) - p.body.cy, dz = (pos.z - o) - p.body.cz;
    xx[e] = __fmul_rn(dx, dx);
    yy[e] = __fmul_rn(dy, dy);
    zz[e] = __fmul_rn(dz, dz);
  }
#pragma unroll
  for (int i = 1; i < Q; ++i)
    if (__fadd_rn(__fadd_rn(xx[L::ex(i) + 1], yy[L::ey(i) + 1]), zz[L::ez(i) + 1]) < p.ball2) solid |= 1u << i;
  return solid;
}

// ---- 3D cell update ---------------------------------------------------------
// Pull-stream (periodic sources, then bounce-back patches: body first with
// Ladd's correction at local rho_w, then walls), moments, Guo forcing with
// the chi penalty, BGK collide, sponge blend, SOLID_EQ. When `force` is set
// (the caller's block can see the body) the cell's force/torque contribution
// is returned in cf.

// What the body and the walls mean for a cell: its distance, the body's
// velocity there, whether it is held at the body's state (SOLID_EQ), and the
// links to patch.
struct Geom3 {
  float phi;
  V3 us;
  unsigned solid, wall;
  bool in_solid;
};

// (x, y, z): the cell in the domain's own coordinates. LINKS = false: of a
// domain without a bounce-back body. WIN: as solid_links_call.
template <int Q, bool LINKS, bool WIN = false>
__device__ __forceinline__ Geom3 classify3(const StepParams &p, int x, int y, int z) {
  using L = Lattice<Q>;
  const int nx = p.nx, ny = p.ny, nz = p.nzg;
  const V3 pos = {(float)x, (float)y, (float)z};
  Geom3 g{1e30f, {0.f, 0.f, 0.f}, 0u, 0u, false};
  bool see = p.has_body;
  if (see && p.nbox_on) {
    int dx = x - p.nbox[0], dy = y - p.nbox[2], dz = z - p.nbox[4];
    dx += dx < 0 ? nx : 0;
    dy += dy < 0 ? ny : 0;
    dz += dz < 0 ? nz : 0;
    see = dx <= p.nbox[1] - p.nbox[0] && dy <= p.nbox[3] - p.nbox[2] && dz <= p.nbox[5] - p.nbox[4];
  }
  if (see) {
    g.phi = phi3(pos, p.body, p.win);
    g.us = body_velocity3(pos, p.body, p.win);
  }
  const bool bbody = LINKS && p.has_body && p.bb;
  // A cell held at the body's state uses nothing it pulls, so its links need
  // no patch. For the others a link reaches a solid source only from within
  // |e| <= sqrt(3) of the surface, as a signed distance is 1-Lipschitz.
  g.in_solid = p.solid_eq && bbody && g.phi < 0.f;
  if (g.in_solid) return g;
  if (bbody && g.phi < 2.5f) g.solid = solid_links<Q, WIN>(p, pos);
  const bool at_wall = (p.wall_x && (x == 0 || x == nx - 1)) || (p.wall_y && (y == 0 || y == ny - 1)) ||
                       (p.wall_z && (z == 0 || z == nz - 1));
  if (at_wall) {
#pragma unroll
    for (int i = 1; i < Q; ++i) {
      const int sx = x - L::ex(i), sy = y - L::ey(i), sz = z - L::ez(i);
      const bool out = (p.wall_x && (sx < 0 || sx >= nx)) || (p.wall_y && (sy < 0 || sy >= ny)) ||
                       (p.wall_z && (sz < 0 || sz >= nz));
      if (out) g.wall |= 1u << i;
    }
  }
  return g;
}

// A 3D cell's position in window coordinates.
__device__ __forceinline__ V3 window_pos(const StepParams &p, const V3 &pos) {
  return {win_coord1(pos.x, win_offset1(p.body.cx, p.win.anchor[0], p.win.n[0]), p.win.n[0]),
          win_coord1(pos.y, win_offset1(p.body.cy, p.win.anchor[1], p.win.n[1]), p.win.n[1]),
          win_coord1(pos.z, win_offset1(p.body.cz, p.win.anchor[2], p.win.n[2]), p.win.n[2])};
}

// The sponge weight of a 3D cell (p.sponge_w > 0), from its position in window
// coordinates: under a moving window the band travels with the body.
__device__ __forceinline__ float sponge3(const StepParams &p, const V3 &pos) {
  const float dx = p.sax ? fminf(pos.x, (float)(p.nx - 1) - pos.x) : 1e30f;
  const float dy = p.say ? fminf(pos.y, (float)(p.ny - 1) - pos.y) : 1e30f;
  const float dz = p.saz ? fminf(pos.z, (float)(p.nzg - 1) - pos.z) : 1e30f;
  return sponge_weight_inv(fminf(dx, fminf(dy, dz)), p.sponge_inv);
}

// Everything after the pull gather, for one cell: bounce-back patches,
// moments, forcing, collision into `sink`, mac, force. `fi` is the domain's
// base in the input arena (own-cell loads of the bounce-back patches).
template <int Q, typename S, class Sink, bool TRT = false, bool LINKS = true>
__device__ __forceinline__ void cell3_core(const S *__restrict__ fi, float (&f)[Q], float *__restrict__ mac,
                                           const StepParams &p, const Geom3 &g, int x, int y, int z, bool force,
                                           CellForce &cf, Sink &sink) {
  using L = Lattice<Q>;
  // z indexes the stored planes; the physics (body, walls, sponge, reach
  // box) sees the domain's own z, which for a slab is offset by p.zoff in a
  // domain p.nzg planes deep (both the identity for a whole domain)
  const int nx = p.nx, ny = p.ny, nz = p.nzg;
  const int64_t n = p.n;
  const int cell = (z * ny + y) * nx + x;
  z += p.zoff;
  const V3 pos = {(float)x, (float)y, (float)z};
  const float phi = g.phi;
  const V3 us = g.us;
  const unsigned solid = LINKS ? g.solid : 0u, wall = g.wall;
  const bool bbody = LINKS && p.has_body && p.bb, in_solid = LINKS && g.in_solid;
  float fbx = 0.f, fby = 0.f, fbz = 0.f;

  // 1b. Bounce-back links, all classified already (classify3): the cell's own
  // populations that the patches read are loaded together, so a near cell
  // waits for one memory latency instead of one per solid link. (The rest
  // direction never patches: its source is the cell itself.)
  {
    if (solid | wall) {
      const bool all = bbody && p.rho_w_local && phi < 2.f;  // rho_w sums every population
      float own[Q];
#pragma unroll
      for (int i = 0; i < Q; ++i)
        own[i] = (all || (((solid | wall) >> L::opp(i)) & 1u)) ? Codec<S>::ld(fi + (int64_t)i * n + cell, i, p.pk)
                                                                 : 0.f;
      float rhoW = 1.f;
      if (all) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < Q; ++i) s += own[i];
        rhoW = s;
      }
#pragma unroll
      for (int i = 1; i < Q; ++i) {
        const int ex = L::ex(i), ey = L::ey(i), ez = L::ez(i);
        const float fopp = own[L::opp(i)];
        if ((solid >> i) & 1u) {
          const float corr =
              2.f * L::w(i) * rhoW * ((float)ex * us.x + (float)ey * us.y + (float)ez * us.z) * kInvCS2;
          f[i] = fopp + corr;
          if (phi >= 0.f) {
            const float m = 2.f * fopp + corr;
            fbx += -(float)ex * m;
            fby += -(float)ey * m;
            fbz += -(float)ez * m;
          }
        } else if ((wall >> i) & 1u) {
          f[i] = fopp;
        }
      }
    }
  }

  // 2. Moments.
  float rho, mx, my, mz;
  moments<L, Q>(f, rho, mx, my, mz);
  const float rhoDen = fmaxf(rho, 1e-6f);
  const float inv = 1.0f / rhoDen;
  const float uxs = mx * inv, uys = my * inv, uzs = mz * inv;

  // 3. Solid coupling and Guo forcing: u = u* + F / (2 rho).
  const float chi = (p.has_body && !p.bb) ? chi_from_phi(phi, p.chi_eps) : 0.f;
  const float rc = rho * chi;
  const float Fx = __fmaf_rn(rc, us.x - uxs, p.fx);
  const float Fy = __fmaf_rn(rc, us.y - uys, p.fy);
  const float Fz = __fmaf_rn(rc, us.z - uzs, p.fz);
  const float hinv = 0.5f * inv;
  const float ux = fmaf(Fx, hinv, uxs);
  const float uy = fmaf(Fy, hinv, uys);
  const float uz = fmaf(Fz, hinv, uzs);

  float spw = 0.f;
  if (p.sponge_w > 0.f) spw = sponge3(p, p.win.on ? window_pos(p, pos) : pos);

  // 4. Collide + sponge blend, 5. solid interior held at feq(1, u_body).
  if (!in_solid) {
    collide_store<L, Q, Sink, TRT>(f, rho, ux, uy, uz, Fx, Fy, Fz, p.omega, spw, p.ftarget, sink, p.trt_dw);
  } else {
    const float ussq = us.x * us.x + us.y * us.y + us.z * us.z;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const float w = L::w(i);
      const float eu = (float)L::ex(i) * us.x + (float)L::ey(i) * us.y + (float)L::ez(i) * us.z;
      sink.put(i, w * (1.f + 3.f * eu + 4.5f * eu * eu - 1.5f * ussq));
    }
  }
  if (p.write_mac) {
    float4 m = in_solid ? make_float4(1.f, us.x, us.y, us.z) : make_float4(rho, ux, uy, uz);
    reinterpret_cast<float4 *>(mac + 4 * p.base)[cell] = m;
  }

  // Force on the body from this cell (bounce-back links were summed above).
  if (force) {
    if (bbody) {
      if (p.swept && fabsf(phi) < p.swept_band) {
        const bool solid_now = phi < 0.f;
        const bool solid_next = phi3_ahead(pos, p.body, 1.f, p.win) < 0.f;
        if (solid_now != solid_next) {
          float cx = 0.f, cy = 0.f, cz = 0.f;
#pragma unroll
          for (int i = 0; i < Q; ++i) {
            const float v = Codec<S>::ld(fi + (int64_t)i * n + cell, i, p.pk);
            cx += v * (float)L::ex(i);
            cy += v * (float)L::ey(i);
            cz += v * (float)L::ez(i);
          }
          if (!solid_now) { fbx += cx; fby += cy; fbz += cz; }
          else { fbx += -cx; fby += -cy; fbz += -cz; }
        }
      }
    } else if (p.has_body) {
      const float c2 = chi_from_phi(phi, p.chi_eps);
      if (c2 >= 1e-6f) {
        const float rc2 = rho * c2;
        fbx = -(rc2 * (us.x - uxs));
        fby = -(rc2 * (us.y - uys));
        fbz = -(rc2 * (us.z - uzs));
      }
    }
    const V3 r = body_delta(pos, p.body, p.win);
    const float rx = r.x, ry = r.y, rz = r.z;
    cf.fx = fbx; cf.fy = fby; cf.fz = fbz;
    cf.tx = ry * fbz - rz * fby;
    cf.ty = rz * fbx - rx * fbz;
    cf.tz = rx * fby - ry * fbx;
  }
}


// Pull gather of one cell from the periodic sources.
template <int Q, typename S>
__device__ __forceinline__ void gather3(const S *__restrict__ fi, const StepParams &p, int x, int y, int z,
                                        float (&f)[Q]) {
  using L = Lattice<Q>;
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  const int64_t n = p.n;
  const int nxny = nx * ny;
  const int cell = z * nxny + y * nx + x;
  // Offset of the pull source for e = +1 / -1 on each axis, periodic.
  const int xo_p = x == 0 ? nx - 1 : -1, xo_m = x == nx - 1 ? 1 - nx : 1;
  const int yo_p = y == 0 ? (ny - 1) * nx : -nx, yo_m = y == ny - 1 ? (1 - ny) * nx : nx;
  const int zo_p = z == 0 ? (nz - 1) * nxny : -nxny, zo_m = z == nz - 1 ? (1 - nz) * nxny : nxny;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int ex = L::ex(i), ey = L::ey(i), ez = L::ez(i);
    const int off = (ex == 1 ? xo_p : (ex == -1 ? xo_m : 0)) + (ey == 1 ? yo_p : (ey == -1 ? yo_m : 0)) +
                    (ez == 1 ? zo_p : (ez == -1 ? zo_m : 0));
    f[i] = Codec<S>::ld(plane_cell(fi + (int64_t)i * n, cell + off), i, p.pk);
  }
}

// TRT: the collision is the two-relaxation-time one; callers pass
// p.trt_dw != 0 (see collide_store).
// LINKS: the domain may have a bounce-back body. Its links are decided before
// the gather is issued, as they may take a call, which would have to save the
// populations in flight. Without one (a penalty body, whose distance every
// cell takes) the gather comes first and hides the distance; and without the
// call the update does not spill at the step's 64 registers.
// WIN: as solid_links_call.
template <int Q, typename S, bool TRT = false, bool LINKS = true, bool WIN = false>
__device__ __forceinline__ void cell3(const S *__restrict__ fin, S *__restrict__ fout,
                                      float *__restrict__ mac, const StepParams &p, int x, int y,
                                      int z, bool force, CellForce &cf) {
  const S *fi = fin + p.base;
  Geom3 g;
  if (LINKS) g = classify3<Q, true, WIN>(p, x, y, z + p.zoff);
  float f[Q];
  gather3<Q, S>(fi, p, x, y, z, f);
  if (!LINKS) g = classify3<Q, false>(p, x, y, z + p.zoff);
  MemSink<S> sink{fout + p.base, p.n, (z * p.ny + y) * p.nx + x, p.pk};
  cell3_core<Q, S, MemSink<S>, TRT, LINKS>(fi, f, mac, p, g, x, y, z, force, cf, sink);
}

// cell3 with the collision and the kind of body picked from the domain's
// parameters (warp-uniform branches), for kernels that do not instantiate per
// collision.
template <int Q, typename S>
__device__ __forceinline__ void cell3_any(const S *__restrict__ fin, S *__restrict__ fout,
                                          float *__restrict__ mac, const StepParams &p, int x, int y,
                                          int z, bool force, CellForce &cf) {
  const bool links = p.has_body && p.bb;
  if (p.trt_dw != 0.f) {
    if (links) cell3<Q, S, true, true>(fin, fout, mac, p, x, y, z, force, cf);
    else cell3<Q, S, true, false>(fin, fout, mac, p, x, y, z, force, cf);
  } else {
    if (links) cell3<Q, S, false, true>(fin, fout, mac, p, x, y, z, force, cf);
    else cell3<Q, S, false, false>(fin, fout, mac, p, x, y, z, force, cf);
  }
}

// A cell that only fluid can reach: no body link within reach (or no body),
// no wall on any of its links, and not in the force reduction. For such a
// cell cell3() finds phi = 1e30, u_s = 0 and chi = 0, so its Guo force is the body force alone (rho chi (u_s - u*) = +-0, and
// +-0 + F = F) and nothing is patched; this is that path with the dead
// tests taken out, to the bit. WIN: the domain has a moving window.
template <int Q, typename S, bool TRT = false, bool WIN = false>
__device__ __forceinline__ void cell3_fluid(const S *__restrict__ fin, S *__restrict__ fout,
                                            float *__restrict__ mac, const StepParams &p, int x, int y, int z) {
  using L = Lattice<Q>;
  const S *fi = fin + p.base;
  float f[Q];
  gather3<Q, S>(fi, p, x, y, z, f);
  float rho, mx, my, mz;
  moments<L, Q>(f, rho, mx, my, mz);
  const float inv = 1.0f / fmaxf(rho, 1e-6f);
  const float uxs = mx * inv, uys = my * inv, uzs = mz * inv;
  const float hinv = 0.5f * inv;
  const float ux = fmaf(p.fx, hinv, uxs);
  const float uy = fmaf(p.fy, hinv, uys);
  const float uz = fmaf(p.fz, hinv, uzs);
  float spw = 0.f;
  if (p.sponge_w > 0.f) {
    const V3 pos = {(float)x, (float)y, (float)(z + p.zoff)};
    spw = sponge3(p, WIN ? window_pos(p, pos) : pos);
  }
  const int cell = (z * p.ny + y) * p.nx + x;
  MemSink<S> sink{fout + p.base, p.n, cell, p.pk};
  collide_store<L, Q, MemSink<S>, TRT>(f, rho, ux, uy, uz, p.fx, p.fy, p.fz, p.omega, spw, p.ftarget, sink,
                                       p.trt_dw);
  if (p.write_mac) reinterpret_cast<float4 *>(mac + 4 * p.base)[cell] = make_float4(rho, ux, uy, uz);
}

// Force contribution of one cell without the collision (a free body's
// force pass).
template <int Q, typename S>
__device__ __forceinline__ void cell3_force(const S *__restrict__ fin, const StepParams &p, int x, int y, int z,
                                            CellForce &cf) {
  const S *fi = fin + p.base;
  const Geom3 g = classify3<Q, true>(p, x, y, z + p.zoff);
  float f[Q];
  gather3<Q, S>(fi, p, x, y, z, f);
  NullSink sink;
  cell3_core<Q, S>(fi, f, nullptr, p, g, x, y, z, true, cf, sink);
}

// ---- 2D cell update (D2Q9) ---------------------------------------------------

// Pull gather of one D2Q9 cell from its periodic sources.
template <typename S>
__device__ __forceinline__ void gather2(const S *__restrict__ fi, const StepParams &p, int x, int y, float (&f)[9]) {
  using L = Lattice<9>;
  const int W = p.nx, H = p.ny;
  const int64_t n = p.n;
  const int cell = y * W + x;
  const int xo_p = x == 0 ? W - 1 : -1, xo_m = x == W - 1 ? 1 - W : 1;
  const int yo_p = y == 0 ? (H - 1) * W : -W, yo_m = y == H - 1 ? (1 - H) * W : W;
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const int ex = L::ex(i), ey = L::ey(i);
    const int off = (ex == 1 ? xo_p : (ex == -1 ? xo_m : 0)) + (ey == 1 ? yo_p : (ey == -1 ? yo_m : 0));
    f[i] = Codec<S>::ld(fi + (int64_t)i * n + (cell + off), i, p.pk);
  }
}

template <typename S>
__device__ __forceinline__ void cell2_core(const S *__restrict__ fin, float (&f)[9], S *__restrict__ fout,
                                           float *__restrict__ mac, const StepParams &p, int x, int y, bool force,
                                           CellForce &cf);

template <typename S>
__device__ __forceinline__ void cell2(const S *__restrict__ fin, S *__restrict__ fout,
                                      float *__restrict__ mac, const StepParams &p, int x, int y,
                                      bool force, CellForce &cf) {
  float f[9];
  gather2<S>(fin + p.base, p, x, y, f);
  cell2_core<S>(fin, f, fout, mac, p, x, y, force, cf);
}

// Everything after the gather for one D2Q9 cell: bounce-back and wall
// patches, moments, forcing, collision, mac, force.
template <typename S>
__device__ __forceinline__ void cell2_core(const S *__restrict__ fin, float (&f)[9], S *__restrict__ fout,
                                           float *__restrict__ mac, const StepParams &p, int x, int y, bool force,
                                           CellForce &cf) {
  using L = Lattice<9>;
  const int W = p.nx, H = p.ny;
  const int64_t n = p.n;
  const S *fi = fin + p.base;
  S *fo_ = fout + p.base;
  const int cell = y * W + x;
  const float fW = (float)W, fH = (float)H;
  const float px = (float)x, py = (float)y;
  float rx = 0.f, ry = 0.f, usx = 0.f, usy = 0.f, phi = 1e30f;
  // outside the reach box (p.nbox) no link ends in the body and chi is 0:
  // the distance (two divisions, a square root, for an ellipse the Newton
  // steps) is not evaluated there
  bool see = p.has_body;
  if (see && p.nbox_on) see = x >= p.nbox[0] && x <= p.nbox[1] && y >= p.nbox[2] && y <= p.nbox[3];
  if (see) {
    rx = wrap_delta(px - p.body.cx, fW);
    ry = wrap_delta(py - p.body.cy, fH);
    usx = __fmaf_rn(-p.body.wz, ry, p.body.vx);
    usy = __fmaf_rn(p.body.wz, rx, p.body.vy);
    phi = phi2(px, py, p.body, fW, fH);
  }
  const bool bbody = p.has_body && p.bb;
  const bool near = bbody && phi < 2.5f;
  const bool at_wall = p.wall_y && (y == 0 || y == H - 1);
  float fbx = 0.f, fby = 0.f;
  if (near || at_wall) {
    const int xm = x == 0 ? W - 1 : x - 1, xp = x == W - 1 ? 0 : x + 1;
    const int ym = y == 0 ? H - 1 : y - 1, yp = y == H - 1 ? 0 : y + 1;
    // Every link is classified first, then the cell's own populations that the
    // patches read are loaded together: a warp of near cells, whose links
    // differ from lane to lane, waits for one memory latency instead of one
    // per direction. An unrotated circle's links are found as the sphere's
    // (solid_links): squares shared, compared with p.ball2.
    unsigned solid = 0u, wall = 0u;
    if (near && phi2_is_circle(p.body)) {
      float xx[3], yy[3];
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const float dx = wrap_delta((float)(e == 2 ? xm : (e == 0 ? xp : x)) - p.body.cx, fW);
        const float dy = wrap_delta((float)(e == 2 ? ym : (e == 0 ? yp : y)) - p.body.cy, fH);
        xx[e] = __fmul_rn(dx, dx);
        yy[e] = __fmul_rn(dy, dy);
      }
#pragma unroll
      for (int i = 0; i < 9; ++i)
        if (__fadd_rn(xx[L::ex(i) + 1], yy[L::ey(i) + 1]) < p.ball2) solid |= 1u << i;
    } else if (near) {
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const int sx = L::ex(i) == 1 ? xm : (L::ex(i) == -1 ? xp : x);
        const int sy = L::ey(i) == 1 ? ym : (L::ey(i) == -1 ? yp : y);
        if (phi2((float)sx, (float)sy, p.body, fW, fH) < 0.f) solid |= 1u << i;
      }
    }
    if (at_wall) {
#pragma unroll
      for (int i = 0; i < 9; ++i)
        if (y - L::ey(i) < 0 || y - L::ey(i) >= H) wall |= 1u << i;
    }
    if (solid | wall) {
      float own[9];
#pragma unroll
      for (int i = 0; i < 9; ++i)
        own[i] = ((solid | wall) >> L::opp(i)) & 1u ? Codec<S>::ld(fi + (int64_t)i * n + cell, i, p.pk) : 0.f;
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const float ex = (float)L::ex(i), ey = (float)L::ey(i), fopp = own[L::opp(i)];
        if ((solid >> i) & 1u) {
          const float corr = __fmul_rn(2.f * L::w(i) * (ex * usx + ey * usy), kInvCS2);
          f[i] = __fadd_rn(fopp, corr);
          if (phi >= 0.f) {
            const float m = __fmaf_rn(2.f, fopp, corr);
            fbx += -ex * m;
            fby += -ey * m;
          }
        } else if ((wall >> i) & 1u) {
          const float corr = __fmul_rn(2.f * L::w(i) * ex * (y - L::ey(i) < 0 ? p.wall_u0 : p.wall_u1), kInvCS2);
          f[i] = __fadd_rn(fopp, corr);
        }
      }
    }
  }
  float rho, mxs, mys, mzs;
  moments<L, 9>(f, rho, mxs, mys, mzs);
  const float rhoDen = fmaxf(rho, 1e-6f);
  const float inv = 1.0f / rhoDen;
  const float uxs = mxs * inv, uys = mys * inv;
  const float chi = (see && !p.bb) ? chi_from_phi(phi, p.chi_eps) : 0.f;
  const float Fx = rho * chi * (usx - uxs) + p.fx;
  const float Fy = rho * chi * (usy - uys) + p.fy;
  const float hinv = 0.5f * inv;
  const float ux = fmaf(Fx, hinv, uxs);
  const float uy = fmaf(Fy, hinv, uys);

  float spw = 0.f;
  if (p.sponge_w > 0.f) {
    const float dx = fminf(px, (float)(W - 1 - x));
    const float dy = fminf(py, (float)(H - 1 - y));
    spw = sponge_weight_inv(fminf(dx, dy), p.sponge_inv);
  }
  const bool in_solid = p.solid_eq && bbody && phi < 0.f;
  if (!in_solid) {
    MemSink2<S> sink{fo_, n, cell, p.pk};
    collide_store<L, 9>(f, rho, ux, uy, 0.f, Fx, Fy, 0.f, p.omega, spw, p.ftarget, sink);
  } else {
    const float ussq = usx * usx + usy * usy;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const float w = L::w(i);
      const float eu = (float)L::ex(i) * usx + (float)L::ey(i) * usy;
      Codec<S>::st(fo_ + (int64_t)i * n + cell, w * 1.0f * (1.f + 3.f * eu + 4.5f * eu * eu - 1.5f * ussq), i, p.pk);
    }
  }
  if (p.write_mac && mac) reinterpret_cast<float4 *>(mac + 4 * p.base)[cell] = make_float4(rho, ux, uy, 0.f);

  if (force) {
    if (!bbody && see) {
      const float c2 = chi_from_phi(phi, p.chi_eps);
      if (c2 >= 1e-6f) {
        fbx = -(rho * c2 * (usx - uxs));
        fby = -(rho * c2 * (usy - uys));
      }
    }
    cf.fx = fbx;
    cf.fy = fby;
    cf.tz = rx * fby - ry * fbx;
  }
}

// One D2Q9 cell that no body reaches, outside any force region:
// cell2_core with the tests that cannot fire taken out (no solid link,
// chi = 0 and u_s = 0, so the Guo force is the body force) and only the
// moving-wall patch of a wall row kept, the same arithmetic in the same
// order, so the same bits.
template <typename S>
__device__ __forceinline__ void cell2_fluid(const S *__restrict__ fin, float (&f)[9], S *__restrict__ fout,
                                            float *__restrict__ mac, const StepParams &p, int x, int y) {
  using L = Lattice<9>;
  const int W = p.nx, H = p.ny;
  const int cell = y * W + x;
  if (p.wall_y && (y == 0 || y == H - 1)) {
    const S *fi = fin + p.base;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const int ex = L::ex(i), ey = L::ey(i), o = L::opp(i);
      const int ysrc = y - ey;
      if (ysrc < 0 || ysrc >= H) {
        const float wu = ysrc < 0 ? p.wall_u0 : p.wall_u1;
        const float corr = __fmul_rn(2.f * L::w(i) * (float)ex * wu, kInvCS2);
        f[i] = __fadd_rn(Codec<S>::ld(fi + (int64_t)o * p.n + cell, o, p.pk), corr);
      }
    }
  }
  float rho, mxs, mys, mzs;
  moments<L, 9>(f, rho, mxs, mys, mzs);
  const float rhoDen = fmaxf(rho, 1e-6f);
  const float inv = 1.0f / rhoDen;
  const float uxs = mxs * inv, uys = mys * inv;
  const float chi = 0.f, usx = 0.f, usy = 0.f;
  const float Fx = rho * chi * (usx - uxs) + p.fx;
  const float Fy = rho * chi * (usy - uys) + p.fy;
  const float hinv = 0.5f * inv;
  const float ux = fmaf(Fx, hinv, uxs);
  const float uy = fmaf(Fy, hinv, uys);
  float spw = 0.f;
  if (p.sponge_w > 0.f) {
    const float dx = fminf((float)x, (float)(W - 1 - x));
    const float dy = fminf((float)y, (float)(H - 1 - y));
    spw = sponge_weight_inv(fminf(dx, dy), p.sponge_inv);
  }
  MemSink2<S> sink{fout + p.base, p.n, cell, p.pk};
  collide_store<L, 9>(f, rho, ux, uy, 0.f, Fx, Fy, 0.f, p.omega, spw, p.ftarget, sink);
  if (p.write_mac) reinterpret_cast<float4 *>(mac + 4 * p.base)[cell] = make_float4(rho, ux, uy, 0.f);
}

}  // namespace lbm
