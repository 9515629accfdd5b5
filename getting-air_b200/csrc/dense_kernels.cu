// Dense-grid kernels for sm_100a: the fused pull-stream / BGK / Guo-forcing
// step with its body-force reduction, equilibrium seeding, storage
// conversion and the FP64 conserved-totals reduction.
//
// Reference arithmetic:
//   3D step    common_d3_step.wgsl:224-400
//   3D force   common_d3_force.wgsl:171-283 (momentum exchange with local
//              rho_w and the swept-cell term, or the chi penalty)
//   2D step    lbm_step.wgsl:137-270
//   2D force   lbm_force.wgsl (main)
//   initEq     common_d3_step.wgsl:206-222
//   totals     amr2d-gpu.mjs:698-736 readConservedTotals
//
// Layout in HBM: f is Q planes, plane-major, `f[i * n + cell]` with
// cell = (z*NY + y)*NX + x -- the reference's layout, which is also the one
// that gives every warp a coalesced 128-byte row per plane. One thread owns
// one cell: it decides which of its links the body or a wall cuts (in a block
// that either can reach; the others skip this), issues the Q pull loads
// (periodic sources), patches the few cut links, collides in registers and
// writes the Q planes of its own cell. The mac field is written only when the
// host asks for it (the last step of a batch), not every step.
//
// The body force is summed INSIDE the step: the reference runs a separate
// full-grid force pass before each step over the same pre-streaming f_in,
// and every quantity it needs (f_opp at the cell, the streamed rho and u*)
// is already in this kernel's registers. Only the launch blocks whose cells
// can touch the body reduce; each writes one FP64 partial, and the partials
// are summed in a fixed order after the launch, so the result is
// deterministic: by blocks of their own in front of the next step's grid when
// steps follow one another (add_sum_layers), else by a small launch of the
// same blocks. The kernel boundary is what orders the partials before the sum.
// A last-block ticket inside the step needs a release fence per partial, and
// under the step's full write traffic each fence held its CTA for
// microseconds; one block with cells summing all partials first waits on
// dozens of rounds of loads; and a one-block launch after every step costs its
// launch gaps (measured at 256x128x128: +9 %, +10 % and +7 % of the step
// against no force at all, and +1 % for the sum in the next launch).

#include <algorithm>

#include "dense_block.cuh"

namespace lbm {

namespace {

// ---- dense fused steps -------------------------------------------------------
// One thread per cell, kStepThreads (64) cells per CTA: of a row, grid
// (NX/64, NY, NZ), the row and plane straight from blockIdx, or of the
// plane's cells as one run (choose_step_map).

// A copy of the launch's parameters in shared memory with the body pose,
// swept-cell band and reach box of this step taken from the device
// (free-body launches, where the pose is produced on the device).
__device__ __forceinline__ void stage_pose(const StepParams &p, StepParams &sp) {
  const unsigned *src = reinterpret_cast<const unsigned *>(&p);
  unsigned *dst = reinterpret_cast<unsigned *>(&sp);
  for (int k = threadIdx.x; k < (int)(sizeof(StepParams) / 4); k += blockDim.x) dst[k] = src[k];
  __syncthreads();
  if (threadIdx.x == 0) {
    const BodyPose &bp = *p.pose_in;
    sp.body = bp.body;
    sp.nbox_on = bp.nbox_on;
    for (int k = 0; k < 6; ++k) sp.nbox[k] = bp.nbox[k];
    sp.swept = bp.swept;
    sp.swept_band = bp.swept_band;
  }
  __syncthreads();
}

// A block that no body, wall, force region or window touches runs the fluid
// update; the others the general one, with the body's links and the walls
// classified before the gather (Geom3). FP32 is bound by HBM (D3Q19: 152 bytes
// a cell), 16-bit storage by instruction issue, small domains by the latency
// of the force region's blocks. 256x128x128 sphere, us per step, before and
// after the explicit collision, these kinds, the dedicated sum blocks, the
// tight reach box and (16-bit) the 32-bit offsets:
//             FP32             FP16             BF16
//   D3Q19  107.1 -> 102.6   106.6 -> 98.7    106.6 -> 99.4
//   D3Q27  153.9 -> 146.2   154.3 -> 136.0   154.6 -> 135.6
// and a D3Q19 FP32 sphere in 64^3 13.1 -> 9.9 (8.3 with publish_force's short
// sum). (Two cells a thread in packed
// arithmetic, and planes staged by bulk copies, both ran slower: more
// registers, so fewer warps to hide the gather.)
// WIN: a domain with a moving window, whose fluid blocks take the sponge in
// window coordinates (an instantiation of its own: in the other it would cost
// 1 to 2 %) and whose links see which image of the body they lead to
// (solid_links_call). us per step of a windowed FP32 sphere with every block
// general, with fluid blocks, and with those links: 128^3 72.7, 67.2, 62.9;
// 256x128x128 129.2, 117.6, 112.9.
template <int Q, typename S, bool TRT, bool WIN>
__global__ void __launch_bounds__(kStepThreads, Q == 27 ? (kStepMinBlocks * 3) / 4 : kStepMinBlocks)
    d3_step(const S *__restrict__ fin, S *__restrict__ fout, float *__restrict__ mac,
            const __grid_constant__ StepParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");  // a no-op unless launched by launch_pdl
  if (sum_previous(p)) return;
  const BlockMap m = block_map(p, kStepThreads);
  const int c = m.c0 + threadIdx.x;
  int x, y;
  block_cell(p, m, c, x, y);
  if (block_kind(p, m, kStepThreads) == kFluid) {
    if (c < m.lim) cell3_fluid<Q, S, TRT, WIN>(fin, fout, mac, p, x, y, m.bz);
    return;
  }
  CellForce cf;
  if (c < m.lim) cell3<Q, S, TRT, true, WIN>(fin, fout, mac, p, x, y, m.bz, m.region, cf);
  if (m.region) publish_force<kStepThreads>(cf, p.partials, m.part);
}

// The step of a penalty body, which reaches every cell through chi: the
// general update everywhere, without the links' code (cell3). Through d3_step,
// whose general update decides links before it gathers, such a step was up to
// 13 % slower than with the gather first; us per step of d3_step and of this
// kernel: D3Q19 sphere FP32 128^3 61.3 -> 53.8, 256x128x128 118.7 -> 103.9, FP16
// 128^3 62.9 -> 55.4, spheroid 96.4 -> 86.8, D3Q27 rounded box 89.5 -> 81.8.
template <int Q, typename S, bool TRT>
__global__ void __launch_bounds__(kStepThreads, Q == 27 ? (kStepMinBlocks * 3) / 4 : kStepMinBlocks)
    d3_step_penalty(const S *__restrict__ fin, S *__restrict__ fout, float *__restrict__ mac,
                    const __grid_constant__ StepParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (sum_previous(p)) return;
  const BlockMap m = block_map(p, kStepThreads);
  const int c = m.c0 + threadIdx.x;
  int x, y;
  block_cell(p, m, c, x, y);
  CellForce cf;
  if (c < m.lim) cell3<Q, S, TRT, false>(fin, fout, mac, p, x, y, m.bz, m.region, cf);
  if (m.region) publish_force<kStepThreads>(cf, p.partials, m.part);
}

// The step of a free body: the pose comes from the device (written by the
// force pass just before); no force reduction. Blocks beyond the pose's
// reach box run the fluid update with the launch's own parameters; the
// others stage them with the pose in shared memory. (Evaluating the body's
// distance at every cell, as before the pose carried its reach box, was
// most of the step: a spheroid's takes an arctangent and three Newton
// steps of sines and cosines. A spheroid in 96x64x64 with its force pass, bound
// by the latter's chain of sums: 116.0 -> 46.7 us per step.)
template <int Q, typename S, bool TRT>
__global__ void __launch_bounds__(kStepThreads, Q == 27 ? 10 : 12)
    d3_step_free(const S *__restrict__ fin, S *__restrict__ fout, float *__restrict__ mac,
                 const __grid_constant__ StepParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __shared__ StepParams sp;
  const BodyPose &bp = *p.pose_in;
  const BlockMap m = block_map(p, kStepThreads);
  const int c = m.c0 + threadIdx.x;
  int x, y;
  block_cell(p, m, c, x, y);
  if (!p.win.on && block_kind(p, m, kStepThreads, bp.nbox_on, bp.nbox) == kFluid) {
    if (c < m.lim) cell3_fluid<Q, S, TRT>(fin, fout, mac, p, x, y, m.bz);
    return;
  }
  stage_pose(p, sp);
  CellForce cf;
  if (c < m.lim) cell3<Q, S, TRT>(fin, fout, mac, sp, x, y, m.bz, false, cf);
}

// Integrates the free body under the force just summed and publishes the
// next pose with its force box (clipped to the launch capacity; a body
// outside the domain keeps one block so the integrator still runs).
__device__ __noinline__ void integrate_and_publish(BodyDyn *dyn, const double *force, BodyPose *next) {
  const double F[3] = {force[0], force[1], force[2]}, T[3] = {force[3], force[4], force[5]};
  body_step(dyn->st, F, T, dyn->opt);
  BodyPose np;
  np.body = body_pose(dyn->shape, dyn->st);
  int box[6];
  const bool any = body_cell_box(np.body, dyn->q, dyn->nx, dyn->ny, dyn->nz, dyn->bounceback, dyn->swept_force,
                                 dyn->chi_eps, box, &np.swept, &np.swept_band, dyn->win);
  np.nbox_on = dyn->bounceback;
  reach_box3(box, any, dyn->nx, dyn->ny, dyn->nz, np.nbox);
  if (!any) {
    const float c[3] = {np.body.cx, np.body.cy, np.body.cz};
    const int len[3] = {dyn->nx, dyn->ny, dyn->nz};
    for (int a = 0; a < 3; ++a) {
      const int v = (int)fminf(fmaxf(c[a], 0.f), (float)(len[a] - 1));
      box[2 * a] = box[2 * a + 1] = v;
    }
  }
  if (force_box(box, dyn->nx, dyn->ny, dyn->nz, dyn->cap, np.box)) dyn->overflow += 1;
  *next = np;
}

// Free-body force pass: the cells of the current force box as one run, one
// per thread (the launch covers the largest box; blocks past this step's
// cells leave at once and take no part in the reduction). The last block to
// finish sums the partials and integrates the body, a chain that the step
// waits for: with a block per 64 cells of a row of the grid the box of a
// 16-cell body had a thousand partials, whose sum by one warp took most of
// the pass; as one run it has about a hundred.
template <int Q, typename S>
__global__ void __launch_bounds__(kForceThreads)
    d3_force_pass(const S *__restrict__ fin, const __grid_constant__ StepParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __shared__ StepParams sp;
  const int *b = p.pose_in->box;
  const int lx = b[1], ly = b[3], cells = lx * ly * b[5];
  if ((int)blockIdx.x * kForceThreads >= cells) return;
  const int lo[3] = {b[0], b[2], b[4]};
  stage_pose(p, sp);
  const int k = blockIdx.x * kForceThreads + threadIdx.x;
  ForceAcc acc;
  if (k < cells) {
    const int row = k / lx, pl = row / ly;
    int x = lo[0] + k - row * lx, y = lo[1] + row - pl * ly, z = lo[2] + pl;
    x -= x >= sp.nx ? sp.nx : 0;
    y -= y >= sp.ny ? sp.ny : 0;
    z -= z >= sp.nz ? sp.nz : 0;
    CellForce cf;
    cell3_force<Q, S>(fin, sp, x, y, z, cf);
    acc.add(cf);
  }
  const int parts = (cells + kForceThreads - 1) / kForceThreads;
  const bool last = reduce_force<kForceThreads>(acc, sp.partials, sp.counter, parts, blockIdx.x, sp.force_out);
  if (last && threadIdx.x == 0) integrate_and_publish(sp.dyn, sp.force_out, sp.pose_out);
}

// The D2Q9 step: 64 cells of a row per block. Where no body reaches the block
// and it lies outside the force region, the fluid update (which keeps the
// walls), else the general one. A 2D grid is small (512^2: 19 MB, in L2) and
// its step mostly latency: the launch, and per cell the body's distance,
// which outside its reach box (for a penalty body where chi is not 0) is not
// evaluated. us per step before (every cell general, no programmatic launch)
// and after: 512^2 FP32 12.4 -> 6.5, FP16 12.3 -> 7.5, 1000x600 16.4 -> 8.4,
// 200x150 10.3 -> 5.7, 2048x1024 34.2 -> 31.4; with publish_force's short sum
// 5.0, 5.9, 8.2, 4.0 and 31.7. (64 registers: at 40, 512^2
// takes 7.2 and 2048x1024, bound by HBM, 27.1. Two cells a thread: 8.5 and 46.)
template <typename S>
__global__ void __launch_bounds__(kStepThreads, kStepMinBlocks)
    d2_step(const S *__restrict__ fin, S *__restrict__ fout, float *__restrict__ mac,
            const __grid_constant__ StepParams p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (sum_previous<kStepThreads, true>(p)) return;
  const int bx = blockIdx.x, lo = bx * kStepThreads, hi = lo + kStepThreads - 1;
  int by = (int)blockIdx.y - p.sum_layers + p.rot;
  by -= by >= p.ny ? p.ny : 0;
  const int x = lo + (int)threadIdx.x;
  const bool region = p.force_on && bx >= p.rbx0 && bx < p.rbx1 && by >= p.rby0 && by < p.rby1;
  const bool reach = p.has_body && (!p.nbox_on || (lo <= p.nbox[1] && hi >= p.nbox[0] && by >= p.nbox[2] && by <= p.nbox[3]));
  if (!reach && !region) {
    if (x >= p.nx) return;
    float f[9];
    gather2<S>(fin, p, x, by, f);
    cell2_fluid<S>(fin, f, fout, mac, p, x, by);
    return;
  }
  CellForce cf;
  if (x < p.nx) cell2<S>(fin, fout, mac, p, x, by, region, cf);
  if (region) {
    const int rx = p.rbx1 - p.rbx0;
    publish_force<kStepThreads>(cf, p.partials, (by - p.rby0) * rx + (bx - p.rbx0));
  }
}

// The force of a step that no following launch sums: the same blocks, with
// the same arithmetic, as those in front of a following step's grid.
__global__ void __launch_bounds__(kStepThreads)
    force_finish(const double *__restrict__ partials, int nparts, double *__restrict__ groups,
                 unsigned int *__restrict__ counter, double *__restrict__ out) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  sum_partials_grouped<kStepThreads>(partials, nparts, groups, counter, out, blockIdx.x);
}

// ---- seeding and storage conversion ----------------------------------------

// f at equilibrium of the mac field; UNIFORM: of the one state `mu`, which
// is also written to every cell of mac (a uniform seed needs no host data).
template <int Q, typename S, bool UNIFORM = false>
__global__ void init_eq(const float4 *__restrict__ mac, S *__restrict__ f, int64_t n, const Pack pk,
                        float4 mu = {}, float4 *__restrict__ mac_out = nullptr) {
  using L = Lattice<Q>;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    const float4 m = UNIFORM ? mu : mac[c];
    if (UNIFORM) mac_out[c] = mu;
    const float rho = m.x, ux = m.y, uy = m.z, uz = Q == 9 ? 0.f : m.w;
    const float usq = Q == 9 ? (ux * ux + uy * uy) : (ux * ux + uy * uy + uz * uz);
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const float eu = (float)L::ex(i) * ux + (float)L::ey(i) * uy + (float)L::ez(i) * uz;
      const float v = L::w(i) * rho * (1.f + 3.f * eu + 4.5f * eu * eu - 1.5f * usq);
      Codec<S>::st(f + (int64_t)i * n + c, v, i, pk);
    }
  }
}

template <int Q, typename S>
__global__ void pack_planes(const float *__restrict__ src, S *__restrict__ dst, int64_t n, const Pack pk) {
  using L = Lattice<Q>;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x)
#pragma unroll
    for (int i = 0; i < Q; ++i) Codec<S>::st(dst + (int64_t)i * n + c, src[(int64_t)i * n + c], i, pk);
}

template <int Q, typename S>
__global__ void unpack_planes(const S *__restrict__ src, float *__restrict__ dst, int64_t n, const Pack pk) {
  using L = Lattice<Q>;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x)
#pragma unroll
    for (int i = 0; i < Q; ++i) dst[(int64_t)i * n + c] = Codec<S>::ld(src + (int64_t)i * n + c, i, pk);
}

// ---- conserved totals ------------------------------------------------------
// Per cell the reference sums the f32 populations in f64 (JS numbers):
// rho, rho u, then mass += rho - 1. Same here, with FP64 partial sums per
// block and a fixed-order final sum.

constexpr int kTotalsBlocks = 148 * 4;

template <int Q, typename S>
__global__ void __launch_bounds__(kReduceThreads)
    totals_kernel(const S *__restrict__ f, int64_t n, int64_t stride, const Pack pk, double *partials,
                  unsigned int *counter, double *out) {
  using L = Lattice<Q>;
  double mass = 0.0, px = 0.0, py = 0.0, pz = 0.0, bad = 0.0;
  double rmin = 1e300, rmax = -1e300, u2max = 0.0;
  for (int64_t c = blockIdx.x * (int64_t)kReduceThreads + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * kReduceThreads) {
    double rho = 0.0, mx = 0.0, my = 0.0, mz = 0.0;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const double v = (double)Codec<S>::ld(f + (int64_t)i * stride + c, i, pk);
      rho += v;
      mx += v * L::ex(i);
      my += v * L::ey(i);
      mz += v * L::ez(i);
    }
    if (!isfinite(rho + mx + my + mz)) {
      bad += 1.0;
      continue;
    }
    mass += rho - 1.0;
    px += mx;
    py += my;
    pz += mz;
    rmin = fmin(rmin, rho);
    rmax = fmax(rmax, rho);
    u2max = fmax(u2max, (mx * mx + my * my + mz * mz) / (rho * rho));
  }
  // Sums via the shared block_sum; min/max folded through negation tricks
  // would lose determinism guarantees for ties, so they are reduced apart.
  __shared__ double sm[kTotalsSlots * (kReduceThreads / 32)];
  double v[5] = {mass, px, py, pz, bad};
  block_sum<5, kReduceThreads>(v, sm);
  double mm[3] = {rmin, -rmax, -u2max};
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mm[k] = fmin(mm[k], __shfl_down_sync(0xffffffffu, mm[k], o));
  __shared__ double smm[3 * (kReduceThreads / 32)];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int k = 0; k < 3; ++k) smm[k * (kReduceThreads / 32) + warp] = mm[k];
  __syncthreads();
  if (warp == 0) {
    for (int k = 0; k < 3; ++k) {
      double t = lane < kReduceThreads / 32 ? smm[k * (kReduceThreads / 32) + lane] : 1e300;
      for (int o = 16; o > 0; o >>= 1) t = fmin(t, __shfl_down_sync(0xffffffffu, t, o));
      mm[k] = t;
    }
  }
  __shared__ bool s_last;
  if (threadIdx.x == 0) {
    double *pp = partials + (int64_t)blockIdx.x * kTotalsSlots;
    pp[0] = v[0]; pp[1] = v[1]; pp[2] = v[2]; pp[3] = v[3];
    pp[4] = mm[0]; pp[5] = mm[1]; pp[6] = mm[2]; pp[7] = v[4];
    __threadfence();
    const unsigned int t = atomicAdd(counter, 1u);
    s_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (threadIdx.x == 0) {
    double s0 = 0, s1 = 0, s2 = 0, s3 = 0, s7 = 0, m4 = 1e300, m5 = 1e300, m6 = 1e300;
    for (unsigned int j = 0; j < gridDim.x; ++j) {
      const double *pp = partials + (int64_t)j * kTotalsSlots;
      s0 += __ldcg(pp + 0); s1 += __ldcg(pp + 1); s2 += __ldcg(pp + 2); s3 += __ldcg(pp + 3);
      m4 = fmin(m4, __ldcg(pp + 4)); m5 = fmin(m5, __ldcg(pp + 5)); m6 = fmin(m6, __ldcg(pp + 6));
      s7 += __ldcg(pp + 7);
    }
    out[0] = s0; out[1] = s1; out[2] = s2; out[3] = s3;
    out[4] = m4; out[5] = -m5; out[6] = sqrt(-m6 < 0 ? 0.0 : -m6); out[7] = s7;
    *counter = 0u;
  }
}

// Expands the body once per (Q, storage) pair with Q and S bound.
#define LBM_DISPATCH(q, storage, ...)                                           \
  switch ((q) * 4 + (storage)) {                                                 \
    case 9 * 4 + 0: { constexpr int Q = 9; using S = float; __VA_ARGS__; } break;        \
    case 9 * 4 + 1: { constexpr int Q = 9; using S = __half; __VA_ARGS__; } break;       \
    case 9 * 4 + 2: { constexpr int Q = 9; using S = __nv_bfloat16; __VA_ARGS__; } break; \
    case 19 * 4 + 0: { constexpr int Q = 19; using S = float; __VA_ARGS__; } break;      \
    case 19 * 4 + 1: { constexpr int Q = 19; using S = __half; __VA_ARGS__; } break;     \
    case 19 * 4 + 2: { constexpr int Q = 19; using S = __nv_bfloat16; __VA_ARGS__; } break; \
    case 27 * 4 + 0: { constexpr int Q = 27; using S = float; __VA_ARGS__; } break;      \
    case 27 * 4 + 1: { constexpr int Q = 27; using S = __half; __VA_ARGS__; } break;     \
    case 27 * 4 + 2: { constexpr int Q = 27; using S = __nv_bfloat16; __VA_ARGS__; } break; \
    default: return cudaErrorInvalidValue;                                       \
  }                                                                              \
  return cudaGetLastError();

int grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  return (int)(b < 148 * 8 ? (b < 1 ? 1 : b) : 148 * 8);
}

}  // namespace

void launch_force_sum(const double *partials, int parts, double *groups, unsigned int *counter, double *out,
                      cudaStream_t st) {
  launch_pdl(dim3(sum_groups(parts)), dim3(kStepThreads), st, force_finish, partials, parts, groups, counter, out);
}

namespace {
cudaError_t launch_step_kernel(int q, int storage, const void *f_in, void *f_out, float *mac, const StepParams &p,
                               cudaStream_t st) {
  if (q != 9 && p.pose_in) {
    LBM_DISPATCH(q, storage, {
      auto run = [&](auto k) {
        launch_pdl(step_grid(p), dim3(kStepThreads), st, k, (const S *)f_in, (S *)f_out, mac, p);
      };
      if constexpr (Q != 9) {
        if (p.trt_dw != 0.f) run(d3_step_free<Q, S, true>);
        else run(d3_step_free<Q, S, false>);
      }
    });
  }
  StepParams r = p;
  dim3 grid = step_grid(p);
  if (q == 9) grid = dim3((p.nx + kStepThreads - 1) / kStepThreads, p.ny, 1);
  if (p.force_on) r.rot = q == 9 ? p.rby0 : std::max(0, p.rbz0 - p.zoff - p.zlo);
  // (A whole plane in front of a D2Q9 grid is mostly blocks that start and
  // leave, 0.4 ns each: 2048x1024 took 49 us per step, 34 without it.)
  if (!add_sum_layers(r, grid, q == 9))
    launch_force_sum(p.prev_partials, p.prev_parts, p.groups, p.counter, p.force_out, st);
  LBM_DISPATCH(q, storage, {
    auto run = [&](auto k) { launch_pdl(grid, dim3(kStepThreads), st, k, (const S *)f_in, (S *)f_out, mac, r); };
    if constexpr (Q == 9) {
      run(d2_step<S>);
    } else if (p.has_body && !p.bb) {
      if (p.trt_dw != 0.f) run(d3_step_penalty<Q, S, true>);
      else run(d3_step_penalty<Q, S, false>);
    } else if (p.win.on) {
      if (p.trt_dw != 0.f) run(d3_step<Q, S, true, true>);
      else run(d3_step<Q, S, false, true>);
    } else {
      if (p.trt_dw != 0.f) run(d3_step<Q, S, true, false>);
      else run(d3_step<Q, S, false, false>);
    }
  });
}
}  // namespace

cudaError_t launch_step(int q, int storage, const void *f_in, void *f_out, float *mac,
                        const StepParams &p, cudaStream_t st) {
  // a free body's step takes no force (its force pass does)
  if (p.pose_in && p.force_on) return cudaErrorInvalidValue;
  if (p.force_on && (!p.partials || !p.groups || !p.counter || !p.force_out)) return cudaErrorInvalidValue;
  if (p.prev_parts && (!p.prev_partials || !p.groups || !p.counter || !p.force_out)) return cudaErrorInvalidValue;
  const cudaError_t e = launch_step_kernel(q, storage, f_in, f_out, mac, p, st);
  if (e != cudaSuccess || !p.force_on || p.defer_force) return e;
  launch_force_sum(p.partials, force_parts(q, p), p.groups, p.counter, p.force_out, st);
  return cudaGetLastError();
}

cudaError_t launch_force_pass(int q, int storage, const void *f_in, const StepParams &p, int parts, cudaStream_t st) {
  if (q == 9 || !p.pose_in || !p.pose_out || !p.dyn) return cudaErrorInvalidValue;
  LBM_DISPATCH(q, storage, {
    if constexpr (Q != 9) launch_pdl(dim3(parts), dim3(kForceThreads), st, d3_force_pass<Q, S>, (const S *)f_in, p);
  });
}

cudaError_t launch_init_eq(int q, int storage, const float *mac_in, void *f_out, int64_t n, const Pack &pk,
                           cudaStream_t st) {
  LBM_DISPATCH(q, storage, init_eq<Q, S><<<grid_for(n, 256), 256, 0, st>>>((const float4 *)mac_in, (S *)f_out, n, pk));
}

cudaError_t launch_init_uniform(int q, int storage, const float rho_u[4], float *mac_out, void *f_out, int64_t n,
                                const Pack &pk, cudaStream_t st) {
  const float4 mu = make_float4(rho_u[0], rho_u[1], rho_u[2], rho_u[3]);
  LBM_DISPATCH(q, storage, (init_eq<Q, S, true><<<grid_for(n, 256), 256, 0, st>>>(nullptr, (S *)f_out, n, pk, mu,
                                                                                 (float4 *)mac_out)));
}

cudaError_t launch_pack(int q, int storage, const float *f32, void *f_store, int64_t n, const Pack &pk,
                        cudaStream_t st) {
  LBM_DISPATCH(q, storage, pack_planes<Q, S><<<grid_for(n, 256), 256, 0, st>>>(f32, (S *)f_store, n, pk));
}

cudaError_t launch_unpack(int q, int storage, const void *f_store, float *f32, int64_t n, const Pack &pk,
                          cudaStream_t st) {
  LBM_DISPATCH(q, storage, unpack_planes<Q, S><<<grid_for(n, 256), 256, 0, st>>>((const S *)f_store, f32, n, pk));
}

int totals_blocks() { return kTotalsBlocks; }

cudaError_t launch_totals(int q, int storage, const void *f, int64_t n, const Pack &pk, double *partials,
                          unsigned int *counter, double *out, cudaStream_t st, int64_t stride) {
  if (stride <= 0) stride = n;
  LBM_DISPATCH(q, storage, (totals_kernel<Q, S><<<kTotalsBlocks, kReduceThreads, 0, st>>>((const S *)f, n, stride, pk, partials, counter, out)));
}

}  // namespace lbm
