// Launch parameters and entry points of the dense-grid kernels.
#pragma once

#include <cstdint>
#include <utility>

#include <cuda_runtime.h>
#include "../../include/lbm.h"
#include "body.cuh"

namespace lbm {

// How 16-bit storage encodes a population: s = (f - off[i]) * scale, stored
// rounded to nearest even; f = s * inv + off[i]. off[i] is the equilibrium of
// the domain's far field, feq_i(rho = 1, u = U_far) (f-pack mode 2 with the
// rest state replaced by the free stream: the stored value is the flow's
// deviation from it), and scale = 2^10 for FP16 keeps small deviations out
// of the subnormal range. Unused by FP32 storage.
// noff[i] = -off[i] * scale (exact: scale is a power of two), so that the
// encode is one fused multiply-add, fma(f, scale, noff[i]) = (f - off) *
// scale to the bit.
constexpr float kF16Scale = 1024.0f;  // 2^10, the FP16 storage scale
struct Pack {
  float off[27];
  float noff[27];
  float scale, inv;
};

// Per-step constants of the fused stream-collide kernels. Mirrors the
// override constants of common_d3_step.wgsl:125-213 / lbm_step.wgsl:36-135.
struct StepParams {
  int nx, ny, nz;       // stored extent (a slab's nz counts its two ghost planes)
  // A z-slab of a larger domain (lbm_create_slab): stored plane z is the
  // domain's plane z + zoff, the domain is nzg planes deep, and the step
  // covers the stored planes [zlo, nz - zlo) (zlo = 1: the ghost planes
  // below and above are filled by the halo exchange). A whole domain has
  // zoff = 0, nzg = nz, zlo = 0.
  int zoff, nzg, zlo;
  int64_t n;            // plane stride of the arena the domain lives in (cells)
  int64_t base;         // arena index of the domain's cell 0
  float omega;          // 1 / tau
  float trt_dw;         // omega_- - omega of the TRT collision; 0 = BGK
  float fx, fy, fz;     // uniform Guo body force
  int wall_x, wall_y, wall_z;
  float wall_u0, wall_u1;  // D2Q9 moving y-walls
  int has_body, bb, solid_eq, rho_w_local, swept;
  float swept_band;     // |phi| below which a cell can change hands in one step
  float chi_eps;
  float sponge_w, sponge_inv;  // band width and its reciprocal
  int sax, say, saz;
  float ftarget[27];    // sponge far-field equilibrium per direction (rho = 1)
  lbm_body body;
  float ball2;          // the smallest square whose root reaches body.a (ball_square)
  Win win;              // moving window (3D); win.on = 0 without one
  // The cell box outside which the body changes no cell, so the SDF and the
  // body velocity need not be evaluated there (nbox_on = 0: evaluate
  // everywhere): no link reaches it (bounce-back; read modulo the grid in
  // 3D), or chi is 0 to the bit (D2Q9 penalty; reach_box2).
  int nbox_on;
  int nbox[6];
  int write_mac;
  // Force reduction: the blocks of the launch grid that can see the body.
  int force_on;
  int rbx0, rbx1, rby0, rby1, rbz0, rbz1;
  double *partials;        // 8 doubles per region block
  unsigned int *counter;   // last-block ticket, returns to 0 after each step
  double *force_out;       // 8 doubles: fx fy fz tx ty tz nonfinite 0
  // Dense steps sum their partials after the launch (sum_partials_grouped,
  // with `counter` as its ticket and `groups` as its first-level sums): with
  // defer_force = 0 launch_step() follows the step with a launch that does
  // it; with defer_force = 1 it is left to the next launch on the stream,
  // which sums the prev_parts partials at prev_partials (add_sum_layers).
  double *groups;
  int defer_force;
  int prev_parts;
  const double *prev_partials;
  int clear_ticket;        // the step zeroes `counter` first (no prev_parts)
  Pack pk;                 // 16-bit storage encoding
  // Multi-domain launches: the domain's first tile, and the tile range
  // [ft0, ft1) (relative to tile0) whose cells can see the body.
  int tile0, ft0, ft1;
  // Free body (dense 3D only; all NULL otherwise): the pose this launch
  // reads (and for a force pass, the pose its last block writes) and the
  // integrator state.
  const BodyPose *pose_in;
  BodyPose *pose_out;
  BodyDyn *dyn;
  // Launch mapping of the dense 3D step (choose_step_map): whether the blocks
  // cut a plane's cells as one run (flat) or each row by itself. magic: for
  // the division of a plane's cell index by nx (row_magic), 0 where it would
  // not be exact.
  int flat;
  unsigned magic;
  // Layers (along z; D2Q9: rows) of blocks in front of the grid that only sum
  // the previous launch's force partials (add_sum_layers).
  int sum_layers;
  // The plane (3D) or row (D2Q9) that the launch's first blocks take: the
  // force region's first, so that its blocks, whose chain of link tests, own
  // populations and block sums is the longest, do not start last.
  int rot;
};

// The smallest FP32 number whose (correctly rounded) square root is at least
// a: sqrt(t) - a < 0 is t < ball_square(a). (0 for a <= 0.)
float ball_square(float a);

// Row of cell c of a plane of nx-cell rows: umulhi(c, magic) with
// magic = ceil(2^32 / nx), exact while c * nx < 2^32.
LBM_HD unsigned row_magic(int nx) { return (unsigned)(((1ull << 32) + (unsigned)nx - 1) / (unsigned)nx); }

// Launch shape of the dense step (threads per CTA along x, and the CTAs per
// SM the register budget is sized for). Compile-time so the tuning sweep can
// build variants; the defaults are the measured best.
#ifndef LBM_STEP_THREADS
#define LBM_STEP_THREADS 64
#endif
#ifndef LBM_STEP_MIN_BLOCKS
#define LBM_STEP_MIN_BLOCKS 16
#endif
constexpr int kStepThreads = LBM_STEP_THREADS;
constexpr int kStepMinBlocks = LBM_STEP_MIN_BLOCKS;

// The launch blocks of the dense step grid (kStepThreads cells along x, one
// row per block in y and z) that cover an inclusive cell box: per axis the
// first block and first + count, read modulo the grid -- the box of a windowed
// axis can cross the periodic seam (where its cells, not its blocks, wrap: the
// last block of a row may hold fewer cells). A box as long as the axis, or
// whose two ends share a block, covers all of it.
inline void box_region(const int box[6], int nx, int ny, int nz, int r[6]) {
  const int unit[3] = {kStepThreads, 1, 1};
  const int len[3] = {nx, ny, nz};
  for (int a = 0; a < 3; ++a) {
    const int nb = (len[a] + unit[a] - 1) / unit[a], cells = box[2 * a + 1] - box[2 * a] + 1;
    int lo = box[2 * a] % len[a];
    if (lo < 0) lo += len[a];
    const int hi = lo + cells - 1;
    int first = lo / unit[a];
    int count = (hi < len[a] ? hi / unit[a] : nb + (hi - len[a]) / unit[a]) - first + 1;
    if (cells >= len[a] || count >= nb) { first = 0; count = nb; }
    r[2 * a] = first;
    r[2 * a + 1] = first + count;
  }
}
// Force partials summed per block by sum_partials_grouped, and the number of
// such blocks. A dense step of a small body has about a hundred partials: in
// one block the sum is one chain of loads and a block tree, in two or three
// it also has a fence, a ticket and a second chain.
constexpr int kSumGroup = 64, kSumOne = 256;
LBM_HD int sum_groups(int nparts) { return nparts <= kSumOne ? 1 : (nparts + kSumGroup - 1) / kSumGroup; }

// Number of force partials (launch blocks of the force region) of a dense step.
inline int force_parts(int q, const StepParams &p) {
  return (p.rbx1 - p.rbx0) * (p.rby1 - p.rby0) * (q == 9 ? 1 : p.rbz1 - p.rbz0);
}
// Whether launch block (bx, by) of the domain's plane zg, in a dense 3D step of
// gx * gy blocks a plane, is in the force region, and its partial. The region is
// read modulo the grid, as it can cross a windowed seam. A slab's, its own
// share of the domain's planes, has no seam: a plane below it wraps past it.
// (`part` means nothing outside the region. Returning -1 there instead of a
// separate truth value made the 256x128x128 FP16 step 0.7 % slower.)
LBM_HD bool region_part(const StepParams &p, int bx, int by, int zg, int gx, int gy, int &part) {
  int dx = bx - p.rbx0, dy = by - p.rby0, dz = zg - p.rbz0;
  dx += dx < 0 ? gx : 0;
  dy += dy < 0 ? gy : 0;
  dz += dz < 0 ? p.nzg : 0;
  const int rx = p.rbx1 - p.rbx0, ry = p.rby1 - p.rby0, rz = p.rbz1 - p.rbz0;
  part = (dz * ry + dy) * rx + dx;
  return p.force_on && dx < rx && dy < ry && dz < rz;
}
// The blocks that sum the previous step's force take no cells: a sum is a
// chain of loads, a block tree, a fence and a ticket of some microseconds, and
// a step of a small domain (2.7 us without a body at 32^3) would wait for it
// in the blocks that also have cells. `layer`: the blocks of one layer.
inline int sum_layers_for(const StepParams &p, unsigned layer) {
  return p.prev_parts ? (int)((sum_groups(p.prev_parts) + layer - 1) / layer) : 0;
}
// Puts the blocks that sum p.prev_parts in front of a step's launch grid: rows
// in front of a D2Q9 grid (rows = true), layers in front of a 3D one. False,
// and the sum taken out of `p`, where the sum is better a launch of its own
// (launch_force_sum): the grid has no room for the layers, or a 3D layer has
// more than kSumLayer blocks. Most of a layer's blocks only start and leave, 0.4
// ns each, and the launch costs 3 to 5 us: us per step of D3Q19 with a small
// body, with the layer and with the launch, FP32 and FP16, 600x500x5 (4688
// blocks) 40.8 and 44.5, 41.5 and 45.2; 1000x1000x8 (15,625) 198.1 and 197.7,
// 184.2 and 183.3; 1024x1024x8 (16,384) 207.5 and 203.1, 191.7 and 187.2;
// 2048x512x6 (16,384) 157.8 and 154.3, 146.8 and 143.0. (The sum in the grid's
// own first blocks, before their cells: 2 us less for such domains, and 1 %
// more for all others, as the kernel then held the sum and the update in one
// path.)
constexpr unsigned kSumLayer = 12288;
inline bool add_sum_layers(StepParams &p, dim3 &grid, bool rows) {
  unsigned &along = rows ? grid.y : grid.z;
  const unsigned layer = rows ? grid.x : grid.x * grid.y;
  const int layers = sum_layers_for(p, layer);
  if (p.prev_parts && (along + (unsigned)layers > 65535u || (!rows && layer > kSumLayer))) {
    p.sum_layers = p.prev_parts = 0;
    return false;
  }
  p.sum_layers = layers;
  along += layers;
  return true;
}
// Launch grid of a dense 3D step (without the sum layers).
inline dim3 step_grid(const StepParams &p) {
  const int nz = p.nz - 2 * p.zlo;
  if (p.flat) return dim3((unsigned)(((int64_t)p.nx * p.ny + kStepThreads - 1) / kStepThreads), 1, nz);
  return dim3((p.nx + kStepThreads - 1) / kStepThreads, p.ny, nz);
}
constexpr int kReduceThreads = 256;
constexpr int kForceSlots = 8;
constexpr int kTotalsSlots = 8;

// A launch that may begin while the previous kernel on the stream drains
// (programmatic dependent launch): the step and force-sum kernels wait at
// their first instruction (griddepcontrol.wait) until that kernel has
// completed and its writes are visible, so the order is the stream's; what
// overlaps is the new grid's launch and scheduling with the old one's tail.
// Measured on B200 for one-step calls: 0.124 -> 0.120 ms per step, and with
// a force readback after each 0.129 -> 0.124 ms.
template <typename... K, typename... A>
inline cudaError_t launch_pdl(dim3 g, dim3 b, cudaStream_t st, void (*k)(K...), A &&...args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = g;
  lc.blockDim = b;
  lc.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return cudaLaunchKernelEx(&lc, k, std::forward<A>(args)...);
}

// storage: 0 fp32, 1 fp16 offset, 2 bf16 offset
cudaError_t launch_step(int q, int storage, const void *f_in, void *f_out, float *mac,
                        const StepParams &p, cudaStream_t st);
// The sum of `parts` force partials (sum_partials_grouped) as a launch of its
// own, for a step that no following launch sums.
void launch_force_sum(const double *partials, int parts, double *groups, unsigned int *counter, double *out,
                      cudaStream_t st);
// Free-body force pass: the cells near the body (pose p.pose_in), FP64
// force/torque into p.force_out, then the body integrated into p.pose_out.
// `parts` is the launch grid (the largest box's cells, kForceThreads a block).
constexpr int kForceThreads = 128;
cudaError_t launch_force_pass(int q, int storage, const void *f_in, const StepParams &p, int parts, cudaStream_t st);
cudaError_t launch_init_eq(int q, int storage, const float *mac_in, void *f_out, int64_t n, const Pack &pk,
                           cudaStream_t st);
// The equilibrium of one state (rho, ux, uy, uz) in every cell, with that
// state written to mac: the same bits as launch_init_eq of a uniform field.
cudaError_t launch_init_uniform(int q, int storage, const float rho_u[4], float *mac_out, void *f_out, int64_t n,
                                const Pack &pk, cudaStream_t st);
cudaError_t launch_pack(int q, int storage, const float *f32, void *f_store, int64_t n, const Pack &pk,
                        cudaStream_t st);
cudaError_t launch_unpack(int q, int storage, const void *f_store, float *f32, int64_t n, const Pack &pk,
                          cudaStream_t st);
// Totals over the current f, FP64; `partials` holds totals_partials() * 8
// doubles, `counter` one zeroed unsigned int.
int totals_blocks();
// n cells from f (a plane stride of `stride` cells, n when 0).
cudaError_t launch_totals(int q, int storage, const void *f, int64_t n, const Pack &pk, double *partials,
                          unsigned int *counter, double *out, cudaStream_t st, int64_t stride = 0);

// One launch of a batch step over tile positions k0 .. k1-1 of `order`
// (batch.cu); `fluid` selects the lean D2Q9 kernel.
cudaError_t launch_batch_step(int q, int storage, int threads, int ctas, cudaStream_t st, const void *fin,
                              void *fout, float *mac, const StepParams *doms, const int2 *tiles, const int *order,
                              int k0, int k1, int cells_per_tile, int write_mac, bool fluid);

}  // namespace lbm
