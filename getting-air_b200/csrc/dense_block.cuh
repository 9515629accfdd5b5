// What the launch blocks of the dense 3D steps decide before their cells: the
// previous step's force sum, the mapping of the block to cells, the share in
// the force region and the kind of update its cells need.
#pragma once

#include "cell_update.cuh"

namespace lbm {

// The previous step's force, by the blocks of the launch's first layers (2D:
// rows); true for such a block, which has no cells.
template <int THREADS = kStepThreads, bool ROWS = false>
__device__ __forceinline__ bool sum_previous(const StepParams &p) {
  const int b = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  if (p.clear_ticket && b == 0 && threadIdx.x == 0) *p.counter = 0u;
  if ((int)(ROWS ? blockIdx.y : blockIdx.z) >= p.sum_layers) return false;
  if (b < sum_groups(p.prev_parts))
    sum_partials_grouped<THREADS>(p.prev_partials, p.prev_parts, p.groups, p.counter, p.force_out, b);
  return true;
}

// Whether a cell of [lo, hi] lies in the interval [a, a + len] read modulo
// n (a in [0, n); len < 0 is empty): the reach-box test of cell3_core for a
// whole span of cells.
__device__ __forceinline__ bool span_hits(int lo, int hi, int a, int len, int n) {
  if (len >= n - 1) return true;
  const int b = a + len;
  return (lo <= b && hi >= a) || (lo + n <= b && hi + n >= a);
}

// What a launch block of the 3D step must evaluate, decided once per block
// (warp-uniform): kGeneral runs cell3 for every cell; kFluid runs
// cell3_fluid, for blocks that take no part in the force reduction, have no
// cell within reach of a bounce-back body (or no body) and touch no wall.
// (Under a moving window the fluid update needs the body's position: a free
// body's step, whose launch does not have it, takes kGeneral.) Penalty bodies reach every cell through chi and always
// take kGeneral (the dense step has a kernel of its own for them). (A third kind without the sponge blend, for blocks beyond
// the sponge band, had fewer instructions per update but a slower step: a
// third hot copy of the update raised instruction-fetch and memory stalls.)
enum BlockKind { kGeneral = 0, kFluid = 1 };

// The block's cells are [lo, hi] of the rows [y0, y1] of plane z (lo = 0 and
// hi = nx - 1 where they span several rows).
// The tests in the order that leaves most blocks early.
__device__ __forceinline__ int block_kind(const StepParams &p, int lo, int hi, int y0, int y1, int z, bool region,
                                          int nbox_on, const int *nbox) {
  if (region) return kGeneral;
  if (p.has_body) {
    if (!p.bb || !nbox_on) return kGeneral;
    if (span_hits(z, z, nbox[4], nbox[5] - nbox[4], p.nzg) && span_hits(y0, y1, nbox[2], nbox[3] - nbox[2], p.ny) &&
        span_hits(lo, hi, nbox[0], nbox[1] - nbox[0], p.nx))
      return kGeneral;
  }
  if ((p.wall_x && (lo == 0 || hi == p.nx - 1)) || (p.wall_y && (y0 == 0 || y1 == p.ny - 1)) ||
      (p.wall_z && (z == 0 || z == p.nzg - 1)))
    return kGeneral;
  return kFluid;
}

// The cells of a launch block and its place in the force region.
struct BlockMap {
  int c0, lim;        // first cell and end: of row by, or (flat) of the plane
  int by, bz, zg;     // row (row mapping), stored plane, the domain's plane
  bool region;        // takes part in the force reduction, as
  int part;           // this partial
};

// bz skips a slab's ghost plane below; zg is the domain's plane, which the
// force region (region_part) and the block kind are in.
__device__ __forceinline__ BlockMap block_map(const StepParams &p, int bcells) {
  BlockMap m;
  m.by = blockIdx.y;
  const int planes = (int)gridDim.z - p.sum_layers;
  int pz = (int)blockIdx.z - p.sum_layers + p.rot;
  pz -= pz >= planes ? planes : 0;
  m.bz = pz + p.zlo;
  m.zg = m.bz + p.zoff;
  m.c0 = blockIdx.x * bcells;
  m.lim = p.flat ? p.nx * p.ny : p.nx;
  m.region = region_part(p, blockIdx.x, m.by, m.zg, gridDim.x, gridDim.y, m.part);
  return m;
}

// Position of cell c (an index of the block's row or plane).
__device__ __forceinline__ void block_cell(const StepParams &p, const BlockMap &m, int c, int &x, int &y) {
  if (p.flat) {
    y = (int)__umulhi((unsigned)c, p.magic);
    x = c - y * p.nx;
  } else {
    y = m.by;
    x = c;
  }
}

__device__ __forceinline__ int block_kind(const StepParams &p, const BlockMap &m, int bcells, int nbox_on,
                                          const int *nbox) {
  const int c1 = min(m.c0 + bcells, m.lim) - 1;
  int lo, hi, y0, y1;
  block_cell(p, m, m.c0, lo, y0);
  block_cell(p, m, c1, hi, y1);
  if (y0 != y1) { lo = 0; hi = p.nx - 1; }
  return block_kind(p, lo, hi, y0, y1, m.zg, m.region, nbox_on, nbox);
}
__device__ __forceinline__ int block_kind(const StepParams &p, const BlockMap &m, int bcells) {
  return block_kind(p, m, bcells, p.nbox_on, p.nbox);
}

}  // namespace lbm
