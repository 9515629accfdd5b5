"""The launch mapping of the dense 3D step, on the CPU: the host functions the
kernels and the sessions share, compiled into a small program.

For every domain, body and slab, the launch blocks of the force region have
the partials 0 .. force_parts - 1, each exactly once, and every cell of the
body's force box lies in one of them: a block outside must write no partial,
and a step reads as many as it has blocks. And the blocks in front of the grid
that sum the previous step's partials hold each group of them once, the rest
each block of the grid once.
"""
import subprocess

import pytest

PROGRAM = r"""
#include <cstdio>
#include <string>
#include <vector>
#include "host_params.cuh"
using namespace lbm;

static int fail(const lbm_config &c, const char *what, int z0, int nzl) {
  std::printf("%s: %d x %d x %d, body %g at %g %g %g, slab %d + %d\n", what, c.nx, c.ny, c.nz, c.body.a, c.body.cx,
              c.body.cy, c.body.cz, z0, nzl);
  return 1;
}

// slab: planes [z0, z0 + nzl) of the domain (nzl 0: all of it)
static int check(const lbm_config &c, int z0, int nzl) {
  std::string why;
  if (validate_config(&c, why)) return fail(c, why.c_str(), z0, nzl);
  StepParams p{};
  fill_step_params(c, (int64_t)c.nx * c.ny * c.nz, 0, p);
  set_body_regions(c, p, true);
  if (nzl) set_slab(z0, nzl, p);
  const dim3 g = step_grid(p);
  const int parts = p.force_on ? force_parts(c.q, p) : 0;
  std::vector<int> seen(parts, 0);
  int box[6];
  StepParams t = p;
  const bool any = force_cell_box(c, t, box);
  const int len[3] = {c.nx, c.ny, c.nz};
  auto inside = [&](int a, int v) {
    int d = (v - box[2 * a]) % len[a];
    return (d < 0 ? d + len[a] : d) <= box[2 * a + 1] - box[2 * a];
  };
  for (int z = 0; z < (int)g.z; ++z)
    for (int y = 0; y < (int)g.y; ++y)
      for (int x = 0; x < (int)g.x; ++x) {
        const int zg = z + p.zlo + p.zoff;
        int part;
        const bool region = region_part(p, x, y, zg, g.x, g.y, part);
        if (region && (part < 0 || part >= parts)) return fail(c, "partial out of range", z0, nzl);
        if (region && seen[part]++) return fail(c, "partial twice", z0, nzl);
        bool hit = false;  // a cell of the force box in the block
        const int first = x * kStepThreads, lim = p.flat ? c.nx * c.ny : c.nx;
        for (int k = first; k < first + kStepThreads && k < lim; ++k) {
          const int cx = p.flat ? k % c.nx : k, cy = p.flat ? k / c.nx : y;
          hit = hit || (any && inside(0, cx) && inside(1, cy) && inside(2, zg));
        }
        if (hit && !region) return fail(c, "force cell without a partial", z0, nzl);
      }
  for (int k = 0; k < parts; ++k)
    if (!seen[k]) return fail(c, "partial without a block", z0, nzl);
  return 0;
}

// The launch with the sum of `parts` partials in front of the grid.
static int check_sum(const lbm_config &c, int parts) {
  StepParams p{};
  fill_step_params(c, (int64_t)c.nx * c.ny * c.nz, 0, p);
  const bool rows = c.q == 9;
  const dim3 g0 = rows ? dim3((c.nx + kStepThreads - 1) / kStepThreads, c.ny, 1) : step_grid(p);
  dim3 g = g0;
  p.prev_parts = parts;
  if (!add_sum_layers(p, g, rows)) {
    if (parts && !p.prev_parts && g.x == g0.x && g.y == g0.y && g.z == g0.z) return 0;
    return fail(c, "a sum left out changes the grid", 0, parts);
  }
  const int groups = sum_groups(parts);
  std::vector<int> sums(groups, 0);
  std::vector<char> cells((size_t)g0.x * g0.y * g0.z, 0);
  for (int z = 0; z < (int)g.z; ++z)
    for (int y = 0; y < (int)g.y; ++y)
      for (int x = 0; x < (int)g.x; ++x) {
        const int64_t b = x + (int64_t)g.x * (y + (int64_t)g.y * z);
        if ((rows ? y : z) < p.sum_layers) {
          if (b < groups && sums[b]++) return fail(c, "group twice", 0, parts);
          continue;
        }
        const int by = rows ? y - p.sum_layers : y, bz = rows ? z : z - p.sum_layers;
        if (by >= (int)g0.y || bz >= (int)g0.z || cells[((size_t)bz * g0.y + by) * g0.x + x]++)
          return fail(c, "block outside the grid or twice", 0, parts);
      }
  for (int k = 0; k < groups; ++k)
    if (parts && sums[k] != 1) return fail(c, "group without a block", 0, parts);
  for (char k : cells)
    if (k != 1) return fail(c, "cells without a block", 0, parts);
  return 0;
}

int main() {
  for (int parts : {0, 1, 64, 256, 257, 5000, 70000})
    for (int q : {9, 19})
      for (auto &d : {std::vector<int>{40, 24, 26}, {64, 20, 30}, {1024, 300, 4}, {100, 90, 3}, {7, 9, 2000}, {256, 128, 128},
                      {2048, 3, 3}, {2048, 512, 6}, {1000, 1000, 3}}) {
        lbm_config c;
        lbm_config_default(&c, q, d[0], d[1], q == 9 ? 1 : d[2]);
        if (check_sum(c, parts)) return 1;
      }
  lbm_config deep;
  lbm_config_default(&deep, 19, 12, 12, 65532);
  if (check_sum(deep, 612)) return 1;
  const int dims[][3] = {{40, 24, 26}, {64, 20, 30}, {128, 12, 17}, {130, 30, 9}, {7, 9, 40}, {192, 5, 3}, {100, 10, 12}};
  const float at[][3] = {{0.33f, 0.5f, 0.5f}, {0.05f, 0.1f, 0.95f}, {0.9f, 0.9f, 0.02f}, {0.5f, 0.5f, 0.75f}, {0.5f, 3.0f, 0.5f}};
  int n = 0;
  for (auto &d : dims)
    for (auto &f : at)
      for (float a : {1.0f, 3.2f, 6.0f})
        for (int kind = 0; kind < 4; ++kind) {
          lbm_config c;
          lbm_config_default(&c, 19, d[0], d[1], d[2]);
          c.has_body = 1;
          c.use_bounceback = kind != 1;
          c.body.a = a; c.body.b = 0.7f * a; c.body.c = 1.2f * a; c.body.r = 0.1f * a;
          c.body.shape = kind == 2 ? LBM_SHAPE_ROUNDBOX : LBM_SHAPE_SPHERE;
          c.body.cx = f[0] * d[0]; c.body.cy = f[1] * d[1]; c.body.cz = f[2] * d[2];
          if (kind == 3) {
            c.window[0] = c.window[2] = 1;
            c.sponge_w = 2.0f;
          }
          if (check(c, 0, 0)) return 1;
          ++n;
          if (kind == 3) continue;  // a slab takes no window
          for (int R = 1; R <= 4 && R <= d[2]; ++R)
            for (int k = 0; k < R; ++k) {
              const int z0 = d[2] * k / R, z1 = d[2] * (k + 1) / R;
              if (check(c, z0, z1 - z0)) return 1;
              ++n;
            }
        }
  std::printf("ok %d\n", n);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(lbm, tmp_path_factory):
    from getting_air_b200 import build
    d = tmp_path_factory.mktemp("step_map")
    (d / "map.cu").write_text(PROGRAM)
    exe = d / "map"
    subprocess.run([build._nvcc(), "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-ffp-contract=off",
                    "-I", str(build.CSRC), "-o", str(exe), str(d / "map.cu"), str(build.CSRC / "host_params.cu"),
                    str(build.LIB), "-Xlinker", f"-rpath={build.LIB.parent}"], check=True)
    return exe


def test_force_region_blocks_have_the_partials_once(program):
    r = subprocess.run([str(program)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.startswith("ok")
