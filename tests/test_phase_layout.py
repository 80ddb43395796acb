"""The cut of a multigrid level into the blocks of a cooperative phase (mggrid.cuh,
mgbox.cuh; host code, compiled here with the host compiler): over levels of all
proportions, long rows among them, the form that runs has room for each block's
cells and halo, and every shared-memory region it uses is allotted."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "3d_droplet_simulation_2007_gb300", "csrc")
PROGRAM = r"""
#include <cstdio>
#include <random>
#include "mgbox.cuh"
using namespace dsg::mgg;
static int bad = 0, cuts = 0, staged_for_halo = 0, boxes = 0;
static void fail(const char *what, int x, int y, int z) {
  if (bad++ < 10) printf("%s: %d %d %d\n", what, x, y, z);
}
// regions of mggrid.cuh's phase: u of both colours behind 64 bytes, ei and the
// right-hand side of both colours (last form), the residual
template <class T>
static bool level(int x, int y, int z, int sms, int max_cells, int max_halo, bool finest) {
  Args<T> G{};
  if (!plan(G.g, x, y, z, sms, sizeof(T), max_cells, max_halo) || !layout(G)) return false;
  const Boxes &g = G.g;
  cuts++;
  const int f = form(g), room = f == 1 ? 2 : f == 8 ? 8 : 4;
  const size_t own = (size_t)g.hx * g.ry * g.np, u_end = 64 / sizeof(T) + 2 * (size_t)g.half();
  if (sizeof(T) == 8 && f != 1) fail("one form only in FP64", x, y, z);
  if (own > 256u * f || g.words() > 256 * room) fail("cells or halo", x, y, z);
  if (u_end * sizeof(T) > 0x10000) fail("16-bit offsets", x, y, z);
  if ((size_t)G.o_er < u_end || (size_t)G.o_res < G.o_er + (f > 4 ? 4 * own : 0)) fail("ei and right-hand side", x, y, z);
  if ((G.o_res + (size_t)x * g.ry * g.np) * sizeof(T) > G.shared || G.shared > kMaxShared) fail("shared memory", x, y, z);
  if (g.blocks() > sms) fail("blocks", x, y, z);
  if (f == 8 && g.cells <= 4) staged_for_halo++;
  for (int b = 0; b < g.py; b++)
    if (g.y0(b + 1) - g.y0(b) > g.ry || g.y0(b + 1) <= g.y0(b)) fail("rows", x, y, z);
  for (int b = 0; b < g.pz; b++)
    if (g.z0(b + 1) - g.z0(b) > g.np || g.z0(b + 1) <= g.z0(b)) fail("planes", x, y, z);
  if (g.y0(g.py) != y || g.z0(g.pz) != z) fail("the whole level", x, y, z);
  return true;
}
static void box(int x, int y, int z, int sms) {
  Args<float> G{};
  if (!plan_box(G, x, y, z, sms)) return;
  boxes++;
  const Boxes &g = G.g;
  const size_t items = (size_t)(g.hx / 4) * g.ry * g.np, u = 8 * (size_t)g.half();
  if (kBoxHead + 2 * u + 8 * items > G.shared || G.shared > kBoxShared) fail("box: shared memory", x, y, z);
  if (g.words() / 4 > kBoxHalo * kBoxThreads) fail("box: halo", x, y, z);
  if (g.half() / 4 > 0x10000 || (size_t)g.hx / 2 * (g.ry + g.np) >= 0x10000) fail("box: 16-bit table", x, y, z);
  if (g.blocks() > sms || (g.hx & 3)) fail("box: cut", x, y, z);
}
int main() {
  std::mt19937 r(1);
  auto side = [&](int most) {  // even, spread over the logarithm
    const double e = std::uniform_real_distribution<double>(1.0, std::log2((double)most))(r);
    return 2 * (int)(std::exp2(e) / 2);
  };
  for (int n = 0; n < 4000; n++) {
    const int x = side(1024), y = side(512), z = side(512), sms = n % 3 ? 148 : n % 2 ? 128 : 64;
    if ((long long)x * y * z > (1 << 24)) continue;
    const bool g = level<float>(x, y, z, sms, 8, 8, n & 1);
    level<double>(x, y, z, sms, 1, 2, n & 1);
    if (!g) box(x, y, z, sms);
  }
  level<float>(256, 32, 32, 148, 8, 8, false);
  printf("cuts %d, last form for the halo %d, boxes %d, bad %d\n", cuts, staged_for_halo, boxes, bad);
  return bad || cuts < 500 || staged_for_halo < 5 || boxes < 50;
}
"""


def test_forms_have_room(tmp_path):
    cxx = shutil.which("g++")
    cuda = "/usr/local/cuda/include"
    if cxx is None or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    src, exe = tmp_path / "cuts.cpp", tmp_path / "cuts"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I" + CSRC, "-I" + cuda, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
