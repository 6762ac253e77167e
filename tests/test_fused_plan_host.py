"""The layout of the field solve's joined phases (fused_plan in csrc/pb_poisson.cuh), on the host: over
grids, block counts and level counts, what each block of k_poisson_runs and k_poisson_tiles lays out
in shared memory (the sizes that fused_tables takes) fits what the plan asks for, the tiles cover
level 2 once, every virtual warp has a warp, and every patch index that the kernels form lies in its
array.  And which kernel a solve takes: runs on the small grids, tiles on the larger ones, the general
kernel where neither fits."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "thruster_cx_code_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "pb_poisson.cuh"
using namespace pb;

static void levels(int ny, int nx, int max_coarse, MgLevel* L, int* n) {
  *n = 0;
  while (true) {
    L[*n] = MgLevel{};
    L[*n].ny = ny; L[*n].nx = nx;
    ++*n;
    if ((long)ny * nx <= max_coarse || ny < 4 || nx < 4 || *n >= 15) return;
    ny = ny / 2 + 1;
    nx = nx / 2 + 1;
  }
}

#define NEED(c) do { if (!(c)) { printf("BAD %s: %d x %d, %d levels, %d blocks, block %d\n", #c, ny, nx, nl, nblk, b); exit(1); } } while (0)

// one block's layout; returns the floats it takes ahead of the coarse rows
static long block_floats(const FusedPlan& P, const MgLevel* L, int nl, int nvb, int nblk, int b, std::vector<int>& seen) {
  const int ny = L[0].ny, nx = L[0].nx, N = ny * nx;
  const bool runs = P.runs != 0;
  const MgLevel &L1 = L[1], &L2 = L[2];
  const int vw = nvb * 32, c0 = (int)((long long)b * vw / nblk), c1 = (int)((long long)(b + 1) * vw / nblk);
  NEED(c1 - c0 <= 32);
  int h = 0, w = 0, I0 = 0, J0 = 0;
  if (b < P.ty * P.tx) {
    const int ty = b / P.tx, tx = b - ty * P.tx;
    I0 = ty * L2.ny / P.ty; J0 = tx * L2.nx / P.tx;
    h = (ty + 1) * L2.ny / P.ty - I0; w = (tx + 1) * L2.nx / P.tx - J0;
    for (int y = I0; y < I0 + h; ++y) for (int x = J0; x < J0 + w; ++x) ++seen[y * L2.nx + x];
  }
  const int hw = h * w, halo = runs ? FUSED_HALO : FUSED_HALO_TILE, halo1 = runs ? 3 : 5;
  const int H = 4 * h + halo, W = 4 * w + halo, H1 = 2 * h + halo1, W1 = 2 * w + halo1;
  const int np = hw ? H * W : 0, n1 = hw ? H1 * W1 : 0;
  // the block's own nodes lie on its tile's patch, and their neighbours two away too
  if (hw && !runs) {
    for (int y = 4 * I0; y < std::min(ny, 4 * (I0 + h)); ++y) NEED(y - (4 * I0 - 7) >= 3 && y - (4 * I0 - 7) + 3 < H);
    for (int x = 4 * J0; x < std::min(nx, 4 * (J0 + w)); ++x) NEED(x - (4 * J0 - 7) >= 3 && x - (4 * J0 - 7) + 3 < W);
  }
  // level 1 reads s two rows and columns around its place; level 2 five by five nodes of level 1
  if (hw) {
    NEED(2 * (H1 - 1) + 3 + 2 < H && 2 * (W1 - 1) + 3 + 2 < W);
    NEED(2 * (h - 1) + 4 < H1 && 2 * (w - 1) + 4 < W1);
  }
  const int nv = nvb * 1024, b0 = 32 * c0, b1 = nv + 32 * c0;
  const int l0 = std::max(0, std::min(N, 32 * c1) - b0), l1 = std::max(0, std::min(N, nv + 32 * c1) - b1);
  const int w0 = l0 + 4, w1 = l1 + 4, n0 = l0 ? 5 * w0 : 0, n = runs ? n0 + (l1 ? 5 * w1 : 0) : 0;
  long f = 4L * np + 3L * n1 + 27L * hw + 3L * n + (runs ? n : np) + n + (runs ? n : 0);
  for (int l = 2; l < nl; ++l) f += 32 * ((((long)L[l].ny * L[l].nx + 31) / 32 + nblk - 1) / nblk);
  long nz = 0;
  if (!runs && hw) {
    const int Ya = std::max(0, 2 * I0 - 1), Yb = std::min(L1.ny - 1, 2 * (I0 + h) + 1);
    const int Xa = std::max(0, 2 * J0 - 1), Xb = std::min(L1.nx - 1, 2 * (J0 + w) + 1), sw = Xb - Xa + 1;
    const int W2 = w + 4, n2 = (h + 4) * W2;
    nz = (long)(Yb - Ya + 1) * sw;
    for (int k = 0; k < nz; ++k) {
      const int y = Ya + k / sw, x = Xa + k % sw;
      const int p1 = (y - 2 * I0 + 2) * W1 + x - 2 * J0 + 2, p2 = ((y >> 1) - I0 + 2) * W2 + (x >> 1) - J0 + 2;
      NEED(p1 - W1 - 1 >= 0 && p1 + W1 + 1 < n1 && p1 < 32768);
      NEED(p2 - W2 - 1 >= 0 && p2 + W2 + 1 < n2 && p2 < 65536);
    }
    for (int k = 0; k < np; ++k) {
      const int ly = k / W, lx = k - ly * W, y = 4 * I0 - 7 + ly, x = 4 * J0 - 7 + lx, py = ly - 7, px = lx - 7;
      if (y < 0 || y >= ny || x < 0 || x >= nx) continue;
      const bool own = py >= 0 && py < 4 * h && px >= 0 && px < 4 * w;
      if (py >= -2 && py < 4 * h + 2 && px >= -2 && px < 4 * w + 2) {
        const int Y = y >> 1, X = x >> 1, m01 = (x & 1) && X + 1 < L1.nx, m10 = (y & 1) && Y + 1 < L1.ny;
        const int z = (Y - Ya) * sw + X - Xa;
        NEED(z >= 0 && X - Xa + m01 < sw && z + m10 * sw + m01 < nz);
      }
      if (py >= -1 && py < 4 * h + 1 && px >= -1 && px < 4 * w + 1) NEED(k - W >= 0 && k + W < np);
      if (own) NEED(k - W >= 0 && k + W < np);
    }
    f += 2L * n2 + np;
  } else if (!runs) {
    f += np;
  }
  if (runs) {
    int seg_u[4], seg_c0[4], seg_w[4];
    long seg_at[4], seg_n[4];
    for (int q = 0; q < 4; ++q) {
      const int o = q >> 1, l = o ? l1 : l0, bb = o ? b1 : b0;
      const int y = bb / nx + (q & 1), x0 = bb - (bb / nx) * nx, first = nx - x0;
      const int ua = q & 1 ? first : 0, ub = q & 1 ? l : std::min(l, first);
      seg_u[q] = ua; seg_at[q] = nz; seg_c0[q] = seg_w[q] = 0; seg_n[q] = 0;
      if (ub <= ua) continue;
      const int xa = std::max(0, (q & 1 ? 0 : x0) - 2), xb = std::min(nx - 1, (q & 1 ? 0 : x0) + (ub - ua) - 1 + 2);
      const int Ya = std::max(0, y - 2) >> 1, Yb = std::min(L1.ny - 1, (std::min(ny - 1, y + 2) >> 1) + 1);
      const int Xa = xa >> 1, Xb = std::min(L1.nx - 1, (xb >> 1) + 1), sw = Xb - Xa + 1;
      NEED(ub - ua <= nx);
      seg_c0[q] = Ya << 16 | Xa; seg_w[q] = sw; seg_n[q] = (long)(Yb - Ya + 1) * sw;
      nz += seg_n[q];
    }
    for (int k = 0; k < n; ++k) {
      const bool o = k >= n0;
      const int q = o ? k - n0 : k, rw = o ? w1 : w0, ly = q / rw, lx = q - ly * rw, bb = o ? b1 : b0;
      const int j = bb + (ly - 2) * nx + lx - 2, g = 2 * o + (lx - 2 >= seg_u[2 * o + 1] && seg_w[2 * o + 1] > 0);
      const int x0 = bb - (bb / nx) * nx, xx = g & 1 ? lx - 2 - seg_u[g] : x0 + lx - 2;
      if (j < 0 || j >= N || xx < 0 || xx >= nx) continue;
      const int y = j / nx, x = j - y * nx, Y = y >> 1, X = x >> 1;
      const int m01 = (x & 1) && X + 1 < L1.nx, m10 = (y & 1) && Y + 1 < L1.ny;
      const int z = (Y - (seg_c0[g] >> 16)) * seg_w[g] + X - (seg_c0[g] & 0xFFFF);
      NEED(z >= 0 && z + m10 * seg_w[g] + m01 < seg_n[g]);
      if (ly >= 1 && ly <= 3 && lx >= 1 && lx <= rw - 2) NEED(k - rw >= 0 && k + rw < n);
    }
    for (int o = 0; o < 2; ++o)
      for (int u = 0; u < (o ? l1 : l0); ++u) {
        const int rw = o ? w1 : w0, k = (o ? n0 : 0) + 2 * rw + u + 2;
        NEED(k - rw >= 0 && k + rw < n);
      }
  }
  return f + 20 * nz;
}

int main(int argc, char** argv) {
  if (argc > 1) {  // ny nx blocks periodic max_coarse: the kernel
    MgLevel L[MG_MAX_LEVELS];
    int nl;
    const int ny = atoi(argv[1]), nx = atoi(argv[2]), nblk = atoi(argv[3]), mc = atoi(argv[5]);
    levels(ny, nx, mc, L, &nl);
    const FusedPlan P = fused_plan(L, nl, atoi(argv[4]) != 0, 2, 50, mg_virtual_blocks((long)ny * nx, 148), nblk, mc * 5 / 4);
    printf("%s\n", !P.smem ? "general" : P.runs ? "runs" : "tiles");
    return 0;
  }
  const int ys[] = {8, 9, 17, 33, 48, 54, 64, 65, 68, 81, 85, 99, 128, 129, 160, 200, 257, 258, 321, 400};
  const int xs[] = {8, 15, 33, 65, 137, 195, 256, 257, 284, 321, 374, 512, 568, 801, 1025, 1135, 2049};
  const int bs[] = {9, 18, 61, 74, 147, 148};
  const int mcs[] = {40, 300, 1536, 4096};
  long runs = 0, tiles = 0;
  for (int ny : ys) for (int nx : xs) for (int nblk : bs) for (int mc : mcs) {
    MgLevel L[MG_MAX_LEVELS];
    int nl, b = -1;
    levels(ny, nx, mc, L, &nl);
    const int nvb = mg_virtual_blocks((long)ny * nx, 148), ncap = std::min(MG_MAX_COARSE, mc * 5 / 4);
    const FusedPlan P = fused_plan(L, nl, false, 2, 50, nvb, nblk, ncap);
    if (!P.smem) continue;
    ++(P.runs ? runs : tiles);
    NEED(P.ty * P.tx <= nblk && P.smem <= FUSED_SMEM_MAX && P.croom >= 0);
    std::vector<int> seen((size_t)L[2].ny * L[2].nx, 0);
    for (b = 0; b < nblk; ++b) {
      const long f = block_floats(P, L, nl, nvb, nblk, b, seen);
      NEED(4 * (size_t)(f + P.croom) <= P.smem);
    }
    for (int v : seen) NEED(v == 1);
  }
  printf("ok %ld %ld\n", runs, tiles);
  return runs > 100 && tiles > 100 ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("fused")
    src, exe = d / "fused.cpp", d / "fused"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", CSRC, str(src), "-o", str(exe)], check=True, capture_output=True,
                   text=True)
    return str(exe)


def test_blocks_fit_their_plan(driver):
    out = subprocess.run([driver], check=False, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.parametrize("ny,nx,blocks,periodic,max_coarse,kernel", [
    (65, 284, 148, 0, 1536, "runs"), (53, 229, 148, 0, 1536, "runs"), (85, 374, 148, 0, 1536, "runs"),
    (129, 568, 148, 0, 1536, "tiles"), (257, 1025, 148, 0, 1536, "tiles"), (229, 1014, 148, 0, 300, "tiles"),
    (65, 284, 147, 0, 1536, "runs"), (65, 284, 18, 0, 1536, "tiles"), (65, 284, 3, 0, 1536, "general"),
    (65, 284, 148, 1, 1536, "general"), (401, 1601, 148, 0, 1536, "general"), (513, 2049, 148, 0, 1536, "general")])
def test_kernel_of_a_solve(driver, ny, nx, blocks, periodic, max_coarse, kernel):
    out = subprocess.run([driver] + [str(v) for v in (ny, nx, blocks, periodic, max_coarse)], check=True,
                         capture_output=True, text=True, timeout=60)
    assert out.stdout.strip() == kernel
