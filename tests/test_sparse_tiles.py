"""Tiles of the sparse factorisation's products (csrc/sparse_tiles.h, compiled for
the host): over fronts of k own and m boundary DOFs in launches sized for larger
fronts beside them, every accepted tile starts inside the product and every entry
to be updated is in exactly one accepted tile -- the trailing update of each panel
(everything right of and below it except F22) and F22's own product.  Fronts
without a boundary (the root, or a disconnected part of the mesh) among them."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <vector>
#include "sparse_tiles.h"
using namespace fem25::sp;

// tiles of one front's product in a launch of `count` tiles and tile columns [c0, c0 + cn)
static bool mark(int M, int corner, int count, int c0, int cn, std::vector<int> &hit) {
  for (int tile = 0; tile < count; tile++) {
    int m0 = -1, n0 = -1;
    if (!gemm_tile(M, corner, tile, c0, cn, &m0, &n0)) continue;
    if (m0 < 0 || n0 < 0 || m0 >= M || n0 >= M) return false;
    for (int c = n0; c < n0 + kGt && c < M; c++)
      for (int r = m0; r < m0 + kGt && r < M; r++)
        if (r < corner || c < corner) hit[r + (size_t)c * M]++;
  }
  return true;
}

int main() {
  const int nb = 32, ks[] = {1, 31, 32, 33, 64, 97, 100, 129}, ms[] = {0, 1, 31, 32, 33, 70};
  for (int k : ks)
    for (int m : ms)
      for (int more : {0, 1, 65}) {  // another front of the launch is larger
        const int n = k + m;
        for (int jb = 0; jb < k + more; jb += nb) {
          if (jb >= k) continue;  // the kernel leaves fronts that are done
          const int K = nb < k - jb ? nb : k - jb, M = n - jb - K, corner = k - jb - K;
          const int tr = (n + more - jb + kGt - 1) / kGt;
          std::vector<int> hit((size_t)M * M, 0);
          if (!mark(M, corner, tr, 0, 1, hit) || !mark(M, corner, tr * (tr - 1), 1, tr - 1, hit))
            return std::printf("trailing tile outside: k %d m %d jb %d\n", k, m, jb), 1;
          for (int c = 0; c < M; c++)
            for (int r = 0; r < M; r++)
              if (hit[r + (size_t)c * M] != (r < corner || c < corner))
                return std::printf("trailing entry: k %d m %d jb %d\n", k, m, jb), 1;
        }
        const int tm = (m + more + kGt - 1) / kGt;
        std::vector<int> hit((size_t)m * m, 0);
        if (!mark(m, m, tm * tm, 0, tm, hit)) return std::printf("F22 tile outside: m %d\n", m), 1;
        for (int h : hit)
          if (h != 1) return std::printf("F22 entry: m %d\n", m), 1;
      }
  return 0;
}
"""


def test_product_tiles(tmp_path):
    src, exe = tmp_path / "tiles.cpp", tmp_path / "tiles"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "fem25_b200", "csrc"),
                    "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
