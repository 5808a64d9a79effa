"""Host-side checks of the tile layout (a C++ program built from the package's
own sources): renumbering the local vertices for the shared-memory banks keeps
every corner's vertex and is undone by sorted_labels, for tiles of one element
to full ones; and pair_tiles gives every tile to one SM, the larger of an SM's
two among the largest ones of the plan."""

from __future__ import annotations

import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parent.parent
CSRC = ROOT / "apple_gb300" / "csrc"

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <random>
#include "agb_internal.h"
using namespace agb;

static int spread(int points, int cells, int tile_elems, std::mt19937& rng) {
  std::vector<int32_t> c(4 * (size_t)cells);
  std::vector<double> centroid(3 * (size_t)cells), D(9 * (size_t)cells, 0.0), z(cells, 0.0);
  for (int e = 0; e < cells; ++e)
    for (int k = 0; k < 4; ++k) {
      c[4 * e + k] = (int)((e + 10 * k + rng() % 10) % points);  // neighbours
      if (k < 3) centroid[3 * e + k] = (double)e + 0.1 * k;
    }
  TilePlan p;
  if (build_tiles(cells, c.data(), centroid.data(), D.data(), z.data(), z.data(), tile_elems, &p)) return 1;
  TilePlan q = p;
  spread_banks(&q);
  if (q.tile_estart != p.tile_estart || q.group_estart != p.group_estart || q.elem_user != p.elem_user) return 2;
  for (int t = 0; t < p.n_tiles; ++t) {
    const int vs = p.tile_vstart[t], nv = p.tile_vstart[t + 1] - vs;
    for (int b = 0; b < nv; b += 32) {  // a permutation inside blocks of 32
      std::vector<int32_t> x(q.tv_vid.begin() + vs + b, q.tv_vid.begin() + vs + std::min(nv, b + 32));
      std::sort(x.begin(), x.end());
      if (!std::equal(x.begin(), x.end(), p.tv_vid.begin() + vs + b)) return 3;
    }
    for (int e = p.tile_estart[t]; e < p.tile_estart[t + 1]; ++e)
      for (int k = 0; k < 4; ++k)
        if (q.tv_vid[vs + ((q.ids[e] >> (8 * k)) & 255)] != p.tv_vid[vs + ((p.ids[e] >> (8 * k)) & 255)]) return 4;
  }
  std::vector<int32_t> tv;
  std::vector<uint32_t> ids;
  sorted_labels(q, &tv, &ids);
  return tv == p.tv_vid && ids == p.ids ? 0 : 5;
}

static int pairs(int tiles, int sms, std::mt19937& rng) {
  TilePlan p;
  p.n_tiles = tiles;
  p.tile_gstart.assign(1, 0);
  for (int t = 0; t < tiles; ++t) p.tile_gstart.push_back(p.tile_gstart.back() + 1 + (int)(rng() % 30));
  const std::vector<int32_t> order = pair_tiles(p, sms);
  if ((int)order.size() != 2 * sms) return 1;
  std::vector<int> seen(tiles, 0), size;
  for (int t = 0; t < tiles; ++t) size.push_back(p.tile_gstart[t + 1] - p.tile_gstart[t]);
  std::vector<int> ranked = size;
  std::sort(ranked.rbegin(), ranked.rend());
  for (int k = 0; k < sms; ++k) {
    const int a = order[2 * k], b = order[2 * k + 1];
    for (int t : {a, b})
      if (t >= 0 && (t >= tiles || seen[t]++)) return 2;
    if (a >= 0 && size[a] < ranked[std::min(sms, tiles) - 1]) return 3;
    if (b >= 0 && (a < 0 || size[b] > size[a])) return 4;
  }
  for (int t = 0; t < tiles; ++t)
    if (!seen[t]) return 5;
  return 0;
}

int main() {
  std::mt19937 rng(3);
  for (int cells : {1, 2, 31, 33, 700, 3000})
    for (int points : {40, 64, 3000})
      for (int te : {1, 8, 256, 0})
        if (int e = spread(points, cells, te, rng)) { printf("spread %d %d %d: %d\n", points, cells, te, e); return 1; }
  for (int tiles : {1, 151, 152, 153, 250, 303, 304})
    if (int e = pairs(tiles, 152, rng)) { printf("pairs %d: %d\n", tiles, e); return 2; }
  return 0;
}
"""


def test_layout(tmp_path):
    cpp = tmp_path / "check.cpp"
    cpp.write_text(PROGRAM)
    exe = tmp_path / "check"
    cuda = pathlib.Path("/usr/local/cuda/include")
    subprocess.run(["g++", "-O1", "-g", "-fsanitize=address,undefined", "-std=c++17", f"-I{CSRC}", f"-I{cuda}", str(cpp),
                    str(CSRC / "prep.cpp"), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
