"""The order in which the wave kernel's pairs take tiles, its own source compiled for the host: every tile once, and a tile worked out past the end --
the loops step before they test -- divides by nothing that can be zero."""
import os
import re
import subprocess

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ditto_b200", "csrc", "mlp_waves_kernel_sm100.cu")

MAIN = r"""
int main(int argc, char** argv) {
  WavesParams p;
  p.blocks_per_batch = atoi(argv[1]);
  p.blocks = p.blocks_per_batch * atoi(argv[2]);
  const int columns = atoi(argv[3]);
  p.tiles = p.blocks * columns;
  p.per_group = kGroup * columns;
  p.second = atoi(argv[4]);
  const int pairs = min(p.tiles, 74);
  std::vector<int> seen(p.tiles, 0);
  for (int q = 0; q < pairs; ++q) {
    Tile x = tile_at(p, q);
    for (int t = q; t < p.tiles; t += pairs, x = tile_at(p, t)) {
      if (x.rb < 0 || x.rb >= p.blocks || x.n < 0 || x.n >= columns || x.b != x.rb / p.blocks_per_batch || x.row != x.rb % p.blocks_per_batch * 256) return 1;
      ++seen[x.rb * columns + x.n];
    }
  }
  for (int n : seen) if (n != 1) return 2;
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    text = open(SOURCE).read()
    code = re.search(r"struct Tile \{.*?\n(?=\}  // namespace)", text, re.S).group(0)
    assert "Tile tile_at(const WavesParams& p, int t)" in code
    path = tmp_path_factory.mktemp("order")
    (path / "order.cpp").write_text("#include <algorithm>\n#include <cstdlib>\n#include <vector>\nusing std::max;\nusing std::min;\n#define __device__\n#define __forceinline__ inline\nconstexpr int kGroup = 8;\n"
                                    "struct WavesParams { int blocks_per_batch, blocks, tiles, per_group, second; };\n" + code + MAIN)
    subprocess.run(["g++", "-std=c++17", "-O0", str(path / "order.cpp"), "-o", str(path / "order")], check=True)
    return str(path / "order")


# row blocks an entry, entries, columns of tiles: one tile; a last group that is full and one that is not; fewer tiles than pairs; many rounds
@pytest.mark.parametrize("shape", [(1, 1, 1), (8, 1, 1), (8, 1, 16), (16, 1, 5), (9, 1, 16), (64, 1, 16), (64, 1, 4), (13, 1, 20), (3, 24, 12), (2, 4, 37)])
@pytest.mark.parametrize("second", [0, 1])
def test_every_tile_once(program, shape, second):
    assert subprocess.run([program, *map(str, shape), str(second)]).returncode == 0
