"""The rule that picks the tile of the W8A8 tensor-core GEMM (csrc/qx_int8_tiles.h): the tiles that measured fastest, and
no tile that its own count of cycles puts behind the largest one."""

import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "quixicore-cpu_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "qx_int8_tiles.h"
int main() {
  long long m, n, k;
  int only;
  while (std::scanf("%lld %lld %lld %d", &m, &n, &k, &only) == 4) {
    const qx::Int8Tile t = qx::choose_int8_tile(m, n, k, 148, only);
    long long tiles = 0;
    const int na = only != 0 ? only : 2, bn = m < 256 ? static_cast<int>((m + 31) / 32 * 32) : 256;
    std::printf("%d %d %lld %lld\n", t.na, t.bn, qx::int8_tile_cycles(m, n, k, t.na, t.bn, 148, &tiles),
                qx::int8_tile_cycles(m, n, k, na, bn, 148, &tiles));
  }
}
"""


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    folder = tmp_path_factory.mktemp("tiles")
    source, program = folder / "tiles.cpp", folder / "tiles"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(source), "-o", str(program)], check=True)

    def run(shapes):
        lines = "".join("%d %d %d %d\n" % shape for shape in shapes)
        done = subprocess.run([str(program)], input=lines, capture_output=True, text=True, check=True)
        return [tuple(int(v) for v in line.split()) for line in done.stdout.splitlines()]
    return run


# (256 channels where 128 with as many tokens took 2 to 13 % longer; smaller tiles where they took half to nine tenths)
@pytest.mark.parametrize("m,n,k,tile", [
    (4096, 14336, 4096, (2, 256)), (2048, 28672, 8192, (2, 256)), (2790, 18669, 6560, (2, 256)), (243, 30851, 976, (2, 256)),
    (118, 25456, 4016, (2, 128)), (512, 14336, 4096, (2, 256)), (1024, 14336, 4096, (2, 256)), (300, 14336, 4096, (2, 160)), (1300, 9000, 2048, (1, 224)),
    (200, 2048, 8192, (1, 64)), (512, 1024, 4096, (1, 64)), (2048, 1024, 1024, (1, 128)), (36, 8192, 4096, (1, 64))])
def test_measured_shapes(choose, m, n, k, tile):
    assert choose([(m, n, k, 0)])[0][:2] == tile


def test_never_behind_the_largest_tile(choose):
    rng = random.Random(3)
    shapes = [(int(2 ** rng.uniform(0, 13)), int(2 ** rng.uniform(0, 16)), 16 * int(2 ** rng.uniform(0, 12)), rng.randrange(3))
              for _ in range(3000)]
    for (m, n, k, only), (na, bn, cycles, largest) in zip(shapes, choose(shapes)):
        assert na == only or (only == 0 and na in (1, 2))
        assert bn % 32 == 0 and 32 <= bn <= 256 and (bn == 32 or bn - 32 < m), (m, n, k, only, na, bn)
        assert cycles * 46 <= largest * 50, (m, n, k, only, na, bn)
