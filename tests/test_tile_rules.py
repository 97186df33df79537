"""The rules that cut grids into tiles (csrc/tiles.h), compiled as plain C++: each choice is the best by the
rule's own cost for the blocks that take the tiles."""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <cstdio>
#include "tiles.h"
int main() {
    int x, y, z, wave, lo, off, near;
    while (std::scanf("%d %d %d %d %d %d %d", &x, &y, &z, &wave, &lo, &off, &near) == 7) {
        if (near == -2) {  // the wave in MiB of free memory
            std::printf("%u 0\n", pm::cavity_row_pitch(x, y, z, (size_t)wave << 20));
            continue;
        }
        if (near < 0) {
            std::printf("%d 0\n", pm::choose_hall_zc(x, y, z, 148u, (unsigned)wave, lo));
            continue;
        }
        const unsigned w = pm::yee_tile_blocks((unsigned)wave, near != 0);
        const int zc = pm::choose_zc(x, y, z, w, lo, off);
        std::printf("%d %u\n", zc, pm::grid_for(pm::make_tiles(x, y, z, zc), w));
    }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    cc = shutil.which("g++")
    if not cc:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("tiles")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([cc, "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "pantometry_b200", "csrc"),
                    str(d / "main.cpp"), "-o", str(d / "main")], check=True)

    def run(queries):
        text = "\n".join(" ".join(str(v) for v in q) for q in queries)
        out = subprocess.run([str(d / "main")], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(int(v) for v in line.split()) for line in out.splitlines()]

    return run


def _tiles(x, y, z, zc):
    return -(-x // 32) * -(-y // 8) * -(-z // zc)


@pytest.mark.parametrize("near", [0, 1], ids=["tiles", "beside a box"])
@pytest.mark.parametrize("wave,lo", [(444, 3), (296, 4), (1, 3)])
def test_a_cavitys_chunk_is_the_best_for_the_blocks_that_take_its_tiles(rules, wave, lo, near):
    r = random.Random(5)
    sizes = [(384, 296, 17), (65, 33, 257), (64, 64, 257), (193, 33, 257), (60, 47, 147), (2, 2, 2)]
    sizes += [tuple(r.randint(2, 260) for _ in range(3)) for _ in range(400)]
    blocks = max(1, wave - near)
    for (x, y, z), (zc, grid) in zip(sizes, rules([(*s, wave, lo, 1, near) for s in sizes])):
        def cost(c):
            return (-(-_tiles(x, y, z, c) // blocks) + 0.25) * (c + 1)

        assert grid == min(blocks, _tiles(x, y, z, zc))
        chunks = range(lo - 1, min(65, z + lo), lo)
        assert zc in chunks and cost(zc) == min(cost(c) for c in chunks), (x, y, z, zc)


@pytest.mark.parametrize("wave,lo", [(444, 2), (296, 2), (296, 8)])
def test_a_halls_chunk_is_the_best_by_its_rounds_and_its_sms_planes(rules, wave, lo):
    r = random.Random(6)
    sizes = [(255, 64, 64), (128, 128, 128), (33, 33, 200), (3, 3, 3), (2, 2, 2)]
    sizes += [tuple(r.randint(2, 260) for _ in range(3)) for _ in range(400)]
    for (x, y, z), (zc, _) in zip(sizes, rules([(*s, wave, lo, 0, -1) for s in sizes])):
        def cost(c):
            t = _tiles(x, y, z, c)
            return (0.75 * -(-t // 148) + 0.25 * (t / 148) + -(-t // wave)) * (c + 0.8)

        chunks = range(lo, min(8 * lo + 1, z + lo), lo)
        assert zc in chunks and cost(zc) <= min(cost(c) for c in chunks) * (1 + 1e-12), (x, y, z, zc)


def test_a_cavitys_rows_widen_only_where_all_it_may_allocate_fits(rules):
    r = random.Random(7)
    sizes = [(384, 384, 384), (383, 383, 383), (2047, 1447, 1446), (1619, 1625, 1625), (1, 1, 1), (1275, 1275, 1275)]
    sizes += [tuple(r.randint(1, 1400) for _ in range(3)) for _ in range(200)]
    for free in (0, 16, 1 << 14, 170 << 10):  # MiB
        for (x, y, z), (pitch, _) in zip(sizes, rules([(*s, free, 0, 0, -2) for s in sizes])):
            wide, narrow = (x + 8) // 8 * 8, (x + 4) // 4 * 4
            lattice = wide * (y + 1) * (z + 1)
            fits = lattice < 1 << 32 and 48 * 4 * lattice <= free << 20
            assert pitch == (wide if fits else narrow), (x, y, z, free)
            assert pitch >= x + 1
