"""The grid of the cell sort without allocation, for devices and shares of any number of SMs (CPU)."""
import subprocess

from conftest import ROOT

MAX_PARTICLES = 1 << 18

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "noalloc_grid.h"
int main(int argc, char** argv) {
    for (int k = 1; k + 1 < argc; k += 2) {
        auto g = slf::noalloc_grid(uint32_t(std::atoi(argv[k])), uint32_t(std::atoi(argv[k + 1])));
        std::printf("%u %d\n", g.blocks, int(g.held));
    }
}
"""


def test_every_call_gets_a_grid_that_runs_at_once_and_reaches_every_particle(tmp_path):
    (tmp_path / "grid.cpp").write_text(PROGRAM)
    binary = str(tmp_path / "grid")
    subprocess.run(["g++", "-std=c++17", "-I", f"{ROOT}/solunar_b200/csrc", str(tmp_path / "grid.cpp"), "-o", binary],
                   check=True)
    cases = [(n, room) for n in (1, 256, 257, 2048, 2049, 100003, MAX_PARTICLES)
             for room in (0, 1, 2, 16, 127, 128, 132, 148, 256, 1000)]
    out = subprocess.run([binary, *(str(v) for c in cases for v in c)], check=True, capture_output=True, text=True)
    grids = [tuple(map(int, line.split())) for line in out.stdout.splitlines()]
    assert len(grids) == len(cases)
    for (n, room), (blocks, held) in zip(cases, grids):
        assert 1 <= blocks <= max(1, min(room, 256)), (n, room)
        assert held == (blocks * 512 * 4 >= n), (n, room)  # four particles a thread in registers, or a stride
        assert blocks == 1 or (blocks - 1) * 256 < n, (n, room)  # no block without particles
        if room >= 128:
            assert held, (n, room)
