"""Which device scheduling flags let a world's wait poll (CPU), and a world under each of them (GPU)."""
import subprocess
import sys

import pytest

from conftest import ROOT
from solunar_b200.build import _cuda_include

AUTO, SPIN, YIELD, BLOCKING, MAP_HOST = 0, 1, 2, 4, 8


def test_waits_poll_only_where_the_runtime_spins(tmp_path):
    (tmp_path / "rule.cpp").write_text('''#include <cstdio>
#include <cstdlib>
#include "status_wait.h"
int main(int argc, char** argv) {
    for (int k = 1; k < argc; ++k) std::printf("%d ", int(slf::polls_under(unsigned(std::atoi(argv[k])))));
}
''')
    binary = str(tmp_path / "rule")
    subprocess.run(["g++", "-std=c++17", "-I", f"{ROOT}/solunar_b200/csrc", "-I", _cuda_include(),
                    str(tmp_path / "rule.cpp"), "-o", binary], check=True)
    flags = [AUTO, SPIN, YIELD, BLOCKING]
    flags += [f | MAP_HOST for f in flags]
    out = subprocess.run([binary, *map(str, flags)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["1", "1", "0", "0"] * 2


@pytest.mark.gpu
def test_worlds_step_alike_under_every_flag(gpu_lib):
    program = """
import sys
from cuda.bindings import driver
driver.cuInit(0)
assert driver.cuDevicePrimaryCtxSetFlags(0, int(sys.argv[1]))[0] == 0
from solunar_b200 import FluidSettings, FluidWorld
w = FluidWorld(FluidSettings())
w.add_box_container((0, 0, 0), (1, 1, 1))
w.fill_box((0, 0, 0), (0.5, 0.5, 0.5))
for _ in range(3):
    w.step(1e-2)
print(w.state_hash())
"""
    hashes = {subprocess.run([sys.executable, "-c", program, str(flags)], check=True, capture_output=True, text=True,
                             cwd=ROOT).stdout for flags in (AUTO, SPIN, YIELD, BLOCKING)}
    assert len(hashes) == 1 and "" not in hashes
