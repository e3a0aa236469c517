"""The density pass's division by the kernel radius, in two fmas (div_radius2 in kernels.cu), against IEEE
division over every significand of the numerator: for radii in use, for the largest and smallest
significands, and for random ones.  Powers of two scale both alike, so one binade stands for all (CPU).
"""
import subprocess

import numpy as np

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
static float f32(uint32_t bits) { float f; std::memcpy(&f, &bits, 4); return f; }
int main(int argc, char** argv) {
    for (int k = 1; k < argc; ++k) {
        const float r = f32(uint32_t(std::strtoul(argv[k], nullptr, 10))), y = 1.0f / r;
        long wrong = 0;
        for (uint32_t m = 0; m < (1u << 23); ++m) {
            const float a = f32(0x3f800000u | m), q = a * y;
            wrong += std::fma(std::fma(-r, q, a), y, q) != a / r;
        }
        std::printf("%ld\n", wrong);
    }
}
"""


def test_two_fmas_divide_by_any_radius_as_the_division_does(tmp_path):
    (tmp_path / "division.cpp").write_text(PROGRAM)
    binary = str(tmp_path / "division")
    subprocess.run(["g++", "-std=c++17", "-O3", "-march=native", "-ffp-contract=off", str(tmp_path / "division.cpp"),
                    "-o", binary], check=True)
    used = [s * k for s in (0.01, 0.0166, 0.02, 0.03, 0.05) for k in (1.5, 2.0, 2.5, 3.0, 4.0)]
    used = np.array(used + [2.0 ** -13, 1.0, 1024.0], dtype=np.float32).view(np.uint32)
    one = 0x3F800000
    edges = one + np.concatenate([np.arange(48), (1 << 23) - 1 - np.arange(96)])
    middle = one + np.random.default_rng(3).integers(0, 1 << 23, 128)
    radii = [str(int(b)) for b in np.concatenate([used, edges, middle])]
    out = subprocess.run([binary, *radii], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0"] * len(radii)
