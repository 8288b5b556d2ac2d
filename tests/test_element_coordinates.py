"""The division by which the stage kernels find an element's place in a box: nwb::set_divider
itself, compiled for the host, and the kernels on boxes with long axes."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

HOST = r"""
#include "nwb_internal.h"
#include <cstdio>
#include <random>
int main() {
    std::mt19937_64 g(11);
    const unsigned top = 1u << 25;
    for (int k = 0; k < 3000; ++k) {
        const unsigned d = k < 600 ? k + 1 : k < 602 ? top - (k - 600) : 1 + g() % top;
        unsigned mul;
        int shift;
        nwb::set_divider(static_cast<int>(d), &mul, &shift);
        for (int t = 0; t < 400; ++t) {
            unsigned long long n = t % 2 ? g() % top : (g() % (top / d + 1)) * d - t % 4 / 2;
            if (t < 2) n = t ? top - 1 : 0;
            if (n >= top) continue;
            // as struct_coords() has it
            if (static_cast<int>((n * mul) >> shift) != static_cast<int>(n / d)) return printf("%llu / %u\n", n, d), 1;
        }
    }
    return printf("ok\n"), 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++") or not os.path.exists(f"{CUDA}/include/cuda_runtime.h"),
                    reason="no host compiler or CUDA headers")
def test_set_divider_is_exact_below_2_to_25(tmp_path):
    src, exe = tmp_path / "d.cpp", tmp_path / "d"
    src.write_text(HOST)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "nekwave_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", f"{CUDA}/include", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("N", range(2, 11))
@pytest.mark.parametrize("nel,per", [((37, 5, 3), (True, False, True)), ((3, 41, 2), (False, True, False)),
                                     ((1, 7, 29), (True, True, True))])
def test_boxes_with_a_long_axis(gpu, N, nel, per):
    """Axes that are no power of two, structured: against the oracle (rounding and FMA
    contraction only)."""
    from oracle import oracle as O
    from tests.gpu_helpers import random_state, rel_max, solver_for
    m = O.box_mesh(N, nel, (0, 0, 0), (1.0, 1.3, 0.9), per)
    s = solver_for(m, 1.0)
    assert s.info()["structured"] == nel
    u = random_state(m, N)
    s.uploadState(u)
    assert rel_max(s.evalRhs(), O.rhs(m, 1.0, u)) < 1e-12
    s.finalize()
