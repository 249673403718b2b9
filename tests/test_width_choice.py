"""The autotuner's choice among measured window widths (csrc/width_choice.hpp, host code):
the least work within 3% of the fastest, reported with its own time."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# argv: pairs of a width and its time; a width's work is 100 - width.  Prints the choice.
DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include "width_choice.hpp"
int main(int n, char **v)
{
    std::vector<std::pair<int, float>> t;
    for (int i = 1; i + 1 < n; i += 2) t.push_back({std::atoi(v[i]), float(std::atof(v[i + 1]))});
    const auto c = nkr::choose_width(t, [](int w) { return 100.0 - w; });
    std::printf("%d %.3f\n", c.first, c.second);
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("width")
    src, exe = d / "width.cpp", d / "width"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "nkr-zkp_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("times,want", [
    ([(15, 1.0)], (15, 1.0)),
    ([(15, 1.0), (16, 1.02), (17, 1.5)], (16, 1.02)),  # its own time, not the fastest one's
    ([(15, 1.02), (16, 1.0), (17, 1.04)], (16, 1.0)),
    ([(14, 2.0), (15, 1.0), (16, 1.2)], (15, 1.0)),
])
def test_choice_and_its_time(driver, times, want):
    args = [str(x) for t in times for x in t]
    out = subprocess.run([driver] + args, capture_output=True, text=True, check=True).stdout.split()
    assert int(out[0]) == want[0] and abs(float(out[1]) - want[1]) < 1e-6
