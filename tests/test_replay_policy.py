"""When a prove is issued and when it is replayed from a captured graph (csrc/replay.hpp,
host code): the first call issues, the second captures, and a capture or a graph launch
that fails leaves the call and all later ones to the issued path instead of failing them."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# argv: capture status, status of the first launch, of the later ones, of issuing.  Prints
# what each of five calls did and its status.
DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include "replay.hpp"
int main(int, char **v)
{
    const int cap = std::atoi(v[1]), first = std::atoi(v[2]), later = std::atoi(v[3]), iss = std::atoi(v[4]);
    nkr::ReplayPolicy p;
    bool graph = false;
    int launches = 0;
    for (int k = 0; k < 5; ++k) {
        const int s = p.run([&] { return graph; },
                            [&] { std::printf("c"); graph = cap == 0; return cap; },
                            [&] { std::printf("l"); return launches++ ? later : first; },
                            [&] { std::printf("i"); return iss; });
        std::printf("%d ", s);
    }
    std::printf("\n");
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("replay")
    src, exe = d / "replay.cpp", d / "replay"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "nkr-zkp_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("args,want", [
    ((0, 0, 0, 0), "i0 cl0 l0 l0 l0"),   # issue, capture and replay
    ((3, 0, 0, 0), "i0 ci0 i0 i0 i0"),   # the capture fails: issued, not tried again
    ((0, 2, 0, 0), "i0 cli0 i0 i0 i0"),  # the graph does not launch
    ((0, 0, 2, 0), "i0 cl0 li0 i0 i0"),
    ((0, 0, 0, 2), "i2 i2 i2 i2 i2"),    # a prove that fails is no first prove
    ((3, 0, 0, 2), "i2 i2 i2 i2 i2"),
])
def test_replay_policy(driver, args, want):
    out = subprocess.run([driver] + [str(a) for a in args], capture_output=True, text=True, check=True).stdout
    assert out.split() == want.split()
