"""A traversal launch counts its rays, and the ones its warps ask for past the end, in 32 bits: the extension rays of a
chunk join its shadow rays (lights + 1 a path) only where (lights + 2) rays a path stay below that."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "bisemutum-engine_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "pt_device.h"
int main(int argc, char** argv) {
    for (int i = 1; i + 1 < argc; i += 2)
        std::printf("%d\n", (int)bsm::one_trace_launch((uint32_t)strtoull(argv[i], 0, 10), (uint32_t)atoi(argv[i + 1])));
}
"""


@pytest.fixture(scope="module")
def one_launch(tmp_path_factory):
    d = tmp_path_factory.mktemp("queue")
    (d / "q.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++20", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(CUDA, "include"), str(d / "q.cpp"), "-o", str(d / "q")], check=True)

    def ask(pairs):
        out = subprocess.run([str(d / "q"), *[str(x) for p in pairs for x in p]], check=True, capture_output=True,
                             text=True).stdout.split()
        return [x == "1" for x in out]
    return ask


def test_joined_queues_stay_countable(one_launch):
    overrun = 152 * 64 * 32   # a warp's lanes for every warp that 152 SMs can hold
    rng = np.random.default_rng(1)
    pairs = [(p, lights) for lights in range(9)
             for p in (1, 2**27, (2**32 - 1) // (lights + 2), 2**32 // (lights + 1) - 1, 2**32 - 1,
                       *(int(x) for x in 2 ** rng.uniform(20, 31.9, 40)))]
    got = one_launch(pairs)
    assert any(got) and not all(got)
    for (paths, lights), one in zip(pairs, got):
        rays = paths * (lights + 2)
        assert one or rays + overrun >= 2**32 - 2**20, (paths, lights)      # no more apart than need be
        assert not one or rays + overrun < 2**32, (paths, lights)
