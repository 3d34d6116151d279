"""Room for clusters (resident_clusters of csrc/common.cuh), from which the GEMMs choose how many CTAs share a tile: a size
that the GPU does not have, or of which the runtime does not tell, has no room, so that a call takes another cut
instead of a launch that fails."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "server-benchmark_b200", "csrc")
PROGRAM = """
#include <cstdio>
#include "common.cuh"
__global__ void kernel() {}
int main() {
  static std::atomic<int> cache[awq::kMaxCluster + 1];
  // the kernel has not asked for the sizes above 8, which not every GPU has
  for (const int S : {2, 8, 16, 16, 17, 0}) std::printf("%d ", awq::resident_clusters(kernel, S, 128, 0, cache));
  for (const int S : {2, 16}) std::printf("%d ", (int)cache[S]);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    folder = tmp_path_factory.mktemp("room")
    (folder / "room.cu").write_text(PROGRAM)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", CSRC, "-o",
                    str(folder / "room"), str(folder / "room.cu")], check=True)
    return str(folder / "room")


def rooms(program, **env):
    out = subprocess.run([program], check=True, capture_output=True, text=True, env=dict(os.environ, **env))
    return [int(v) for v in out.stdout.split()]


def test_no_answer_is_no_room_and_not_kept(program):
    assert rooms(program, CUDA_VISIBLE_DEVICES="") == [0] * 6 + [0, 0]


@pytest.mark.gpu
def test_sizes_the_kernel_may_not_have(program):
    two, eight, sixteen, again, *beyond, kept, kept16 = rooms(program)
    assert two >= eight > 0 and kept == two
    assert sixteen == again == 0 and beyond == [0, 0] and kept16 <= 0
