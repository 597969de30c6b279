"""The side streams of a batch's small launches, compiled against a fake of the
CUDA calls they make: a lane runs nothing unless it waits for the fork (the
batch's upload) first, and every lane that ran something is joined."""
import shutil
import subprocess
from pathlib import Path

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "batch_lanes.hpp"

static int fail_wait = 0;      // the wait (counted from 1) that fails, 0: none
static int waits = 0;
static long next_handle = 100;
extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)++next_handle; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)++next_handle; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { printf("record %ld on %ld\n", (long)e, (long)s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    if (++waits == fail_wait) return cudaErrorInvalidValue;
    printf("wait %ld for %ld\n", (long)s, (long)e);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { printf("sync %ld\n", (long)s); return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
struct Ctx {
    static constexpr int kLanes = 3;
    cudaStream_t stream = (cudaStream_t)1;
    cudaStream_t lane[kLanes] = {};
    cudaEvent_t fork = nullptr, join[kLanes] = {};
    bool profile = false;
};
int main(int, char** argv) {
    fail_wait = atoi(argv[1]);
    Ctx c;
    {
        tgp::BatchLanes<Ctx> lanes(&c, 8);
        for (int i = 0; i < 8; ++i) {
            lanes.next();
            printf("launch on %ld\n", (long)c.stream);
        }
        if (!lanes.join()) return 1;
    }
    printf("end on %ld fork %ld\n", (long)c.stream, (long)c.fork);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("lanes")
    (d / "lanes.cpp").write_text(PROGRAM)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = Path(nvcc).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", f"-I{cuda}", f"-I{ROOT / 'turbogp_b200' / 'csrc'}", str(d / "lanes.cpp"), "-o",
                    str(d / "lanes")], check=True)
    return d / "lanes"


@pytest.mark.parametrize("fail_wait", range(0, 4))
def test_a_lane_waits_for_the_fork_before_its_first_launch(program, fail_wait):
    out = subprocess.run([str(program), str(fail_wait)], capture_output=True, text=True, check=True).stdout.splitlines()
    main, fork = "1", out[-1].split()[-1]
    assert out[-1].startswith("end on 1 ")
    behind, ran = set(), set()
    for line in out:
        w = line.split()
        if w[0] == "wait" and w[3] == fork:
            behind.add(w[1])
        if w[0] == "launch":
            ran.add(w[2])
            assert w[2] == main or w[2] in behind, line
    joined = {line.split()[3] for line in out if line.startswith("record")} - {main}
    assert joined == ran - {main}
    assert len(ran) == 4   # a failed wait is tried again at the lane's next turn
