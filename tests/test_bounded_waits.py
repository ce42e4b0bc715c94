"""The temporally blocked kernels' bounded wait, compiled for the host against scripted
copies and a scripted clock: no thread gives up without the error flag, and none gives up on
copies that have landed."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "meep_torch_b200", "csrc")

HOST = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#define __device__
#define __forceinline__ inline
struct TbCtl { uint64_t bar; };
struct { unsigned x; } threadIdx;
constexpr unsigned long long WAIT_NS = 1000;
// polls before `lands` fail; the clock jumps by `jump` once, at its second reading
static long polls, lands, reads;
static unsigned long long now, jump;
static bool mbar_try_wait(uint64_t *, uint32_t) { return ++polls > lands; }
static unsigned long long gtimer() { now += 1 + (++reads == 2 ? jump : 0); return now; }
static int atomicExch(int *p, int v) { int o = *p; *p = v; return o; }
%s
int main(int argc, char **argv) {
    threadIdx.x = atoi(argv[1]);
    lands = atol(argv[2]);
    jump = atoll(argv[3]);
    TbCtl ctl{};
    int err = 0;
    const bool ok = tb_wait(ctl, 0, &err);
    printf("%%d %%d\n", (int)ok, err);
}
"""


@pytest.fixture(scope="module")
def wait(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    src = open(os.path.join(CSRC, "yee2d_tb.cuh")).read()
    fn = re.search(r"__device__ __forceinline__ bool tb_wait\(.*?\n}\n", src, re.S).group(0)
    d = tmp_path_factory.mktemp("wait")
    (d / "w.cpp").write_text(HOST % fn)
    subprocess.run(["g++", "-O1", "-o", str(d / "w"), str(d / "w.cpp")], check=True)

    def run(thread, lands, jump):
        out = subprocess.run([str(d / "w"), str(thread), str(lands), str(jump)],
                             capture_output=True, text=True, check=True, timeout=60).stdout
        return tuple(int(v) for v in out.split())
    return run


@pytest.mark.parametrize("thread", [0, 1, 31, 1023])
def test_expired_wait_raises_the_flag_in_any_thread(wait, thread):
    assert wait(thread, 1 << 40, 0) == (0, 1)


@pytest.mark.parametrize("thread", [0, 7, 1023])
def test_landed_copies_are_taken(wait, thread):
    assert wait(thread, 0, 0) == (1, 0)          # at once
    assert wait(thread, 40, 0) == (1, 0)         # while waiting
    # between a poll and a reading of the clock that lies past the limit
    assert wait(thread, 2, 5000) == (1, 0)
