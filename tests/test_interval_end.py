"""The end of an interval of a chain (end_interval, lgpu_interval_end.h) on the host: a
block of threads, one warp of which comes late, leaves what a single thread leaves:
the scalars in the interval's own row and no other, the next interval's control block
or the chain's end, the interval's scalars cleared."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = next((d for d in (os.environ.get("CUDA_HOME", ""), "/usr/local/cuda")
             if d and os.path.exists(os.path.join(d, "include", "cuda_runtime.h"))), None)
pytestmark = pytest.mark.skipif(shutil.which("g++") is None or CUDA is None, reason="needs g++ and the CUDA headers")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = tmp_path_factory.mktemp("end") / "interval_end_check"
    subprocess.check_call(["g++", "-std=c++20", "-O2", "-pthread", "-I", os.path.join(ROOT, "loki-mc_gb300", "csrc"),
                           "-I", os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "interval_end_check.cpp"),
                           "-o", str(exe)])

    def run(*args):
        r = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=60)
        return r.stdout.strip()
    return run


@pytest.mark.parametrize("threads,late", [(128, 0), (128, 1), (128, 2), (128, 3), (1024, 2), (32, 0)])
@pytest.mark.parametrize("go,pos,n,e,sampled,want", [
    (1, 0, 3, 4.0, 1, "ok 1 1 1"),    # the chain goes on
    (1, 14, 16, 8.0, 1, "ok 15 1 15"),
    (1, 2, 3, 4.0, 1, "ok 3 0 2"),    # its last interval
    (1, 1, 3, 8.5, 1, "ok 2 0 1"),    # an energy for the host
    (1, 0, 1, 4.0, 0, "ok 1 0 0"),    # no sample
    (0, 1, 3, 4.0, 1, "ok -1 0 1"),   # stopped before: nothing is touched
])
def test_a_late_warp_changes_nothing(check, threads, late, go, pos, n, e, sampled, want):
    assert check(threads, late, go, pos, n, e, sampled) == want
