"""The chunk size of the batched samples (even_chunk, lgpu_chunks.h) on the host: while
one round of chunks over the blocks takes all electrons, the smallest chunk that
leaves one to a block; beyond that the even share of the rounds that are needed."""
import math
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
BLOCKS, MOST, LEAST = 152, 65535, 1024


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = tmp_path_factory.mktemp("chunk") / "chunk_size_check"
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "loki-mc_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "chunk_size_check.cpp"), "-o", str(exe)])
    return lambda n: [int(x) for x in subprocess.check_output([str(exe), *map(str, (BLOCKS, MOST, LEAST, *n))]).split()]


@pytest.mark.parametrize("n", [
    [1], [1024], [1025], [LEAST * BLOCKS], [LEAST * BLOCKS + 1], [MOST * BLOCKS], [MOST * BLOCKS - 1],
    [10000 + 645 * k for k in range(32)], [20000] * 32, [-500000, 30000, 7], [1] * 152, [65535] * 152, [65536, 65535],
])
def test_one_round(check, n):
    chunk, made, made_smaller, _ = check(n)
    assert LEAST <= chunk <= MOST and made <= BLOCKS
    assert chunk == LEAST or made_smaller > BLOCKS


@pytest.mark.parametrize("n", [
    [MOST * BLOCKS + 1], [500000] * 32, [65536] * 77, [int(10000 * 200 ** (k / 63)) for k in range(64)], [2] * 153,
])
def test_several_rounds(check, n):
    chunk, _, _, fewest = check(n)
    assert fewest > BLOCKS
    rounds = max(1, math.ceil(sum(n) / (BLOCKS * MOST)))
    assert chunk == min(MOST, max(LEAST, math.ceil(sum(n) / (BLOCKS * rounds))))
