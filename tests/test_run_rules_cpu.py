"""The limits of the row runs (runrules.h), compiled for the host: what the kernels
compute in 32 bits against Python's integers, up to the largest operands."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("rules") / "librules.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-shared", "-fPIC",
                    "-I", os.path.join(ROOT, "nsp_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "run_rules.cpp"), "-o", so], check=True)
    return C.CDLL(so)


def lengths():
    big = 1 << 27
    yield [big] * 32 + [5]                      # 2^32 + 5
    yield [big] * 31 + [big - 3] + [5]
    yield [(1 << 31) - 1] * 2 + [2 + 7]         # 2^32 + 7
    yield [1 << 26] * 64 + [1]
    yield [1 << 30] * 4 + [1536]
    yield [1536]
    yield [1537]
    yield [12] * 128
    yield [12] * 127 + [13]
    yield [0] * 128
    rng = np.random.default_rng(1)
    for _ in range(300):
        n = int(rng.integers(1, 129))
        top = int(2 ** rng.uniform(0, 31)) - 1
        yield [int(x) for x in rng.integers(0, max(top, 1), n)]


def test_products_of_a_row_do_not_wrap(rules):
    limit = rules.max_ip()
    for lens in lengths():
        assert len(lens) <= rules.max_a()
        got = rules.row_products((C.c_int * len(lens))(*lens), len(lens))
        assert got == min(sum(lens), limit + 1), lens


@pytest.mark.parametrize("warps", [8, 16])
def test_a_block_gives_up_as_a_whole(rules, warps):
    """A wait runs out while the warps of a block look at the flag one after the
    other: all of them stop, or none."""
    for after in range(-1, warps):
        assert rules.warps_that_stop(warps, after) in (0, warps), after
    assert rules.warps_that_stop(warps, warps) == 0
    assert rules.warps_that_stop(warps, 0) == warps


def test_tiles_of_distant_rows_do_not_wrap(rules):
    """Every distance between rows that a 32-bit row pointer allows: values counted
    exactly, or refused; nothing is refused that would fit 110 KB of shared memory
    and the 15 bits that a program word has for it."""
    rng = np.random.default_rng(2)
    steps = [1, 3, 27, 128, 32767, 32768, 1 << 24, (1 << 24) + 3, 1 << 25, 1 << 26, (1 << 27) + 3, 1 << 28,
             1 << 30, (1 << 31) - 1] + [int(2 ** rng.uniform(0, 31)) for _ in range(200)]
    for step in steps:
        for rows in range(1, 129):
            for n in (1, 128):
                exact = (rows - 1) * step + n
                got = rules.tile_values(step, rows, n)
                if got < 0:
                    assert exact * 4 > 110000 and step >= 1 << 15, (step, rows)
                else:
                    assert got == exact < 1 << 23, (step, rows)
