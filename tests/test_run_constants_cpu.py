"""The numbers that test_row_run_cpu restates are those of the kernels' sources."""
import math
import os
import re

import test_row_run_cpu as rules

from conftest import ROOT


def source(name):
    with open(os.path.join(ROOT, "nsp_b200", "csrc", name)) as f:
        return f.read()


def test_constants():
    text = source("runrules.h") + source("internal.h") + source("rowrun.cu")
    got = dict(re.findall(r"constexpr int (k\w+) = (\d+);", text))
    want = {"kMaxLag": rules.MAX_LAG, "kShiftMaxLen": rules.MAX_LEN, "kRunMaxA": rules.MAX_A,
            "kRunMaxIp": rules.MAX_IP, "kRunMin": rules.RUN_MIN, "kRunBlock": rules.BLOCK,
            "kRunSmallIp": rules.SMALL_IP, "kSegReach": rules.REACH}
    assert {k: int(got[k]) for k in want} == want


def test_kernel_sizes():
    found = re.findall(r"struct RunCfg<(\d)> \{.*?WARPS = (\d+),.*?SMEM = ([\d* ]+),", source("rowrun.cu"),
                       re.S)
    sizes = {large == "1": (math.prod(int(x) for x in smem.split("*")), int(warps)) for large, warps, smem in found}
    assert sizes == rules.CLASS
