"""Memory order of the early (programmatic dependent) launches, in the sources: a
kernel that may be placed while the one before it still runs waits for it before
anything else, and reads what that kernel writes by ordinary loads.  A kernel that
read first, or through the read-only path, could see stale values on some runs
only, so this is checked here and not by running one."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "gpluto_dev_b200", "csrc")


def source(name):
    s = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", s)


def files():
    return sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h")))


def test_trigger_and_wait_stand_together():
    n = 0
    for f in files():
        s = source(f)
        n += len(re.findall("griddepcontrol", s))
        pair = re.findall(r"__forceinline__ void step_order\(\) \{\s*asm volatile\("
                          r"\"griddepcontrol.launch_dependents;\" ::: \"memory\"\);\s*asm volatile\("
                          r"\"griddepcontrol.wait;\" ::: \"memory\"\);\s*\}", s)
        n -= 2 * len(pair)
    assert n == 0      # no trigger and no wait outside step_order


def kernels():
    s = source("gp_launch.cu")
    return sorted(set(re.findall(r"\blaunch\([\w.]+, (\w+)<", s)))


def test_every_early_kernel_is_known():
    assert {"sweeps_kernel", "sweep_x_kernel", "sweep_m_kernel", "finish_kernel"} <= set(kernels())
    assert all(k.endswith("_kernel") for k in kernels())


@pytest.mark.parametrize("name", kernels())
def test_early_kernels_wait_first(name):
    """Nothing but declarations without an initial value and constants before step_order()."""
    s = source("gp_kernels.cuh")
    m = re.search(r"\b" + name + r"\(StageArgs<CTT> a[^)]*\) \{(.*?)step_order\(\);", s, re.S)
    assert m, name
    for statement in m.group(1).split(";"):
        t = " ".join(statement.split())
        assert t == "" or t.startswith(("constexpr ", "__shared__ ", "using ")), t


def test_no_read_only_path():
    """The table of constants in gp_crmath.cuh is the one thing read through it."""
    for f in files():
        s = source(f)
        if f == "gp_crmath.cuh":
            s = s.replace("__ldg(&kSinCosTable[j][k])", "")
        assert "__ldg" not in s and "global.nc" not in s, f
        if f == "gp_kernels.cuh":   # the start-up map alone is never launched early
            s = re.sub(r"__global__ void prim2cons_kernel\([^)]*\)", "", s)
            assert "__restrict__" not in s
