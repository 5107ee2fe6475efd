"""Loads and launch order of the step kernels, by reading their source: a step
overwrites the momenta it reads, and a dependent launch is resident while the
launch before it still writes, so the read-only data path (which is defined for
memory that nothing writes during the kernel) is not theirs."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scp_b200", "csrc")
# the diagnostics walker only reads, and is never a dependent launch
READ_ONLY = {"diag_walk.cuh"}
FILES = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu*")))


def code(name):
    """Source without comments."""
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


@pytest.mark.parametrize("name", [f for f in FILES if f not in READ_ONLY])
def test_no_read_only_loads(name):
    assert not re.findall(r"ld\.global\.nc|__ldg\s*\(|__restrict__", code(name))


def test_dependent_launches_wait_first():
    """Every kernel launched as a dependent waits for the launch before it
    ahead of its first work item."""
    launched = set()
    for f in FILES:
        text = code(f)
        launched |= set(re.findall(r"launch_step_kernel\(\s*(\w+_kernel)\b", text))
        if "launch_step_kernel(fn," in text:   # chosen by step_fn / step2_fn / step_diag_fn
            launched |= {"step_kernel", "step_diag_kernel", "step2_kernel"}
    assert launched == {"step_kernel", "step_diag_kernel", "step2_kernel", "walk_kernel", "r6_kernel"}
    for kernel in launched:
        body = [m for f in FILES for m in re.findall(
            r"\b%s\([^)]*\)\s*\{(.*?)\n\}" % kernel, code(f), flags=re.S)]
        assert len(body) == 1, kernel
        assert 0 <= body[0].find("griddep_wait()") < body[0].find("for_each_piece"), kernel
