"""Rules of the kernels that are launched while their predecessor drains (cato_ctl.cuh,
launch_overlapped), read from the sources: a race would not show in every run."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "fvleg_2d_gb300", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def test_overlapped_kernels_use_no_read_only_loads():
    # the read-only path promises data that is constant from the kernel's start on, which is
    # before its predecessor has written it
    for name in ("cato_stage.cuh", "cato_batch.cuh", "cato_ctl.cuh"):
        code = _code(name)
        for word in ("__ldg", "ld.global.nc", "__restrict__", "ldcs("):
            assert word not in code, (name, word)


def test_tiles_do_not_launch_the_next_kernel():
    # a persistent kernel makes many tiles: the trigger belongs after its last one
    for name in ("cato_stage.cuh", "cato_batch.cuh"):
        code = _code(name)
        for m in re.finditer(r"launch_next\(\)", code):
            before = code[:m.start()]
            assert before.rfind("__global__") > before.rfind("__device__"), (name, before[-300:])
