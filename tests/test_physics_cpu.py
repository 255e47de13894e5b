"""The stage arithmetic (fvleg_2d_gb300/csrc/cato_physics.cuh) compiled for the host with g++:
the routines that leave work out against the general forms they stand for, bit for bit, over
ordinary and extreme values (tests/physics_check.cpp)."""
import os
import shutil
import subprocess

import pytest

from fvleg_2d_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def families(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    exe = str(tmp_path_factory.mktemp("physics") / "physics_check")
    subprocess.run([gxx, "-O1", "-std=c++17", "-ffp-contract=off", "-I", cuda,
                    os.path.join(HERE, "physics_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "200000"], capture_output=True, text=True, timeout=600)
    out = {}
    for ln in r.stdout.splitlines():
        f = ln.split()
        if " tested " in ln:
            out[f[0]] = (int(f[2]), int(f[4]), r.stdout)
    return out


@pytest.mark.parametrize("family", [
    "mlp3", "mlp5", "roe_sensor", "tvd2", "add_1em16", "one_plus", "to_df", "f2d_int", "div_normal"])
def test_bit_identical_to_the_general_form(families, family):
    tested, bad, log = families[family]
    assert tested >= 100_000 and bad == 0, log
