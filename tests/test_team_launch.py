"""What a call does when the cooperative step's launch does not go as usual: the test's process puts
launchers of its own (team/launch_shim.cu) before the library's."""
import os
import subprocess
import sys

import pytest

from sayram2d_gb300 import build

pytestmark = pytest.mark.gpu
TEAM = os.path.join(os.path.dirname(os.path.abspath(__file__)), "team")


@pytest.fixture(scope="module")
def shim(capi, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("shim") / "launch_shim.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", build.CSRC,
                    "-I", os.path.join(build.ROOT, "include"), os.path.join(TEAM, "launch_shim.cu"), "-o", so, "-ldl"],
                   check=True)
    return so


def _child(shim, scenario):
    r = subprocess.run([sys.executable, os.path.join(TEAM, "launch_child.py"), shim, scenario], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "scenario ok" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("scenario", ["first", "second", "bins", "split", "timing", "noalloc first", "noalloc second",
                                      "server"])
def test_a_refused_launch_goes_on_as_separate_kernels(shim, scenario):
    _child(shim, scenario)


@pytest.mark.parametrize("scenario", ["gave up", "gave up split", "gave up autotune", "gave up noalloc",
                                      "gave up server"])
def test_a_wait_that_runs_out(shim, scenario):
    """The barriers of one launch get no polls: its blocks leave, and the host is told."""
    _child(shim, scenario)


@pytest.mark.parametrize("scenario", ["side by side", "beside separate kernels"])
def test_calls_side_by_side_share_the_chip(shim, scenario):
    _child(shim, scenario)
