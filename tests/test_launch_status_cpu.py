"""A failed launch is reported by the call that made it and by no later one: the launch helpers over a fake of the CUDA runtime."""
import ctypes
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    from pam_b200 import build
    import pathlib
    cuda = pathlib.Path(build._nvcc()).resolve().parents[1] / "include"
    out = tmp_path_factory.mktemp("launch") / "liblaunch.so"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", f"-isystem{cuda}", "-x", "c++", "-o", str(out),
                           str(ROOT / "tests" / "launch_status_shim.cpp")])
    return ctypes.CDLL(str(out))


@pytest.mark.parametrize("entry", ["shim_failed_launch", "shim_failed_call"])
@pytest.mark.parametrize("error", [1, 2, 9, 701])
def test_the_next_call_does_not_report_it_again(shim, entry, error):
    status, recorded, after = (ctypes.c_int(7) for _ in range(3))
    getattr(shim, entry)(error, *(ctypes.byref(v) for v in (status, recorded, after)))
    assert (status.value, recorded.value, after.value) == (-5, error, 0)
