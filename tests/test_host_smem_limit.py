"""The shared-memory limit of a kernel, raised by several threads at once (csrc/smem_limit.h, compiled for the host)."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("shim") / "libsmem_limit.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", "-o", out,
                           "-I", os.path.join(ROOT, "permutohedral_lattice_b200", "csrc"),
                           os.path.join(ROOT, "tests", "helpers", "smem_limit_shim.cpp")])
    return ctypes.CDLL(out)


@pytest.mark.parametrize("sizes", [[100, 20], [20, 100, 50, 70], [100, 100, 100]])
def test_no_thread_finds_less_than_it_asked_for(shim, sizes):
    calls = ctypes.c_int(0)
    assert shim.raise_from_threads((ctypes.c_int * len(sizes))(*sizes), len(sizes), ctypes.byref(calls)) == 0
    assert 1 <= calls.value <= len(set(sizes))


def test_a_failed_driver_call_is_not_taken_for_granted(shim):
    assert shim.raise_after_failure() == 0
