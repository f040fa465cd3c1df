"""The engine's host code on a recording stand-in for the device (cpp/engine_on_fake_device.cpp): what it does when a call
fails in the middle of a flush."""
from __future__ import annotations

import os
import subprocess

import pytest

import build_ext
from conftest import PKG, REPO


@pytest.fixture(scope="module")
def exe(built):
    out = os.path.join(PKG, "_build", "cpp_tests")
    os.makedirs(out, exist_ok=True)
    inc = ["-I" + os.path.join(REPO, "include"), "-I" + build_ext.CSRC, "-I" + os.path.join(build_ext.CUDA_HOME, "include")]
    path = os.path.join(out, "engine_on_fake_device")
    objs = [os.path.join(build_ext.OBJ, s + ".o") for s in build_ext.CXX_SOURCES]
    # kernels that no scenario reaches stay undefined
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-w", *inc, "-x", "c++", os.path.join(build_ext.CSRC, "llg_engine.cu"),
                        os.path.join(REPO, "tests", "cpp", "engine_on_fake_device.cpp"), "-x", "none", *objs, "-o", path,
                        "-no-pie", "-Wl,--unresolved-symbols=ignore-all"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return path


def run(exe, *args):
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


@pytest.mark.parametrize("call", ["weights", "copy", "record", "wait", "block"])
def test_a_failing_call_leaves_nothing_in_flight(exe, call):
    run(exe, call)
