"""Steps taken once on each device (csrc/gb_device_once.h): every device gets
its own, whatever other devices did, a step that threw is taken again, and
kernel attributes, which hold for one device, are only set by such steps."""
import ctypes
import os
import re
import subprocess
import threading

import pytest

from conftest import PKG, REPO

CSRC = os.path.join(PKG, "csrc")


@pytest.fixture()
def once(tmp_path):
    so = str(tmp_path / "device_once.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread", "-I", CSRC, "-o", so,
                           os.path.join(REPO, "tests", "device_once_harness.cpp")])
    return ctypes.CDLL(so)


def test_each_device_takes_the_step(once):
    for device in (0, 1, 63, 1, 0):
        assert once.take(device, 0) == 0
    assert [once.taken(d) for d in (0, 1, 2, 63)] == [1, 1, 0, 1]
    assert once.take(64, 0) == 2 and once.take(-1, 0) == 2


def test_a_step_that_threw_is_taken_again(once):
    assert once.take(3, 1) == 1 and once.taken(3) == 0
    assert once.take(3, 0) == 0 and once.taken(3) == 1
    assert once.take(3, 1) == 0 and once.taken(3) == 1


def test_threads_take_it_once(once):
    threads = [threading.Thread(target=lambda: [once.take(d, 0) for d in range(8)]) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert [once.taken(d) for d in range(8)] == [1] * 8


def test_attributes_are_set_per_device():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        src = open(os.path.join(CSRC, name)).read()
        assert "std::once_flag" not in src, name
        # the one checked call; its users stand in a device_once step
        calls = len(re.findall(r"cudaFuncSetAttribute\(", src))
        assert calls == (1 if name == "gb_runtime.cuh" else 0), name
        for body in re.findall(r"\n\{\n(.*?)\n\}", src, re.S):
            if "allow_dynamic_smem(" in body and "cudaFuncSetAttribute" not in body:
                assert re.search(r"device_once once;\n\s*once\.run\(current_device\(\), \[", body), name
