"""The rule by which a queued force is written by its kernel or copied (psl_destination.h),
compiled for the host: a destination that a kernel could only write with a fault is copied."""
import ctypes
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BASE, SIZE = 0x7F0000000000, 4096


@pytest.fixture(scope="module")
def rule():
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    build = os.path.join(REPO, "tests", "_build")
    os.makedirs(build, exist_ok=True)
    so = os.path.join(build, "destination_host.so")
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(REPO, "periodicshiftlbm_b200", "csrc"),
                    os.path.join(REPO, "tests", "native", "destination_host.cpp"), "-o", so], check=True)
    fn = ctypes.CDLL(so).kernel_may_write_host
    u64 = ctypes.c_uint64
    fn.argtypes = [ctypes.c_int, ctypes.c_int, u64, u64, u64, ctypes.c_uint, u64, u64, ctypes.c_int]

    def ask(offset, device_memory=1, memory_device=0, mapped=None, size=SIZE, access=3, start=BASE, bytes_=24):
        address = BASE + offset
        return bool(fn(device_memory, memory_device, address if mapped is None else mapped, start, size, access, address,
                       bytes_, 0))

    return ask


@pytest.mark.parametrize("offset,fits", [(0, True), (8, True), (SIZE - 24, True), (SIZE - 16, False), (SIZE - 8, False),
                                         (SIZE, False), (SIZE + 8, False), (-8, False)])
@pytest.mark.parametrize("device_memory", [0, 1])
def test_all_three_doubles_lie_in_the_range(rule, offset, fits, device_memory):
    assert rule(offset, device_memory) is fits


def test_short_unknown_or_unwritable_ranges_are_copied(rule):
    assert not rule(0, size=16)
    assert not rule(0, size=0, start=0)  # the driver does not know the range
    assert not rule(0, access=1)  # registered read-only
    assert not rule(0, access=0)
    assert not rule(0, mapped=0)  # not mapped into this device
    assert not rule(0, mapped=BASE + 4)  # misaligned


def test_another_devices_memory_is_copied(rule):
    assert not rule(0, device_memory=1, memory_device=1)
    assert rule(0, device_memory=0, memory_device=1)  # pinned host memory made while that device was current
