"""The threads of large host copies against a stand-in for the CUDA runtime whose
streams run their work only when something waits for it, and where
cudaStreamPerThread is another stream in every thread: the copies keep the order of
the caller's stream, return errors and give their slabs back."""
import ctypes
import os
import subprocess

import pytest

from rgsplat_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
MIB = 1 << 20


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("hostcopy") / "hostcopy.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    # -Bsymbolic: the stand-in's functions, also where the process has loaded the real ones
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic", "-I" + cuda, "-I" + build.CSRC,
                    "-I" + build.INCLUDE, "-x", "c++", os.path.join(build.CSRC, "hostcopy.cu"),
                    os.path.join(HERE, "hostcopy_fake.cpp"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    for f in (lib.fake_ordered, lib.fake_failing):
        f.argtypes = [ctypes.c_size_t, ctypes.c_int] + ([ctypes.c_int] if f is lib.fake_failing else [])
    lib.fake_user(1)
    assert lib.fake_ordered(32 * MIB, 0) == 0  # from here on the slabs exist
    assert lib.fake_registered() == 1
    yield lib
    lib.fake_user(-1)
    assert lib.fake_registered() == 0


@pytest.mark.parametrize("per_thread", [0, 1])
@pytest.mark.parametrize("nbytes", [1, 8 * MIB - 1, 8 * MIB, 8 * MIB + 1, 9 * MIB + 3, 16 * MIB, 40 * MIB + 17])
def test_order_of_the_callers_stream(lib, nbytes, per_thread):
    for _ in range(3):
        assert lib.fake_ordered(nbytes, per_thread) == 0


@pytest.mark.parametrize("to_host", [0, 1])
@pytest.mark.parametrize("good", [0, 1, 7, 15, 16, 17, 39])
def test_error(lib, good, to_host):
    assert lib.fake_failing(40 * MIB, good, to_host) == 0
    assert lib.fake_ordered(20 * MIB, 0) == 0


def test_last_context_goes_during_a_capture(lib):
    """Another thread's capture in the global mode refuses cudaHostUnregister to a
    thread that is not in the relaxed mode; the block is given back all the same."""
    lib.fake_capturing(1)
    lib.fake_user(-1)
    lib.fake_capturing(0)
    assert lib.fake_dangling() == 0
    assert lib.fake_registered() == 0
    lib.fake_user(1)
    assert lib.fake_ordered(32 * MIB, 0) == 0
    assert lib.fake_registered() == 1


def test_block_that_cannot_be_unregistered(lib):
    """What the driver still holds as page-locked stays mapped, and is used again."""
    lib.fake_no_unregister(1)
    lib.fake_user(-1)
    assert lib.fake_dangling() == 0
    lib.fake_user(1)
    assert lib.fake_ordered(40 * MIB, 0) == 0
    lib.fake_no_unregister(0)
    lib.fake_user(-1)
    assert lib.fake_registered() == 0
    lib.fake_user(1)
    assert lib.fake_ordered(32 * MIB, 0) == 0
    assert lib.fake_registered() == 1
