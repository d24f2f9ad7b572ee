"""The range-restricted reciprocal, quotient and index of csrc/l3d_ieee.h against 1.0f / x, a / b and rintf on
the device: the reciprocal over every float of its range, the index over every float, quotients at
random over theirs."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "luvas.io-3d_b200", "csrc")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("ieee") / "ieee_helpers.so")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "--fmad=false", "-std=c++17", "-Xcompiler",
                    "-fPIC", "-shared", "-I", CSRC, "-o", out, os.path.join(HERE, "ieee_helpers.cu")], check=True)
    return C.CDLL(out)


def counts(f, *args):
    out = (C.c_ulonglong * 2)()
    assert f(*args, out) == 0
    return out[0], out[1]


def test_reciprocal_of_every_float_of_its_range(lib):
    # 251 exponents of 2^23 floats and 2^125 itself, both signs
    assert counts(lib.check_reciprocal) == (2 * (251 * 2**23 + 1), 0)


@pytest.mark.parametrize("seed", range(4))
def test_quotients(lib, seed):
    n, bad = counts(lib.check_quotient, C.c_uint32(seed))
    assert n > 5e8 and bad == 0


@pytest.mark.parametrize("n", [1, 2, 7, 480, 641, 1 << 22])
def test_index_of_every_float(lib, n):
    assert counts(lib.check_index, C.c_uint32(n)) == (2**32, 0)
