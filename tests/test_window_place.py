"""The corner bound of the exact evaluators (csrc/l3d_window.cuh) on the CPU: a window that it calls inside
has no lost sample and every bilinear footprint in the image, one that it calls outside has a lost
sample, for ordinary homographies, ones that graze a border, images one pixel wide or high and
homographies with rows of zeros."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "luvas.io-3d_b200", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("window")
    (d / "cuda_runtime.h").write_text("")
    out = str(d / "window_place.so")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-march=x86-64-v3", "-fPIC", "-shared", "-I", str(d),
                    "-I", CSRC, "-o", out, os.path.join(HERE, "window_place.cpp")], check=True)
    return C.CDLL(out)


def homographies(rng, n, W, H, px, py):
    """Scalings and rotations about the window's image, which lies anywhere around the image's borders, with
    a tilt; a third of them exact (whole numbers and no tilt), a tenth with zeroed rows."""
    s, a = rng.uniform(0.05, 2.0, n), rng.uniform(-np.pi, np.pi, n)
    exact = rng.random(n) < 0.33
    s[exact], a[exact] = rng.integers(0, 3, exact.sum()), rng.integers(0, 4, exact.sum()) * (np.pi / 2)
    at = [rng.choice([-6, -5, 0, 1, 5, 5.5, 6], n) + rng.choice([0, d - 1, d / 2, d - 6], n) for d in (W, H)]
    h = np.zeros((n, 9))
    c, t = np.cos(a), np.sin(a)
    c[exact], t[exact] = np.round(c[exact]), np.round(t[exact])
    h[:, 0], h[:, 1], h[:, 3], h[:, 4] = s * c, -s * t, s * t, s * c
    h[:, 2] = at[0] - h[:, 0] * px - h[:, 1] * py
    h[:, 5] = at[1] - h[:, 3] * px - h[:, 4] * py
    h[:, 6:8] = np.where(exact[:, None], 0.0, rng.normal(scale=2e-3, size=(n, 2)))
    h[:, 8] = 1.0
    w = h[:, 6] * px + h[:, 7] * py
    h[:, 8] -= w
    scale = 10.0 ** rng.uniform(-9, 9, n)
    h[~exact] *= scale[~exact, None]
    zero = rng.random(n) < 0.1
    h[zero, :3] = 0.0
    zero = rng.random(n) < 0.1
    h[zero, 3:6] = 0.0
    odd = rng.random(n) < 0.02
    h[odd, rng.integers(0, 9, odd.sum())] = rng.choice([np.nan, np.inf, -np.inf, 3e38, 1e-42], odd.sum())
    with np.errstate(over="ignore"):
        return h.astype(np.float32)


@pytest.mark.parametrize("side,dilation", [(6, 2), (11, 1)])
@pytest.mark.parametrize("size", [(1, 1), (1, 40), (40, 1), (2, 2), (11, 12), (64, 48), (1001, 7)])
def test_places_stand_for_every_sample(lib, side, dilation, size):
    W, H = size
    n = 40000
    rng = np.random.default_rng(W * 100 + H + side)
    px, py = rng.integers(0, 800, n).astype(np.float32), rng.integers(0, 600, n).astype(np.float32)
    h = np.ascontiguousarray(homographies(rng, n, W, H, px, py))
    pxy = np.ascontiguousarray(np.stack([px, py], -1))
    for ulps in (-1, 0, 1):
        counts = np.zeros(5, np.int32)
        lib.window_places(n, h.ctypes.data_as(C.c_void_p), pxy.ctypes.data_as(C.c_void_p), side, dilation, W, H, ulps,
                          counts.ctypes.data_as(C.c_void_p))
        assert counts[3] == 0 and counts[4] == 0, counts
        assert counts[1] > n // 20 and counts[2] > n // 200
        assert counts[0] > n // 200 or min(W, H) < 11
