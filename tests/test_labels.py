"""Component labels (csrc/l3d_labels.h, the kernels of removeSmallComponents, mesh.ts:37-87) on the CPU under
random orders of their loads and stores: whatever the order, every vertex of a component ends with one
and the same label."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "luvas.io-3d_b200", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("labels") / "label_orders.so")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-I", CSRC, "-o", out,
                    os.path.join(HERE, "label_orders.cpp")], check=True)
    lib = C.CDLL(out)
    lib.label_orders.argtypes = [C.c_uint32, C.c_void_p, C.c_uint32, C.c_void_p, C.c_uint32]
    lib.label_rank.argtypes, lib.label_rank.restype = [C.c_uint32], C.c_uint32
    return lib


def run(lib, label, edges, seed):
    e = np.ascontiguousarray(edges, np.uint32).reshape(-1)
    assert lib.label_orders(label.size, label.ctypes.data, e.size // 2, e.ctypes.data, seed) == 0
    return label


@pytest.mark.parametrize("n", [1, 2, 4, 5, 6, 9, 33])
def test_a_chain_flattens_to_its_root(lib, n):
    rank = sorted(range(n), key=lib.label_rank)
    for seed in range(1500):
        label = np.zeros(n, np.uint32)
        for i, v in enumerate(rank):  # each vertex leads to the one of next lower rank
            label[v] = rank[max(i - 1, 0)]
        assert (run(lib, label, [], seed) == rank[0]).all(), (seed, label)


@pytest.mark.parametrize("n,edges", [(3, 2), (12, 10), (40, 36), (60, 120)])
def test_random_graphs_have_one_label_per_component(lib, n, edges):
    for seed in range(300):
        rng = np.random.default_rng(seed)
        e = rng.integers(0, n, (edges, 2))
        label = run(lib, np.arange(n, dtype=np.uint32), e, seed)
        want = np.arange(n)  # the smallest vertex of each component
        for _ in range(n):
            for a, b in e:
                want[a] = want[b] = min(want[a], want[b])
        pairs = set(zip(label.tolist(), want.tolist()))
        assert len(pairs) == len(set(label.tolist())) == len(set(want.tolist())), (seed, label)
