"""Lengths of the probe chains that the slot hash gives for keys in lattices, planes, lines and clusters and for bits of
floats, by the very source of the device function compiled for the host."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

SOURCE = os.path.join(os.path.dirname(__file__), "..", "torch-ash_b200", "csrc", "common.cuh")


@pytest.fixture(scope="module")
def hash_keys(tmp_path_factory):
    text = open(SOURCE).read()
    body = re.search(r"__device__ __forceinline__ uint32_t hash_key\(.*?\n}\n", text, re.S).group(0)
    where = tmp_path_factory.mktemp("hash")
    code = ("#include <cstdint>\n#define __device__\n#define __forceinline__ inline\n" + body +
            'extern "C" void hash_all(const int* k, uint32_t* h, long n) {\n'
            "    for (long i = 0; i < n; ++i) h[i] = hash_key(k[4 * i], k[4 * i + 1], k[4 * i + 2], k[4 * i + 3]);\n}\n")
    (where / "h.cpp").write_text(code)
    lib = str(where / "h.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-o", lib, str(where / "h.cpp")], check=True)
    fn = ctypes.CDLL(lib).hash_all

    def hashes(columns):
        n = len(columns[0])
        keys = np.zeros((n, 4), np.int32)
        for d, c in enumerate(columns):
            keys[:, d] = c.astype(np.int64).astype(np.int32)
        assert len(np.unique(keys, axis=0)) == n
        out = np.empty(n, np.uint32)
        fn(keys.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(n))
        return out

    return hashes


def chains(h):
    """Mean and longest distance of a key from its home slot: linear probing in the table of the smallest capacity."""
    n = len(h)
    slots = 1 << int(np.ceil(np.log2(2 * n)))
    home = np.sort(h & np.uint32(slots - 1)).astype(np.int64)
    away = np.maximum.accumulate(home - np.arange(n)) + np.arange(n) - home
    return float(away.mean()), int(away.max())


def lattice(sides, strides):
    axes = np.meshgrid(*[(np.arange(s) - s // 2) << a for s, a in zip(sides, strides)], indexing="ij")
    return [a.ravel() for a in axes]


def random_chains(n, seed=0):
    return chains(np.random.default_rng(seed).integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32))


def check(h, room=1.05):
    """No longer than random slots' but for chance: the mean over 2^18 keys and more scatters by 2 %, the longest by a few."""
    mean, most = chains(h)
    of_random = [random_chains(len(h), s) for s in range(3)]
    assert mean <= room * max(m for m, _ in of_random), (mean, of_random)
    assert most <= 2 * max(m for _, m in of_random), (most, of_random)


# strides of powers of two, alike and mixed, up to 2^18 in each column
@pytest.mark.parametrize("strides", [(0, 0, 0), (4, 4, 4), (9, 9, 9), (13, 13, 13), (18, 18, 18), (18, 0, 0), (0, 18, 0), (0, 0, 18),
                                     (16, 8, 0), (0, 8, 16), (18, 4, 18), (2, 17, 9), (12, 18, 3), (18, 18, 0), (7, 0, 15)])
def test_lattices(hash_keys, strides):
    check(hash_keys(lattice((64, 64, 64), strides)))


@pytest.mark.parametrize("strides", [(22, 8, 24), (24, 14, 24), (22, 22, 22), (24, 24, 24)])
def test_lattices_of_the_widest_strides(hash_keys, strides):
    """Columns of which only the uppermost bits differ, mixed: up to a third longer on average."""
    check(hash_keys(lattice((64, 64, 64), strides)), room=1.35)


@pytest.mark.parametrize("sides,strides", [((1024, 1024), (0, 0)), ((1024, 1024), (10, 0)), ((1024, 1024), (3, 17)),
                                           ((1, 512, 512), (0, 0, 0)), ((512, 1, 512), (0, 0, 9)), ((1 << 20,), (0,)),
                                           ((1 << 20,), (8,)), ((1, 1, 1 << 20), (0, 0, 0)), ((32, 32, 32, 32), (0, 0, 0, 0)),
                                           ((16, 16, 16, 64), (8, 8, 8, 8))])
def test_planes_lines_and_four_columns(hash_keys, sides, strides):
    check(hash_keys(lattice(sides, strides)))


@pytest.mark.parametrize("step", [(1, 1, 1), (1, -1, 0), (3, 5, 7), (1, 1024, 1 << 20), (3000, 1000, 1)])
def test_diagonals(hash_keys, step):
    if max(step) < 1024:
        i = np.arange(1 << 19)
        check(hash_keys([i * s for s in step]))
    else:      # short runs along the first column, on a diagonal
        i, j = np.arange(2000)[:, None], np.arange(200)
        check(hash_keys([(i * step[0] + j).ravel(), (i * step[1] + 0 * j).ravel(), (i * step[2] + 0 * j).ravel()]))


def test_bits_of_floats_and_clusters(hash_keys):
    rng = np.random.default_rng(1)
    whole = np.unique(rng.integers(-60, 61, (400_000, 3)), axis=0).astype(np.float32).view(np.int32)
    check(hash_keys(list(whole.T)))
    ball = np.round(24 * rng.standard_normal((1, 2000, 3))).astype(np.int64)
    balls = (rng.integers(-(2**17), 2**17, (200, 1, 3)) + ball).reshape(-1, 3)
    check(hash_keys(list(np.unique(balls, axis=0).T)))


def test_the_measure_sees_a_linear_hash():
    """A linear combination of the columns, kept as it is: lattices of wide strides crowd into few slots."""
    x, y, z = [c.astype(np.int64).astype(np.uint32) for c in lattice((64, 64, 64), (16, 16, 16))]
    with np.errstate(over="ignore"):
        h = x * np.uint32(0x9E3779B1) + y * np.uint32(0x85EBCA77) + z * np.uint32(0xC2B2AE3D)
    assert chains(h)[0] > 2 * random_chains(len(h))[0]
