"""The layouts of the FP32 source location (csrc/srcloc_shape.cuh): the rule on the
host, and values against FP64 where it changes."""
import ctypes
import os
import subprocess

import pytest

import hmclab_gb300 as H
import test_srcloc_edges as edges

_SOURCE = r"""
#include "srcloc_shape.cuh"
extern "C" int shape(int64_t E, int64_t S, int64_t C) {
  const hmc::SrclocShape s = hmc::srcloc_shape(E, S, C);
  return 100 * s.blocks + s.lanes;
}
"""


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    d = tmp_path_factory.mktemp("srcloc_shape")
    (d / "s.cpp").write_text(_SOURCE)
    csrc = os.path.join(os.path.dirname(H.__file__), "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", csrc, str(d / "s.cpp"), "-o", str(d / "s.so")],
                   check=True)
    f = ctypes.CDLL(str(d / "s.so")).shape
    f.argtypes = [ctypes.c_int64] * 3
    return lambda *a: divmod(f(*a), 100)


def test_every_layout_covers_the_events(shape):
    for E in (1, 7, 8, 9, 10, 16, 17, 25, 64, 65, 130, 1000):
        for S in (1, 29, 30, 99, 100, 1000):
            for C in (1, 32, 2500, 8192, 28_800, 28_801, 65_504, 65_505, 10**6):
                blocks, lanes = shape(E, S, C)
                assert 1 <= blocks <= min(8, -(-E // 8)) and 1 <= lanes <= 8 and (lanes == 8 or E > 8)


def test_full_chips_take_fewer_blocks_and_even_lanes(shape):
    """Eight lanes and up to eight blocks everywhere were up to 1.9 times as slow as one block of 16 lanes here."""
    assert shape(64, 4, 30_000) == (1, 8) and shape(9, 700, 30_000) == (2, 5) and shape(25, 61, 100_000) == (1, 7)
    assert shape(12, 20, 8192) == (2, 6) and shape(130, 4, 8192) == (2, 8) and shape(64, 20, 5000) == (3, 8)
    assert shape(20, 200, 8192) == (3, 8) and shape(130, 200, 8192) == (8, 8) and shape(17, 200, 8192) == (3, 6)
    # few chains, many stations: as measured before
    assert shape(32, 200, 8192) == (4, 8) and shape(130, 200, 200) == (8, 8) and shape(1, 12, 1000) == (1, 8)


@pytest.mark.gpu
@pytest.mark.parametrize("E,S,C", [(9, 61, 2500), (10, 20, 8192), (12, 29, 30_000), (25, 30, 5000), (33, 4, 9000), (130, 5, 8192),
                                   (9, 99, 28_801), (9, 100, 28_769), (20, 10, 65_505), (17, 513, 700)])
@pytest.mark.parametrize("infer", [True, False])
def test_against_the_host(E, S, C, infer):
    edges.test_against_the_host(E, S, C, infer)
