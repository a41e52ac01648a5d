"""The line search of the tile kernel (search_after, sbk_tile_search.cuh), one
element's record and one lane's code: compiled for the host and driven trial
by trial."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "springback-precomp_b200", "csrc")
NEWTON, SHRINK, SECTION, RETURN, NORM, BEST = range(6)
GO_ON, ACCEPT, HAND_ON = 0, 1, 2

RUNTIME = """
#pragma once
#include <cmath>
#include <cstring>
#define __host__
#define __device__
#define __noinline__
#define __forceinline__ inline
#define __longlong_as_double(v) [](long long i) { double d; std::memcpy(&d, &i, 8); return d; }(v)
typedef struct CUstream_st* cudaStream_t;
using std::isfinite;
using std::fmin;
using std::fmax;
double __shfl_xor_sync(unsigned, double, int, int);
"""

HARNESS = """
#include "sbk_tile_search.cuh"
struct Record {
  double r[9], alpha[9], at[9], dir[9], r0[9], res;
  int stage;
  sbk::TileSearch search;
};
extern "C" int after(Record* e, int evaluated, double full, int met, int reduced) {
  return sbk::search_after(*e, e->search, evaluated != 0, full, met != 0, reduced != 0);
}
"""


class Search(ctypes.Structure):
    _fields_ = [(n, ctypes.c_double) for n in ("phi0", "reach", "s0", "f0", "s1", "f1", "step", "best", "best_step")] + \
               [(n, ctypes.c_int) for n in ("count", "halvings", "side", "last_is_best")]


class Record(ctypes.Structure):
    _fields_ = [(n, ctypes.c_double * 9) for n in ("r", "alpha", "at", "dir", "r0")] + \
               [("res", ctypes.c_double), ("stage", ctypes.c_int), ("search", Search)]


@pytest.fixture(scope="module")
def after(tmp_path_factory):
    d = tmp_path_factory.mktemp("search")
    (d / "cuda_runtime.h").write_text(RUNTIME)
    (d / "harness.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + str(d), "-I" + CSRC,
                    "-I" + os.path.join(ROOT, "include"), str(d / "harness.cpp"), "-o", str(d / "search.so")], check=True)
    f = ctypes.CDLL(str(d / "search.so")).after
    f.argtypes = [ctypes.POINTER(Record), ctypes.c_int, ctypes.c_double, ctypes.c_int, ctypes.c_int]
    return f


def record(slope):
    """An element whose full step (1 along the first mode) was refused; slope: d . r at the step's start."""
    e = Record(res=1.0, stage=NEWTON)
    e.dir[0], e.r0[0] = 1.0, slope
    return e


def step(e):
    return e.at[0] - e.alpha[0]


def test_norm_search_hands_on_a_best_point_that_fails_again(after):
    for evaluated, want in ((1, ACCEPT), (0, HAND_ON)):
        e = record(1.0)  # no descent: the norm decides
        e.r[0] = 2.0
        assert after(e, 1, 2.0, 0, 0) == GO_ON and e.stage == NORM and step(e) == 0.5
        assert after(e, 0, np.nan, 0, 0) == GO_ON and step(e) == 0.25
        assert after(e, 1, 0.99999, 0, 0) == GO_ON and step(e) == 0.125  # the best, too little to stop at
        for k in range(4, 9):
            assert after(e, 0, np.nan, 0, 0) == GO_ON and e.stage == NORM and step(e) == 0.5 ** k
        assert after(e, 0, np.nan, 0, 0) == GO_ON and e.stage == BEST and step(e) == 0.25
        assert after(e, evaluated, 0.99999, 0, 0) == want


def test_section_search_hands_on_a_last_point_that_fails_again(after):
    for evaluated, want in ((1, ACCEPT), (0, HAND_ON)):
        e = record(-1.0)
        e.r[0] = 4.0  # the slope turns within the step
        assert after(e, 1, 4.0, 0, 0) == GO_ON and e.stage == SECTION
        e.r[0] = -0.9  # still down: the interval's new start
        last = step(e)
        assert after(e, 1, 0.9, 0, 0) == GO_ON and e.stage == SECTION
        for _ in range(6):
            assert step(e) > last and after(e, 0, np.nan, 0, 0) == GO_ON and e.stage == SECTION
        assert after(e, 0, np.nan, 0, 0) == GO_ON and e.stage == RETURN and step(e) == last
        assert after(e, evaluated, 0.9, 0, 0) == want


def test_searches_that_find_nothing_hand_on(after):
    e = record(-1.0)
    for k in range(1, 9):
        assert after(e, 0, np.nan, 0, 0) == GO_ON and e.stage == SHRINK and step(e) == 0.5 ** k
    assert after(e, 0, np.nan, 0, 0) == HAND_ON
    e = record(-1.0)
    e.r[0] = 4.0
    assert after(e, 1, 4.0, 0, 0) == GO_ON
    for _ in range(7):
        assert after(e, 0, np.nan, 0, 0) == GO_ON and e.stage == SECTION
    assert after(e, 0, np.nan, 0, 0) == HAND_ON
    assert after(record(1.0), 1, 0.5, 0, 1) == ACCEPT and after(record(1.0), 1, 1e-30, 1, 0) == ACCEPT
