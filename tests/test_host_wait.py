"""The wait for results in pinned memory (csrc/host_wait.h), compiled for the CPU: results that arrive late, in any
order or never, and what the look at the stream says then."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from raster_b200 import build

DRIVER = r"""
#include "host_wait.h"
// The stream of the test: `answers` are what the looks at it say in turn; before look number k the words written[k] ..
// written[k + 1] - 1 of `order` receive their results.
extern "C" int run(uint32_t* res, long n, uint32_t* y, const int* answers, const long* written, const long* order, const uint32_t* value,
                   int* looks, int* missing) {
    bool m = true;
    *looks = 0;
    int rc = rstq::await_results(res, n, y, [&]() -> int32_t {
        for (long k = written[*looks]; k < written[*looks + 1]; ++k) res[order[k]] = value[order[k]];
        return answers[(*looks)++];
    }, &m);
    *missing = m;
    return rc;
}
"""
NOT_YET = 0x7FE5A5A5


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("wait")
    (d / "driver.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-O3", "-std=c++17", "-shared", "-fPIC", "-I", build.CSRC, str(d / "driver.cpp"), "-o", str(d / "w.so")], check=True)
    fn = C.CDLL(str(d / "w.so")).run

    def call(n, answers, batches, ready=()):
        value = np.arange(1, n + 1, dtype=np.uint32)
        res = np.full(n, NOT_YET, np.uint32)
        res[list(ready)] = value[list(ready)]
        order = np.array([i for b in batches for i in b] + [0], np.int64)
        written = np.cumsum([0] + [len(b) for b in batches]).astype(np.int64)
        y, a = np.zeros(n, np.uint32), np.array(answers + [-99], np.int32)
        looks, missing = C.c_int(), C.c_int()
        rc = fn(*(x.ctypes.data_as(C.c_void_p) if isinstance(x, np.ndarray) else x for x in
                  (res, C.c_long(n), y, a, written, order, value)), C.byref(looks), C.byref(missing))
        return rc, y, looks.value, missing.value, value
    return call


@pytest.mark.parametrize("n", [1, 31, 32, 33, 100, 4096])
def test_results_that_are_there_need_no_look(run, n):
    rc, y, looks, missing, value = run(n, [], [], range(n))
    assert (rc, looks, missing) == (0, 0, 0) and np.array_equal(y, value)


@pytest.mark.parametrize("n", [1, 33, 100, 4096])
def test_results_that_arrive_while_the_stream_is_busy(run, n):
    idx = np.random.default_rng(n).permutation(n)
    batches = [b.tolist() for b in np.array_split(idx, 3)]
    rc, y, looks, missing, value = run(n, [1, 1, 1], batches)
    assert (rc, looks, missing) == (0, 3 if n > 1 else 1, 0) and np.array_equal(y, value)


@pytest.mark.parametrize("n,never", [(100, 0), (100, 99), (100, 97), (96, 64), (1, 0)])   # first, last, inside a partial group of 32
def test_a_result_that_never_arrives_ends_with_the_stream(run, n, never):
    rest = [i for i in range(n) if i != never]
    rc, y, looks, missing, value = run(n, [1, 1, 0], [[], rest, []])
    assert (rc, looks, missing) == (0, 3, 1)
    assert y[never] == NOT_YET and np.array_equal(y[rest], value[rest])


def test_results_that_arrive_with_the_end_of_the_stream(run):
    rc, y, looks, missing, value = run(70, [1, 0], [[3], [i for i in range(70) if i != 3]])
    assert (rc, looks, missing) == (0, 2, 0) and np.array_equal(y, value)


def test_a_failure_ends_the_wait(run):
    rc, y, looks, missing, value = run(70, [1, -1], [list(range(40)), []])
    assert (rc, looks) == (-1, 2)
