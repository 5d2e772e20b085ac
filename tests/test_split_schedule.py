"""The split chained SOR's schedule on the CPU: the kernels' own rules
(csrc/frg_split_schedule.h) in a model of their waits (split_model.cpp).  From three
columns on, for every strip and warp division in use: no wait that never ends, no state
or coefficient read before it is written."""
import ctypes
import os
import subprocess

import pytest

from test_chain_schedule import passes_model

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pyflowreg_gb300", "csrc")
WHAT = {1: "a wait never ends", 2: "a fold takes the wrong pixel", 3: "read before written", 4: "slot overwritten"}
# (strips per CTA, fold warps per strip) of the float64 and float32 forms
DIVISIONS = [(1, 4), (1, 6), (1, 8), (2, 4), (2, 6), (4, 2), (4, 3), (4, 4)]


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("model") / "split_model.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, os.path.join(HERE, "split_model.cpp"),
                    "-o", so], check=True)
    return ctypes.CDLL(so)


def _run(model, h, w, M, FC, iterations, lag):
    ps = passes_model(iterations, lag, 5)
    n = len(ps)
    G = (ctypes.c_int * n)(*[g for g, _ in ps])
    cont = (ctypes.c_int * n)(*[int(m < 0) for _, m in ps])
    rc = model.split_model(h, w, M, FC, n, G, cont)
    assert rc == 0, f"{w} columns, {h} rows, M={M}, FC={FC}, lag {lag}: {WHAT[rc]}"


@pytest.mark.parametrize("M,FC", DIVISIONS)
@pytest.mark.parametrize("w", list(range(3, 13)) + [20])
def test_waits_end_and_values_are_there(model, w, M, FC):
    for h in (1, 31, 33, 64, 130, 300):
        _run(model, h, w, M, FC, 15, 5)


@pytest.mark.parametrize("lag", [1, 2, 3, 6, 11, 16])
@pytest.mark.parametrize("w", list(range(3, 11)))
def test_folds_take_the_entering_pixels(model, w, lag):
    """Passes shorter than the stride of a fold warp: several pass boundaries between two of its steps."""
    for M, FC in DIVISIONS:
        for h in (1, 20, 33, 70):
            _run(model, h, w, M, FC, 23, lag)


def test_strips_fit_the_cluster(model):
    """Every level of up to 2048 rows fits a cluster of 16 CTAs, and one of 1024 rows the 8 that any device takes."""
    for strips in range(1, 65):
        for most, reach in ((16, 64), (8, 32)):
            m = model.split_strips_per_cta(strips, most)
            assert m == next((k for k in (1, 2, 4) if -(-strips // k) <= most), 0)
            assert (m > 0) == (strips <= reach)
