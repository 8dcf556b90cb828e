"""rows_share_new_pages (csrc/step_pages.h, host only): which decode batches have rows that read what other rows of the same step
write, against a restatement over sets, for random tables over a small pool and for a pool far larger than its filter."""
import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SOURCE = r"""
#include "step_pages.h"
extern "C" int shares(const int *tables, int width, const int *cached, int n, int block_size) {
    std::vector<glmasr_BlockTable> bts((size_t)n);
    for (int i = 0; i < n; ++i) bts[i].h_table = const_cast<int *>(tables) + (size_t)i * width;
    return glmasr::rows_share_new_pages(bts.data(), cached, n, block_size) ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def shares(tmp_path_factory):
    d = tmp_path_factory.mktemp("step_pages")
    (d / "s.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", ROOT + "/glm_asr_stack_b200/csrc", "-o", str(d / "s.so"),
                    str(d / "s.cpp")], check=True, capture_output=True)
    lib = ctypes.CDLL(str(d / "s.so"))

    def call(tables, cached, block_size):
        t, c = np.ascontiguousarray(tables, np.int32), np.ascontiguousarray(cached, np.int32)
        p = ctypes.POINTER(ctypes.c_int)
        return bool(lib.shares(t.ctypes.data_as(p), t.shape[1], c.ctypes.data_as(p), len(c), block_size))
    return call


def restated(tables, cached, bs):
    new = [int(t[c // bs]) for t, c in zip(tables, cached)]
    old = [set(int(b) for b in t[:c // bs]) for t, c in zip(tables, cached)]        # a page listed twice in one row counts too
    return len(new) > 1 and (len(set(new)) < len(new) or any(b in o for b in new for o in old))


@pytest.mark.parametrize("pool", [12, 60, 400, 5_000_000])
def test_against_sets(shares, pool):
    rng = np.random.default_rng(pool)
    hits = 0
    for _ in range(300):
        n, bs = int(rng.integers(1, 9)), int(rng.choice([1, 4, 16]))
        cached = rng.integers(0, 5 * bs, n)
        tables = rng.integers(0, pool, (n, 6)) if pool < 1000 else rng.integers(0, pool // 4096, (n, 6)) * 4096 + 7   # one filter bit
        got = shares(tables, cached, bs)
        assert got == restated(tables, cached, bs)
        hits += got
    assert 0 < hits < 300 or pool == 12


def test_separate_and_shared_prefix(shares):
    tables = np.arange(256 * 28).reshape(256, 28)
    cached = np.full(256, 27 * 16 + 3)
    assert not shares(tables, cached, 16)
    tables[:, :20] = tables[0, :20]                        # a full prefix shared by all: read by many, written by none
    assert not shares(tables, cached, 16)
    tables[9, 27] = tables[200, 27]
    assert shares(tables, cached, 16)
