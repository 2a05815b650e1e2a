"""The factorisation of multiplier tables over 4-bit floats (csrc/amsim_factor.h): exact for every shipped table, and
quick to give up on tables that have none (it runs whenever a table is opened)."""
import ctypes as C
import os
import subprocess
import time

import numpy as np
import pytest

from conftest import ROOT, SMALL_LUTS, lut_path

SOURCE = r'''
#include "amsim_factor.h"
extern "C" int factor(const uint8_t* entries, int m, uint8_t* f, uint8_t* g, double* unit, int* shape) {
  const amsim::CodeTables c = amsim::factor_table(entries, m);
  *unit = c.unit;
  shape[0] = c.rows_f; shape[1] = c.rows_g;
  for (size_t i = 0; i < c.f.size(); ++i) f[i] = c.f[i];
  for (size_t i = 0; i < c.g.size(); ++i) g[i] = c.g[i];
  return c.slots;
}
'''
LEVELS = np.array([0, .5, 1, 1.5, 2, 3, 4, 6])
LEVELS = np.concatenate([LEVELS, -LEVELS])


@pytest.fixture(scope="module")
def factor(tmp_path_factory):
    d = tmp_path_factory.mktemp("factor")
    (d / "f.cc").write_text(SOURCE)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "approxtrain_b200", "csrc"),
                           "-o", str(d / "f.so"), str(d / "f.cc")])
    lib = C.CDLL(str(d / "f.so"))

    def run(entries, m):
        f, g, unit, shape = np.zeros(129 * 64, np.uint8), np.zeros(129 * 64, np.uint8), C.c_double(), (C.c_int * 2)()
        t = time.perf_counter()
        slots = lib.factor(entries.astype(np.uint8).ctypes.data_as(C.c_void_p), m, f.ctypes.data_as(C.c_void_p),
                           g.ctypes.data_as(C.c_void_p), C.byref(unit), shape)
        t = time.perf_counter() - t

        def codes(x, rows):
            x = x[:rows * slots // 2].reshape(rows, slots // 2)
            out = np.empty((rows, slots))
            out[:, 0::2], out[:, 1::2] = LEVELS[x & 15], LEVELS[x >> 4]
            return np.repeat(out, (1 << m) // rows, axis=0)
        product = codes(f, shape[0]) @ codes(g, shape[1]).T * unit.value if slots else None
        return slots, product, t
    return run


def _values(entries, m):
    return np.ldexp(1.0 + (entries & ((1 << m) - 1)) / (1 << m), entries >> m)


@pytest.mark.parametrize("lut,slots", [("ACC_7", 128), ("MBM_7", 64), ("MIT_7", 128), ("MBM_5", 32), ("MIT_5", 32), ("MBM_3", 32),
                                       ("MIT_3", 32), ("MBM_1", None), ("MIT_1", 32)])
def test_shipped_tables(factor, lut, slots):
    m = int(lut.split("_")[1])
    raw = np.fromfile(lut_path(lut), np.uint8).astype(int).reshape(1 << m, 1 << m)
    entries = ((raw >> 7) << m) + (raw & 0x7f)
    got, product, _ = factor(entries, m)
    assert slots is None or got == slots
    if got:
        assert np.array_equal(product, _values(entries, m))


@pytest.mark.parametrize("seed", range(3))
def test_giving_up_is_quick(factor, seed):
    """Steps between rows are codes, the first row is not within reach of what they leave."""
    n = np.random.default_rng(seed).integers(0, 40, 128)
    i, j = np.meshgrid(np.arange(128), np.arange(128), indexing="ij")
    entries = np.minimum(i + j + n[j], 255)
    slots, product, seconds = factor(entries, 7)
    assert slots == 0 or np.array_equal(product, _values(entries, 7))
    assert seconds < 0.6, seconds    # 0.1 to 0.15 here; 1.9 with every column of every pair worked out
