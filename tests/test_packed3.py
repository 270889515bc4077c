"""Packed3 (tl_math.cuh, compiled for the host): three FP64 values in 16 bytes,
each rounded to nearest at 30 bits of its fraction."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests.test_device_math_host import CSRC, CUDA_INCLUDE

SOURCE = r"""
#include "tl_math.cuh"
using namespace tl;
extern "C" void pk(const double* in, double* out, int n) {
  for (int i = 0; i < n; ++i) {
    const V3<double> v = unpack3(pack3(V3<double>{in[3 * i], in[3 * i + 1], in[3 * i + 2]}));
    out[3 * i] = v.x;
    out[3 * i + 1] = v.y;
    out[3 * i + 2] = v.z;
  }
}
"""


@pytest.fixture(scope="module")
def packed(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are missing")
    d = tmp_path_factory.mktemp("packed")
    (d / "pk.cc").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-Wno-unknown-pragmas", f"-I{CUDA_INCLUDE}",
                    f"-I{CSRC}", "-o", str(d / "pk.so"), str(d / "pk.cc")], check=True)
    lib = C.CDLL(str(d / "pk.so"))

    def run(values):
        a = np.ascontiguousarray(values, np.float64).reshape(-1, 3)
        out = np.empty_like(a)
        lib.pk(C.c_void_p(a.ctypes.data), C.c_void_p(out.ctypes.data), a.shape[0])
        return out

    return run


def test_values_are_rounded_to_31_significant_bits(packed):
    rng = np.random.default_rng(1)
    v = rng.standard_normal((4000, 3)) * 10.0 ** rng.uniform(-300, 300, (4000, 3))
    got = packed(v)
    assert np.all(np.abs(got - v) <= 2.0 ** -31 * np.abs(v))
    assert not np.any(got.view(np.uint64) & np.uint64((1 << 22) - 1))
    assert np.array_equal(packed(got).view(np.uint64), got.view(np.uint64))  # what is rounded stays


def test_each_component_has_its_own_low_bits(packed):
    fine = 1.0 + 2.0 ** -30
    for k in range(3):
        v = np.array([2.0, -4.0, 8.0])
        v[k] *= fine
        assert np.array_equal(packed(v)[0], v)


def test_special_values(packed):
    tiny, big = np.finfo(np.float64).tiny, np.finfo(np.float64).max
    v = np.array([[0.0, -0.0, np.inf], [-np.inf, tiny, -tiny], [1e-310, big * (1.0 - 2.0 ** -20), -1.0]])
    got = packed(v)
    assert np.array_equal(np.signbit(got), np.signbit(v))
    assert np.array_equal(got[0], v[0]) and np.array_equal(got[1], v[1])
    assert abs(got[2, 0] - v[2, 0]) <= 5e-324 * 2.0 ** 21 and got[2, 2] == -1.0
    nan = np.array([0x7ff8000000000000, 0xffffffffffffffff, 0x7fffffffffffffff], np.uint64).view(np.float64)
    assert np.isnan(packed(nan)).all()
