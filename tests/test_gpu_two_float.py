"""GPU: the two-float numbers of the residual sums and the Chebyshev recurrence
against FP64.  A double splits into a float and a remainder of at most half its
last place, 48 bits or more together; sums and products of two such pairs err
by a few units of 2^-46, quotients by the square of an FP32 reciprocal's error
(2^-44).  Comparisons are those of the pairs' exact values."""
import os
import subprocess

import numpy as np
import pytest

from xpbd_gpu import _native

pytestmark = pytest.mark.gpu

OUT = np.dtype([("split", "<f4", 2), ("sum", "<f8"), ("prod", "<f8"), ("quot", "<f8"), ("wide", "<f8"),
                ("narrow", "<f4"), ("less", "<i4")], align=True)


@pytest.fixture(scope="module")
def ops(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("two_float") / "two_float")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "two_float.cu")
    subprocess.run([_native._nvcc(), *_native.ARCH_FLAGS, "-std=c++17", "-O2", src, "-o", exe], check=True, timeout=300)

    def run(a, b=None, f=None):
        a = np.asarray(a, dtype=np.float64)
        b = np.ones_like(a) if b is None else np.asarray(b, dtype=np.float64)
        f = np.ones(len(a), dtype=np.float32) if f is None else np.asarray(f, dtype=np.float32)
        blob = np.int32(len(a)).tobytes() + a.tobytes() + b.tobytes() + f.tobytes()
        r = subprocess.run([exe], input=blob, stdout=subprocess.PIPE, check=True, timeout=120)
        return np.frombuffer(r.stdout, dtype=OUT)
    return run


def _doubles(n, seed, lo=-30.0, hi=30.0):
    r = np.random.default_rng(seed)
    return r.choice([-1.0, 1.0], n) * r.uniform(1.0, 2.0, n) * np.exp2(np.round(r.uniform(lo, hi, n)))


def _value(split):
    return split[:, 0].astype(np.float64) + split[:, 1].astype(np.float64)


def test_a_split_is_normalised_and_holds_48_bits(ops):
    a = np.concatenate([_doubles(20000, 1), _doubles(5000, 2, -74, -60), _doubles(5000, 3, 100, 126),
                        1.0 + np.arange(-512, 512) * 2.0 ** -30, 0.5 - np.arange(512) * 2.0 ** -53, [0.0]])
    s = ops(a)["split"]
    v = _value(s)
    assert (np.abs(v - a) <= 2.0 ** -48 * np.abs(a)).all()
    # |lo| <= ulp(hi) / 2: the high part is the value rounded to nearest
    np.testing.assert_array_equal(s[:, 0], v.astype(np.float32))


def test_comparisons_are_those_of_the_values(ops):
    a = np.concatenate([np.repeat(_doubles(200, 4), 100)])
    b = a * (1.0 + np.tile(np.arange(-50, 50), 200) * 2.0 ** -29)
    r, q = ops(a, b), ops(b, a)
    va, vb = _value(r["split"]), _value(q["split"])
    np.testing.assert_array_equal(r["less"] != 0, va < vb)
    np.testing.assert_array_equal(q["less"] != 0, vb < va)


def test_operations(ops):
    a, b = _doubles(20000, 5), _doubles(20000, 6)
    r = ops(a, b)
    assert (np.abs(r["sum"] - (a + b)) <= 2.0 ** -44 * np.maximum(np.abs(a), np.abs(b))).all()
    assert (np.abs(r["prod"] - a * b) <= 2.0 ** -44 * np.abs(a * b)).all()
    assert (np.abs(r["quot"] - 1.0 / b) <= 2.0 ** -42 / np.abs(b)).all()


def test_narrow_rounds_like_a_conversion(ops):
    a = np.concatenate([_doubles(20000, 7, -140, 126), 1.0 + np.arange(-64, 64) * 2.0 ** -25, [0.0, np.inf, -np.inf]])
    np.testing.assert_array_equal(ops(a)["narrow"], a.astype(np.float32))


def test_every_float_widens_exactly(ops):
    """Denormal floats too: a material adjoint of 1e-40 is a summand like any other."""
    r = np.random.default_rng(8)
    f = np.concatenate([r.integers(0, 1 << 32, 20000, dtype=np.uint64).astype(np.uint32).view(np.float32),
                        np.arange(1, 2000, dtype=np.uint32).view(np.float32),
                        np.array([0.0, -0.0, np.inf, -np.inf, 1e-40, -1e-45, 1.17549435e-38], dtype=np.float32)])
    f = f[~np.isnan(f)]
    w = ops(np.ones(len(f)), f=f)["wide"]
    np.testing.assert_array_equal(w, f.astype(np.float64))
    np.testing.assert_array_equal(np.signbit(w), np.signbit(f))
