"""The scalar steps of the on-chip CG (csrc/tg_scalar.cuh) on the CPU: quotients
from a reciprocal, and sums of squares as integers at the scale of the last total."""
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include <cstring>
#include "tg_scalar.cuh"
using namespace tg;
template <typename R> static double total(const R* v, int n, double last, int* ok) {
  const int ref = fx_total_ref(last);
  unsigned long long lo = 0, hi = 0;
  for (int i = 0; i < n; i++) {
    const FxTerm q = fx_term(v[i], ref);
    lo += q.low + ((unsigned long long)q.mid << 26);
    hi += q.top;
  }
  hi += lo >> 52;
  double t;
  *ok = fx_total_value((unsigned)lo & 0x3ffffff, (unsigned)(lo >> 26) & 0x3ffffff, (unsigned)hi, ref, t);
  return t;
}
int main() {
  double h[4];
  static double d[4096]; static float f[4096];
  while (fread(h, sizeof h, 1, stdin) == 1) {  // kind, n or a, last or b
    double out[2] = {0, 0};
    int ok = 1;
    if (h[0] == 0) { out[0] = div_newton(h[1], h[2]); out[1] = div_corrected(h[1], h[2], 1.0 / h[2]); if (h[3] != 0) out[0] = div_newton<false>(h[1], h[2]); }
    else {
      const int n = (int)h[1];
      if (fread(d, 8, n, stdin) != (size_t)n) return 1;
      for (int i = 0; i < n; i++) f[i] = (float)d[i];
      out[0] = h[0] == 1 ? total(d, n, h[2], &ok) : total(f, n, h[2], &ok);
      out[1] = ok;
    }
    fwrite(out, sizeof out, 1, stdout);
  }
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("sc")
    (d / "h.cu").write_text(HARNESS)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                    f"-I{ROOT}/thirring2d_gb300/csrc", f"-I{ROOT}/include", "-o", str(d / "h"), str(d / "h.cu")],
                   check=True, capture_output=True)

    def run(data):
        out = subprocess.run([str(d / "h")], input=data, capture_output=True, check=True).stdout
        return np.frombuffer(out).reshape(-1, 2)
    return run


@pytest.mark.parametrize("spread", [1, 200, 800])
def test_quotients_are_within_an_ulp(harness, spread):
    """One residual correction of a quotient that is right to 2^-44: the result is
    within (1/2 + 2^-40) ulp of the exact one; 0.75 ulp allowed."""
    rng = np.random.default_rng(spread)
    a = rng.uniform(1, 2, 3000) * 2.0 ** rng.integers(-100, 100, 3000)
    b = rng.uniform(1, 2, 3000) * 2.0 ** rng.integers(-spread, spread + 1, 3000)
    b[:4] = [1.0, np.nextafter(2, 1), np.nextafter(1, 2), 1.5]
    got = harness(np.stack([np.zeros_like(a), a, b, np.zeros_like(a)], 1).tobytes())
    for x, y, g in zip(a, b, got):
        q = Fraction(x) / Fraction(y)
        for v in g:
            assert abs(Fraction(v) - q) <= Fraction(3, 4) * Fraction(math.ulp(float(v)))


def test_uncorrected_quotients(harness):
    """An FP32 reciprocal (seed error under 2^-22) and one Newton step: 2^-43 relative."""
    rng = np.random.default_rng(8)
    a, b = rng.uniform(1, 2, 1000), rng.uniform(1, 2, 1000) * 2.0 ** rng.integers(-300, 300, 1000)
    got = harness(np.stack([np.zeros_like(a), a, b, np.ones_like(a)], 1).tobytes())[:, 0]
    assert np.all(np.abs(got * b / a - 1) < 2.0 ** -43)


def test_divisions_outside_the_range_are_plain(harness):
    a = np.array([1.0, 1.0, 0.0, 3.0, -2.0, 1.0, 5.0])
    b = np.array([0.0, np.inf, 0.0, np.nan, -4.0, 1e-300, 1e300])
    got = harness(np.stack([np.zeros_like(a), a, b, np.zeros_like(a)], 1).tobytes())[:, 0]
    with np.errstate(all="ignore"):
        assert np.array_equal(got, a / b, equal_nan=True)


@pytest.mark.parametrize("kind", [1, 2])
@pytest.mark.parametrize("n", [1, 31, 64, 4096])
@pytest.mark.parametrize("growth", [1e-3, 0.13, 0.5, 1.0, 1.9, 20.0, 1e4])
def test_integer_sums(harness, kind, n, growth):
    """Terms rounded at 2^-62 of the last total (n halves of that), one rounding of the
    total to 53 of its top 56 bits: accepted sums are within (n 2^-62 / growth +
    2^-51) relative; a total of an eighth of the last one or more is accepted
    unless one term alone exceeds it."""
    rng = np.random.default_rng([kind, n, int(growth * 1000)])
    for scale in (1.0, 1e-20, 1e12):
        v = rng.exponential(size=n) * scale
        v[rng.random(n) < 0.2] = 0.0
        v[0] = scale
        if kind == 2:
            v = v.astype(np.float32).astype(np.float64)
        exact = sum(Fraction(float(x)) for x in v)
        last = float(exact) / growth
        t, ok = harness(np.array([kind, n, last, 0.0]).tobytes() + v.tobytes())[0]
        if growth >= 0.13 and v.max() < 2 * last:
            assert ok
        if growth <= 1e-3:
            assert not ok
        if ok:
            assert abs(Fraction(float(t)) - exact) <= exact * (Fraction(n) / (Fraction(growth) * 2 ** 61) + Fraction(1, 2 ** 51))


@pytest.mark.parametrize("kind", [1, 2])
def test_sums_that_are_refused(harness, kind):
    """NaN and Inf terms, and a last total that gives no scale."""
    for bad, last in ((np.nan, 10.0), (np.inf, 10.0), (1.0, 0.0), (1.0, np.inf), (1.0, np.nan), (1.0, 1e-300)):
        v = np.ones(32)
        v[7] = bad
        assert harness(np.array([kind, 32, last, 0.0]).tobytes() + v.tobytes())[0, 1] == 0


@pytest.mark.parametrize("scale", [1e-37, 1e-38, 1e-40, 1e-43])
def test_integer_sums_of_denormal_floats(harness, scale):
    """FP32 terms below 2^-126 are whole multiples of 2^-149 and keep their value: the
    bound of test_integer_sums at growth 1."""
    rng = np.random.default_rng(3)
    v = (rng.exponential(size=500) * scale).astype(np.float32).astype(np.float64)
    exact = sum(Fraction(float(x)) for x in v)
    t, ok = harness(np.array([2, len(v), float(exact), 0.0]).tobytes() + v.tobytes())[0]
    assert ok and abs(Fraction(float(t)) - exact) <= exact * (Fraction(len(v), 2 ** 61) + Fraction(1, 2 ** 51))
