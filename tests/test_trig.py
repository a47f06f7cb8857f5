"""Sine and cosine on the integer pipes (csrc/tg_trig.cuh), on the CPU: the functions
are host-callable, so a harness evaluates them and the results are held to exact
series in rational arithmetic.  Bounds: the fixed-point values are within 8 * 2^-64
absolute, and FP64 results round once or twice more (1.5 ulp of the result, at
least 8 * 2^-64)."""
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include "tg_trig.cuh"
using namespace tg;
int main() {  // records: kind, angle or integer -> four doubles
  double r[2];
  while (fread(r, sizeof r, 1, stdin) == 1) {
    double out[4] = {0, 0, 0, 0};
    if (r[0] < 2) {  // a link with sign 1 (kind 0) or -1 (kind 1): W, W from the limbs
      double2 w; FxLink q;
      fx_link_of(r[1], r[0] == 0 ? 1 : -1, w, q);
      const double2 v = fx_link_value(q);
      out[0] = w.x; out[1] = w.y; out[2] = v.x; out[3] = v.y;
    } else if (r[0] == 2) {
      out[0] = one_minus_cos(r[1]);
      FxTrig t;
      out[1] = fx_trig(r[1], t);
    } else {
      fx_sincos_turn((unsigned long long)r[1], out[0], out[1]);
    }
    fwrite(out, sizeof out, 1, stdout);
  }
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("trig")
    (d / "h.cu").write_text(HARNESS)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                    f"-I{ROOT}/thirring2d_gb300/csrc", f"-I{ROOT}/include", "-o", str(d / "h"), str(d / "h.cu")],
                   check=True, capture_output=True)

    def run(kind, x):
        rec = np.stack([np.full(len(x), float(kind)), np.asarray(x, float)], 1)
        out = subprocess.run([str(d / "h")], input=rec.tobytes(), capture_output=True, check=True).stdout
        return np.frombuffer(out).reshape(-1, 4)
    return run


B = 220  # bits of the exact arithmetic


def _atan_inv(n):
    x = (1 << B) // n
    s, k = x, 1
    while x:
        x //= n * n
        k += 2
        s += -(x // k) if (k // 2) % 2 else x // k
    return s


PI = Fraction(4 * (4 * _atan_inv(5) - _atan_inv(239)), 1 << B)


def sincos(a):
    """(sin a, cos a) of a rational angle, to about 2^-190."""
    k = round(a / (PI / 2))
    r = a - k * PI / 2
    x = (r.numerator << B) // r.denominator
    x2 = (x * x) >> B
    s, c, ts, tc, n = x, 1 << B, x, 1 << B, 1
    while ts or tc:
        tc = -(tc * x2 >> B) // ((2 * n - 1) * (2 * n))
        ts = -(ts * x2 >> B) // ((2 * n) * (2 * n + 1))
        s, c, n = s + ts, c + tc, n + 1
        if abs(ts) <= 1 and abs(tc) <= 1:
            break
    s, c = Fraction(s, 1 << B), Fraction(c, 1 << B)
    return [(s, c), (c, -s), (-s, -c), (-c, s)][k % 4]


ANGLES = {
    "md": lambda rng: rng.normal(0, 0.5, 1500),
    "turns": lambda rng: rng.uniform(-50, 50, 1500),
    "large": lambda rng: rng.uniform(-1, 1, 500) * 2.0 ** 19.9,
    "small": lambda rng: rng.normal(size=800) * 2.0 ** rng.integers(-80, -5, 800),
    "quadrants": lambda rng: (np.arange(-40, 41)[:, None] * math.pi / 4
                              + np.array([0, 1e-15, -1e-15, 1e-9, -1e-9, 2e-4])).ravel(),
}


@pytest.mark.parametrize("kind", ANGLES)
def test_links_and_action(harness, kind):
    a = ANGLES[kind](np.random.default_rng(1))
    unit = Fraction(8, 2 ** 64)
    for sign, code in ((1, 0), (-1, 1)):
        for x, (wc, ws, qc, qs) in zip(a, harness(code, a)):
            s, c = sincos(Fraction(float(x)))
            for got, fixed, want in ((wc, qc, sign * c / 2), (ws, qs, sign * s / 2)):
                tol = Fraction(3, 2) * Fraction(math.ulp(float(got)))
                assert abs(Fraction(float(got)) - want) <= max(tol, unit)
                # limbs: even multiples of 2^-60, read back in FP64
                assert abs(Fraction(float(fixed)) - want) <= Fraction(3, 2 ** 60) + Fraction(math.ulp(float(fixed)))
    for x, (v, ok, _, _) in zip(a, harness(2, a)):
        assert ok == 1
        assert abs(Fraction(float(v)) - (1 - sincos(Fraction(float(x)))[1])) <= unit + Fraction(math.ulp(float(v)))


def test_small_angles_keep_their_relative_accuracy(harness):
    a = np.random.default_rng(2).normal(size=500) * 2.0 ** np.random.default_rng(3).integers(-300, 0, 500)
    a = a[np.abs(a) < 0.78]
    for x, (_, ws, _, _) in zip(a, harness(0, a)):
        s = sincos(Fraction(float(x)))[0] / 2 if abs(x) > 2.0 ** -60 else Fraction(float(x)) / 2
        assert abs(Fraction(float(ws)) / s - 1) <= Fraction(3, 2 ** 53)


def test_angles_outside_the_range(harness):
    """2^20 and beyond, Inf and NaN: the library's functions."""
    x = np.array([2.0 ** 20, -3e7, 1e300, np.inf, -np.inf, np.nan])
    out = harness(0, x)
    for v, row in zip(x, out):
        if np.isfinite(v):
            assert abs(row[0] - 0.5 * math.cos(v)) < 1e-15 and abs(row[1] - 0.5 * math.sin(v)) < 1e-15
        else:
            assert np.isnan(row).all()
    assert (harness(2, x)[:, 1] == 0).all()
    assert harness(2, np.array([0.0, -0.0]))[:, 0].tolist() == [0.0, 0.0]
    assert harness(0, np.array([0.0]))[0].tolist() == [0.5, 0.0, 0.5, 0.0]


def test_turns(harness):
    v = np.concatenate((np.random.default_rng(4).integers(0, 2 ** 53, 1500), [0, 1, 2 ** 53 - 1, 2 ** 50, 2 ** 51 - 1, 2 ** 51,
                                                                              2 ** 52, 3 * 2 ** 50])).astype(float)
    for x, (c, s, _, _) in zip(v, harness(3, v)):
        es, ec = sincos(2 * PI * (2 * int(x) + 1) / 2 ** 54)
        for got, want in ((c, ec), (s, es)):
            assert abs(Fraction(float(got)) - want) <= Fraction(8, 2 ** 64) + Fraction(math.ulp(float(got)))


def test_links_near_the_axes_keep_their_relative_accuracy(harness):
    """Near the multiples of pi/2 the small part of W is within 2 ulp (4 of 2^-53) of itself."""
    rng = np.random.default_rng(5)
    k = np.concatenate((np.arange(-40, 41), rng.integers(-600000, 600000, 150)))
    near = np.concatenate([k * (math.pi / 2), k * (math.pi / 2) + rng.normal(size=len(k)) * 2.0 ** rng.integers(-45, -6, len(k))])
    near = near[np.abs(near) < 2.0 ** 20]
    for x, (wc, ws, _, _) in zip(near, harness(0, near)):
        s, c = sincos(Fraction(float(x)))
        for got, want in ((wc, c / 2), (ws, s / 2)):
            assert abs(Fraction(float(got)) - want) <= Fraction(4, 2 ** 53) * abs(want)


def test_turns_near_the_axes_keep_their_relative_accuracy(harness):
    rng = np.random.default_rng(6)
    v = np.concatenate([q * 2 ** 51 + s * rng.integers(0, 2 ** int(b), 20) for q in range(5) for b in (1, 5, 20, 40, 44, 45, 46, 50)
                        for s in (1, -1)])
    v = v[(v >= 0) & (v < 2 ** 53)].astype(float)
    for x, (c, s, _, _) in zip(v, harness(3, v)):
        es, ec = sincos(2 * PI * (2 * int(x) + 1) / 2 ** 54)
        for got, want in ((c, ec), (s, es)):
            assert abs(Fraction(float(got)) - want) <= Fraction(4, 2 ** 53) * abs(want)
