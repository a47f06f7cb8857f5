"""The FP64 operator's integer arithmetic (csrc/tg_fixed.cuh), run on the CPU:
its functions are host-callable, so a small harness evaluates one site from
given operands and the result is held to exact rational arithmetic.

Bound: with P the largest |part| of the five operands (times its operator
constant), the integer sum is within 4 units of 2^-56 P of the exact value
(eight dropped low*low products of at most 1/4 unit, one rounding of the cross
products, truncations of 2^-60), the link constants within 8 * 2^-60 P of the
FP64 links, and the final rounding is half an ulp of a result of at most 5 P:
together under 5 * 2^-53 P."""
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include "tg_fixed.cuh"
using namespace tg;
template <int D, bool MU0> static bool site(const OpK<double>& k, const double2* p, const double2* w, double2& o) {
  return fx_dslash<D, MU0>(k, to_fx(p[0]), to_fx(p[1]), to_fx(p[2]), to_fx(p[3]), to_fx(p[4]), to_fx_link(w[0]),
                           to_fx_link(w[1]), to_fx_link(w[2]), to_fx_link(w[3]), o);
}
int main() {  // records: m, cf, cb, dag, mu0, 5 operands, 4 links -> ok, re, im
  double r[23];
  while (fread(r, sizeof r, 1, stdin) == 1) {
    const double2 *p = (const double2*)(r + 5), *w = (const double2*)(r + 15);
    const OpK<double> k = make_opk(r[0], r[1], r[2], r[4] != 0);
    double2 o{0, 0};
    const bool ok = r[3] != 0 ? (r[4] != 0 ? site<1, true>(k, p, w, o) : site<1, false>(k, p, w, o))
                              : (r[4] != 0 ? site<0, true>(k, p, w, o) : site<0, false>(k, p, w, o));
    const double out[3] = {ok ? 1.0 : 0.0, o.x, o.y};
    fwrite(out, sizeof out, 1, stdout);
  }
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("fx")
    (d / "h.cu").write_text(HARNESS)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                    f"-I{ROOT}/thirring2d_gb300/csrc", f"-I{ROOT}/include", "-o", str(d / "h"), str(d / "h.cu")],
                   check=True, capture_output=True)

    def run(records):
        out = subprocess.run([str(d / "h")], input=np.ascontiguousarray(records).tobytes(), capture_output=True,
                             check=True).stdout
        return np.frombuffer(out).reshape(-1, 3)
    return run


def exact(rec):
    """The site's value and P, in rationals, from the FP64 operands."""
    f = [Fraction(float(v)) for v in rec]
    dag, mu0 = rec[3] != 0, rec[4] != 0
    m, cf, cb = f[0], f[1], f[2]
    if mu0:
        cf, cb = (Fraction(-1), Fraction(1)) if dag else (Fraction(1), Fraction(-1))
    sx = -1 if dag else 1
    p, w = [f[5 + 2 * i:7 + 2 * i] for i in range(5)], [f[15 + 2 * i:17 + 2 * i] for i in range(4)]
    x, y = m * p[0][0], m * p[0][1]
    for (wr, wi), (a, b), c, conj in zip(w, p[1:], (cf, cb, sx, -sx), (1, -1, 1, -1)):
        wi = wi * conj
        x += c * (wr * a - wi * b)
        y += c * (wr * b + wi * a)
    P = max(max(abs(a), abs(b)) * abs(c) for (a, b), c in zip(p, (m, cf, cb, 1, 1)))
    return x, y, P


@pytest.mark.parametrize("dag", [0, 1])
@pytest.mark.parametrize("m,mu", [(0.05, 0.0), (0.0, 0.0), (-3.7, 0.0), (1e-9, 0.0), (0.1, 0.2), (2.5, 1.3)])
@pytest.mark.parametrize("spread", [0, 6, 70, 500])
def test_site_within_bound(harness, dag, m, mu, spread):
    rng = np.random.default_rng([dag, spread, int(1000 * mu)])
    n = 400
    rec = np.zeros((n, 23))
    ep, em = math.exp(mu), math.exp(-mu)
    rec[:, :5] = [m, -em if dag else ep, ep if dag else -em, dag, mu == 0.0]
    rec[:, 5:15] = rng.normal(size=(n, 10)) * 2.0 ** rng.integers(-spread, spread + 1, (n, 10))
    rec[::7, 5:15] = np.where(rng.random((len(rec[::7]), 10)) < 0.5, 0.0, rec[::7, 5:15])   # exact zeros among them
    rec[:, 15:23:2], rec[:, 16:23:2] = (0.5 * f(rng.uniform(-4, 4, (n, 4))) for f in (np.cos, np.sin))
    rec[::11, 15:19] = 0.0                                                                  # open-boundary links
    got = harness(rec)
    for r, (ok, x, y) in zip(rec, got):
        ex, ey, P = exact(r)
        if not ok:
            assert P < Fraction(2) ** -800
            continue
        bound = 5 * Fraction(2) ** -53 * P
        assert abs(Fraction(x) - ex) <= bound and abs(Fraction(y) - ey) <= bound


def test_out_of_range_operands_are_refused(harness):
    """Operands, constants and links that need the FP64 form: all zero, denormal,
    huge, Inf, NaN; one such operand among ordinary ones where it matters."""
    base = np.zeros(23)
    base[:5] = [0.1, 1.0, -1.0, 0, 1]
    base[5:15] = 1.0
    base[15:23] = 0.25
    rows, want = [base.copy()], [1]

    def case(ok, at, value):
        r = base.copy()
        r[at] = value
        rows.append(r)
        want.append(ok)
    case(0, slice(5, 15), 0.0)
    case(0, slice(5, 15), 1e-310)
    for bad in (np.inf, -np.inf, np.nan, 1e305):
        for i in range(5, 15):
            case(0, i, bad)
    for bad in (np.inf, np.nan):
        for i in range(15, 23):
            case(0, i, bad)
        case(0, 0, bad)
    for i in range(5, 15):
        case(1, i, 1e-310)      # beside ordinary operands it is below the sum's resolution
    r = base.copy()
    r[0] = 0.0                  # m = 0 times Inf is NaN in FP64 too
    r[5] = np.inf
    rows.append(r)
    want.append(0)
    assert harness(np.array(rows))[:, 0].astype(int).tolist() == want


def test_integers_are_exact(harness):
    """Small integers times halves and quarters come out exactly, zeros included."""
    rng = np.random.default_rng(3)
    rec = np.zeros((200, 23))
    rec[:, :5] = [0.25, 1.0, -1.0, 0, 1]
    rec[:, 5:15] = rng.integers(-8, 9, (200, 10))
    rec[:, 15:23] = rng.choice([-0.5, 0.0, 0.5, 0.25], (200, 8))
    rec[0, 5:15:2] = 2.0
    rec[0, 6:15:2] = 0.0
    rec[0, 16:23:2] = 0.0       # real links, real operands: the imaginary part is 0
    for r, (ok, x, y) in zip(rec, harness(rec)):
        ex, ey, P = exact(r)
        if ok:
            assert abs(Fraction(x) - ex) <= Fraction(2) ** -50 and abs(Fraction(y) - ey) <= Fraction(2) ** -50
    assert harness(rec)[0, 2] == 0.0
