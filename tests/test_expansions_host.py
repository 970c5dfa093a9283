"""The device math of the expansions and of the wide triangles, emulated on the
host and held against exact values (no GPU).

* the 64-entry phasor table (dfmath.cuh: cis_tab_df) in FP32: 1.5e-7 per
  component, the bound the 256-entry table was held to;
* e^{ix} - 1 from its own table (cis_tab_m1) in FP32: the constant, the
  polynomial, its product and the last sum round once each at the scale of the
  nearest table entry or of the result, so 2^-22 (|entry| + |result|) bounds it;
* the 16-term expansions in FP64 at the bounds on k rho that moments.h states:
  the n-th term is at most x^n / n! of the amplitude, so what is dropped stays
  below x^16 / 16! / (1 - x / 17), which must be less than one FP32 rounding of
  the amplitude (2^-24);
* the wide form of the triangles' phases against divided differences.
"""
import math
import os
import re

import numpy as np
import pytest

mp = pytest.importorskip("mpmath")
f32 = np.float32
N = 64
C = 2 * np.pi / N
C1, C2, C3, C4 = f32(C), f32(C ** 2 / 2), f32(C ** 3 / 6), f32(C ** 4 / 24)
SHIFT = f32(12582912.0)
SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pointint_gb300", "csrc", "moments.h")
X_TRI, X_SURF = (float(re.search(rf"MOMENT_X_{k} = ([0-9.]+)f", open(SOURCE).read()).group(1)) for k in ("TRI", "SURF"))


def dropped(x):
    return x ** 16 / math.factorial(16) / (1 - x / 17)


def test_expansion_bounds_stay_below_one_rounding():
    assert dropped(X_TRI) < 2.0 ** -24 and dropped(X_SURF) < 2.0 ** -24


TAB = np.stack([np.cos(C * np.arange(N)), np.sin(C * np.arange(N))], 1).astype(f32)
TABM = np.stack([-2 * np.sin(C * np.arange(N) / 2) ** 2, np.sin(C * np.arange(N))], 1).astype(f32)


def fma(a, b, c):
    return f32(np.float64(a) * np.float64(b) + np.float64(c))


def split(v):
    return f32(v), f32(v - np.float64(f32(v)))


def frac_terms(f):
    f2 = f32(f * f)
    return f32(f2 * fma(f2, C4, -C2)), f32(f * fma(f2, -C3, C1))


def cis_tab_df(kt, sm):
    t = fma(kt[0], sm[0], SHIFT)
    f = fma(kt[1], sm[0], fma(kt[0], sm[1], fma(kt[0], sm[0], -f32(t - SHIFT))))
    cm, sn = frac_terms(f)
    x, y = TAB[int(np.array(t, dtype=f32).view(np.int32)) & (N - 1)]
    return fma(x, cm, fma(-y, sn, x)), fma(y, cm, fma(x, sn, y))


def cis_tab_m1(kt, d):
    t = fma(kt, d, SHIFT)
    cm, sn = frac_terms(fma(kt, d, f32(SHIFT - t)))
    x, y = TABM[int(np.array(t, dtype=f32).view(np.int32)) & (N - 1)]
    return f32(x + fma(x, cm, fma(-y, sn, cm))), f32(y + fma(y, cm, fma(x, sn, sn))), math.hypot(x, y)


def test_phasor_table_of_64_entries():
    rng = np.random.default_rng(0)
    worst = 0.0
    for _ in range(4000):
        k, s = 10 ** rng.uniform(-2, 3.9), rng.uniform(-1, 1) * 10 ** rng.uniform(-3, 1.1)
        kt, sm = split(k * N / (2 * np.pi)), split(s)
        x = C * (np.float64(kt[0]) + np.float64(kt[1])) * (np.float64(sm[0]) + np.float64(sm[1]))
        re, im = cis_tab_df(kt, sm)
        worst = max(worst, abs(re - np.cos(x)), abs(im - np.sin(x)))
    assert worst <= 1.5e-7, worst


def test_phasor_minus_one_keeps_its_relative_accuracy():
    rng = np.random.default_rng(1)
    for _ in range(6000):
        kt = f32(10 ** rng.uniform(-2, 4) * N / (2 * np.pi))
        d = f32(10 ** rng.uniform(-9, 0.5))
        if float(kt) * float(d) > 1e6:
            continue
        x = C * float(kt) * float(d)
        re, im, ta = cis_tab_m1(kt, d)
        scale = 2.0 ** -22 * (ta + 2 * abs(math.sin(0.5 * x)))
        assert abs(re + 2 * math.sin(0.5 * x) ** 2) <= scale and abs(im - math.sin(x)) <= scale, (kt, d)


def triangle_exact(p):
    """Second divided difference of e^{iz} at three phases."""
    mp.mp.dps = 40
    a, b, c = (mp.mpf(float(v)) for v in p)
    d = lambda u, v: (mp.expj(v) - mp.expj(u)) / (v - u)
    return complex((d(b, c) - d(a, b)) / (c - a))


@pytest.mark.parametrize("shape", ["rim", "random"])
def test_triangle_expansion_at_its_bound(shape):
    x, rng, worst = X_TRI, np.random.default_rng(2), 0.0
    for _ in range(60):
        p = x * (1 - 1e-3 * rng.random(3)) if shape == "rim" else x * rng.uniform(-1, 1, 3)
        if np.abs(np.subtract.outer(p, p))[np.triu_indices(3, 1)].min() < 1e-6:
            continue
        an = qn = hn = 1.0
        s = -0.5 + 0j
        for n in range(1, 16):
            an = p[0] * an
            qn = p[1] * qn + an
            hn = p[2] * hn + qn
            s += 1j ** (n + 2) * hn / math.factorial(n + 2)
        worst = max(worst, abs(s - triangle_exact(p)) / 0.5)
    assert worst <= dropped(x), worst


@pytest.mark.parametrize("kind", ["disk", "gauss"])
def test_surfel_expansion_at_its_bound(kind):
    from scipy.special import j1
    x, rng, worst = X_SURF, np.random.default_rng(3), 0.0
    for _ in range(400):
        p = x * rng.random()                       # the element's own reach
        s = (x - p) * (1 if rng.random() < 0.5 else rng.uniform(-1, 1))
        u = [1.0, s]
        if kind == "disk":
            for n in range(1, 15):
                u.append(((2 * n + 3) * s * u[n] + (p * p - s * s) * u[n - 1]) / ((n + 1) * (n + 3)))
            exact = np.exp(1j * s) * (2 * j1(p) / p if p > 0 else 1.0)
        else:
            q = 0.5 * (p / 2.5) ** 2               # reach = 2.5 sigma
            for n in range(1, 15):
                u.append((s * u[n] + 2 * q * u[n - 1]) / (n + 1))
            exact = np.exp(1j * s - q)
        val = sum((1j) ** n * u[n] for n in range(16))
        worst = max(worst, abs(val - exact))
    assert worst <= dropped(x), worst


def test_wide_triangle_form():
    """e[u, v, w] = e^{iv} (M1/G1 + conj(M2)/G2)/(k^2 D) and the derivatives, in
    FP64, against divided differences at spreads from 1 to 40."""
    rng = np.random.default_rng(4)
    mp.mp.dps = 40
    for _ in range(60):
        u, v, w = sorted(rng.uniform(0, 1, 3) * 10 ** rng.uniform(0.5, 1.6))
        g1, g2 = w - v, v - u
        if min(g1, g2) < 1e-3:
            continue
        M1, M2 = np.exp(1j * g1) - 1, np.exp(1j * g2) - 1
        D = g1 + g2
        F = np.exp(1j * v) * (M1 / g1 + np.conj(M2) / g2) / D
        assert abs(F - triangle_exact((u, v, w))) <= 1e-11
        W = lambda g: (1j * np.exp(1j * g) - (np.exp(1j * g) - 1) / g) / g
        Dw = np.exp(1j * v) * (W(g1) - F / np.exp(1j * v)) / D
        h = mp.mpf(10) ** -12
        ex = lambda a, b, c: ((mp.expj(c) - mp.expj(b)) / (c - b) - (mp.expj(b) - mp.expj(a)) / (b - a)) / (c - a)
        a, b, c = mp.mpf(u), mp.mpf(v), mp.mpf(w)
        assert abs(Dw - complex((ex(a, b, c + h) - ex(a, b, c - h)) / (2 * h))) <= 1e-10
