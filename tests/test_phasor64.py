"""The phasor table's index and fraction (dfmath.cuh: cis_tab_df, cis_tab_m1_df2)
at negative and large phases, emulated in FP32 on the host with the constants
read from the source: 64 entries, |y| < 2^22 in units of 1/64 turn (|x| < 4.1e5
rad), four-term polynomials.  1.5e-7 per component, the bound of the other table
tests; e^{ix} - 1, up to 2 in size, rounds at twice the scale, one sum more: 2.5e-7.
"""
import os
import re

import numpy as np
import pytest

f32 = np.float32
SOURCE = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pointint_gb300", "csrc",
                           "dfmath.cuh")).read()


def constant(name):
    return f32(re.search(rf"#define {name} ([-0-9.e]+)f", SOURCE).group(1))


N = int(re.search(r"PHASOR_ENTRIES = (\d+)", SOURCE).group(1))
C1, C2, C3, C4 = (constant("PI_TURN64" + s) for s in ("", "_C2", "_C3", "_C4"))
SHIFT = constant("PI_ROUND_SHIFT")
ANGLES = 2 * np.pi * np.arange(N) / N
TAB = np.stack([np.cos(ANGLES), np.sin(ANGLES)], 1).astype(f32)
TABM = np.stack([-2 * np.sin(ANGLES / 2) ** 2, np.sin(ANGLES)], 1).astype(f32)


def fma(a, b, c):
    return f32(np.float64(a) * np.float64(b) + np.float64(c))


def split(v):
    return f32(v), f32(v - np.float64(f32(v)))


def index_and_turn(kt, sm):
    t = fma(kt[0], sm[0], SHIFT)
    f = fma(kt[1], sm[0], fma(kt[0], sm[1], fma(kt[0], sm[0], f32(SHIFT - t))))
    f2 = f32(f * f)
    return int(np.array(t, dtype=f32).view(np.int32)) & (N - 1), f32(f2 * fma(f2, C4, -C2)), f32(f * fma(f2, -C3, C1))


def cis_tab_df(kt, sm):
    i, cm, sn = index_and_turn(kt, sm)
    x, y = TAB[i]
    return fma(x, cm, fma(-y, sn, x)), fma(y, cm, fma(x, sn, y))


def cis_tab_m1(kt, sm):
    i, cm, sn = index_and_turn(kt, sm)
    x, y = TABM[i]
    return f32(x + fma(x, cm, fma(-y, sn, cm))), f32(y + fma(y, cm, fma(x, sn, sn)))


def test_constants():
    c = 2 * np.pi / N
    assert N == 64 and SHIFT == f32(1.5 * 2 ** 23)
    for got, want in zip((C1, C2, C3, C4), (c, c ** 2 / 2, c ** 3 / 6, c ** 4 / 24)):
        assert got == f32(want)


@pytest.mark.parametrize("y", [-0.0, -0.49, -0.51, -1.0, -31.5, -63.6, -64.0, -64.5, -1e6 + 0.3, 3.49, 63.5, 2 ** 21 + 7.0,
                               2.0 ** 22 - 0.75, -(2.0 ** 22) + 0.75])
def test_index_wraps(y):
    kt, sm = split(y), (f32(1.0), f32(0.0))
    x = 2 * np.pi * y / N
    re, im = cis_tab_df(kt, sm)
    assert abs(re - np.cos(x)) <= 1.5e-7 and abs(im - np.sin(x)) <= 1.5e-7
    re, im = cis_tab_m1(kt, sm)
    assert abs(re + 2 * np.sin(x / 2) ** 2) <= 2.5e-7 and abs(im - np.sin(x)) <= 2.5e-7


def test_negative_phases_over_the_range():
    rng = np.random.default_rng(0)
    worst = 0.0
    for _ in range(3000):
        k, s = 10 ** rng.uniform(-2, 4.4), -rng.random() * 10 ** rng.uniform(-3, 1.1)
        if k * -s > 4.0e5:
            continue
        kt, sm = split(k * N / (2 * np.pi)), split(s)
        x = 2 * np.pi / N * (np.float64(kt[0]) + np.float64(kt[1])) * (np.float64(sm[0]) + np.float64(sm[1]))
        re, im = cis_tab_df(kt, sm)
        worst = max(worst, abs(re - np.cos(x)), abs(im - np.sin(x)))
    assert worst <= 1.5e-7, worst
