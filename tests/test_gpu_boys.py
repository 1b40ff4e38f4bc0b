"""Known-answer test of the device Boys function (csrc/boys.cuh) that every ERI kernel evaluates.

Golden values (tests/golden/boys_values.npz, make_boys_golden.py): F_0 .. F_9 at 481 values of T in
[0, 60] from the reference's Boys::calculateBoys (src/Boys.cpp:14-71) and from mpmath at 40 digits.

Tolerances:
* FP64, T <= 30 (Taylor expansion about the nearest grid point, downward recursion): 1e-14 relative to
  the exact value.
* FP64, T > 30: the reference and this engine both switch to the asymptotic form F_0 = sqrt(pi/T)/2,
  F_{m+1} = (m + 1/2) F_m / T, which drops terms of order e^{-T}; the device must agree with the
  reference's values to 1e-13 relative, and with the exact values to 1e-14 of F_0(T) absolute.
* FP32: 1e-6 relative for T <= 30 (float rounding, 6e-8 per operation, dominates the 2.6e-9 truncation
  of the 5-term expansion), and above 30, against the reference's asymptotic values, 2.5e-7 (m + 1) + 3e-7
  relative for order m (float rounding of each upward step).
"""
import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _golden():
    import os

    return dict(np.load(os.path.join(GOLDEN, "boys_values.npz")))


@pytest.mark.parametrize("m_max", [0, 1, 4, 8, 9])
def test_gpu_boys_fp64_known_answers(m_max):
    from hfgpu.engine import boys_eval

    g = _golden()
    T, ex, rf = g["T"], g["F_exact"][:, :m_max + 1], g["F_ref"][:, :m_max + 1]
    F = boys_eval(m_max, T)
    lo = T <= 30.0
    assert np.max(np.abs(F[lo] - ex[lo]) / ex[lo]) <= 1e-14
    hi = ~lo
    assert np.max(np.abs(F[hi] - rf[hi]) / rf[hi]) <= 1e-13
    # The asymptotic form drops e^{-T} / (2T) in each of the m upward steps (each step scales earlier
    # errors by (k + 1/2) / T < 1 for T > 30): |F_m - exact| <= m e^{-T} / (2T) plus rounding.
    m = np.arange(m_max + 1)[None, :]
    bound = m * (np.exp(-T[hi]) / (2 * T[hi]))[:, None] + 1e-14 * ex[hi]
    assert np.all(np.abs(F[hi] - ex[hi]) <= bound)


@pytest.mark.parametrize("m_max", [0, 2, 5, 8])
def test_gpu_boys_fp32_known_answers(m_max):
    from hfgpu.engine import boys_eval

    g = _golden()
    T, ex, rf = g["T"], g["F_exact"][:, :m_max + 1], g["F_ref"][:, :m_max + 1]
    F = boys_eval(m_max, T, fp32=True)
    lo = T <= 30.0
    assert np.max(np.abs(F[lo] - ex[lo]) / ex[lo]) <= 1e-6
    # Above 30 each upward step (m + 1/2) / T * F_m rounds about three times in float (6e-8 each), on top
    # of rsqrtf's F_0: 2.5e-7 per order plus 3e-7.
    m = np.arange(m_max + 1)[None, :]
    assert np.all(np.abs(F[~lo] - rf[~lo]) / rf[~lo] <= 2.5e-7 * (m + 1) + 3e-7)


def test_gpu_boys_rejects_bad_arguments():
    from hfgpu.engine import HfgError, boys_eval

    with pytest.raises(HfgError):
        boys_eval(10, [1.0])
    with pytest.raises(HfgError):
        boys_eval(2, [-1.0])
    with pytest.raises(HfgError):
        boys_eval(2, [float("nan")])


def boys_series(m_max, T):
    """F_0(T) .. F_m_max(T) in long double: e^-T sum_k (2T)^k / ((2m+1)(2m+3) .. (2m+2k+1)), all terms positive."""
    T = np.asarray(T, np.longdouble)
    out = []
    for m in range(m_max + 1):
        term = 1 / np.full(T.shape, 2 * m + 1, np.longdouble)
        total = term.copy()
        for k in range(1, 220):  # at T = 31 the terms fall below 1e-20 of the sum after 150
            term = term * 2 * T / (2 * m + 2 * k + 1)
            total += term
        out.append(total * np.exp(-T))
    return np.stack(out, axis=-1)


@pytest.mark.parametrize("m_max", range(10))
def test_gpu_scaled_boys_known_answers(m_max):
    """c s^m F_m(T) of the FP64 thread, chunk and gradient kernels at grid points, in the middle and at both edges of the
    cells (h = 1/32), at 0 and around the switch to the asymptotic form at 30: 1e-14 relative, as for boys_eval (stated in
    boys.cuh: 2e-15).  T is what the device's own s and R2 give, in long double."""
    from hfgpu.engine import boys_scaled

    rng = np.random.default_rng(m_max)
    i = np.arange(961)
    T = np.concatenate([i / 32, (i[:-1] + 0.5) / 32 * (1 - 1e-7), (i[:-1] + 0.5) / 32 * (1 + 1e-7), rng.random(2000) * 30,
                        rng.random(200) * 1e-6, 30 - np.logspace(-15, -1, 40)])
    T = np.concatenate([T, T, T])
    rho = np.concatenate([np.full(T.size // 3, r) for r in (0.17, 1.0, 3.4e4)])  # diffuse, unit and tight exponents
    s, R2, c = -2 * rho, T / rho, rng.choice([-1, 1], T.size) * 10.0 ** rng.uniform(-12, 4, T.size)
    T = -s.astype(np.longdouble) * R2 / 2
    lo = T < 29.999  # nearer the switch either branch may run: its dropped e^-T is allowed for below
    F = boys_scaled(m_max, c, s, R2)
    m = np.arange(m_max + 1)
    exact = (c.astype(np.longdouble)[:, None] * s.astype(np.longdouble)[:, None] ** m) * boys_series(m_max, T)
    rel = np.abs((F - exact) / exact).astype(float)
    assert rel[lo].max() <= 1e-14
    # Asymptotic: F_0 and each upward step drop e^-T / (2T) or less, taken as a part of F_m near the switch.
    T2 = np.concatenate([30 + np.logspace(-3, 0, 40), [35.0, 60.0, 1e3, 1e9]])
    s2, R22 = np.full(T2.size, -1.7), T2 / 0.85
    F2 = boys_scaled(m_max, 2.5, s2, R22)
    Tl = -s2.astype(np.longdouble) * R22 / 2
    asym = np.empty((T2.size, m_max + 1), np.longdouble)
    asym[:, 0] = 2.5 * np.sqrt(np.longdouble("3.14159265358979323846264338327950288") / Tl) / 2
    for k in range(m_max):
        asym[:, k + 1] = asym[:, k] * (k + 0.5) / Tl * s2
    assert np.max(np.abs((F2 - asym) / asym)) <= 1e-14
    near = ~lo
    Fm = np.abs(boys_series(m_max, T[near]))
    drop = ((m + 1) * (np.exp(-T[near]) / (2 * T[near]))[:, None] / Fm).astype(float)
    assert np.all(rel[near] <= 1e-14 + 1.01 * drop)


def test_gpu_scaled_boys_rejects_bad_arguments():
    from hfgpu.engine import HfgError, boys_scaled

    for m_max, c, s, R2 in ((10, 1.0, -1.0, 1.0), (2, 1.0, 1.0, 1.0), (2, 1.0, -1.0, -1.0), (2, float("nan"), -1.0, 1.0)):
        with pytest.raises(HfgError):
            boys_scaled(m_max, [c], [s], [R2])
