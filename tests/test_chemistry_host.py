"""The device chemistry compiled for the host: its FP64 fits against 40 digits, and the test of
an update against the quotient that the reference forms (update(), hydrogen_only/mod.rs:444-461).
"""
import ctypes
import subprocess

import numpy as np
import pytest

from subsweep_gb300 import build

UNIT = 2.0 ** -53


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = tmp_path_factory.mktemp("chemistry") / "chemistry.so"
    src = build.ROOT / "tests" / "chemistry_host.cpp"
    subprocess.run([build.CXX, *build.HOST_FLAGS, f"-I{build.CSRC}", "-shared", "-o", str(out), str(src)], check=True,
                   timeout=300)
    return ctypes.CDLL(str(out))


def ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def test_fits_are_exact_to_a_few_roundings(host):
    mp = pytest.importorskip("mpmath")
    t = np.exp(np.linspace(np.log(1e2), np.log(1e6), 4001))
    alpha, dalpha, cooling = (np.empty_like(t) for _ in range(3))
    host.fits(len(t), ptr(t), ptr(alpha), ptr(dalpha), ptr(cooling))
    # (the constants are the doubles that the program has)
    with mp.workdps(40):
        def off(got, want):
            return abs(float((mp.mpf(float(got)) - want) / want))
        cm3, erg_cm3 = mp.mpf(1e-6), mp.mpf(1e-13)
        err = np.zeros((3, len(t)))
        for i, v in enumerate(t):
            v = mp.mpf(float(v))
            lam = 315614 / v
            p = (lam / mp.mpf(2.74)) ** mp.mpf(0.407)
            a = mp.mpf(2.753e-14) * lam ** mp.mpf(1.5) / (1 + p) ** mp.mpf(2.242) * cm3
            c, d = mp.mpf(0.407), mp.mpf(2.242)
            # d alpha / d lambda (175-194) times d lambda / d t
            poly = c * d * p - mp.mpf(1.5) * p - mp.mpf(1.5)
            slope = mp.mpf(2.753e-14) * -mp.sqrt(lam) / (1 + p) ** (d + 1) * poly * cm3 * (-315614 / v ** 2)
            q = (lam / mp.mpf(2.25)) ** mp.mpf(0.376)
            r = (mp.mpf(3.435e-30) * v * lam ** mp.mpf(1.97) / (1 + q) ** mp.mpf(3.72) + mp.mpf(1.42e-27) * mp.sqrt(v))
            err[:, i] = off(alpha[i], a), off(dalpha[i], slope), off(cooling[i], r * erg_cm3)
    # alpha: lambda^1.5 to 3.5 roundings (one in lambda, a half more by its root, a root, a product),
    # (1 + p)^2.242 at p < 10 to fewer than 2.242 * 2.8 + 1, and three more; at most 14 in all, and
    # far fewer on the average
    assert err[0].max() < 14 * UNIT and err[0].mean() < 2 * UNIT, (err[0].max(), err[0].mean())
    assert err[1].max() < 24 * UNIT and err[1].mean() < 4 * UNIT, (err[1].max(), err[1].mean())
    # the logarithm of lambda, up to 8, scales the roundings of the two exponentials and of the
    # power: 1.97 * 8 * 0.5 + 3.72 * (0.376 * 8 * 0.5 + 2) and five more
    assert err[2].max() < 26 * UNIT, err[2].max()


def test_small_changes_are_those_of_the_quotient(host):
    rng = np.random.default_rng(5)
    n = 200_000
    value = rng.choice([1.0, -1.0], n) * 10.0 ** rng.uniform(-12, 7, n)
    safety = rng.choice([0.1, 0.05, 0.3, 1e-3, 1.0, 3e15, 4.6e15, 1e17, 1e300, np.inf, np.nan, 0.0], n)
    with np.errstate(all="ignore"):
        change = value * safety * (1.0 + rng.integers(-6, 7, n) * UNIT)
        change[::5] = value[::5] * 10.0 ** rng.uniform(-20, 20, len(change[::5]))
        special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-300, 1e308])
        value[::97] = rng.choice(special, len(value[::97]))
        change[::89] = rng.choice(special, len(change[::89]))
        relative = np.fmin(np.abs(change / value), 1.0 / np.finfo(float).eps)
        expected = ~(relative > safety)
    got = np.empty(n, np.uint8)
    host.small_enough(n, ptr(value), ptr(change), ptr(safety), ptr(got))
    np.testing.assert_array_equal(got.astype(bool), expected)
