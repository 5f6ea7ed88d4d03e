"""CPU: the identities behind the nonlinear term's transforms (fft_dev.cuh,
fft_nl.cu), in exact integers and in numpy."""
import random

import numpy as np
import pytest

LENGTHS = (16, 24, 32, 48, 64, 96, 128, 192, 256)


def _split(x, shift=0):
    """fx_split: the limbs (x1, x0) of x 2^shift, x0 a signed 32-bit integer."""
    y = x << shift
    assert -(1 << 63) <= y < 1 << 63
    lo = ((y + (1 << 31)) & 0xFFFFFFFF) - (1 << 31)
    hi = (y - lo) >> 32
    assert -(1 << 31) <= hi < 1 << 31
    return hi, lo


def _prod2(x, w, y, v):
    """fx_prod2 on limbs: every intermediate must fit the register it has."""
    fits = lambda a, b: -(1 << (b - 1)) <= a < 1 << (b - 1)  # noqa: E731
    lo = ((x[1] * w[1]) >> 32) + ((y[1] * v[1]) >> 32)
    assert fits(lo, 32)
    m = lo + (1 << 31)
    for a, b in ((x[0], w[1]), (x[1], w[0]), (y[0], v[1]), (y[1], v[0])):
        m += a * b
        assert fits(m, 64)
    h = m >> 32
    for a, b in ((x[0], w[0]), (y[0], v[0])):
        h += a * b
        assert fits(h, 64)
    return h


def test_limb_products_round_once():
    rng = random.Random(5)
    worst = 0
    for i in range(20000):
        ang = rng.uniform(0, 2 * np.pi) if i % 4 else rng.choice((0.0, np.pi / 2, np.pi, 3 * np.pi / 2))
        wx, wy = round(np.cos(ang) * 2.0 ** 62), round(np.sin(ang) * 2.0 ** 62)
        # a modulus below 2^61, as every value that meets a table entry has
        r, t = 2.0 ** rng.uniform(0, 60.9), rng.uniform(0, 2 * np.pi)
        x, y = round(r * np.cos(t)), round(r * np.sin(t))
        lx, ly = _split(x, 2), _split(y, 2)
        w, v = _split(wx), _split(wy)
        if abs(w[1]) == 1 << 31 or abs(v[1]) == 1 << 31:
            continue  # stored one unit off (pack_limbs)
        nv = (-v[0], -v[1])
        for got, exact in ((_prod2(lx, w, ly, nv), x * wx - y * wy), (_prod2(ly, w, lx, v), y * wx + x * wy)):
            err = abs((got << 62) - exact)  # in units of 2^-62
            worst = max(worst, err)
    assert worst <= (1 << 61) + (1 << 32)  # half a unit and two floors of 2^-31


@pytest.mark.parametrize("n", LENGTHS)
def test_pair_packing_and_exchange(n):
    """Z[k] = S + i P, Z[N-k] = conj S + i conj P packs the half spectrum of 2N
    real points for one inverse length-N transform; the forward transform is
    the inverse one with re and im exchanged; 2 X[k] = E + P, 2 X[N-k] =
    conj E - conj P unpacks it."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal(2 * n)
    X = np.fft.rfft(x)
    w = np.exp(2j * np.pi * np.arange(n) / (2 * n))
    Z = np.zeros(n, complex)
    for k in range(n // 2):
        a, b = X[k], X[n - k]
        S, D = a + np.conj(b), a - np.conj(b)
        P = w[k] * D
        Z[k] = S + 1j * P
        if k:
            Z[n - k] = np.conj(S) + 1j * np.conj(P)
    Z[n // 2] = 2 * np.conj(X[n // 2])
    z = np.fft.ifft(Z) * n / (2 * n)
    assert np.max(np.abs(z.real - x[0::2])) < 1e-13 and np.max(np.abs(z.imag - x[1::2])) < 1e-13
    swap = lambda a: a.imag + 1j * a.real  # noqa: E731
    F = swap(np.fft.ifft(swap(z)) * n)
    assert np.max(np.abs(F - np.fft.fft(z))) < 1e-11
    Y = np.zeros(n + 1, complex)
    for k in range(n // 2):
        za, zb = F[k], F[(n - k) % n]
        E, P = za + np.conj(zb), np.conj(w[k]) * (-1j) * (za - np.conj(zb))
        Y[k] = (E + P) / 2
        Y[n - k] = (np.conj(E) - np.conj(P)) / 2
    Y[n // 2] = np.conj(F[n // 2])
    assert np.max(np.abs(Y - X)) < 1e-11
