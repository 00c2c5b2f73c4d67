"""Roundings of the spectral sums and of the energy-spectrum bins, on fields
whose exact sums are known in rational arithmetic."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = Fraction(1, 2 ** 53)       # one rounding of a double
TINY = 1 + Fraction(1, 2 ** 40)  # second-order terms


def _field(N, prec, om):
    from palinstrophy_gb300.turbo_simulator import Field

    F = Field(N, prec, 1e3, 0.3)
    F.set_state(om.astype(F.cdt))
    F.set_scalars(dt=1e-3)
    return F


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_energy_of_one_mode_is_rounded_once(prec):
    """E of a field with one mode is w om^2 / K2: the square of a 24-bit integer
    is exact, so the quotient's rounding is the only one."""
    N = 128
    rng = np.random.default_rng(1)
    for _ in range(150):
        kx, kz = int(rng.integers(0, N // 2)), int(rng.integers(-N // 2 + 1, N // 2))
        if kx == kz == 0:
            continue
        a = int(rng.integers(1 << 23, 1 << 24))
        om = np.zeros((N, N // 2), np.complex128)
        om[kz % N, kx] = a
        F = _field(N, prec, om)
        E = F.diagnostics()["E"]
        F.close()
        exact = Fraction((1 if kx in (0, N // 2 - 1) else 2) * a * a, kx * kx + kz * kz)
        assert abs(Fraction(E) - exact) <= U * TINY * exact, (kx, kz)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_spectrum_bins_of_one_mode_are_rounded_twice(prec):
    """One mode in each of many bins (a bin per value of K2): the quotient's
    rounding and the scale's."""
    N, k_nyq = 128, 64.0
    rng = np.random.default_rng(2)
    om = np.zeros((N, N // 2), np.complex128)
    mode = {}
    for kx in range(N // 2):
        for kz in range(N // 2):
            k2 = kx * kx + kz * kz
            if k2 > 0 and k2 not in mode and k2 < 3000:
                mode[k2] = (kx, int(rng.integers(1 << 23, 1 << 24)))
                om[kz, kx] = mode[k2][1]
    nbins, r_max = 400000, 2.0 ** 0.5
    F = _field(N, prec, om)
    e, _ = F.energy_spectrum(nbins, r_max, k_nyq)
    F.close()
    bins = {k2: int(np.floor(np.sqrt(float(k2)) / k_nyq / r_max * nbins)) for k2 in mode}
    assert len(set(bins.values())) == len(mode)
    scale2 = Fraction(N * 3 // 2) ** 4
    for k2, (kx, a) in mode.items():
        exact = (2 if kx else 1) * Fraction(a * a, k2) * scale2
        assert abs(Fraction(float(e[bins[k2]])) - exact) <= 2 * U * TINY * exact, k2


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_pairs_of_modes_are_summed_without_a_bias(prec):
    """Z adds exact terms (integer squares) in compensated sums, rounded where a
    block hands on its sum and at the end.  With all pairs of modes kz, -kz
    alike, a rounding of a pair's own sum would show in all of them with one
    sign: pairs are taken whose sum lies 0.4 to 0.5 units below a double.  The two
    roundings that remain are spread over +-U, so the mean of 60 fields is
    within 0.4 U of zero (five standard deviations); the pairs' would be 0.8 U."""
    N, nh = 32, 16
    rng = np.random.default_rng(4)
    kx = np.arange(nh)[None, :]
    kz = np.where(np.arange(N) < nh, np.arange(N), np.arange(N) - N)[:, None]
    w = np.where((kx == 0) | (kx == nh - 1), 1, 2) * np.ones_like(kz)
    err = []
    while len(err) < 60:
        a = int(rng.integers(1 << 23, 17 << 19))
        b = Fraction(int(rng.integers(1 << 23, 1 << 24)), 1 << int(rng.integers(4, 7)))
        pair = Fraction(a) ** 2 + b ** 2
        if not Fraction(4, 5) <= (Fraction(float(pair)) - pair) / pair / U:
            continue
        om = np.where(kz > 0, float(a), float(b)) * np.ones((1, nh))
        om[nh] = om[0] = 0.0
        F = _field(N, prec, om)
        Z = F.diagnostics()["Z"]
        F.close()
        exact = pair * int(w[1:nh].sum())
        err.append((exact - Fraction(Z)) / exact / U)
    assert max(abs(x) for x in err) <= 2 * TINY
    assert abs(sum(err) / len(err)) <= Fraction(2, 5)
