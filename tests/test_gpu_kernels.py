"""Kernels at the sizes and call orders where their tiles and dispatch rules change."""
import numpy as np
import pytest

from oracle import dns_oracle as do
from oracle import pao_generator as pg

pytestmark = pytest.mark.gpu


def _field(N, prec, g, dt=1e-3):
    from palinstrophy_gb300.turbo_simulator import Field

    F = Field(N, prec, 1e3, 0.3)
    F.set_state(g["om2"], None, g["uc_low"])
    F.set_scalars(dt=dt, cn=1.0, cnm1=0.0, visc=1e-3, cflnum=0.3)
    return F


@pytest.mark.parametrize("N", [32, 64, 384, 512, 1536])
def test_methods_alternate(N):
    """fnm1 crosses from one stepper to the other through the butterfly-major
    order: an RK3 call takes only om in and hands fnm1 back to a CNAB2 call."""
    g = pg.generate(N, 5.0, 1e3, 7, "KM3")
    F = _field(N, "fp64", g)
    S = do.OracleState(N, g["om2"], g["uc_low"], 1e-3, 0.3)
    S.dt, S.cn, S.cnm1 = 1e-3, 1.0, 0.0
    do.step2a(S)
    for method, step, n in (("CNAB2", do.cnab2, 2), ("LS_IMEX_RK3", do.rk3, 2), ("CNAB2", do.cnab2, 3)):
        F.step(method, n, update=0)
        for _ in range(n):
            step(S)
    # FP64 parity of the repository's step tests
    assert do.rel_l2(S.om2, F.om2()) <= 1e-12
    assert do.rel_l2(S.fnm1, F.fnm1()) <= 1e-10
    F.close()


def _long_double_step(om, dt, nu):
    """u, fn and om2 of one CNAB2 step (cnm1 = 0) in NumPy's long double."""
    import scipy.fft as sf

    L = np.longdouble
    N = om.shape[0]
    nh, M = N // 2, 3 * N // 2
    kx = np.arange(nh).astype(L)[None, :]
    kz = np.where(np.arange(N) < nh, np.arange(N), np.arange(N) - N).astype(L)[:, None]
    k2 = kx * kx + kz * kz
    inv = 1 / np.where(k2 > 0, k2, 1)
    om = om.astype(np.clongdouble)

    def phys(b):
        X = np.zeros((M, M // 2 + 1), np.clongdouble)
        X[:nh, :nh], X[N:, :nh] = b[:nh], b[nh:]
        return sf.irfft2(X, s=(M, M), norm="forward")

    def gather(s):
        return np.concatenate((s[:nh, :nh], s[N:, :nh]))

    u, v = phys(-1j * kz * inv * om), phys(1j * kx * inv * om)
    fn = (kz * kx * gather(sf.rfft2(u * u - v * v)) + (kz * kz - kx * kx) * gather(sf.rfft2(u * v))) / L(M) ** 2
    fn[nh] = 0
    h = L(nu) * L(dt) / 2
    return u, fn, ((1 - k2 * h) * om + L(dt) * fn) / (1 + k2 * h)


def _spectrum(N, kind):
    rng = np.random.default_rng(N)
    nh = N // 2
    k = np.hypot(np.arange(nh)[None, :], np.fft.fftfreq(N, 1.0 / N)[:, None])
    k[0, 0] = 1.0
    om = np.exp(2j * np.pi * rng.random((N, nh)))
    om *= {"k-1": 1.0 / k, "steep": np.exp(-0.5 * k), "white": 1.0}[kind]
    om[nh] = om[0, 0] = 0.0
    om[nh + 1:, 0] = np.conj(om[1:nh, 0][::-1])
    return om


@pytest.mark.parametrize("kind", ["k-1", "steep", "white"])
@pytest.mark.parametrize("N", [32, 64, 128, 256, 384])
def test_fixed_point_transforms_are_no_worse_than_fp64(N, kind):
    """The FP64 form's block fixed-point transforms against long double: the
    velocity and the nonlinear term are as close to it as an FP64 transform's
    (the oracle's, in NumPy / SciPy double), the update as close as FP64 rounds."""
    from palinstrophy_gb300.turbo_simulator import Field

    dt, nu = 1e-3, 1e-3
    om = _spectrum(N, kind)
    u, fn, on = _long_double_step(om, dt, nu)
    F = Field(N, "fp64", 1e3, 0.3)
    F.set_state(om)
    F.set_scalars(dt=dt, cn=1.0, cnm1=0.0, visc=nu, cflnum=0.3)
    F.step2a()
    gu = F.ur(0)
    F.step("CNAB2", 1)
    kx = np.arange(N // 2)[None, :]
    kz = np.where(np.arange(N) < N // 2, np.arange(N), np.arange(N) - N)[:, None]
    k2 = np.where(kx * kx + kz * kz > 0, kx * kx + kz * kz, 1)
    S = do.OracleState(N, om, np.stack([-1j * kz * om / k2, 1j * kx * om / k2]), nu, 0.3)
    S.dt, S.cn, S.cnm1 = dt, 1.0, 0.0
    do.step2a(S)

    def err(x, ref):
        return float(np.linalg.norm((x.astype(ref.dtype) - ref).ravel().astype(np.complex128))
                     / np.linalg.norm(ref.ravel().astype(np.complex128)))

    ou = err(S.ur_full[0], u)
    do.cnab2(S)
    # a transform rounds at least once per pass: never asked to be below 2 eps
    eps = np.finfo(np.float64).eps
    assert err(gu, u) <= max(ou, 2 * eps)
    assert err(F.fnm1(), fn) <= max(err(S.fnm1, fn), 2 * eps)
    assert err(F.om2(), on) <= max(err(S.om2, on), 2 * eps)
    F.close()


@pytest.mark.parametrize("scale", [1e-290, 1e-160, 1e-30, 1e30, 1e140])
@pytest.mark.parametrize("N", [32, 256])
def test_fixed_point_follows_the_field_scale(N, scale):
    """A power-of-two scaled field gives the scaled velocity exactly (as long as
    no stored value is subnormal)."""
    from palinstrophy_gb300.turbo_simulator import Field

    s = 2.0 ** np.round(np.log2(scale))
    om = _spectrum(N, "k-1")
    got = []
    for f in (1.0, s):
        F = Field(N, "fp64", 1e3, 0.3)
        F.set_state(om * f)
        F.step2a()
        got.append((F.ur(0), F.ur(1)))
        F.close()
    for a, b in zip(*got):
        assert np.array_equal(a * s, b)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("N", [32, 512])
def test_fixed_point_non_finite_fields(N, bad):
    """A NaN or an infinity in the field reaches every value of the next one and
    the diagnostics report it; a zero field stays zero."""
    from palinstrophy_gb300.turbo_simulator import Field

    om = _spectrum(N, "k-1")
    om[3, 2] = bad
    F = Field(N, "fp64", 1e3, 0.3)
    F.set_state(om)
    F.set_scalars(dt=1e-3, visc=1e-3)
    F.step("CNAB2", 2)
    # the nonlinear term of the row kz = -N/2 is zero by definition
    assert not np.isfinite(np.delete(F.om2(), N // 2, axis=0)[:, 1:]).any()
    assert F.diagnostics()["nonfinite"] == 1
    F.close()
    F = Field(N, "fp64", 1e3, 0.3)
    F.set_state(np.zeros_like(om))
    F.set_scalars(dt=1e-3, visc=1e-3)
    F.step("LS_IMEX_RK3", 2)
    assert not F.om2().any() and not F.ur(0).any()
    F.close()


@pytest.mark.parametrize("nbins, r_max, k_nyq", [(1, 1.0, 16.0), (7, 0.3, 10.0), (32, 2.0**0.5, 16.0),
                                                 (1000, 2.0**0.5, 192.0), (513, 5.0, 3.0), (64, 1e-3, 1e-3)])
@pytest.mark.parametrize("N, prec", [(32, "fp32"), (384, "fp64")])
def test_energy_spectrum_bins(N, prec, nbins, r_max, k_nyq):
    """Bins as intervals of the integer K2 against the per-mode formula, at
    widths from many modes a bin to many bins a mode."""
    from palinstrophy_gb300.turbo_simulator import Field

    om = _spectrum(N, "k-1").astype(np.complex64 if prec == "fp32" else np.complex128)
    F = Field(N, prec, 1e3, 0.3)
    F.set_state(om)
    e, c = F.energy_spectrum(nbins, r_max, k_nyq)
    F.close()
    nh = N // 2
    kx = np.arange(nh, dtype=np.float64)[None, :]
    kz = np.where(np.arange(N) < nh, np.arange(N), np.arange(N) - N).astype(np.float64)[:, None]
    k2 = kx * kx + kz * kz
    with np.errstate(over="ignore"):
        b = np.clip(np.floor(np.sqrt(k2) / k_nyq / r_max * nbins), 0, nbins - 1).astype(np.int64)
    w = np.where(kx > 0, 2, 1) * (k2 > 0)
    o = om.astype(np.complex128)
    p = w * (o.real**2 + o.imag**2) / np.where(k2 > 0, k2, 1.0) * (1.5 * N) ** 4
    assert np.array_equal(c, np.bincount(b.ravel(), w.ravel(), nbins).astype(np.int64))
    ref = np.bincount(b.ravel(), p.ravel(), nbins)
    # positive terms: at most N^2/2 additions of one rounding each, on both sides
    assert np.all(np.abs(e - ref) <= N * N * np.finfo(np.float64).eps * ref)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("N", [32, 96 * 4, 1024])
def test_spectral_sums(N, prec):
    """E, L, Z, P of k_spectral against exactly rounded sums (math.fsum): the
    terms carry a few FP64 roundings each, the sums none."""
    import math

    from palinstrophy_gb300.turbo_simulator import Field

    om = _spectrum(N, "k-1").astype(np.complex64 if prec == "fp32" else np.complex128)
    om[0, 0] = 0.25
    F = Field(N, prec, 1e3, 0.3)
    F.set_state(om)
    F.set_scalars(dt=1e-3)
    d = F.diagnostics()
    F.close()
    nh = N // 2
    kx = np.arange(nh, dtype=np.float64)[None, :]
    kz = np.where(np.arange(N) < nh, np.arange(N), np.arange(N) - N).astype(np.float64)[:, None]
    k2 = kx * kx + kz * kz
    w = np.where((kx == 0) | (kx == nh - 1), 1.0, 2.0) * np.ones_like(k2)
    o = om.astype(np.complex128)
    p = w * (o.real**2 + o.imag**2)
    m = k2 > 0
    E = math.fsum((p[m] / k2[m]).ravel())
    S = math.fsum((p[m] / k2[m] / np.sqrt(k2[m])).ravel())
    for key, ref in (("E", E), ("L", 2.0 * math.pi * S / E), ("Z", math.fsum(p.ravel()) - p[0, 0]),
                     ("P", math.fsum((k2 * p).ravel()))):
        assert abs(d[key] - ref) <= 16 * np.finfo(np.float64).eps * ref, key


@pytest.mark.parametrize("scale", [1e-42, 1e-30, 1.0, 1e16])
@pytest.mark.parametrize("N", [32, 384, 1024, 2048])
def test_mean_square_velocity(N, scale):
    """The diagnostic sum of u^2 + v^2 of an FP32 field against the exactly
    rounded sum of its squares (exact in FP64): the sum is off by a rounding per
    group and by its shifted-out bits, U by half of that, its square root and
    quotient.  Scales: subnormal and small velocities, ordinary ones, large ones."""
    import math

    from palinstrophy_gb300.turbo_simulator import Field

    om = (_spectrum(N, "k-1") * scale).astype(np.complex64)
    F = Field(N, "fp32", 1e3, 0.3)
    F.set_state(om)
    F.set_scalars(dt=1e-3)
    U = F.diagnostics()["U"]
    F.step2a()
    u, v = (np.asarray(F.ur(i), np.float64).ravel() for i in (0, 1))
    F.close()
    ref = math.sqrt(math.fsum(u * u + v * v) / u.size)
    assert ref > 0.0
    assert abs(U - ref) <= 4 * np.finfo(np.float64).eps * ref
