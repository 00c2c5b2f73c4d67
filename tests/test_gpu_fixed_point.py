"""The FP64 form's fixed-point transforms at four passes a line and on fields
whose modes are all in phase, where the passes' values grow the most."""
import numpy as np
import pytest

from oracle import dns_oracle as do
from test_gpu_kernels import _long_double_step, _spectrum

pytestmark = pytest.mark.gpu


def _coherent(N, kind):
    nh = N // 2
    kz = np.where(np.arange(N) < nh, np.arange(N), np.arange(N) - N)[:, None]
    # a point vortex, and a field whose velocity u adds up at one point
    om = (np.ones((N, 1)) if kind == "vortex" else 1j * kz) * np.ones((1, nh), np.complex128)
    om[nh] = om[0, 0] = 0.0
    return om


@pytest.mark.parametrize("N, kind", [(1024, "k-1"), (256, "vortex"), (256, "jet"), (512, "jet"), (1024, "jet")])
def test_transforms_are_closer_than_double_ones(N, kind):
    """Velocity and nonlinear term against long double: no further off than the
    oracle's, which are SciPy's double transforms."""
    from palinstrophy_gb300.turbo_simulator import Field

    dt, nu = 1e-3, 1e-3
    om = _spectrum(N, kind) if kind == "k-1" else _coherent(N, kind)
    u, fn, _ = _long_double_step(om, dt, nu)
    kx = np.arange(N // 2)[None, :]
    kz = np.where(np.arange(N) < N // 2, np.arange(N), np.arange(N) - N)[:, None]
    k2 = np.where(kx * kx + kz * kz > 0, kx * kx + kz * kz, 1)
    S = do.OracleState(N, om, np.stack([-1j * kz * om / k2, 1j * kx * om / k2]), nu, 0.3)
    S.dt, S.cn, S.cnm1 = dt, 1.0, 0.0
    do.step2a(S)

    def err(x, ref):
        return float(np.linalg.norm((x.astype(ref.dtype) - ref).ravel().astype(np.complex128))
                     / np.linalg.norm(ref.ravel().astype(np.complex128)))

    eu = err(S.ur_full[0], u)
    do.cnab2(S)
    ef = err(S.fnm1, fn)
    F = Field(N, "fp64", 1e3, 0.3)
    v = F.variant()
    for row, col in [(r, 0) for r in range(v["n_rows"])] + [(0, c) for c in range(1, v["n_cols"])]:
        F.set_variant(row, col)
        F.set_state(om)
        F.set_scalars(dt=dt, cn=1.0, cnm1=0.0, visc=nu, cflnum=0.3)
        F.step2a()
        gu = F.ur(0)
        F.step("CNAB2", 1)
        d = F.variant()["desc"]
        print(d, err(gu, u), eu, err(F.fnm1(), fn), ef)
        assert err(gu, u) <= eu, d
        assert err(F.fnm1(), fn) <= ef, d
    F.close()
