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
