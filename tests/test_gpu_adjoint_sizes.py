"""The adjoint at every grid it is compiled for, each with kernels and plans of
its own, and in segments shorter than the checkpoint interval."""
import numpy as np
import pytest

from oracle import pao_generator as pg
from oracle import torch_step as tsr

pytestmark = pytest.mark.gpu

DT, VISC = 2e-3, 2e-4


def _field(N, prec, om):
    from palinstrophy_gb300.turbo_simulator import Field

    F = Field(N, prec, 1.0 / VISC, 0.5)
    F.set_state(om, None, None)
    F.set_scalar("visc", VISC)
    F.set_scalar("dt", DT)
    return F


@pytest.fixture(scope="module")
def reference():
    cache = {}

    def get(N):
        if N not in cache:
            om = pg.generate(N, 5.0, 5e3, 7, "PAO")["om2"].astype(np.complex128)
            cache[N] = (om, *tsr.loss_and_grad(om, N, DT, VISC, 5))
        return cache[N]

    return get


# the bounds of the repository's gradient test at N = 64
@pytest.mark.parametrize("ckpt", [2, 5])
@pytest.mark.parametrize("N", [32, 64, 128, 256, 512])
def test_fp64_gradient_equals_autograd(reference, N, ckpt):
    om, L_ref, g_ref = reference(N)
    F = _field(N, "fp64", om)
    L, g = F.adjoint_palinstrophy(5, ckpt)
    F.close()
    assert abs(L - L_ref) <= 1e-12 * L_ref
    assert np.linalg.norm(g - g_ref) <= 1e-10 * np.linalg.norm(g_ref)


@pytest.mark.parametrize("graphs", ["1", "0"])
def test_segments_of_least_memory_give_the_same_gradient(monkeypatch, graphs):
    """64 steps of N = 512 in FP64 with a checkpoint every 64 would hold 1.2 GB of
    velocity planes: the call cuts them into 13 segments, the last one shorter.
    The forward sweep is the same, so loss and field are; a segment that is run
    again starts from the velocity of its om, which the sweep before had from its
    column pass, so the gradient agrees to rounding (the bound of the repository's
    test of the interval)."""
    monkeypatch.setenv("PAL_ADJOINT_GRAPHS", graphs)
    N = 512
    om = pg.generate(N, 5.0, 5e3, 7, "PAO")["om2"].astype(np.complex128)
    got = []
    for ckpt in (16, 64):
        F = _field(N, "fp64", om)
        got.append((*F.adjoint_palinstrophy(64, ckpt), F.om2(), F.scalars()["t"]))
        F.close()
    (L, g, om_end, t), (L2, g2, om_end2, t2) = got
    assert L == L2 and t == t2 and np.array_equal(om_end, om_end2)
    assert np.linalg.norm(g - g2) <= 1e-12 * np.linalg.norm(g)
