"""The diagnostics' sums of squares (pal_sums.cuh), run on the host against
exact rational arithmetic."""
import os
import struct
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    from palinstrophy_gb300.build import CSRC, _nvcc

    exe = str(tmp_path_factory.mktemp("sums") / "sums_host")
    subprocess.run([_nvcc(), "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-Xcompiler", "-ffp-contract=off",
                    "-I" + CSRC, os.path.join(HERE, "sums_host.cu"), "-o", exe], check=True)

    def run(lines):
        out = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True, check=True).stdout
        return [sum(Fraction(struct.unpack("<d", struct.pack("<Q", int(w, 16)))[0]) for w in line.split())
                for line in out.splitlines()]

    return run


def _groups():
    rng = np.random.default_rng(3)
    out = [np.zeros(16, np.float32)]
    for spread in (0, 4, 12, 24, 33, 60):  # binary orders of magnitude within a group
        for scale in (-140, -60, 0, 60, 127 - spread):
            v = rng.uniform(1.0, 2.0, (40, 16)) * 2.0 ** rng.integers(-spread, 1, (40, 16))
            out.extend((v * 2.0 ** scale).astype(np.float32) * rng.choice((-1, 1), (40, 16)).astype(np.float32))
    # one large value and fifteen whose squares leave almost a whole unit behind
    for k in range(20, 31):
        for m in (2 - 2.0 ** -23, 1 + 2.0 ** -23, 1 + 2.0 ** -12):
            g = np.full(16, m * 2.0 ** -k, np.float32)
            g[5] = 1.0
            out.append(g)
    return out


def test_squares_of_float_points_are_summed_beyond_double(sums):
    """Eight points a group: closer to the exact sum than points rounded to
    double one by one may be (2^-53 of the sum); what the integers leave out is
    below 2^-56."""
    gs = _groups()
    got = sums(["g " + " ".join(f"{b:x}" for b in g.view(np.uint32)) for g in gs])
    assert len(got) == len(gs)
    for g, s in zip(gs, got):
        exact = sum(Fraction(float(v)) ** 2 for v in g)
        assert abs(s - exact) <= exact / 2 ** 56, g


@pytest.mark.parametrize("n", [1, 3, 4, 48])
def test_squares_of_double_points_are_compensated_one_by_one(sums, n):
    """n equal points add up to n times the rounded point: a compensated sum's
    own error is of the order n 2^-106, a plain chain of four has roundings of
    2^-53 in it."""
    rng = np.random.default_rng(n)
    uv = rng.standard_normal((300, 2)) * 2.0 ** rng.integers(-20, 20, (300, 1))
    got = sums([f"p {n} " + " ".join(f"{b:x}" for b in p.view(np.uint64)) for p in uv])
    for (u, v), s in zip(uv, got):
        point = Fraction(float(Fraction(u) ** 2 + Fraction(float(v * v))))
        assert abs(s - n * point) <= n * point / 2 ** 100
