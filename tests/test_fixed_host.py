"""The fixed-point passes have room for every radix that a plan can take."""
import math
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_pass_leaves_64_bits(tmp_path):
    """Inputs of a pass have components below 2^b, so moduli below 2^(b + 1/2).
    A twiddle product keeps its sums inside 64 bits for moduli below 2^62.8, a
    butterfly's outputs (R times an input) have to stay below that too."""
    from palinstrophy_gb300.build import CSRC, _nvcc

    exe = str(tmp_path / "fixed_host")
    subprocess.run([_nvcc(), "-std=c++17", "-O0", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I" + CSRC, os.path.join(HERE, "fixed_host.cu"), "-o", exe], check=True)
    rows = [tuple(map(int, ln.split())) for ln in
            subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()]
    assert len(rows) == 9
    for R, b, b_dit, b_pad in rows:
        # positions N/2 .. M - N/2 of a padded line are zero: segment j of R holds (3 j .. 3 j + 3) N / 2R
        inputs = sum(not (3 * j >= R and 3 * j + 3 <= 2 * R) for j in range(R))
        assert math.log2(inputs) + b_pad + 0.5 <= 62.8, R
        assert math.log2(R) + b + 0.5 <= 62.8, R
        assert b_dit + 0.5 <= 62.8, R   # what the DIT twiddles multiply
        assert b_dit - 2 <= b, R        # they divide by 4
