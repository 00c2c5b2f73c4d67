"""Length and memory of the adjoint's segments."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
GIB = 1 << 30


def test_segment_memory(tmp_path):
    """ckpt_every is taken as it is up to 1 GiB; beyond, a call needs no more
    memory than om checkpoints every ckpt_every steps with the om of a segment's
    stages do, but for the padded planes' factor at the interval that is best
    for those (2 sqrt(27 n) om planes for 2 sqrt(6 n))."""
    from palinstrophy_gb300.build import CSRC

    exe = str(tmp_path / "segments_host")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC, os.path.join(HERE, "segments_host.cpp"), "-o", exe],
                   check=True)
    calls = [(n, c, N, e) for N in (32, 64, 128, 256, 512) for e in (8, 16)
             for n in (1, 2, 7, 64, 200, 5000, 50000, 1000000) for c in (1, 2, 20, 100, 333, 10000)]
    text = "\n".join(f"{n} {c} {N // 2 * (3 * N // 2) * e}" for n, c, N, e in calls)
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
    for (n, c, N, e), line in zip(calls, out):
        seg, got = map(int, line.split())
        assert 1 <= seg <= n
        om = N // 2 * N * e
        before = om * (2 * -(-n // c) + 3 * c)
        s = min(n, c)
        if (2 * (-(-n // s) - 1) + 6 * s) * om * 3 // 2 <= GIB:
            assert seg == s
        assert got <= max(GIB, 27 ** 0.5 / 6 ** 0.5 * before + 8 * om), (n, c, N, e)
