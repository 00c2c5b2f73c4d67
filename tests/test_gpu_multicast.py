"""Row candidates that load by TMA cluster multicast run in one-GPU programs only."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
N = 8192


def _run(code, **env):
    clean = {k: v for k, v in os.environ.items() if k not in ("WORLD_SIZE", "LOCAL_WORLD_SIZE", "PAL_TUNE_FILE")}
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300,
                         env={**clean, **env})
    assert out.returncode == 0, out.stderr[-2000:]
    return out.stdout.split("\n")


def test_jobs_of_several_processes_take_no_multicast_candidate(built_lib, tmp_path):
    """One process of a job of two (as torchrun marks it): neither the autotuner
    nor a tuning file nor a choice by index gives it a multicast candidate."""
    tune = tmp_path / "tune.txt"
    code = ("from palinstrophy_gb300 import _lib as L\n"
            "from palinstrophy_gb300.turbo_simulator import Field\n"
            f"F = Field({N}, 'fp32', 1e5, 0.1)\n"
            "v = F.variant()\n"
            "print(v['desc'])\n"
            "for r in range(v['n_rows']):\n"
            "    try:\n"
            "        F.set_variant(r, 0)\n"
            "        print(F.variant()['desc'])\n"
            "    except L.PalError as e:\n"
            "        print('refused', e.code == L.PAL_ERR_STATE)\n"
            "F.close()\n")
    rows = [d.split("row[")[1].split("]")[0] for d in _run(code) if "row[" in d][1:]
    assert any(" mc " in r for r in rows)  # a one-GPU program may choose it
    mc = next(r for r in rows if " mc " in r)
    tune.write_text(f"fp32 {N} {mc}|16.32.24 x512\n")
    out = _run(code, WORLD_SIZE="2", PAL_TUNE_FILE=str(tune))
    assert not any(" mc " in line for line in out)
    assert out.count("refused True") == sum(" mc " in r for r in rows)


def test_shards_take_no_multicast_candidate(built_lib):
    """A shard of an ensemble over several processes, even where this process
    tuned to a multicast candidate before and no launcher is to be seen."""
    code = ("from palinstrophy_gb300 import _lib as L, ensemble_shards as es\n"
            "from palinstrophy_gb300.turbo_simulator import Ensemble, Field\n"
            f"F = Field({N}, 'fp32', 1e4, 0.5)\n"
            "F.close()\n"
            f"es.run_ensemble_shard([{N}, {N}], [1, 2], 0, 2, nsteps=1)\n"
            f"E = Ensemble([{N}])\n"
            f"print(E.variant({N}))\n"
            "E.close()\n")
    out = _run(code)
    assert "row[" in out[0] and " mc " not in out[0]


def test_forms_without_multicast_give_the_same_field(built_lib):
    """The multicast candidate and the one without it load the same rows into
    the same arithmetic, so that a job on several GPUs loses no digit."""
    from palinstrophy_gb300.turbo_simulator import Field

    rng = np.random.default_rng(8)
    om = np.zeros((N, N // 2), np.complex64)
    om[1:9, :8] = rng.standard_normal((8, 8)) + 1j * rng.standard_normal((8, 8))
    got = {}
    F = Field(N, "fp32", 1e3, 0.3)
    for r in range(F.variant()["n_rows"]):
        F.set_variant(r, 0)
        d = F.variant()["desc"]
        if "cluster tma-in mc tma-out]" in d or "cluster tma-in tma-out]" in d:
            F.set_state(om)
            F.set_scalars(dt=1e-3, visc=1e-3)
            F.step("CNAB2", 1)
            got[d] = F.om2()
    F.close()
    a, b = got.values()
    assert np.array_equal(a, b)
