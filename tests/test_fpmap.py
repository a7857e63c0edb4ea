"""The return map in pairs of floats (code_mpm_gb300/csrc/fpmap.h, the FP32 form's fallback path) on the CPU, against
the map in long double and the map in double: the same header is compiled into pass 2."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not available")
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_pairs_round_like_the_map_in_double(tmp_path, seed):
    """Outputs rounded once are off by 1/sqrt(12) ulp RMS; a thousandth more leaves room for the sample.  48 bits leave
    about 2^-20 of an ulp of error before the rounding, times the cancellation of small corrections (a factor of about
    100 on the average state here), so the pairs and the double map round differently in about 1e-4 of the outputs at
    most.  The elastic / plastic decision is the same."""
    exe = str(tmp_path / "fpmap_check")
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "csrc", "fpmap_check.c"), "-lm"],
                   check=True)
    r = subprocess.run([exe, "2000000", str(seed)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    w = r.stdout.split()
    got = {k: float(w[i + 1]) for i, k in enumerate(w) if k in ("differ", "plastic", "branch", "outputs")}
    rms, rms_double = (float(w[i + 1]) for i, k in enumerate(w) if k == "rms")
    assert rms <= 0.288675 * 1.001 and abs(rms / rms_double - 1.0) <= 1e-4, r.stdout
    assert got["differ"] < 1e-4 and got["branch"] == 0, r.stdout
    assert 0.2 < got["plastic"] < 0.8 and got["outputs"] > 1e7, r.stdout
