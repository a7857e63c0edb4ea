"""Where the FP32 form's fallback map in pairs of floats is taken, and what it is worth there, on the CPU: the header
that pass 2 is built from.

Every pair operation is good to 2^-46 of its operands, of which the longest chain has some sixteen in a row, so an output
is off by its own rounding and at most 2^-42 of the largest stress in hand (as a strain: over the modulus), whatever
the material, the units and the state; and finite.  States near the surface of ordinary materials all fit.
"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not available")
@pytest.mark.parametrize("seed", [1, 2])
def test_states_that_fit_are_mapped_right(tmp_path, seed):
    exe = str(tmp_path / "fpmap_range")
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "csrc", "fpmap_range.c"), "-lm"],
                   check=True)
    r = subprocess.run([exe, "2000000", str(seed)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    w = r.stdout.split()
    got = {w[i]: float(w[i + 1]) for i in range(0, len(w), 2)}
    assert got["notfinite"] == 0 and got["side"] == 0, r.stdout
    assert max(got["dsig"], got["deps_p"], got["dR"]) <= 1.0, r.stdout
    assert got["fit"] > 100_000 and got["ordinary"] > 10_000 and got["left"] == 0, r.stdout
