"""Keys (t, d >= 1, t), special ones whose level equals their traveltime: a node whose value equals its group's
level has one, on models with exact ties beside shocks (blocks of round velocity values). The fast form of the
order rule as a brick calls it (prefix_rule_signed in stencil.cuh, compiled for the host) gives the general rule's
value, codes and key bit for bit on every lattice neighbourhood it decides, with and without such keys."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "eikonalsolvers.jl_b200", "csrc")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("tied_keys") / "harness")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC,
                    os.path.join(HERE, "tied_keys_harness.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2])
def test_fast_rule_beside_tied_keys(harness, seed):
    cases = 2_000_000
    out = subprocess.run([harness, str(cases), str(seed)], check=True, capture_output=True, text=True).stdout
    decided, differing, tied = map(int, out.split())
    assert differing == 0
    assert tied > 0.3 * cases and decided > 0.02 * cases
