"""The fast form of the order rule (prefix_rule_fast in stencil.cuh, compiled for the host) gives
the general rule's value, codes and key bit for bit on every random neighbourhood it decides,
and decides most of them: ordinary ones, ones with special keys, ties, far from the source."""
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
    exe = str(tmp_path_factory.mktemp("fast_rule") / "harness")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC,
                    os.path.join(HERE, "fast_rule_harness.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("nd", [2, 3])
@pytest.mark.parametrize("specials", [0, 1])
def test_fast_rule_equals_the_general_rule(harness, nd, specials):
    cases = 1_000_000
    out = subprocess.run([harness, str(nd), str(cases), str(10 * nd + specials), str(specials)],
                         check=True, capture_output=True, text=True).stdout
    decided, differing = map(int, out.split())
    assert differing == 0
    assert decided > 0.3 * cases
