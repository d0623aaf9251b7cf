"""The mean of incident radiation in pairs of floats (diffuse_mean) against long
double, beside the same quotient in doubles: as accurate over all magnitudes, and
the same for what is not finite or overflows."""
import os
import shutil
import subprocess

import pytest


@pytest.fixture(scope="module")
def ranges(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = tmp_path_factory.mktemp("mean") / "mean_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off",
                    os.path.join(root, "tests", "cpp", "mean_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    return {line.split()[0]: [float(x) for x in line.split()[1:]]
            for line in out.splitlines() if not line.startswith("#")}


@pytest.mark.parametrize("name", ["radiation", "bright", "dim", "no_sky", "few", "large_counts", "tiny",
                                  "tiniest", "huge", "mixed"])
def test_as_accurate_as_doubles(ranges, name):
    """Half a unit of the last place is the rounding to float; the pair's own error
    is some 2^-46, a double's 2^-52: 2^-20 units on top for both."""
    pair, plain, differ = ranges[name]
    assert plain <= 0.5 + 2.0 ** -20
    assert pair <= 0.5 + 2.0 ** -20
    assert differ <= 5  # halfway cases of 100,000


def test_values_that_are_not_finite(ranges):
    assert ranges["odd"][0] == 0
