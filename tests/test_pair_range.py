"""The range guard of the float-pair weights, built for the host: no window passes it with a
result that is not finite, and conversions keep NaN and infinities."""
import os
import subprocess

import pytest

from hypar_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("pair") / "pair_range_host")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", B.CSRC, "-o", exe,
                           os.path.join(HERE, "pair_range_host.cpp")])
    return [ln.split() for ln in subprocess.check_output([exe], text=True).splitlines()]


def test_accepted_windows_are_finite(lines):
    for wt, accepted, wrong in lines[:5]:
        assert int(accepted) > 1000, (wt, accepted)
        assert int(wrong) == 0, (wt, wrong, accepted)


def test_conversions_keep_nan_and_infinity(lines):
    assert lines[5] == ["conv", "1"]
