"""The float-pair arithmetic of the interface correction, built for the host.

Bound: an operation on pairs is off by a few 2^-48 of its result (l holds 24 bits below h's
24, its roundings are relative to l); the chain from the differences to the correction has
some ten dependent ones, the smoothness terms entering squared twice, so 2^-43 (16 in units
of 2^-47) of the terms' magnitudes is held, plus the rounding of the FP64 differences
themselves (one unit of the largest value).  Conversions: 2^-48."""
import os
import subprocess

from hypar_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_pair_correction_against_long_double(tmp_path):
    exe = str(tmp_path / "pair_host")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", B.CSRC, "-o", exe,
                           os.path.join(HERE, "pair_host.cpp")])
    lines = [ln.split() for ln in subprocess.check_output([exe], text=True).splitlines()]
    for wt, s, d, share in lines[:5]:
        assert float(s) <= 16.0 and float(d) <= 16.0, (wt, s, d)
        assert float(share) >= 0.75, (wt, share)  # all but the large-unit windows, at least
    assert lines[5][0] == "conv" and float(lines[5][1]) <= 1.0 and lines[5][2] == "1"
