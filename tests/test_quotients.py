"""The on-chip FP64 solver forms its quotients without the division operator, which its results
must match to the bit: the same source against the operator on the CPU, over random and special
significands, the whole exponent range, overflow, subnormals, infinities and NaN."""
import os
import subprocess

import pytest

from tests.test_const_division import _has_fma

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "cuphu_b200", "csrc")


def test_quotients_match_the_operator(tmp_path):
    exe = str(tmp_path / "quotient_check")
    flags = ["-O2", "-std=c++17", "-ffp-contract=off"] + (["-mfma"] if _has_fma() else [])
    try:
        subprocess.run(["g++", *flags, "-I" + CSRC, "-o", exe,
                        os.path.join(HERE, "quotient_check.cpp"), "-lm"], check=True,
                       capture_output=True)
    except OSError as e:
        pytest.skip(f"g++ unavailable: {e}")
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    res = {ln.split()[0]: (int(ln.split()[1]), int(ln.split()[2])) for ln in out.splitlines()}
    assert set(res) == {"scalars", "any", "ends", "pixels"}
    assert all(n > 1_000_000 and bad == 0 for n, bad in res.values()), res
