"""The logarithm and the exponential of the FP64 return hold the errors that their
comment states: 1.01 ulp of the power, 0.55 ulp of the logarithm."""
import os
import subprocess

import helpers

HERE = os.path.dirname(os.path.abspath(__file__))


def test_errors_of_power_and_logarithm(tmp_path):
    with open(os.path.join(helpers.PKG, "csrc", "dnl_math.cuh")) as f:
        source = f.read()
    begin, end = source.index("struct TwoDoubles"), source.index("// The Johnson-Cook law as the return calls it.")
    law = tmp_path / "law.inc"
    law.write_text(source[begin:end])
    exe = str(tmp_path / "law")
    subprocess.run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", f'-DLAW_SOURCE="{law}"', "-o", exe,
                    os.path.join(HERE, "law_functions.cpp"), "-lquadmath"], check=True)
    power, log = map(float, subprocess.run([exe, "1000000"], capture_output=True, text=True, check=True).stdout.split())
    assert 0.9 < power <= 1.01
    assert 0.5 < log <= 0.55
