"""The activation quantiser's divisions by multiplications (csrc/quotients.cuh) against IEEE division, on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotients_have_the_bits_of_a_division(tmp_path):
    exe = str(tmp_path / "quotients")
    subprocess.run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", os.path.join(ROOT, "tests", "host", "quotients_check.cpp"), "-o", exe], check=True, capture_output=True, timeout=300)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout.split()
    bad_scale, bad_by, bad_quant, bad_tiny, n_quant = map(int, out)
    assert (bad_scale, bad_by, bad_quant, bad_tiny) == (0, 0, 0, 0)
    assert n_quant > 5000000
