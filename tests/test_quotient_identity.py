"""The sweeps' quotients by a shared divisor are the IEEE division's, and the
van Leer gradient with two ratios fewer is the reference formula's, bit for
bit: a host program built by nvcc from the device header compares them
(tests/host/quotient_check.cu).  No GPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_shared_divisor_quotients_are_bit_identical():
    exe = os.path.join(HERE, "host", "_build", "quotient_check")
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "host"), exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches 0" in r.stdout
