"""The clamped quotients of the pente-borne fluxes, which divide only where the
clamped value depends on the quotient, are bit-identical to clamping the
division: a host program built by nvcc from the device header compares them
(tests/host/ratio_check.cu).  No GPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_clamped_quotients_are_bit_identical():
    exe = os.path.join(HERE, "host", "_build", "ratio_check")
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "host"), exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches 0" in r.stdout
