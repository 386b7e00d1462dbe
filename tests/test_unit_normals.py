"""The sweeps skip the initial outer normals along an axis where they are
exactly (-1, 1) for every cell; a host program built by nvcc from the device
headers checks that decision against the general formula, cell by cell
(tests/host/normals_check.cu).  No GPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_unit_normals_are_exact():
    exe = os.path.join(HERE, "host", "_build", "normals_check")
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "host"), exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches 0" in r.stdout
