"""Host threads that each drive their own case share the resident-block
figures of the kernels: asked together from cold, each is found once and by
one thread at a time (tests/host/resident_check.cc).  No GPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_threads_share_the_figures():
    exe = os.path.join(HERE, "host", "_build", "resident_check")
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "host"), exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("wrong 0 together 0 "), r.stdout
