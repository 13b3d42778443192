"""The host's wait for a step's lists (csrc/mi8_tagged.h), with a thread in the place of the GPU: a word that does not come ends the wait as soon as the stream is
idle, whichever word it is.  A wait without an end ends the test program by its limit."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_tagged_wait(tmp_path):
    exe = str(tmp_path / "tagged_wait_test")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-Wall", "-pthread", "-o", exe, os.path.join(HERE, "cpp", "tagged_wait_test.cpp")])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and "tagged wait tests passed" in out.stdout, out.stdout + out.stderr
