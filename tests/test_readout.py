"""Reading the transforms' sums chunk by chunk (photonoxide_b200/csrc/readout.h) on the host, the device
played by arrays: whatever call fails on the way, a second read completes the sums, each added once."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_failed_read_is_completed_by_the_next(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "photonoxide_b200", "csrc"),
                    os.path.join(ROOT, "tests", "readout_check.cpp"), "-o", exe], check=True)
    bad, cases = map(int, subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert cases > 20 and bad == 0, f"{bad} of {cases} cases"
