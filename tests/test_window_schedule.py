"""The steps of a window that refresh the SIC current or start a new noise index, on the host
(no GPU): tests/window_schedule_check.cpp."""
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_schedule_is_the_per_step_loops(tmp_path):
    exe = tmp_path / "window_schedule_check"
    # -fwrapv: a sum past the largest int gives a wrong bit instead of anything at all
    subprocess.run(["g++", "-O1", "-fwrapv", "-std=c++17", "-o", str(exe),
                    os.path.join(HERE, "window_schedule_check.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    m = re.search(r"checked (\d+) bad (\d+) refreshes (\d+) noises (\d+)", r.stdout)
    assert m and r.returncode == 0 and int(m.group(2)) == 0, r.stdout + r.stderr
    assert int(m.group(1)) == 400000 and int(m.group(3)) > 10000 and int(m.group(4)) > 10000
