"""The builder's walk on cached draws against a walk that draws from the stream, on the
host (no GPU): tests/walk_words.cpp."""
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_cached_walk_makes_the_streams_draws(tmp_path):
    exe = tmp_path / "walk_words"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "walk_words.cpp")], check=True)
    r = subprocess.run([str(exe), "500"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    m = re.search(r"walks (\d+) mismatches (\d+) cache_overruns (\d+) hits (\d+) lengths (\d+) long (\d+)", r.stdout)
    assert m and int(m.group(1)) == 20000 and int(m.group(2)) == 0
    assert int(m.group(3)) > 0 and int(m.group(4)) > 0
    assert int(m.group(5)) > 100000 and int(m.group(6)) > 0
