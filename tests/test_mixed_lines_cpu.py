"""The mixed-radix line passes' launch shapes (tests/cpp/mixed_lines.cpp), without
a GPU."""
import subprocess

from tests.cpp_build import build


def test_mixed_lines():
    r = subprocess.run([build("mixed_lines")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith("OK")
