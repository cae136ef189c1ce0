"""The mixed-radix plans (tests/cpp/mixed_plan.cpp), without a GPU."""
import subprocess

from tests.cpp_build import build


def test_mixed_plan():
    r = subprocess.run([build("mixed_plan")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith("OK")
