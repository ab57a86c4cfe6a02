"""The exact MPR's root, reciprocal and quotients on the device (tests/cpp/exact_math.cu):
bit for bit the device's correctly rounded operations, and the bound on the seed from
which tests/test_exact_root.py starts."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
CPP = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp")
EXE = os.path.join(CPP, "build", "exact_math")


def test_device_arithmetic(cuda):
    if not os.path.exists(EXE):
        subprocess.run(["make", "-C", CPP], check=True)
    r = subprocess.run([EXE], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.count("TEST PASSED") == 3 and "TEST FAILED" not in r.stdout, r.stdout + r.stderr
