"""The error word of a context is shared with the host while kernels run: kernels set its bits
at system scope, the host takes them atomically, and nothing clears bits of others."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "portablert_gb300", "csrc")


def test_bits_are_taken_once(tmp_path):
    exe = tmp_path / "errword_test"
    src = os.path.join(ROOT, "tests", "cpp", "errword_test.cpp")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-pthread", "-I", CSRC, src, "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout


def test_every_access_goes_through_the_helpers():
    """No kernel touches an error word by a device-scope atomic or a plain store."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        src = open(os.path.join(CSRC, name)).read()
        assert not re.findall(r"atomic\w+\(\s*&?(?:\w+[.>-]+)*(?:d_)?err\b", src), name
        assert not re.findall(r"cudaMemset(?:Async)?\([^;]*d_err", src), name
        assert not re.findall(r"k_\w+<<<[^;]*>>>\(d_err\)", src), name
