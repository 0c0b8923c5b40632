"""Message lengths of the warp-cooperative SHAKE: the words it absorbs, compiled as host code and run
on the CPU, and its callers, none of which may narrow a 32-bit length."""
import glob
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cumayo_b200", "csrc")


def test_absorbed_words_at_every_length(tmp_path):
    from cumayo_b200.build import nvcc
    try:
        cc = nvcc()
    except RuntimeError:
        pytest.skip("nvcc not available")
    exe = tmp_path / "host_shake"
    r = subprocess.run([cc, "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC, "-o", str(exe),
                        os.path.join(ROOT, "tests", "host_shake_test.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.stdout.strip() == "OK", out.stdout


def test_no_caller_casts_a_message_length():
    calls = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        for call in re.findall(r"\b(?:warp_shake<\d+>|\w+\.absorb)\([^;]*;", open(path).read()):
            calls += 1
            assert not re.search(r"\(int\)\s*[\w.\->]*len", call), (os.path.basename(path), call)
    assert calls > 20
