"""The sine and cosine that the baker runs, on the CPU (the header compiles for host and device with identical
IEEE operations): equal to the binary64 path, seldom left to it, and with sums within the 2^-36 that the rounding test
allows for."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
COMPILE = ["g++", "-O2", "-std=c++17", "-pthread", "-ffp-contract=off", "-fno-fast-math"]
CHECK = os.path.join(ROOT, "tests", "native", "sincos_table_check.cpp")
CSRC = os.path.join(ROOT, "dynamiclighting-bevy_gb300", "csrc")
N = 2_000_000


def run(exe):
    fields = subprocess.run([str(exe), str(N)], capture_output=True, text=True, check=True).stdout.split()
    return int(fields[1]), int(fields[3]), int(fields[5]), float(fields[7][2:])


def test_table_path_equals_binary64_and_is_the_one_taken(tmp_path):
    exe = tmp_path / "sincos_table_check"
    subprocess.run([*COMPILE, "-I", CSRC, CHECK, "-o", str(exe)], check=True)
    checked, mismatches, fallbacks, worst = run(exe)
    assert checked > N and mismatches == 0
    assert fallbacks < N // 1000  # the binary64 path is rare
    assert worst < -36.0


@pytest.mark.parametrize("planted", ["a.vh = 0.5f * q;", "if (!(fabsf(x) < 16.0f) || x == 0.0f) return false;"])
def test_a_planted_mistake_is_noticed(tmp_path, planted):
    # the table path switched off, and a cosine's series of half its size
    with open(os.path.join(CSRC, "dl_math.cuh")) as f:
        header = f.read()
    assert header.count(planted) == 1
    header = header.replace(planted, "a.vh = 0.49999f * q;" if planted.startswith("a.vh") else "return false;")
    (tmp_path / "dl_math.cuh").write_text(header)
    exe = tmp_path / "planted"
    subprocess.run([*COMPILE, "-I", str(tmp_path), "-I", CSRC, CHECK, "-o", str(exe)], check=True)
    _, mismatches, fallbacks, worst = run(exe)
    assert mismatches > 0 or fallbacks >= N // 1000
    assert not planted.startswith("a.vh") or worst > -36.0
