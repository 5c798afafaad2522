"""byte_over (csrc/dl_math.cuh), the gathers' division of a photon's bytes, equals the binary32
division for every byte value. CPU only."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_byte_over_equals_the_division(tmp_path):
    exe = tmp_path / "byte_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math",
                    "-I", os.path.join(ROOT, "dynamiclighting-bevy_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "byte_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "mismatches 0" in out.stdout, out.stdout
