"""The traversal's slab test (csrc/dl_slab.hpp, boxes as centre and half extent) against exact
geometry: it never culls a padded box that a ray enters, over every scale of scene and direction,
and prunes boxes behind the ray or beyond its range. CPU only."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_slab_test_never_culls_an_entered_box(tmp_path):
    exe = tmp_path / "slab_check"
    csrc = os.path.join(ROOT, "dynamiclighting-bevy_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I", csrc,
                    os.path.join(ROOT, "tests", "native", "slab_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "missed 0 " in out.stdout, out.stdout + out.stderr
