"""The traversal's slab test (csrc/dl_slab.hpp) never culls a padded box at its faces, edges and corners. CPU only."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_slab_test_never_culls_at_a_boundary(tmp_path):
    exe = tmp_path / "slab_edges_check"
    csrc = os.path.join(ROOT, "dynamiclighting-bevy_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I", csrc,
                    os.path.join(ROOT, "tests", "native", "slab_edges_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.rstrip().endswith("missed 0"), out.stdout + out.stderr
    counts = dict(zip(out.stdout.split()[::2], map(int, out.stdout.split()[1::2])))
    assert min(counts[k] for k in ("faces", "edges", "corners", "grazing", "starting")) > 10000, counts
