"""What dl_session_occluder_bvh returns is what the traversal reads: the comparison of the device's nodes with
the returned boxes notices planted mistakes (CPU), and both builders' trees of every kind pass it (GPU)."""
import os
import subprocess

import pytest

import dynlight_gb300 as dl

from .test_gpu_bvh import CASES

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_node_with_other_boxes_is_noticed(tmp_path):
    exe = tmp_path / "node_check"
    csrc = os.path.join(ROOT, "dynamiclighting-bevy_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I", csrc,
                    os.path.join(ROOT, "tests", "native", "node_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "wrong 0" in out.stdout, out.stdout + out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("host", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_the_devices_nodes_hold_the_returned_boxes(name, host):
    s = dl.Session(*CASES[name](), host_bvh=host)
    try:
        nodes, triangles, depth = s.occluder_bvh()
        assert len(nodes) >= 1 and depth >= 1
    finally:
        s.close()
