"""The formula behind the device's sample tables equals the host's sorted orders for every net. CPU only."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_cells_and_ranks_equal_the_sorted_orders(tmp_path):
    exe = tmp_path / "net_cell_check"
    csrc = os.path.join(ROOT, "dynamiclighting-bevy_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-ffp-contract=off", "-fno-fast-math", "-x", "c++", "-I", csrc,
                    os.path.join(ROOT, "tests", "native", "net_cell_check.cpp"), os.path.join(csrc, "dl_host.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "nets 9 failures 0" in out.stdout, out.stdout
