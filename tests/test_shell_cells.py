"""The work items of the periodic image copies cover exactly the image cells
(tests/hostsim/shell_sim.cc, the kernels' own index functions on the host)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_shell_cells(tmp_path):
    exe = str(tmp_path / "shell_sim")
    subprocess.run(["g++", "-std=c++20", "-O1", "-fsanitize=address", "-I" + os.path.join(ROOT, "rmt3d_b200", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "hostsim", "shell_sim.cc"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
