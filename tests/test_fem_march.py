"""FEM phases that march along z give the bits of the point-by-point phases
(tests/hostsim/march_sim.cc, the kernels' own bodies on the host)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fem_march(tmp_path):
    exe = str(tmp_path / "march_sim")
    subprocess.run(["g++", "-std=c++20", "-O1", "-ffp-contract=off", "-fsanitize=address",
                    "-I" + os.path.join(ROOT, "rmt3d_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                    "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "hostsim", "march_sim.cc"), "-o", exe],
                   check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
