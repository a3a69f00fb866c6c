"""The shared-memory V-cycle's device code (mg_slab.cuh) run on host threads
-- every thread of a small cluster, shared memory as heap blocks under the
address sanitizer, neighbour values and mbarriers emulated -- against the
per-phase cycle of mg_ops.cuh, bit for bit: both solvers, constant and
variable density, FP64 and FP32, walled and periodic axes in every mix, slabs
that do not divide the planes, CTAs without planes, one CTA holding all."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def sim(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("sim") / "slab_sim")
    cmd = ["g++", "-std=c++20", "-O1", "-fsanitize=address", "-ffp-contract=off", "-DRMT3D_HOST_SIM",
           "-I" + os.path.join(ROOT, "rmt3d_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
           "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "hostsim", "slab_sim.cc"), "-o", exe, "-lpthread"]
    subprocess.run(cmd, check=True, capture_output=True)
    return exe


# kind (0 MAC, 1 FEM), variable density, FP64, points, periodic, CTAs, sweeps down and up, first level
@pytest.mark.parametrize("args", [
    "0 0 1 16 16 16 0 0 0 4 2 2 0",
    "1 0 1 17 17 17 0 0 0 4 2 2 0",
    "1 1 0 17 17 17 0 0 0 16 1 1 0",
    "0 1 0 24 16 12 0 0 0 5 2 1 0",
    "1 1 1 25 17 13 0 0 0 5 2 1 0",
    "0 0 1 16 16 16 1 1 1 4 2 2 0",
    "1 0 1 16 16 16 1 1 1 4 2 2 0",
    "0 1 0 16 24 16 0 1 0 3 2 1 0",
    "1 1 1 33 17 24 0 0 1 5 2 0 0",
    "1 0 0 33 33 33 0 0 0 16 1 1 1",
    "0 0 0 32 40 24 0 0 0 16 0 2 0",
    "0 1 1 40 12 24 1 1 0 16 2 2 0",
    "1 1 0 16 33 24 1 0 1 7 2 1 0",
    "0 0 0 12 12 88 0 0 0 16 1 1 0",
    "1 0 0 16 16 16 1 1 1 1 2 2 0",
    "1 1 0 24 24 24 1 1 1 2 1 1 0",
    "1 0 0 57 41 25 0 0 0 16 1 1 1",
    "1 0 1 33 33 33 0 0 0 16 2 1 0",
])
def test_slab_cycle_matches_phases(sim, args):
    r = subprocess.run([sim] + args.split() + ["7"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]


# kind, density, type, points, periodic, CTAs, sweeps, first level; the value sent to
# CTA 1 that is lost: of the first pass, and of the last (of the cycle's 2,000
# or so), after which nothing waits
@pytest.mark.parametrize("args,drop", [
    ("1 0 1 17 17 17 0 0 0 5 2 2 0", 3),
    ("0 1 0 16 16 16 0 0 0 4 1 2 0", 40),
    ("1 1 0 17 17 16 0 0 1 4 2 1 0", 1700),
])
def test_wait_that_gives_up_is_reported(sim, args, drop):
    """A neighbour's value that never arrives: the wait gives up, every thread
    still reaches the end, no mbarrier gets a second arrival in a phase, the
    waiting CTA's planes come out NaN and the solve's control reports it."""
    r = subprocess.run([sim] + args.split() + ["7", str(drop)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]
