"""A new scene runs as much of each V-cycle as fits a cluster's shared memory
(on these grids all of it, the finest level included) in one launch: the same
bits over whole steps as one launch per phase, and fewer launches."""
import time

import numpy as np
import pytest

import helpers as H
import rmt3d_b200 as R
from rmt3d_b200 import scenes

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "w", "p", "q", "dp")


@pytest.mark.parametrize("name", ["cavity16", "stretch24", "varden24", "multi24"])
@pytest.mark.parametrize("precision", [R.FP64, R.MIXED])
def test_whole_cycle_bit_identical(tmp_path, name, precision):
    fx = H.load_fixture(name)
    cfg = H.fixture_cfg(fx, str(tmp_path / (name + ".cfg")))
    got, launches = [], []
    for pts in (None, 0):
        sc = R.Scene.from_cfg(cfg, precision=precision, var_den=int(fx.get("varden", 0)))
        try:
            if pts is not None:
                sc.set_coarse_cluster(pts)
            sc.prepare()
            assert sc.run(3) == R.NORMAL_EXIT
            got.append({f: sc.field(f).copy() for f in FIELDS})
            launches.append(sc.launches())
        finally:
            sc.close()
    for f in FIELDS:
        assert np.array_equal(got[0][f], got[1][f]), f
    assert launches[0] < launches[1]


# the part starts below the finest level (64^3 from 33^3, 96^3 from 48^3 MAC
# and 49^3 FEM in FP32), or is the whole cycle with three planes a CTA (48^3); in a
# box periodic in z alone the sends wrap round the cluster
@pytest.mark.parametrize("n,precision,var_den,periodic", [
    (48, R.MIXED, 0, ""), (48, R.MIXED, 1, ""), (64, R.MIXED, 0, ""), (64, R.FP64, 1, ""), (96, R.MIXED, 0, ""),
    (32, R.FP64, 0, "z"), (48, R.MIXED, 1, "z"), (64, R.MIXED, 0, "z"), (64, R.MIXED, 0, "xyz"), (48, R.MIXED, 1, "y")])
def test_part_bit_identical(tmp_path, n, precision, var_den, periodic):
    t = scenes.stretched_sphere(n) if periodic == "xyz" else scenes.cavity_sphere(n, rho=1.2 if var_den else 1.0)
    t = t.replace("bc_yh 1 1 1 0 0 0", "bc_yh 1 1 1 0.5 0 0")
    cfg = scenes.write(str(tmp_path / "s.cfg"),
                       "".join(q + "\n" for q in t.splitlines() if not (q.startswith("bc_") and q[3] in periodic)))
    got, launches = [], []
    for pts in (None, 0):
        sc = R.Scene.from_cfg(cfg, precision=precision, var_den=var_den)
        try:
            if pts is not None:
                sc.set_coarse_cluster(pts)
            sc.prepare()
            assert sc.run(3) == R.NORMAL_EXIT
            got.append({f: sc.field(f).copy() for f in FIELDS})
            launches.append(sc.launches())
        finally:
            sc.close()
    for f in FIELDS:
        assert np.array_equal(got[0][f], got[1][f]), f
    assert launches[0] < launches[1]


def test_large_group_runs_per_phase(tmp_path):
    """A group of more scenes than their clusters pay for runs its multigrid
    phases as launches over all scenes, new scenes and scenes with a limit
    alike: as fast as when asked to (32 clusters took 1.5 times as long on a
    B200), with the same bits."""
    text = "".join(q + "\n" for q in scenes.cavity(12).splitlines() if not q.startswith("bc_"))
    d = R.desc_from_cfg(scenes.write(str(tmp_path / "p.cfg"), text))
    best, got = [], []
    for pts in (None, 40000, 0):
        b = R.Batch([d] * 32)
        try:
            if pts is not None:
                for i in range(32):
                    R._lib.check(R.lib().rmt3d_scene_set_coarse_cluster(b.scene_handle(i), pts))
            b.prepare()
            b.step(3)
            t = []
            for _ in range(8):
                t0 = time.perf_counter()
                b.step(10)
                t.append(time.perf_counter() - t0)
            best.append(min(t))
            got.append([b.field(31, f) for f in FIELDS])
        finally:
            b.close()
    for f, a, c, e in zip(FIELDS, *got):
        assert np.array_equal(a, e) and np.array_equal(c, e), f
    assert best[0] < 1.25 * best[2] and best[1] < 1.25 * best[2]
