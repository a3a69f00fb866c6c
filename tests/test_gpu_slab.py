"""A new scene runs as much of each V-cycle as fits a cluster's shared memory
(on these grids all of it, the finest level included) in one launch: the same
bits over whole steps as one launch per phase, and fewer launches."""
import numpy as np
import pytest

import helpers as H
import rmt3d_b200 as R

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
