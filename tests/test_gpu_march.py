"""The multigrid phases of a group of six 64^3 cavities march along z (from
400,000 points of work over the group), those of one alone run point by point:
the same bits over whole steps."""
import numpy as np
import pytest

import rmt3d_b200 as R
from rmt3d_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,var_den", [(R.FP64, 0), (R.MIXED, 0), (R.MIXED, 1)])
def test_group_marches_alone_does_not(tmp_path, precision, var_den):
    d = R.desc_from_cfg(scenes.write(str(tmp_path / "c.cfg"), scenes.cavity(64)))
    d.precision, d.var_den = precision, var_den
    sc = R.Scene(d)
    try:
        sc.prepare()
        assert sc.run(2) == R.NORMAL_EXIT
        want = {f: sc.field(f).copy() for f in ("u", "v", "w", "p")}
    finally:
        sc.close()
    b = R.Batch([d] * 6)
    try:
        b.prepare()
        b.step(2)
        for f in want:
            for i in (0, 5):
                assert np.array_equal(b.field(i, f), want[f]), f
    finally:
        b.close()
