"""The one-launch wall ghost fill against the reference's axis-by-axis fill
(fields.hh:765-800) in numpy, exactly: every axis walled, and one axis
periodic, with Dirichlet and Neumann faces."""
import numpy as np
import pytest

import rmt3d_b200 as R
from rmt3d_b200 import scenes

pytestmark = pytest.mark.gpu

BCS = {"xl": (1, 2, 1, 0.0, 0.3, 0.0), "xh": (2, 1, 1, -0.2, 0.1, 0.0), "yl": (1, 1, 2, 0.0, 0.0, 0.1),
       "yh": (1, 2, 1, 0.0, 0.2, 0.0), "zl": (1, 1, 1, 0.0, 0.0, 0.0), "zh": (1, 1, 2, 0.7, 0.2, -0.1)}


@pytest.mark.parametrize("periodic", ["", "y", "x"])
def test_wall_ghosts(tmp_path, periodic):
    n = (24, 16, 20)
    t = scenes.cavity(16, 4).split("bc_xl")[0].replace("sys_size 16 16 16", "sys_size %d %d %d" % n)
    t = t.replace("xyz_bounds 0 1 0 1 0 1", "xyz_bounds 0 1.5 0 1 0 1.25\nwall_pos 0 1.5 0 1 0 1.25")
    for f, b in BCS.items():
        if f[0] not in periodic:
            t += "bc_%s %d %d %d %r %r %r\n" % ((f,) + b)
    sc = R.Scene.from_cfg(scenes.write(str(tmp_path / "w.cfg"), t))
    try:
        sc.prepare()
        assert sc.run(2) == R.NORMAL_EXIT
        h = 1.0 / 16
        for c, name in enumerate("uvw"):
            got = sc.field(name)
            v = got.copy()
            for d, axis in enumerate("xyz"):
                if axis in periodic:
                    continue
                s = np.moveaxis(v, 2 - d, 0)
                for side in (0, 1):
                    b = BCS[axis + "lh"[side]]
                    for layer in (1, 2):
                        gh, mi = (2 - layer, 1 + layer) if side == 0 else (1 + n[d] + layer, 2 + n[d] - layer)
                        dn = 2 * abs(0.5 * h * (2 * layer - 1))
                        s[gh] = 2 * b[3 + c] - s[mi] if b[c] == 1 else (1 if side else -1) * dn * b[3 + c] + s[mi]
            sl = tuple(slice(2, -2) if a in periodic else slice(None) for a in "zyx")
            assert np.array_equal(v[sl], got[sl]), (name, periodic)
    finally:
        sc.close()
