"""Insertion of several particles at once (one operator per coset of the grid rotations, then
their sum) against the same particles one call at a time (all 60 operators each): every
accumulation kind, the plane z = 0 included.

Both round a sample's position to FP32 at up to nx/2 + maxR (2^-18 of a voxel at box 64), on
mirrored axes, so a tap's weight differs by up to 2^-17; the sums over hundreds of taps of
either sign stay within that of each other."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,box,max_res", [("full", 64, 12.0), ("half", 64, 12.0), ("substep", 64, 12.0),
                                              ("full", 48, 8.8)])
def test_together_equals_one_by_one(built, kind, box, max_res):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(n=box, P=7, T=2, step=4.0, max_res=max_res)
    p = ci.default_params(box, apix=4.0, minRes=60.0, maxRes=max_res, ampwg=0.07, subrec=int(kind == "substep"),
                          imgmask=(box // 2 - 2) * 4.0)
    q = parts.copy()
    q["pr"] = 10.0
    q["theta"][1] = q["phi"][1] = q["omega"][1] = 0.0  # its plane is z = 0 itself
    q["pr"][4] = 95.0  # not selected
    out = []
    with ci.Context(0, p) as ctx:
        for groups in ([range(7)], [[i] for i in range(7)], [[0, 1, 2, 3], [4, 5], [6]]):
            ctx.rec_begin_half(q["x"][0], q["y"][0]) if kind == "half" else ctx.rec_begin()
            used = sum(ctx.rec_insert(imgs[list(g)], q[list(g)]) for g in groups)
            assert used == 6
            out.append(ctx.rec_get_partial())
    for got in (out[0], out[2]):
        for a, b in zip(got, out[1]):
            assert np.linalg.norm(a - b) <= 2.0 ** -17 * np.linalg.norm(b)
            assert np.linalg.norm(a[0] - b[0]) <= 2.0 ** -17 * np.linalg.norm(b[0])
