"""A context taken from one box size to another: calls of several passes (each lane has its own transforms)
and the training (whose data are made on a lane) give what a new context gives, to the bit."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu
F = ("theta", "phi", "omega", "x", "y", "pr")


def results(ctx, case, n):
    p, vol, tmpl, timgs, imgs, parts, truth = case
    ctx.set_batch(2)
    ctx.set_lanes(3)
    ctx.load_templates(timgs, tmpl)
    ctx.set_reference_map(vol)
    out = []
    for kw in (dict(pick=0), dict(pick=1, local_range=2.0, local_step=1.0)):
        q = parts.copy()
        c = ctx.contract_search(imgs, q, origin_max=1.0, origin_step=0.5, topk=4, want_cands=True, **kw)
        out += [q[f].copy() for f in F] + [c]
    st = ctx.learn_train(vol, samples=128, batch=32, seed=3, snr=1.0, df_min=1.0, df_max=3.0, origin_max=2.0)
    return out + [np.array([st["loss"]]), ctx.learn_params()]


def test_another_box_size(built):
    import cryoim_gb300 as ci
    cases = {n: small_case(n=n, P=6, T=2, step=6.0, max_res=4.0 * n / 14.5) for n in (64, 50, 72)}
    with ci.Context(0, cases[64][0]) as ctx:
        for n in (64, 50, 72, 64):
            ctx.set_params(cases[n][0])
            got = results(ctx, cases[n], n)
            with ci.Context(0, cases[n][0]) as new:
                want = results(new, cases[n], n)
            for k, (a, b) in enumerate(zip(got, want)):
                np.testing.assert_array_equal(a, b, err_msg=f"box {n}, result {k}")
