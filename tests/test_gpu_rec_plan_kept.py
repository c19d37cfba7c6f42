"""A context keeps its 3D plan and map buffer between reconstructions: the maps are those of a fresh
context, also after the box has changed and on another stream."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


def reconstruct(ctx, imgs, parts):
    ctx.rec_begin()
    ctx.rec_insert(imgs, parts.copy())
    return ctx.rec_finish()


def test_maps_are_those_of_a_fresh_context(built):
    import cryoim_gb300 as ci
    import torch
    cases = []
    for n in (48, 64):
        p, vol, tmpl, timgs, imgs, parts, truth = small_case(n=n, P=3, T=2)
        q = parts.copy()
        q["theta"], q["phi"], q["omega"] = truth[:, 0], truth[:, 1], truth[:, 2]
        with ci.Context(0, p) as ctx:
            cases.append((p, imgs, q, reconstruct(ctx, imgs, q)))
    stream = torch.cuda.Stream()
    with ci.Context(0, cases[0][0]) as ctx:
        for step in (0, 0, 1, 1, 0):
            p, imgs, q, want = cases[step]
            ctx.set_params(p)
            got = reconstruct(ctx, imgs, q)
            # FP32 atomics: the sums' order, not the terms, may differ
            assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
        ctx.set_stream(stream.cuda_stream)
        assert np.abs(reconstruct(ctx, cases[0][1], cases[0][2]) - cases[0][3]).max() <= 1e-5 * np.abs(cases[0][3]).max()
        ctx.set_stream(None)
