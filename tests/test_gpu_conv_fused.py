"""The proposer's tensor-core convolutions at the edges of their tiles: odd heights (a step is
two rows), channel counts that are padded to 8, 16 or 32, blocks that start inside a sample
and cross samples, one row; and the network with the pooling and the ReLU's gates inside the
convolutions at batches of one sample and of several samples per block.  Bounds are those of
the tests whose oracles these are: the same operands, the same FP32 sums in another order."""
import numpy as np
import pytest

from test_gpu_conv_tc import conv_ref, tf32, wgrad_ref
from test_gpu_learn import CM, CONV, MIXK, NR, NT, random_weights, torch_reference
from test_gpu_learn import lctx  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Cin,Cout,H", [
    (1, 1, 32, 1), (3, 1, 16, 7), (70, 1, 16, 33), (2, 8, 16, 5), (3, 8, 32, 1), (5, 16, 16, 3), (7, 24, 32, 2),
    (150, 24, 16, 5), (1, 32, 32, 1), (90, 32, 32, 9), (160, 16, 32, 6),
])
def test_edges_of_the_tiles(built, B, Cin, Cout, H):
    import cryoim_gb300 as ci
    rng = np.random.default_rng(B * 1000 + Cin * 10 + Cout + H)
    x = rng.normal(size=(B, Cin, H, 128)).astype(np.float32)
    W = (rng.normal(size=(Cout, Cin, 3, 3)) / np.sqrt(9 * Cin)).astype(np.float32)
    bias = rng.normal(0, 0.1, Cout).astype(np.float32)
    g = rng.normal(size=(B, Cout, H, 128)).astype(np.float32)
    out, dW, db = ci.conv3_check(x, W, bias, relu=H % 2 == 1, dpre=g, tensor_cores=True)
    ref = conv_ref(tf32(x), tf32(W), bias.astype(np.float64), H % 2 == 1)
    assert np.abs(out - ref).max() < 3e-6 * np.abs(ref).max()
    dref = wgrad_ref(tf32(x), tf32(g))
    assert np.abs(dW - dref).max() < 3e-5 * np.abs(dref).max()
    bref = g.astype(np.float64).sum(axis=(0, 2, 3))
    assert np.abs(db - bref).max() <= 3e-5 * np.abs(bref).max() + 1e-3


@pytest.mark.parametrize("B", [1, 23])
def test_network_with_pooling_inside_the_convolutions(lctx, B):  # noqa: F811
    ctx, p = lctx
    rng = np.random.default_rng(100 + B)
    views = ctx.learn_views()
    V = len(views)
    w = random_weights(ctx.learn_params().size, V, rng)
    ctx.learn_params(w)
    feat = rng.normal(size=(B, NR, NT)).astype(np.float32)
    th, ph = np.radians(views[rng.integers(V, size=B)].astype(np.float64).T)
    truth = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th),
                      rng.integers(NT, size=B).astype(np.float64)], 1).astype(np.float32)
    sc, loss, gr = ctx.learn_forward(feat, truth, views=V)
    only, _, _ = ctx.learn_forward(feat, views=V)  # without the gates of a backward pass
    assert np.array_equal(sc, only)
    rsc, rloss, rgr = torch_reference(w, feat, truth, views.astype(np.float64), 2.0 * p.searchstep, tf32=True)
    assert np.abs(sc - rsc).max() < 1e-4 * np.abs(rsc).max() + 1e-6
    assert np.allclose(loss, rloss, rtol=1e-4, atol=1e-5)
    off = 0
    for sz in [n for ci, co in CONV for n in (co * ci * 9, co)] + [CM * MIXK, CM, V * CM * NT]:
        a, b = gr[off:off + sz], rgr[off:off + sz]
        assert np.abs(a - b).max() <= 5e-3 * np.abs(b).max() + 1e-7
        off += sz
    again = ctx.learn_forward(feat, truth, views=V)[2]
    assert np.array_equal(gr[:off - V * CM * NT], again[:off - V * CM * NT])  # sums in a fixed order
