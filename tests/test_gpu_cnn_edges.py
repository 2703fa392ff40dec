"""The confidence network's tensor-core kernels at the edges of their tiles:
strips and windows of the convolutions (112 and 28 pixels, pairs of rows),
tiles of the weight gradients (64 x 8 pixels), single pixels and rows, several
images per block, blocks that run from one strip into the next.

Against the float64 oracle from the GPU's own stored activations.  Tolerances,
from the formats: a layer's output is an FP32 sum of at most 400 products,
1e-4 of its scale; a stored BF16 activation may round to the other side (one
step, 2^-7 relative, plus that sum's error); a parameter gradient is an FP32
sum over the pixels, 1e-5 relative L2 per tensor.
"""
import numpy as np
import pytest

from oracle import cnn

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (1, 1, 28), (2, 2, 29), (1, 7, 63), (2, 8, 64), (1, 9, 65), (1, 5, 112), (3, 33, 113),
         (1, 4, 225), (40, 3, 30), (2, 37, 141), (1, 160, 190)]
PARTS = (("W1", 0, 2000), ("b1", 2000, 2016), ("W2", 2016, 8416), ("b2", 8416, 8432), ("W3", 8432, 8832),
         ("b3", 8832, 8833))


@pytest.mark.parametrize("n,h,w", SIZES)
def test_layers_and_gradients_at_tile_edges(lib_built, n, h, w):
    import torch
    from fastfusion_b200.confidence import ConfidenceNet, init_params
    net = ConfidenceNet(init_params(4))
    rng = np.random.default_rng(1000 * h + w)
    feat = rng.normal(size=(n, h, w, 8)).astype(np.float32)
    feat[..., 5:] = 0.0
    feat_t = torch.tensor(feat, device="cuda").to(torch.bfloat16).contiguous()
    feat = feat_t.float().cpu().numpy()
    tgt = rng.uniform(0, 5, size=(n, h, w)).astype(np.float32)
    if n * h * w > 4:
        tgt[rng.random(tgt.shape) < 0.1] = -1.0
    b = net.loss_and_grads(feat_t, torch.tensor(tgt, device="cuda"), 1.0 / (n * h * w))
    a1, a2 = (b[k].float().cpu().numpy() for k in ("a1", "a2"))
    P = {k: cnn.bf16(v) for k, v in cnn.unpack(net.state()).items()}
    for got, x, wt, bias in ((a1, feat[..., :5], "W1", "b1"), (a2, a1, "W2", "b2")):
        ref = np.maximum(cnn.conv(x, P[wt], P[bias]), 0)
        tol = 1e-4 * max(1.0, np.abs(ref).max())
        assert (np.abs(got - ref) <= np.abs(ref) * 2.0 ** -7 + tol).all()
        assert (got != cnn.bf16(ref)).mean() <= 0.02
    pred = b["pred"].cpu().numpy()
    ref = cnn.conv(a2, P["W3"], P["b3"])[..., 0]
    assert np.abs(pred - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max())
    g = net.grads.cpu().numpy().astype(np.float64)
    ref = cnn.backward(net.state(), feat, a1, a2, b["dpred"].cpu().numpy())
    for name, o, e in PARTS:
        err = np.linalg.norm(g[o:e] - ref[o:e]) / max(np.linalg.norm(ref[o:e]), 1e-30)
        assert err <= 1e-5, (name, err)
    # the confidence of the same features
    conf = net.forward(feat_t, tau_m=0.03).cpu().numpy()
    assert np.abs(conf - cnn.confidence(pred, 3.0)).max() <= 1e-6


def test_gradients_add_and_keep_infinities(lib_built):
    """Gradients are added to the caller's; an infinite output gradient
    reaches the bias gradient and no finite value appears in its place."""
    import torch
    from fastfusion_b200.confidence import ConfidenceNet, init_params
    net = ConfidenceNet(init_params(5))
    rng = np.random.default_rng(7)
    feat = torch.tensor(rng.normal(size=(1, 20, 70, 8)), device="cuda").to(torch.bfloat16).contiguous()
    tgt = torch.tensor(rng.uniform(0, 5, size=(1, 20, 70)).astype(np.float32), device="cuda")
    net.loss_and_grads(feat, tgt, 1e-3)
    once = net.grads.clone()
    net.loss_and_grads(feat, tgt, 1e-3)
    d = (net.grads - 2 * once).double().norm() / once.double().norm()
    assert float(d) <= 1e-5
    net.grads.zero_()
    tgt[0, 10, 35] = float("inf")  # dpred = -inf there
    net.loss_and_grads(feat, tgt, 1e-3)
    g = net.grads.cpu().numpy()
    assert np.isneginf(g[8832])
    assert not np.isfinite(g[8432:8832]).any()
