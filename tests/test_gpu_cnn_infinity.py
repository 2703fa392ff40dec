"""An activation that overflows to infinity stays within the outputs whose 5x5
windows see it: every other value of each layer keeps its bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,img,r,c", [(1, 40, 150, 0, 20, 75), (1, 41, 150, 0, 17, 127), (1, 40, 300, 0, 22, 128),
                                           (2, 33, 70, 1, 3, 2), (2, 33, 70, 0, 32, 69), (3, 7, 140, 1, 0, 130)])
@pytest.mark.parametrize("value", [3.0e38, float("inf")])
def test_infinite_activation_stays_in_its_windows(lib_built, n, h, w, img, r, c, value):
    import torch
    from fastfusion_b200.confidence import ConfidenceNet, init_params
    params = init_params(6)
    params[:2000] *= 64.0  # (layer 1 overflows at the large finite value too)
    net = ConfidenceNet(params)
    rng = np.random.default_rng(h * w)
    feat = rng.normal(size=(n, h, w, 8)).astype(np.float32)
    feat[..., 5:] = 0.0
    tgt = torch.zeros((n, h, w), device="cuda")

    def run(f):
        f = torch.tensor(f, device="cuda").to(torch.bfloat16).contiguous()
        b = net.loss_and_grads(f, tgt, 1.0)
        layers = [b[k].float().cpu().numpy().reshape(n, h, w, -1).copy() for k in ("a1", "a2", "pred")]
        return layers + [net.forward(f, tau_m=0.03).cpu().numpy().reshape(n, h, w, -1).copy()]

    want = run(feat)
    feat[img, r, c, :5] = value
    got = run(feat)
    assert not np.isfinite(got[0]).all()
    for a, b, reach in zip(got, want, (2, 4, 6, 6)):
        outside = np.ones((n, h, w), bool)
        # (an infinite feature: layer 1 takes kernel columns in pairs, the last with a
        # sixth of weight zero, so one more column to the left)
        left = reach + 1 if np.isinf(value) else reach
        outside[img, max(r - reach, 0):r + reach + 1, max(c - left, 0):c + reach + 1] = False
        assert np.isfinite(b).all()
        assert np.array_equal(a[outside].view(np.uint32), b[outside].view(np.uint32))
