"""The raycaster against its definition, pixel by pixel on the CPU in NumPy
float64: image sizes around a block of pixels, steps shorter and longer than a
voxel, windows that leave the volume, both storages.  Every sample's position is
rounded in float32 on the device, so a pixel whose crossing lies within rounding
of a decision (a sample's sign, a cube's or brick's border) may differ; at least
98 % of the pixels must agree to 0.1 step, and pixels without depth exactly."""
import numpy as np
import pytest

from tests.helpers import MAXCAM, SCALING, circle_frames

pytestmark = pytest.mark.gpu


def _leaf_lookup(f):
    pos, scale, _ = f.leaves()
    d, w, _ = f.bricks()
    table = {}
    for i, (p, s) in enumerate(zip(pos, np.asarray(scale).reshape(-1))):
        table[(int(p[0]), int(p[1]), int(p[2]), int(s))] = i
    return table, d, w, sorted({int(s) for s in np.asarray(scale).reshape(-1)})


def _cast(table, d, w, scales, n, R, t, K, depth, x, y, window, step, thr):
    d0 = np.float64(np.float32(SCALING) * np.float32(depth[y, x]))
    if d0 <= 0:
        return 0.0
    t0 = max(d0 - window, 0.05)
    steps = int((d0 + window - t0) / step) + 1
    ray = np.array([(x - K[2]) / K[0], (y - K[3]) / K[1], 1.0])
    prev, prev_t, band = None, 0.0, 0.0
    for k in range(steps):
        tt = t0 + k * step
        g = R @ (ray * tt) + t
        i = np.rint(g).astype(int)
        s = None
        if (i >= 0).all() and (i < n).all():
            leaf = None
            for sc in scales:
                o = (i // (8 * sc)) * (8 * sc)
                leaf = table.get((int(o[0]), int(o[1]), int(o[2]), sc))
                if leaf is not None:
                    break
            if leaf is not None:
                band = 0.99 * thr * sc
                u = (g - o) / sc
                c = np.floor(u).astype(int)
                if (c >= 0).all() and (c < 7).all():
                    q = [((c[2] + (j >> 2)) * 8 + c[1] + ((j >> 1) & 1)) * 8 + c[0] + (j & 1) for j in range(8)]
                    if (w[leaf, q] > 0).all():
                        a = u - c
                        s = sum((a[0] if j & 1 else 1 - a[0]) * (a[1] if j & 2 else 1 - a[1]) *
                                (a[2] if j & 4 else 1 - a[2]) * float(d[leaf, q[j]]) for j in range(8))
                if s is None:
                    l = np.clip(np.rint(u).astype(int), 0, 7)
                    v = (l[2] * 8 + l[1]) * 8 + l[0]
                    if w[leaf, v] > 0:
                        s = float(d[leaf, v])
        if s is not None and prev is not None and prev < 0 <= s:
            return prev_t + step * -prev / (s - prev)
        if s is not None and prev is None and k > 0 and 0 <= s < band:
            return tt - s
        prev, prev_t = s, tt
    return -1.0


@pytest.mark.parametrize("w,h,step,window,storage", [(160, 120, 0.0025, 0.15, "fp32"), (47, 33, 0.0012, 0.06, "fp32"),
                                                    (17, 9, 0.012, 0.5, "fp32"), (97, 25, 0.0025, 0.1, "fp16")])
def test_raycast_matches_definition(lib_built, w, h, step, window, storage):
    import torch
    from fastfusion_b200 import fusion
    K, frames = circle_frames(0, 3, w, h)
    f = fusion.FusionMipMapCPU(0, 0, 0, 0.005, 0.01, 0, True, leaves_max=100000, branches_max=1 << 21, storage=storage)
    for depth, bgr, R, t in frames:
        f.addMap(depth, fusion.CameraInfo(K, R, t), bgr, SCALING, MAXCAM)
    depth, _, R, t = frames[1]
    depth = depth.copy()
    depth[::7, ::5] = 0
    dd = torch.from_numpy(depth.view(np.int16)).cuda()
    out = torch.empty((h, w), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    f.raycast_depth(dd.data_ptr(), w, h, fusion.CameraInfo(K, R, t), out.data_ptr(), SCALING, window, step)
    f.sync()
    got = out.cpu().numpy()
    st = f.stats()
    table, d, wt, scales = _leaf_lookup(f)
    Rg, tg = R / 0.005, (np.asarray(t) - np.asarray(st["offset"])) / 0.005
    rng = np.random.default_rng(3)
    pix = [(x, y) for y in range(h) for x in range(w)]
    pix = [pix[i] for i in rng.choice(len(pix), min(400, len(pix)), replace=False)]
    good = 0
    for x, y in pix:
        want = _cast(table, d, wt, scales, st["n"], Rg, tg, K, depth, x, y, window, step, 0.01)
        if depth[y, x] == 0:
            assert got[y, x] == 0
        good += abs(got[y, x] - want) <= 0.1 * step
    assert good >= 0.98 * len(pix), good / len(pix)
    assert sum(got[y, x] > 0 for x, y in pix) > len(pix) // 4
