"""The de-duplication's tiles and the list of cells they hand the octree
insert, where they can go wrong: images smaller than a tile, one row or column
past it, wider than many tiles; every pixel its own cell; depths either side of
a cell-size step; pixels at and outside the volume's faces (growth).  Frame by
frame against the oracle: volume, leaf table in index order, queue, octree and
the number of processed pixels; and as one sequence."""
import numpy as np
import pytest

from tests.helpers import MAXCAM, SCALING, queue_set, tree_shape
from tests.test_gpu_fusion import _cam, _compare_frame, _pair

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 40), (40, 1), (31, 16), (32, 17), (33, 32), (65, 33), (1057, 24), (100, 131)]


def _depth(kind, rng, w, h, k):
    if kind == "noise":  # every pixel its own cell
        d = rng.uniform(0.3, 4.2, (h, w))
    elif kind == "step":  # cell sizes change at 1.125 m and 2.125 m
        d = np.where(rng.random((h, w)) < 0.5, 1.125, 2.125) + rng.uniform(-0.004, 0.004, (h, w))
    elif kind == "plane":
        d = np.full((h, w), 0.9 + 0.3 * k)
    else:  # a surface with holes
        d = 1.0 + np.linspace(0, 1.5, w)[None, :] + 0.02 * rng.standard_normal((h, w))
        d[rng.random((h, w)) < 0.2] = 0
    return np.clip(np.rint(d / SCALING), 0, 65535).astype(np.uint16)


def _frames(kind, w, h, n, stride):
    rng = np.random.default_rng(w * 131 + h)
    K = np.array([max(w, 40) * 0.9, max(w, 40) * 0.9, w / 2 - 0.5, h / 2 - 0.5])
    out = []
    for k in range(n):
        a = 0.2 * k
        R = np.array([[np.cos(a), 0, np.sin(a)], [0, 1, 0], [-np.sin(a), 0, np.cos(a)]])
        out.append((_depth(kind, rng, w, h, k), rng.integers(0, 256, (h, w, 3), dtype=np.uint8), R,
                    np.array([stride * k, -0.4 * stride * k, 0.1 * stride * k])))
    return K, out


@pytest.mark.parametrize("kind,stride", [("noise", 0.05), ("step", 0.05), ("plane", 0.02), ("holes", 2.5)])
@pytest.mark.parametrize("w,h", SIZES)
def test_cells_match_oracle(lib_built, port_lib, w, h, kind, stride):
    K, frames = _frames(kind, w, h, 3, stride)
    g, p = _pair(port_lib)
    s, _ = _pair(port_lib)
    for depth, bgr, R, t in frames:
        assert g.addMap(depth, _cam(K, R, t), bgr, SCALING, MAXCAM) == p.add_map(depth, bgr, K, R, t, SCALING, MAXCAM)
        _compare_frame(g, p)
        assert tree_shape(g.tree()) == tree_shape(p.tree())
    s.addMapSequence([f[0] for f in frames], [_cam(K, f[2], f[3]) for f in frames], [f[1] for f in frames], SCALING,
                     MAXCAM)
    for a, b in zip(s.leaves(), g.leaves()):
        assert np.array_equal(a, b)
    assert tree_shape(s.tree()) == tree_shape(g.tree())
    assert queue_set(s.queue()) == queue_set(g.queue())
    assert s.stats()["processed_pixels"] == g.stats()["processed_pixels"]
    for a, b in zip(s.bricks(), g.bricks()):
        assert np.array_equal(a.view(np.uint16), b.view(np.uint16))


@pytest.mark.parametrize("rows", [8, 16, 32])
def test_tile_heights_agree(lib_built, port_lib, rows):
    K, frames = _frames("holes", 129, 97, 3, 0.05)
    g, p = _pair(port_lib)
    g.set_tuning(dedupe_rows=rows)
    for depth, bgr, R, t in frames:
        assert g.addMap(depth, _cam(K, R, t), bgr, SCALING, MAXCAM) == p.add_map(depth, bgr, K, R, t, SCALING, MAXCAM)
        _compare_frame(g, p)
