"""The meshing passes where their shortcuts end: cells whose leaves lie on
different octree levels, samples that fall back to a parent leaf or to nothing,
runs of clean cells between dirty ones, the first update.  Depth images with
steps across several resolutions, holes and noise; the mesh must equal the
oracle's bit for bit after every update, and 16-bit storage must give the same
mesh incrementally as from scratch."""
import numpy as np
import pytest

from tests.helpers import MAXCAM, SCALING
from tests.test_gpu_mesh import _assert_same_mesh, _cam, _gpu

pytestmark = pytest.mark.gpu


def _frames(seed, w, h, n, holes, noise):
    rng = np.random.default_rng(seed)
    K = np.array([w * 0.82, w * 0.82, w / 2 - 0.5, h / 2 - 0.5])  # fx, fy, cx, cy
    out = []
    for k in range(n):
        # a ramp from near to far: every resolution the depth range has, with steps between
        x = np.linspace(0.45, 4.2, w)[None, :] + 0.3 * (np.arange(h)[:, None] * 5 // h)
        d = np.roll(x, 7 * k, axis=1) + noise * rng.standard_normal((h, w))
        for _ in range(holes):
            cx, cy, r = rng.integers(0, w), rng.integers(0, h), rng.integers(2, max(3, h // 6))
            d[max(0, cy - r):cy + r, max(0, cx - r):cx + r] = 0
        depth = np.clip(d / SCALING if SCALING < 1 else d * SCALING, 0, 65535).astype(np.uint16)
        bgr = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
        a = 0.03 * k
        R = np.array([[np.cos(a), 0, np.sin(a)], [0, 1, 0], [-np.sin(a), 0, np.cos(a)]], np.float64)
        out.append((depth, bgr, R, np.array([0.02 * k, 0.01, 0.0])))
    return K, out


@pytest.mark.parametrize("seed,w,h,holes,noise", [(0, 61, 47, 0, 0.0), (1, 61, 47, 6, 0.01), (2, 160, 120, 3, 0.004),
                                                 (3, 97, 131, 12, 0.03), (4, 17, 9, 1, 0.0)])
def test_every_update_matches_oracle(lib_built, port_lib, seed, w, h, holes, noise):
    K, frames = _frames(seed, w, h, 5, holes, noise)
    g = _gpu()
    p = port_lib.PortFusion(leaves_total=271420, branches_total=4793488)
    for depth, bgr, R, t in frames:
        g.addMap(depth, _cam(K, R, t), bgr, SCALING, MAXCAM)
        p.add_map(depth, bgr, K, R, t, SCALING, MAXCAM)
        # the voxels are the map's own: what is compared is the meshing
        p.set_bricks(*g.bricks())
        g.updateMeshes()
        assert g.stats()["mesh_cells"] == p.update_meshes()
        _assert_same_mesh(g.getMeshInterleavedMarchingCubes(), p.mesh())
    # an update with nothing new copies every cell
    g.updateMeshes()
    _assert_same_mesh(g.getMeshInterleavedMarchingCubes(), p.mesh())


@pytest.mark.parametrize("storage", ["fp32", "fp16"])
def test_incremental_equals_first_update(lib_built, storage):
    K, frames = _frames(7, 97, 75, 6, 4, 0.01)
    a, b = _gpu(storage=storage), _gpu(storage=storage)
    for depth, bgr, R, t in frames:
        for m in (a, b):
            m.addMap(depth, _cam(K, R, t), bgr, SCALING, MAXCAM)
        a.updateMeshes()
    b.updateMeshes()
    ma, mb = a.getMeshInterleavedMarchingCubes(), b.getMeshInterleavedMarchingCubes()
    assert len(ma.vertices) > 0
    assert np.array_equal(ma.vertices.view(np.uint32), mb.vertices.view(np.uint32))
    assert np.array_equal(ma.faces, mb.faces)
    assert np.array_equal(ma.colors, mb.colors)


def test_large_cell_lists(lib_built):
    """Cell lists past the size up to which blocks add up the sums before theirs
    (131,072 cells), incrementally and from scratch: every pixel of a noise image
    its own brick."""
    rng = np.random.default_rng(5)
    w, h = 512, 384
    K = np.array([w * 0.9, w * 0.9, w / 2 - 0.5, h / 2 - 0.5])
    a = _gpu(leaves_max=600000, branches_max=1 << 25, storage="fp16")
    b = _gpu(leaves_max=600000, branches_max=1 << 25, storage="fp16")
    for k in range(3):
        depth = np.rint(rng.uniform(0.5, 4.5, (h, w)) / SCALING).astype(np.uint16)
        bgr = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
        for m in (a, b):
            m.addMap(depth, _cam(K, np.eye(3), np.zeros(3)), bgr, SCALING, 5.0)
        a.updateMeshes()
    b.updateMeshes()
    assert a.stats()["mesh_cells"] > 1 << 17
    ma, mb = a.getMeshInterleavedMarchingCubes(), b.getMeshInterleavedMarchingCubes()
    assert len(ma.vertices) > 0
    assert np.array_equal(ma.vertices.view(np.uint32), mb.vertices.view(np.uint32))
    assert np.array_equal(ma.faces, mb.faces)
    assert np.array_equal(ma.colors, mb.colors)
    a.close()
    b.close()
