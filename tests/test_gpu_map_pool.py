"""Maps made one after another share a pool of device memory: what an earlier map
left in it must not show, several threads may make and close maps at once, what
is kept is bounded, and a map too large for the device is still refused and
leaves the next one unharmed."""
import threading

import numpy as np
import pytest

from tests.helpers import MAXCAM, SCALING, circle_frames

pytestmark = pytest.mark.gpu


def _fuse(n=6, wh=(160, 120), leaves=30000, storage="fp32"):
    from fastfusion_b200.fusion import CameraInfo, FusionMipMapCPU
    K, frames = circle_frames(0, n, *wh)
    m = FusionMipMapCPU(0, 0, 0, 0.005, 0.01, 0, True, leaves_max=leaves, branches_max=1 << 21, storage=storage,
                        rcp="exact")
    m.addMapSequence([f[0] for f in frames], [CameraInfo(K, f[2], f[3]) for f in frames], [f[1] for f in frames],
                     SCALING, MAXCAM)
    m.updateMeshes()
    mesh = m.getMeshInterleavedMarchingCubes()
    out = [np.array(x) for x in (*m.bricks(), *m.leaves(), mesh.vertices, mesh.colors, mesh.faces)]
    m.close()
    return out


def _same(a, b):
    return all(x.shape == y.shape and x.tobytes() == y.tobytes() for x, y in zip(a, b))


def test_one_after_another(lib_built):
    want = _fuse()
    for wh, leaves, storage in [((320, 240), 50000, "fp16"), ((97, 61), 20000, "fp32"), ((640, 480), 30000, "fp16")]:
        _fuse(3, wh, leaves, storage)
        assert _same(_fuse(), want)


def test_threads(lib_built):
    want = _fuse()
    bad = []

    def work(k):
        try:
            for i in range(4):
                if (i + k) % 2:
                    _fuse(2, (97, 61), 20000 + 5000 * k, "fp16")
                if not _same(_fuse(), want):
                    bad.append((k, i))
        except Exception as e:  # (reported by the main thread)
            bad.append(repr(e))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_kept_memory_is_bounded(lib_built):
    import torch
    _fuse()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    _fuse(2, leaves=600000)  # 4.3 GB of voxels
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < (1 << 30) + (256 << 20)


def test_too_large_is_refused(lib_built):
    from fastfusion_b200.fusion import FusionMipMapCPU
    want = _fuse()
    with pytest.raises(Exception):
        FusionMipMapCPU(0, 0, 0, 0.005, 0.01, 0, True, leaves_max=60000000, branches_max=1 << 21)  # 430 GB
    assert _same(_fuse(), want)
