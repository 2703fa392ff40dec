"""A sequence whose first frame's confidence network gives up (injected on the
host: the error word is set after the networks, when later frames may have been
placed already): the call reports it, and the map is the one of frames added one by
one of which as many as the sequence placed were not updated -- leaf table, octree,
every voxel, the frames waiting before the call included; the same frames added
again, the ones after them and the mesh are then right."""
import numpy as np
import pytest

from tests.helpers import MAXCAM, SCALING, circle_frames, tree_shape

pytestmark = pytest.mark.gpu


def _same(a, b):
    for x, y in zip((*a.leaves(), *a.bricks()), (*b.leaves(), *b.bricks())):
        assert x.shape == y.shape and x.tobytes() == y.tobytes()
    assert tree_shape(a.tree()) == tree_shape(b.tree())
    sa, sb = a.stats(), b.stats()
    assert (sa["leaves_used"], sa["branches_used"], sa["frames"]) == (sb["leaves_used"], sb["branches_used"],
                                                                      sb["frames"])


@pytest.mark.parametrize("w,h,waiting,n,learned", [(160, 120, 0, 6, True), (160, 120, 3, 6, True),
                                                   (640, 480, 0, 10, True), (640, 480, 5, 10, True),
                                                   (640, 480, 9, 10, True), (160, 120, 3, 6, False)])
def test_network_timeout_leaves_the_map_whole(lib_built, w, h, waiting, n, learned):
    from fastfusion_b200 import confidence
    from fastfusion_b200.fusion import CameraInfo, FFError, FusionMipMapCPU
    K, frames = circle_frames(0, waiting + n + 4, w, h)
    cams = [CameraInfo(K, R, t) for _, _, R, t in frames]
    params, tau = confidence.load_weights()

    def make():
        f = FusionMipMapCPU(0, 0, 0, 0.005, 0.01, 0, True, leaves_max=100000, branches_max=1 << 21, rcp="exact")
        if learned:
            f.set_confidence(params, tau)
        return f

    def add(f, ks):
        return [f.addMap(frames[k][0], cams[k], frames[k][1], SCALING, MAXCAM) for k in ks]

    def sequence(f, ks):
        return f.addMapSequence([frames[k][0] for k in ks], [cams[k] for k in ks], [frames[k][1] for k in ks],
                                SCALING, MAXCAM)

    a, b = make(), make()
    add(a, range(waiting))
    add(b, range(waiting))
    a.inject_error()
    ks = range(waiting, waiting + n)
    with pytest.raises(FFError) as e:
        sequence(a, ks)
    assert e.value.status == 5
    placed = a.stats()["frames"] - waiting
    assert 1 <= placed <= n
    for k in ks[:placed]:
        b.inject_error()
        with pytest.raises(FFError):
            add(b, [k])
    _same(a, b)
    # the failed frames again, and the ones behind them
    assert list(sequence(a, ks)) == add(b, ks)
    _same(a, b)
    assert add(a, range(waiting + n, waiting + n + 4)) == add(b, range(waiting + n, waiting + n + 4))
    _same(a, b)
    assert a.updateMeshes() and b.updateMeshes()
    ma, mb = a.getMeshInterleavedMarchingCubes(), b.getMeshInterleavedMarchingCubes()
    assert len(ma.faces) > 0
    assert np.array_equal(ma.vertices.view(np.uint32), mb.vertices.view(np.uint32))
    assert np.array_equal(ma.colors, mb.colors) and np.array_equal(ma.faces, mb.faces)
    a.close()
    b.close()
