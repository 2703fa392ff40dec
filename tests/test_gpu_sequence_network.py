"""The learned weight in sequences: the frames' networks run in groups (as many
images as the activations' share of the L2 holds); every brick must be the one
of the frames added one by one.  Groups of one,
several groups with a remainder, all frames in one group, intrinsics that differ
from frame to frame, and a sequence longer than one update pass."""
import numpy as np
import pytest

from tests.helpers import MAXCAM, SCALING, circle_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,n", [(160, 120, 5), (640, 480, 7), (1280, 960, 3), (97, 61, 19)])
def test_grouped_networks_equal_single_frames(lib_built, w, h, n):
    from fastfusion_b200 import confidence
    from fastfusion_b200.fusion import CameraInfo, FusionMipMapCPU
    K, frames = circle_frames(0, n, w, h)
    K = np.asarray(K, np.float64).reshape(-1)
    params, tau = confidence.load_weights()

    def make():
        f = FusionMipMapCPU(0, 0, 0, 0.005, 0.01, 0, True, leaves_max=100000, branches_max=1 << 21, rcp="exact")
        f.set_confidence(params, tau)
        return f

    cams = [CameraInfo(K * (1 + 0.002 * k), R, t) for k, (_, _, R, t) in enumerate(frames)]
    one, seq = make(), make()
    for cam, (depth, bgr, _, _) in zip(cams, frames):
        one.addMap(depth, cam, bgr, SCALING, MAXCAM)
    seq.addMapSequence([f[0] for f in frames], cams, [f[1] for f in frames], SCALING, MAXCAM)
    for a, b in zip(seq.bricks(), one.bricks()):
        assert np.array_equal(a.view(np.uint16), b.view(np.uint16))
    one.close()
    seq.close()


def test_injected_timeout_in_a_sequence(lib_built):
    """The first frame of a sequence reports a network wait that gave up: the call
    fails, and the map fuses the following frames again."""
    from fastfusion_b200 import confidence
    from fastfusion_b200.fusion import CameraInfo, FFError, FusionMipMapCPU
    K, frames = circle_frames(0, 6, 160, 120)
    params, tau = confidence.load_weights()
    f = FusionMipMapCPU(0, 0, 0, 0.005, 0.01, 0, True, leaves_max=100000, branches_max=1 << 21, rcp="exact")
    f.set_confidence(params, tau)
    args = [f_[0] for f_ in frames], [CameraInfo(K, f_[2], f_[3]) for f_ in frames], [f_[1] for f_ in frames]
    f.addMapSequence(*(a[:3] for a in args), SCALING, MAXCAM)
    f.inject_error()
    with pytest.raises(FFError) as e:
        f.addMapSequence(*(a[3:5] for a in args), SCALING, MAXCAM)
    assert e.value.status == 5
    f.addMapSequence(*(a[5:] for a in args), SCALING, MAXCAM)
    f.addMapSequence(*(a[:3] for a in args), SCALING, MAXCAM)
    assert f.updateMeshes()
    f.close()
