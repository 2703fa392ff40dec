"""The confidence map that a program reads back is the last frame's, however the
frame was added: one by one, in a sequence (of one pass, of several, after single
frames that wait), with the update deferred or not."""
import numpy as np
import pytest

from tests.helpers import MAXCAM, SCALING, circle_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,n,batch", [(0, 3, 16), (0, 18, 16), (3, 5, 16), (9, 10, 16), (2, 4, 1)])
def test_map_after_a_sequence_is_the_last_frames(lib_built, first, n, batch):
    from fastfusion_b200 import confidence
    from fastfusion_b200.fusion import CameraInfo, FusionMipMapCPU
    K, frames = circle_frames(0, first + n, 160, 120)
    cams = [CameraInfo(K, R, t) for _, _, R, t in frames]
    params, tau = confidence.load_weights()

    def make():
        f = FusionMipMapCPU(0, 0, 0, 0.005, 0.01, 0, True, leaves_max=50000, branches_max=1 << 21, rcp="exact")
        f.set_confidence(params, tau)
        return f

    one, seq = make(), make()
    seq.set_update_batch(batch)
    want = []
    for (depth, bgr, _, _), cam in zip(frames, cams):
        one.addMap(depth, cam, bgr, SCALING, MAXCAM)
        want.append(one.confidence_map())
    assert want[-1].shape == (120, 160) and not np.array_equal(want[-1], want[-2])
    for k in range(first):
        seq.addMap(frames[k][0], cams[k], frames[k][1], SCALING, MAXCAM)
        assert np.array_equal(seq.confidence_map(), want[k])
    seq.addMapSequence([f[0] for f in frames[first:]], cams[first:], [f[1] for f in frames[first:]], SCALING, MAXCAM)
    assert np.array_equal(seq.confidence_map(), want[-1])
    seq.updateMeshes()
    assert np.array_equal(seq.confidence_map(), want[-1])
    one.close()
    seq.close()
