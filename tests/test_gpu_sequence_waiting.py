"""A sequence that begins while single frames of the same map wait for their
update pass: where it does not fit beside them, the call runs their pass first,
and the sequence's marks must not be made while that pass still takes marks
away (small images: the allocation is shorter than the pass)."""
import numpy as np
import pytest

from tests.helpers import MAXCAM, SCALING, circle_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 10, 16, 20])
@pytest.mark.parametrize("waiting", [7, 15])
def test_sequence_after_waiting_frames_equals_frame_by_frame(lib_built, waiting, n):
    from fastfusion_b200.fusion import CameraInfo, FusionMipMapCPU
    K, frames = circle_frames(0, waiting + n, 160, 120)
    cams = [CameraInfo(K, R, t) for _, _, R, t in frames]

    def make():
        return FusionMipMapCPU(0, 0, 0, 0.005, 0.01, 0, True, leaves_max=100000, branches_max=1 << 21, rcp="exact")

    one = make()
    for (depth, bgr, _, _), cam in zip(frames, cams):
        one.addMap(depth, cam, bgr, SCALING, MAXCAM)
    want = one.bricks()
    for _ in range(8):
        s = make()
        for (depth, bgr, _, _), cam in zip(frames[:waiting], cams):
            s.addMap(depth, cam, bgr, SCALING, MAXCAM)
        s.addMapSequence([f[0] for f in frames[waiting:]], cams[waiting:], [f[1] for f in frames[waiting:]], SCALING,
                         MAXCAM)
        for a, b in zip(s.bricks(), want):
            assert np.array_equal(a.view(np.uint16), b.view(np.uint16))
        s.close()
    one.close()
