"""A bound of very many bounces: AUTO leaves the wavefront, which launches every level that the bound
allows, for the megakernel. No path comes near the bound, so both sides of the line render the
same image, exactly."""
import numpy as np
import pytest

from dtrt_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_auto_leaves_the_wavefront_at_many_levels(native):
    out = []
    with native.NativeScene(scenes.config3(257, 257, res=16, nder=1, param_slots=True, nblobs=4)) as s:
        for bounces, schedule in ((1023, 2), (1024, 1), (100000, 1)):  # levels = bounces + 1
            out.append(s.render(seed=4, spp=1, max_bounces=bounces, sppe=0, sppse=0).copy())
            assert s.last_stats()["camera_schedule"] == schedule
        s.set_camera_schedule("wavefront")  # a forced wavefront stays one
        out.append(s.render(seed=4, spp=1, max_bounces=1024, sppe=0, sppse=0).copy())
        assert s.last_stats()["camera_schedule"] == 2
    assert np.abs(out[0]).sum() > 0
    for x in out[1:]:
        assert np.array_equal(x, out[0])
