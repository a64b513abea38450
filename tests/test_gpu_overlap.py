"""Small and middling renders: the primary-edge samples share the last Li launch, Lins records run
beside the edge samples, and short queues are not sorted. A small queue capacity takes the same
samples in many short chunks without sharing, so the images agree up to the order of FP64 sums.
"""
import numpy as np
import pytest

from dtrt_gb300 import native, scenes

pytestmark = pytest.mark.gpu

SCENES = {
    "sphere": lambda w, h, n: scenes.config0(w, h, subdiv=2, nder=n),
    "mesh": lambda w, h, n: scenes.config2(w, h, subdiv=3, nder=n),
}


# one path; a ragged preview; queues on both sides of the sort's threshold
@pytest.mark.parametrize("w,h,spp,sppse,sppe", [(1, 1, 1, 1, 1), (29, 17, 3, 4, 16), (64, 48, 24, 10, 512)])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_shared_launches_equal_short_chunks(name, w, h, spp, sppse, sppe):
    kw = dict(seed=6, spp=spp, max_bounces=4, sppe=sppe, sppse=sppse)
    for nder in (1, 3):
        with native.NativeScene(SCENES[name](w, h, nder)) as s:
            a = s.render(**kw).copy()
            tasks = s.last_stats()["li_tasks"]
            again = s.render(**kw).copy()
            s.set_queue_capacity(1 << 13)
            b = s.render(**kw).copy()
            assert s.last_stats()["li_tasks"] == tasks
        assert np.isfinite(a).all()
        for x in (again, b):
            assert np.linalg.norm(x - a) <= 1e-6 * np.linalg.norm(a)
