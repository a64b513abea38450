"""Large wavefront renders run several batches at once, each on a stream and a workspace of its
own. Against the megakernel (one thread per path, no batches in flight): same paths, so images
agree up to the order of FP64 sums, gradients up to the order of FP32 atomics. Sizes: one path
more than a batch, a ragged last batch, more batches than lanes.
"""
import threading

import numpy as np
import pytest

from dtrt_gb300 import native, scenes

pytestmark = pytest.mark.gpu


def _spec(w, h):
    return scenes.config3(w, h, res=16, nder=1, param_slots=True, nblobs=4)


def _near(a, b, tol):
    assert np.isfinite(a).all() and np.linalg.norm(b) > 0
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("w,h,spp", [(1, 1, (1 << 20) + 1), (61, 33, 1000), (127, 33, 2300)])
def test_lanes_equal_the_megakernel(w, h, spp):
    kw = dict(seed=5, spp=spp, max_bounces=3, sppe=0, sppse=0)
    dimg = np.random.default_rng(2).normal(size=(h, w, 3)).astype(np.float32)
    out = []
    for schedule in ("wavefront", "megakernel"):
        with native.NativeScene(_spec(w, h)) as s:
            s.set_camera_schedule(schedule)
            for _ in range(2):  # the second render reuses streams and workspaces
                r = [s.render(**kw).copy(), s.render_primal(seed=5, spp=spp, max_bounces=3).copy()]
                r += [x.copy() for x in s.render_adjoint(dimg, **kw)]
            out.append(r)
    a, b = out
    for i in range(3):
        _near(a[i], b[i], 1e-6)
    _near(a[3], b[3], 1e-4)


def test_lanes_of_two_threads():
    kw = dict(spp=700, max_bounces=3, sppe=0, sppse=0)
    alone, both = [], [None, None]
    for k in range(2):
        with native.NativeScene(_spec(50 + k, 41)) as s:
            alone.append(s.render(seed=k, **kw).copy())

    def work(k):
        with native.NativeScene(_spec(50 + k, 41)) as s:
            for _ in range(3):
                both[k] = s.render(seed=k, **kw).copy()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        _near(both[k], alone[k], 1e-6)
