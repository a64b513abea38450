"""Forward renders of scenes whose rays carry no derivatives (fixed geometry and camera; only
materials and media vary) run kernels with ray and hit derivatives of width 0. A velocity of
1e-30 on one vertex of the light selects the general kernels on the same scene: same random
decisions, so the images must be equal, and the derivative images equal up to FP32 rounding.
Velocities that are all zero move nothing and keep the width-0 kernels.
"""
import numpy as np
import pytest

from dtrt_gb300 import _abi, native, scenes

pytestmark = pytest.mark.gpu


def _sphere(w, h, nder):
    s = scenes.config0(w, h, subdiv=1, nder=nder)
    s.shapes[0].velocities = None
    s.media[0].d_sigma_t = np.ones(nder, np.float32)
    s.media[0].d_albedo = np.full((nder, 3), 0.5, np.float32)
    s.phases[0] = scenes.PhaseSpec(_abi.PHASE_HG, g=0.4, d_g=np.ones(nder, np.float32))
    return s


def _phong(w, h, nder):
    s = scenes.config2(w, h, subdiv=1, nder=nder)
    s.shapes[0].velocities = None
    s.bsdfs[0] = scenes.BsdfSpec(_abi.BSDF_PHONG, d_diffuse=np.ones((nder, 3), np.float32),
                                 d_exponent=np.ones(nder, np.float32))
    return s


SCENES = {
    "glass": lambda w, h, n: scenes.config1(w, h, res=16, nder=n),
    "rough": lambda w, h, n: _rough(w, h, n),
    "cloud": lambda w, h, n: scenes.config3(w, h, res=17, nder=n, nblobs=6),
    "sphere": _sphere,
    "phong": _phong,
}


def _rough(w, h, nder):
    s = scenes.config1(w, h, res=16, nder=nder)
    s.bsdfs[0].alpha = 0.2
    s.bsdfs[0].d_alpha = np.ones(nder, np.float32)
    return s


@pytest.mark.parametrize("nder", [1, 3, 4, 8])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_width_zero_rays_equal_the_general_kernels(name, nder):
    # one path; a ragged warp; several blocks: on both schedules
    for w, h, spp in ((1, 1, 1), (13, 7, 5), (33, 20, 16)):
        kw = dict(seed=9, spp=spp, max_bounces=7, sppe=16, sppse=2)
        spec = SCENES[name](w, h, nder)
        with native.NativeScene(spec) as s:
            s.set_camera_schedule("wavefront")
            fixed = s.render(**kw).copy()
            s.set_camera_schedule("megakernel")
            mega = s.render(**kw)
            assert np.array_equal(fixed[0], mega[0])
        light = spec.shapes[-1]
        light.velocities = np.zeros((nder * light.vertices.shape[0], 3), np.float32)
        with native.NativeScene(spec) as s:
            s.set_camera_schedule("wavefront")
            assert np.array_equal(fixed, s.render(**kw))
            assert s.last_stats()["edge_records"] == 0
        light.velocities[0, 0] = 1e-30
        with native.NativeScene(spec) as s:
            s.set_camera_schedule("wavefront")
            general = s.render(**kw)
        # a moving grid's accepted density enters the throughput as density / density: one rounding
        np.testing.assert_allclose(fixed[0], general[0], rtol=4e-6, atol=1e-7 * max(1.0, np.abs(general[0]).max()))
        for j in range(1, nder + 1):
            # ten-sample FP32 sums: 2^-24 per operation, some tens of operations, cancellation of up to 10
            for d in (fixed, mega):
                assert np.linalg.norm(d[j] - general[j]) <= 1e-4 * np.linalg.norm(general[j]) + 1e-6, (name, j)
