"""Scenes of opaque surfaces alone take Li kernels without media and null-interface code. A null
BSDF that no shape uses selects the general kernels on the same scene: same random decisions,
so renders agree up to FP32 rounding (a last-bit change of a radiance, summed over a pixel).
"""
import numpy as np
import pytest

from dtrt_gb300 import _abi, native, scenes

pytestmark = pytest.mark.gpu


def _scene(bsdf, w, h, nder):
    s = scenes.config2(w, h, subdiv=2, nder=nder)
    if bsdf == "phong":
        s.bsdfs[0] = scenes.BsdfSpec(_abi.BSDF_PHONG, exponent=12.0)
    elif bsdf == "rough":
        s.bsdfs[0] = scenes.BsdfSpec(_abi.BSDF_ROUGHDIELECTRIC, alpha=0.3)
    return s


def _near(a, b):
    assert np.isfinite(a).all() and np.linalg.norm(a - b) <= 2e-6 * np.linalg.norm(b)


# one path, a ragged warp, several blocks; Li tasks come in pairs, so their number is even
@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 1, 1), (13, 7, 5, 3), (40, 33, 8, 6)])
@pytest.mark.parametrize("bsdf", ["diffuse", "phong", "rough"])
def test_surface_kernels_equal_the_general_ones(bsdf, w, h, spp, depth):
    kw = dict(seed=4, spp=spp, max_bounces=depth, sppe=32, sppse=3)
    dimg = np.random.default_rng(1).normal(size=(h, w, 3)).astype(np.float32)
    for nder in (1, 3, 4, 8):
        out = []
        for general in (False, True):
            spec = _scene(bsdf, w, h, nder)
            if general:
                spec.bsdfs.append(scenes.BsdfSpec(_abi.BSDF_NULL))
            with native.NativeScene(spec) as s:
                r = [s.render(**kw).copy(), s.render_primal(seed=4, spp=spp, max_bounces=depth).copy()]
                if nder == 1:
                    r += [x.copy() for x in s.render_vertex_adjoint(dimg, **kw)]
                out.append(r)
        for a, b in zip(*out):
            _near(a, b)


# Homogeneous media alone: kernels without grid tracking. A 2^3 grid medium that no shape uses
# selects the general ones.
@pytest.mark.parametrize("w,h,spp,depth", [(1, 1, 1, 1), (13, 7, 5, 3), (40, 33, 8, 6)])
def test_homogeneous_kernels_equal_the_general_ones(w, h, spp, depth):
    kw = dict(seed=4, spp=spp, max_bounces=depth, sppe=32, sppse=3)
    for nder in (1, 3, 4, 8):
        out = []
        for general in (False, True):
            spec = scenes.config0(w, h, subdiv=2, nder=nder)
            if general:
                spec.media.append(scenes.MediumSpec(
                    _abi.MEDIUM_HETEROGENEOUS, phase_id=0, density=np.ones((2, 2, 2), np.float32),
                    vol_min=(-1.0,) * 3, vol_max=(1.0,) * 3))
            with native.NativeScene(spec) as s:
                out.append(s.render(**kw).copy())
        _near(*out)
