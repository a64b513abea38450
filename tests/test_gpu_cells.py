"""Density cells (a grid copied so that the 8 corners of a lookup lie together) against voxels: two
media whose grids have different sizes on every axis, so that a swapped axis or a wrong offset shows.
The replay wavefront of a batch and the primal megakernel of a small render read voxels; single
replays and the primal wavefront read cells from 2^16 paths, a replay with a gradient from one
path for 16 voxels. Same paths on both sides: images agree up to the order of FP64 sums,
gradients up to the order of FP32 atomic sums.
"""
import numpy as np
import pytest

from dtrt_gb300 import _abi, scenes

pytestmark = pytest.mark.gpu

VOXELS = 33 * 20 * 51 + 18 * 40 * 47  # 67,500


def _spec(w, h):
    s = scenes.config3(w, h, res=2, nder=1, param_slots=True, nblobs=1)
    rng = np.random.default_rng(5)
    s.shapes.pop(0)
    m = s.media.pop(0)
    for lo, hi, (rx, ry, rz) in (((-0.6, -0.5, -0.5), (0.0, 0.5, 0.5), (33, 20, 51)),
                                 ((0.1, -0.5, -0.4), (0.6, 0.4, 0.5), (18, 40, 47))):
        v, f = scenes.box(lo, hi)
        s.shapes.insert(0, scenes.ShapeSpec(v, f, bsdf_id=0, med_int_id=len(s.media)))
        z, y, x = np.meshgrid(*(np.linspace(0.0, 1.0, r) for r in (rz, ry, rx)), indexing="ij")
        d = 0.2 + x + 0.5 * y * y + 0.3 * z + 0.4 * rng.random((rz, ry, rx))
        s.media.append(scenes.MediumSpec(_abi.MEDIUM_HETEROGENEOUS, phase_id=0, albedo=(0.9, 0.8, 0.7),
                                         density=d.astype(np.float32), vol_min=lo, vol_max=hi, density_scale=4.0,
                                         d_density_scale=m.d_density_scale))
    for e in s.emitters:  # shape ids moved by one
        if hasattr(e, "shape_id"):
            e.shape_id += 1
    return s


def _near(a, b, tol):
    assert np.isfinite(a).all() and np.linalg.norm(b) > 0
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


# the last render on voxels and the first on cells (2^16 paths), a ragged one, and more than 2^19
@pytest.mark.parametrize("w,h,spp", [(64, 33, 31), (64, 32, 32), (61, 43, 29), (64, 64, 129)])
def test_primal_cells_equal_voxels(native, w, h, spp):
    out = []
    for schedule in ("wavefront", "megakernel"):
        with native.NativeScene(_spec(w, h)) as s:
            s.set_camera_schedule(schedule)
            out.append(s.render_primal(seed=3, spp=spp, max_bounces=6).copy())
    _near(*out, 1e-6)


# below and above one path for 16 voxels (4,219 paths); one and several wavefront batches
@pytest.mark.parametrize("w,h,spp", [(32, 16, 8), (33, 16, 8), (61, 33, 33), (64, 64, 300)])
def test_replay_cells_equal_voxels(native, w, h, spp):
    torch = pytest.importorskip("torch")
    dimg = torch.randn((h, w, 3), device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    st = torch.cuda.current_stream().cuda_stream
    with native.NativeScene(_spec(w, h)) as s:
        assert s.gradient_sizes()[0] == VOXELS
        o = s.options(seed=3, spp=spp, max_bounces=6, sppe=0, sppse=0)
        img, grad = torch.zeros((2, h, w, 3), device="cuda"), torch.zeros((2, VOXELS), device="cuda")
        fwd = torch.zeros((2, h, w, 3), device="cuda")
        s.render_adjoint(dimg.data_ptr(), image=img[0].data_ptr(), density_grad=grad[0].data_ptr(), stream=st,
                         device=True, options=o)
        s.render(out=fwd.data_ptr(), stream=st, options=o)
        b = native.Batch([(s, o, dimg.data_ptr(), img[1].data_ptr(), grad[1].data_ptr())], autotune=False,
                         graph=False, stream=st, wavefront=True)
        b.launch(st)
        torch.cuda.synchronize()
        b.close()
    img, grad = img.cpu().numpy(), grad.cpu().numpy()
    first = 33 * 20 * 51
    _near(img[0], img[1], 1e-6)
    for part in (slice(0, first), slice(first, None)):
        _near(grad[0, part], grad[1, part], 1e-4)
    _near(fwd[0].cpu().numpy(), img[1], 1e-6)
