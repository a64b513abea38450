"""Statistics of a render count what ran: kernels of a render small enough to be counted by hand
(one batch on the megakernel, no sorts, no density cells), and primary-edge samples."""
import pytest

from dtrt_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_kernels_of_a_small_moving_render(native):
    with native.NativeScene(scenes.config0(16, 16, subdiv=2)) as s:
        s.render(seed=1, spp=8, max_bounces=5, sppe=16, sppse=4)
        st = s.last_stats()
    assert st["lins_records"] > 0 and st["edge_records"] > 0 and st["primary_edge_samples"] > 0 and st["li_tasks"] > 0
    assert st["batches"] == 1
    assert st["kernel_launches"] == 6  # camera, Lins, edges, primary edges, Li, images


def test_a_render_of_fixed_rays_runs_no_primary_edges(native):
    with native.NativeScene(scenes.config1(16, 16, res=16, nder=3)) as s:
        s.render(seed=1, spp=8, max_bounces=5, sppe=64, sppse=4)
        st = s.last_stats()
    assert st["primary_edge_samples"] == 0 and st["li_tasks"] == 0 and st["ms_primary"] == 0
    assert st["kernel_launches"] == 2  # camera, images
