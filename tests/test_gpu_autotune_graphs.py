"""tr_autotune and graph_iterations: every value above zero is the same program
(two iterations a graph), so the tuner has two to choose from, the caller's
own and none (or two, when the caller's is none). And the small wavefront
renders those graphs run for, against launches one after another."""
import numpy as np
import pytest

from tracer_gb300 import scenes
from tracer_gb300.abi import TR_RENDER_MODE_WAVEFRONT, make_guide

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mine", [0, 6])
def test_tuner_keeps_or_drops_graphs(gpu, mine):
    import torch
    from conftest import tuned
    sc, cam, filt, par = scenes.cornell(24, 24, 1)
    gpu.upload_set([sc])
    film = torch.zeros((24, 24, 4), device="cuda:0")
    torch.cuda.synchronize()
    got = []
    for _ in range(3):
        with tuned(gpu, graph_iterations=mine):
            best, _ = gpu.autotune([(0, cam, filt, par, film.data_ptr())], probe_spp=1)
            got.append(best.graph_iterations)
    assert set(got) <= {0, mine or 2}, got


SMALL = {
    "room": lambda: scenes.occluded_room(64, 48, 4, n_tris=5000),
    "mapped": lambda: scenes.mapped_materials(61, 43, 3),
    "outdoor": lambda: scenes.outdoor(61, 43, 3),
    "disney15": lambda: scenes.disney15_row(61, 43, 3),
}


@pytest.mark.parametrize("guided", [False, True])
@pytest.mark.parametrize("name", sorted(SMALL))
def test_small_wavefront_renders(gpu, name, guided):
    import torch
    from conftest import tuned
    sc, cam, filt, par = SMALL[name]()
    gpu.upload(sc)
    film = []
    if guided:
        gpu.guide_init(3)
    for g in (0, 2):
        with tuned(gpu, graph_iterations=g, render_mode=TR_RENDER_MODE_WAVEFRONT):
            if guided:
                f = torch.zeros((par.height, par.width, 4), device="cuda:0")
                torch.cuda.synchronize()
                st = gpu.render_guided_dev(cam, filt, par, make_guide(0.5, (-8, -8, -8), (8, 8, 8)), f.data_ptr())
                film.append((f.cpu().numpy(), st))
            else:
                film.append(gpu.render(cam, filt, par))
    (a, sa), (b, sb) = film
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for k in ("samples", "extend_rays", "shadow_rays", "shade_items", "occluder_hits"):
        assert getattr(sa, k) == getattr(sb, k), k
