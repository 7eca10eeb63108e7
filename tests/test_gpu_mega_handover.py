"""The persistent kernel when a lane owns pixel after pixel (more than 512 of
them per SM): it claims the next pixel while the last vertex of the one before
still waits for its shadow rays and its film update. Films are the
wavefront's, bit for bit: of one scene, of samples that Russian roulette ends
before their first vertex (min_depth below 0), and of a batch whose
neighbouring pixels belong to scenes that occupy the same space, where an
occluder remembered from one scene must not block a ray of another."""
import numpy as np
import pytest

from tracer_gb300 import scenes
from tracer_gb300.abi import TR_RENDER_MODE_PERSISTENT, TR_RENDER_MODE_WAVEFRONT

pytestmark = pytest.mark.gpu

PER_SM = 1100  # pixels: each lane owns two or three


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("name", ["cornell", "glass_metal", "mapped"])
@pytest.mark.parametrize("min_depth", [-1, 3])
def test_one_scene(gpu, name, min_depth):
    from conftest import tuned
    w, h = _sms(), PER_SM
    sc, cam, filt, par = {"cornell": lambda: scenes.cornell(w, h, 3),
                          "glass_metal": lambda: scenes.cornell(w, h, 3, glass=True, metal=True),
                          "mapped": lambda: scenes.mapped_materials(w, h, 2)}[name]()
    par = scenes.make_params(w, h, par.spp, min_depth, 6, seed_base=11)
    gpu.upload(sc)
    film = []
    for mode in (TR_RENDER_MODE_WAVEFRONT, TR_RENDER_MODE_PERSISTENT):
        with tuned(gpu, render_mode=mode):
            film.append(gpu.render(cam, filt, par))
    assert film[1][1].iterations == 1
    assert _same(film[0][0], film[1][0])
    for k in ("samples", "extend_rays", "shadow_rays"):
        assert getattr(film[0][1], k) == getattr(film[1][1], k), k


def _lit_floor(plates):
    """A floor under a small light; plates hang close below the light (all of
    its light is blocked), over half the floor, or nowhere."""
    b = scenes._Builder()
    white = b.material(scenes.lambert((0.7, 0.7, 0.7)))

    def level(y, x0, x1, z, up, **kw):
        b.quad((x0, y, -z), (x1, y, -z), (x1, y, z), (x0, y, z), (0, 1 if up else -1, 0), white, **kw)

    level(0.0, -2.0, 2.0, 2.0, True)
    if plates == 1:
        level(2.9, -0.7, 0.7, 0.7, False)
    if plates == 2:
        level(1.0, -2.0, 0.0, 2.0, False)
    level(3.0, -0.25, 0.25, 0.25, False, emission=(20.0, 18.0, 15.0))
    return b.finish(max_leaf_prims=2)


@pytest.mark.parametrize("cache", [0, 1])
@pytest.mark.parametrize("kind", ["floors", "rooms"])
def test_batch_of_scenes_in_one_space(gpu, kind, cache):
    """Hundreds of small films of three floors under one light, which a plate
    hides in one of them, and of three rooms with other furniture each."""
    import torch
    from conftest import tuned
    w, h = 29, 31
    n = PER_SM * _sms() // (w * h)
    if kind == "floors":
        sets = [_lit_floor(k) for k in range(3)]
        cam = scenes.make_camera(w / h, (0, 2.0, 4.0), (0, 0, 0), (0, 1, 0), 0.9, 0.0, 1.0)
        max_depth = 1  # a path ends at its first vertex, with that vertex's light samples to come
    else:
        sets = [scenes.occluded_room(8, 8, 1, n_tris=3000, seed=s)[0] for s in range(3)]
        cam = scenes.occluded_room(w, h, 1, n_tris=3000)[1]
        max_depth = 6
    gpu.upload_set(sets)
    filt = scenes.make_filter(0.5, 0.6)
    films = {}
    for mode in (TR_RENDER_MODE_WAVEFRONT, TR_RENDER_MODE_PERSISTENT):
        f = torch.zeros((n, h, w, 4), dtype=torch.float32, device="cuda:0")
        jobs = [(k % 3, cam, filt, scenes.make_params(w, h, 2, -1 if k % 5 == 0 else 2, max_depth, seed_base=1000 * k),
                 f[k].data_ptr()) for k in range(n)]
        torch.cuda.synchronize()
        with tuned(gpu, render_mode=mode, occluder_cache=cache):
            st = gpu.render_batch_dev(jobs)
        films[mode] = (f.cpu().numpy(), st)
    (a, sa), (b, sb) = films[TR_RENDER_MODE_WAVEFRONT], films[TR_RENDER_MODE_PERSISTENT]
    assert sb.iterations == 1 and sa.samples == sb.samples
    if cache:
        assert sb.occluder_hits > 0
    differ = (a.view(np.uint32) != b.view(np.uint32)).any(-1)
    assert not differ.any(), f"{int(differ.sum())} of {differ.size} pixels differ"
    assert sa.extend_rays == sb.extend_rays and sa.shadow_rays == sb.shadow_rays
