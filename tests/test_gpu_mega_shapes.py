"""The persistent kernel's block sizes: few pixels (at most 96 per SM) run in
blocks of 256 threads, more in blocks of 512. Films are those of the
wavefront, bit for bit, on either side of the line and at the smallest
frames."""
import numpy as np
import pytest

from tracer_gb300 import scenes
from tracer_gb300.abi import TR_RENDER_MODE_PERSISTENT, TR_RENDER_MODE_WAVEFRONT

pytestmark = pytest.mark.gpu

SCENES = {
    "cornell": lambda w, h: scenes.cornell(w, h, 2),
    "glass_metal": lambda w, h: scenes.cornell(w, h, 2, max_depth=8, min_depth=2, glass=True, metal=True),
    "grid": lambda w, h: scenes.disney_grid(w, h, 2),
    "mapped": lambda w, h: scenes.mapped_materials(w, h, 2),
}


@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("rows", [0, 95, 96, 97, 300])
def test_block_sizes_keep_the_film(gpu, name, rows):
    import torch
    from conftest import tuned
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    w, h = (1, 1) if rows == 0 else (sms, rows)  # rows pixels per SM
    sc, cam, filt, par = SCENES[name](w, h)
    gpu.upload(sc)
    film = []
    for mode in (TR_RENDER_MODE_WAVEFRONT, TR_RENDER_MODE_PERSISTENT):
        with tuned(gpu, render_mode=mode):
            film.append(gpu.render(cam, filt, par))
    assert film[1][1].iterations == 1
    assert np.array_equal(film[0][0].view(np.uint32), film[1][0].view(np.uint32))
    for k in ("samples", "extend_rays", "shadow_rays"):
        assert getattr(film[0][1], k) == getattr(film[1][1], k), k
