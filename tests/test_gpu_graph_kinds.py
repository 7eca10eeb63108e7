"""The graphs a wavefront render switches between: full iterations, the same
with the occluder cache tested ahead of the shadow rays (once an eighth of
them meet the occluder remembered), and the tail (at most 2^16 live slots).
The same kernels on the same work as one launch after another
(graph_iterations = 0): films bit-identical, work counts equal."""
import numpy as np
import pytest

from tracer_gb300 import scenes
from tracer_gb300.abi import TR_RENDER_MODE_WAVEFRONT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2, 4])
@pytest.mark.parametrize("name,size", [("room", (256, 256)), ("room", (257, 256)), ("room", (500, 301)),
                                       ("outdoor", (311, 257))])
def test_graph_kinds_keep_the_film(gpu, name, size, width):
    from conftest import tuned
    if name == "room":
        sc, cam, filt, par = scenes.occluded_room(*size, 5, n_tris=5000)
    else:
        sc, cam, filt, par = scenes.outdoor(*size, 5)
    gpu.upload(sc)
    with tuned(gpu, graph_iterations=0, render_mode=TR_RENDER_MODE_WAVEFRONT, any_node_width=width):
        ref, st0 = gpu.render(cam, filt, par)
    for g in (1, 8):
        with tuned(gpu, graph_iterations=g, render_mode=TR_RENDER_MODE_WAVEFRONT, any_node_width=width):
            got, st1 = gpu.render(cam, filt, par)
        assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
        for k in ("samples", "extend_rays", "shadow_rays", "shade_items", "occluder_hits"):
            assert getattr(st1, k) == getattr(st0, k), k
    if name == "room":  # enough remembered occluders that the second graph is reached
        assert st0.occluder_hits * 8 >= st0.shadow_rays
