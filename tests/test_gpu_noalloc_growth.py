"""tr_render_dev_noalloc takes device memory at a context's first call after an
upload only (its kernels' code and local memory, which the driver allocates):
none at later calls of other films and path lengths, which run the persistent
kernel in blocks of another size or the wavefront. In a process of its own,
where nothing has been rendered before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r"""
import ctypes as C, sys
import torch
from tracer_gb300 import scenes
from tracer_gb300.abi import TrCamera, TrFilter, TrRenderParams, TrStats
from tracer_gb300.native import GpuContext
ctx = GpuContext(0)
f = ctx.L.tr_render_dev_noalloc
f.restype = C.c_int
f.argtypes = [C.c_void_p, C.POINTER(TrCamera), C.POINTER(TrFilter), C.POINTER(TrRenderParams), C.c_void_p, C.POINTER(TrStats)]
out = torch.zeros((160, 160, 4), dtype=torch.float32, device="cuda:0")
make = getattr(scenes, sys.argv[1])
ctx.upload(make(8, 8, 1)[0])
# a small film, one of more than 96 pixels per SM, paths of more than 256 vertices
for w, h, spp in ((32, 24, 1), (160, 120, 1), (32, 24, 60), (160, 120, 1)):
    _, cam, filt, par = make(w, h, spp)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info(0)[0]
    st = TrStats()
    assert f(ctx.h, C.byref(cam), C.byref(filt), C.byref(par), out.data_ptr(), C.byref(st)) == 0
    print(w, h, spp, st.iterations, free - torch.cuda.mem_get_info(0)[0])
"""


@pytest.mark.parametrize("scene", ["cornell", "outdoor"])
def test_memory_is_taken_by_the_first_call_only(scene):
    r = subprocess.run([sys.executable, "-c", CODE, scene], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    print(r.stdout)
    taken = [int(line.split()[-1]) for line in r.stdout.splitlines()]
    assert len(taken) == 4 and taken[1:] == [0, 0, 0], taken
