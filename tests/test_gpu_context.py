"""GPU: fgs_forward_noalloc in a new primary context.  A process that resets its device gets a new context, into
which the library's kernels are loaded again with none of the attributes they had; calls before and after give
the same bits.  In a process of its own, with plain CUDA allocations: no torch tensor outlives a reset."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_CODE = """
import ctypes as C, sys
import numpy as np
sys.path[:0] = {path!r}
import torch                                   # (brings the CUDA runtime the library links to)
from filtergs_b200 import _lib
from filtergs_b200 import synthetic as S

rt = C.CDLL("libcudart.so.12")
def ok(e):
    assert e == 0, e

def dev(a):
    p = C.c_void_p()
    ok(rt.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)))
    ok(rt.cudaMemcpy(p, C.c_void_p(a.ctypes.data), C.c_size_t(a.nbytes), 1))
    return p

def host(p, a):
    ok(rt.cudaMemcpy(C.c_void_p(a.ctypes.data), p, C.c_size_t(a.nbytes), 2))
    return a

P, W, H = 3000, 200, 136
sc, cam = S.small_scene(P=P, seed=1102, W=W, H=H)
f = lambda a: np.ascontiguousarray(a, np.float32)

def render():
    a = _lib.RasterArgs()
    a.P, a.D, a.M, a.width, a.height = P, 3, 16, W, H
    ins = dict(background=np.zeros(3, np.float32), means3D=f(sc["means3D"]), shs=f(sc["shs"]),
               opacities=f(sc["opacities"]), scales=f(sc["scales"]), rotations=f(sc["rotations"]),
               viewmatrix=f(cam.viewmatrix), projmatrix=f(cam.projmatrix), campos=f(cam.campos))
    for k, v in ins.items():
        setattr(a, k, dev(v))
    a.scale_modifier, a.tan_fovx, a.tan_fovy = 1.0, cam.tanfovx, cam.tanfovy
    a.use_filter = 1
    a.ogfs_epsilon_scale, a.ogfs_epsilon_max, a.ogfs_energy_floor, a.ogfs_radius_ratio_min = 0.2, 0.2, 0.05, 0.7
    outs = [np.zeros(P, np.int32), np.zeros((3, H, W), np.float32), np.zeros((H, W), np.int32),
            np.zeros((H, W), np.float32), np.zeros(P, np.float32)]
    ptrs = [dev(o) for o in outs]
    K = C.c_longlong(-1)
    st = _lib.lib().fgs_forward_noalloc(C.byref(a), *ptrs, C.byref(K), None)
    assert st == _lib.FGS_OK, _lib.status_string(st)
    return int(K.value), [host(p, o) for p, o in zip(ptrs, outs)]

K0, first = render()
assert K0 > 0 and float(np.abs(first[1]).max()) > 0
for _ in range(2):
    ok(rt.cudaDeviceReset())
    K, again = render()
    assert K == K0
    for x, y in zip(again, first):
        assert np.array_equal(x, y)
print("context ok")
"""


def test_noalloc_in_a_new_context(cuda):
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", _CODE.format(path=[here, os.path.dirname(here)])], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "context ok" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
