"""A host that resets the device between two frames: the standalone diffusion call after
cudaDeviceReset does not use the device memory pool of the context that is gone. In a process of
its own, whose context nothing else shares."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, os, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import __graft_entry__
__graft_entry__.package()
from cuda.bindings import runtime as cudart
from film_juicer_b200 import abi, load_library

lib = load_library()
comp = abi.FjDiffusionComponents()
for k in range(9):
    comp.lambda_px[k] = 1.0 + k
    comp.red_weights[k] = comp.green_weights[k] = comp.blue_weights[k] = 1.0 / 9.0
w, h = 96, 64
src = np.random.default_rng(3).uniform(0.0, 2.0, size=(3, h, w)).astype(np.float32)


def check(code):
    code = code[0] if isinstance(code, tuple) else code
    assert int(code) == 0, code


def diffuse(radius):
    err, buf = cudart.cudaMalloc(2 * src.nbytes)
    check(err)
    check(cudart.cudaMemcpy(buf, src.ctypes.data, src.nbytes, cudart.cudaMemcpyKind.cudaMemcpyHostToDevice))
    plane = w * h * 4
    text = abi.ErrorText()
    status = lib.fjb_diffusion(C.byref(comp), radius, 0.3, *[C.c_void_p(int(buf) + c * plane) for c in range(6)], w, w, h,
                               C.c_void_p(0), C.byref(text.buf))
    assert status.category == abi.FJ_STATUS_SUCCESS, status.category
    out = np.empty_like(src)
    check(cudart.cudaMemcpy(out.ctypes.data, int(buf) + src.nbytes, src.nbytes,
                            cudart.cudaMemcpyKind.cudaMemcpyDeviceToHost))
    check(cudart.cudaFree(buf))
    return out


for radius in (3, 12):
    first = diffuse(radius)
    check(cudart.cudaDeviceReset())
    assert np.array_equal(first, diffuse(radius))
    assert not np.array_equal(first, src)
print("done")
"""


def test_diffusion_after_a_device_reset(torch_cuda):
    from conftest import ROOT

    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr
