"""Column passes of the line recursions that take more than one round (columns too long for all
recursions of a channel in shared memory at once) at frame widths where the scratch has no
room beyond its planes, and passes with as many recursions as the scratch has planes.
Oracle and bounds are those of test_line_pairs_gpu.py; the launch count shows that the line
kernels ran."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def planes(w, h, seed):
    rng = np.random.default_rng(seed)
    return [np.ascontiguousarray(p) for p in rng.uniform(0.0, 2.0, size=(3, h, w)).astype(np.float32)]


def launches(torch, call):
    from film_juicer_b200 import load_library

    lib = load_library()
    torch.cuda.synchronize()
    before = lib.fjb_kernel_launches()
    call()
    torch.cuda.synchronize()
    return lib.fjb_kernel_launches() - before


def dir_oracle(sd, plane):
    from oracle import dir as odir
    from oracle import oracle as orc

    h, w = plane.shape
    comps, n, keep = odir.components(sd, w, h)
    out = np.zeros_like(plane)
    blur = orc.load().oracle_dir_blur
    blur.restype = C.c_int
    blur.argtypes = [C.POINTER(odir.OracleDirComp), C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_void_p]
    assert blur(comps, n, C.c_void_p(plane.ctypes.data), w, h, C.c_void_p(out.ctypes.data)) == 0
    del keep
    return out


def check_dir(torch, sd, src, expected_launches):
    from film_juicer_b200 import runtime

    h, w = src[0].shape
    dev = [torch.from_numpy(p).cuda() for p in src]
    out = [torch.empty((h, w), device="cuda") for _ in range(3)]
    f = runtime.DirFilter(sd, w, h)
    assert launches(torch, lambda: f.apply(dev, out)) == expected_launches
    got = [t.cpu().numpy() for t in out]
    f.close()
    for g, p in zip(got, src):
        r = dir_oracle(sd, p)
        assert np.all(np.abs(g - r) <= 1e-6 + 1e-5 * np.abs(r)), float(np.abs(g - r).max())


@pytest.mark.parametrize("w,h", [(1600, 3700), (1601, 3641), (64, 3632)])
def test_four_recursive_components(torch_cuda, w, h):
    from film_juicer_b200 import descriptors

    # sigma 4 and up: starts, rows, starts, columns
    sd = descriptors.spatial_dir_record(5.0, w, h, diffusion_size_um=20.0, tail_um=60.0, tail_weight=0.3)
    check_dir(torch_cuda, sd, planes(w, h, 5), 4)


@pytest.mark.parametrize("legacy", [True, False])
@pytest.mark.parametrize("w,h,bounces", [(640, 360, 5), (643, 361, 5), (640, 360, 4), (800, 3300, 5)])
def test_recursive_bounces_on_three_channels(torch_cuda, prepare, w, h, bounces, legacy):
    """Five bounces take all planes of the scratch; 3300 rows take two rounds of columns."""
    from film_juicer_b200 import runtime
    from oracle import optics

    torch = torch_cuda
    weights = (0.4, 0.25, 0.15, 0.1, 0.1)[:bounces]
    d = prepare.scatter_halation_record(9.11, scatter_amount=0.0, strength=(0.1, 0.05, 0.02), bounce_weights=weights,
                                        legacy=legacy)
    src = planes(w, h, 6)
    dev = [torch.from_numpy(p).cuda() for p in src]
    # rows and columns; at 640x360 four bounces leave room for the taps' plane, which carries
    # the carrier's own share
    assert launches(torch, lambda: runtime.scatter_halation(d, dev)) == (3 if bounces < 5 else 2)
    for t, r in zip(dev, optics.scatter_halation(d, src)):
        g = t.cpu().numpy()
        assert np.all(np.abs(g - r) <= 2e-5 + 2e-5 * np.abs(r)), float(np.abs(g - r).max())
