"""Spatial DIR and scatter/halation on lines at the ends of each form's range: frames of a few
samples (the line form's planes are padded), one pair of rows or columns per CTA from 14529
samples on, the many-launch form in global memory above 29020. The launch count tells the
forms apart. Oracle and bounds are those of test_line_pairs_gpu.py."""
import numpy as np
import pytest

from test_line_rounds_gpu import dir_oracle, launches, planes

pytestmark = pytest.mark.gpu
LINES = [(1, 1), (3, 2), (9, 9), (17, 17), (25, 25), (14528, 5), (14529, 6), (14531, 5), (5, 14532), (9, 14529), (18, 14528), (29020, 3), (8, 29020)]
GLOBAL = [(29024, 4), (3, 29021)]


def check_dir(torch, w, h):
    from film_juicer_b200 import descriptors, runtime

    # all four components recursive, so that the columns take a round each above 14528
    sd = descriptors.spatial_dir_record(5.0, w, h, diffusion_size_um=20.0, tail_um=60.0, tail_weight=0.3)
    src = planes(w, h, w + 2 * h)
    dev = [torch.from_numpy(p).cuda() for p in src]
    out = [torch.empty((h, w), device="cuda") for _ in range(3)]
    f = runtime.DirFilter(sd, w, h)
    count = launches(torch, lambda: f.apply(dev, out))
    f.close()
    for t, p in zip(out, src):
        g, r = t.cpu().numpy(), dir_oracle(sd, p)
        assert np.all(np.abs(g - r) <= 1e-6 + 1e-5 * np.abs(r)), float(np.abs(g - r).max())
    return count


def check_halation(torch, prepare, w, h, legacy):
    from film_juicer_b200 import runtime
    from oracle import optics

    d = prepare.scatter_halation_record(9.11, legacy=legacy)
    src = planes(w, h, w + 3 * h)
    dev = [torch.from_numpy(p).cuda() for p in src]
    count = launches(torch, lambda: runtime.scatter_halation(d, dev))
    for t, r in zip(dev, optics.scatter_halation(d, src)):
        g = t.cpu().numpy()
        assert np.all(np.abs(g - r) <= 2e-5 + 2e-5 * np.abs(r)), float(np.abs(g - r).max())
    return count


@pytest.mark.parametrize("w,h", LINES)
def test_dir_in_the_line_form(torch_cuda, w, h):
    assert check_dir(torch_cuda, w, h) == 4


@pytest.mark.parametrize("w,h", GLOBAL)
def test_dir_in_global_memory(torch_cuda, w, h):
    assert check_dir(torch_cuda, w, h) > 8


@pytest.mark.parametrize("legacy", [False, True])
@pytest.mark.parametrize("w,h", LINES)
def test_halation_in_the_line_form(torch_cuda, prepare, w, h, legacy):
    # taps, rows and columns of the two passes
    assert check_halation(torch_cuda, prepare, w, h, legacy) <= 6


@pytest.mark.parametrize("legacy", [False, True])
@pytest.mark.parametrize("w,h", GLOBAL)
def test_halation_in_global_memory(torch_cuda, prepare, w, h, legacy):
    assert check_halation(torch_cuda, prepare, w, h, legacy) > 8


@pytest.mark.parametrize("w,h", [(9, 9), (33, 18), (129, 129)])
def test_five_recursive_bounces_on_small_frames(torch_cuda, prepare, w, h):
    from film_juicer_b200 import runtime
    from oracle import optics

    d = prepare.scatter_halation_record(9.11, scatter_amount=0.0, strength=(0.1, 0.05, 0.02),
                                        bounce_weights=(0.4, 0.25, 0.15, 0.1, 0.1))
    src = planes(w, h, 7)
    dev = [torch_cuda.from_numpy(p).cuda() for p in src]
    assert launches(torch_cuda, lambda: runtime.scatter_halation(d, dev)) <= 3
    for t, r in zip(dev, optics.scatter_halation(d, src)):
        g = t.cpu().numpy()
        assert np.all(np.abs(g - r) <= 2e-5 + 2e-5 * np.abs(r)), float(np.abs(g - r).max())
