"""The line recursions of scatter/halation and spatial DIR at the sizes where their layout
changes: one sample, lines shorter and longer than the 32 pieces, an odd row or column left
over of a pair, of a row CTA's four rows and of a cluster's eight columns, planes whose rows
are not aligned, and columns too long for all recursions of a channel at once. Oracle and
bounds are those of the stages' own tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIZES = [(1, 1), (2, 3), (8, 4), (9, 5), (31, 33), (33, 31), (64, 64), (65, 67), (97, 130), (161, 8), (7, 161),
         (1283, 21), (21, 1283)]


def planes(w, h, seed):
    rng = np.random.default_rng(seed)
    return [np.ascontiguousarray(p) for p in rng.uniform(0.0, 2.0, size=(3, h, w)).astype(np.float32)]


@pytest.mark.parametrize("legacy", [True, False])
@pytest.mark.parametrize("w,h", SIZES)
def test_halation_sizes(torch_cuda, prepare, w, h, legacy):
    torch = torch_cuda
    from film_juicer_b200 import runtime
    from oracle import optics

    d = prepare.scatter_halation_record(9.11, legacy=legacy)
    src = planes(w, h, 3)
    # rows of an odd stride in one buffer: no row is aligned like the first one
    buf = torch.zeros((3, h, w + 3), device="cuda")
    buf[:, :, :w] = torch.from_numpy(np.stack(src)).cuda()
    runtime.scatter_halation(d, [buf[c, :, :w] for c in range(3)])
    got = buf[:, :, :w].cpu().numpy()
    assert not buf[:, :, w:].any()
    for g, r in zip(got, optics.scatter_halation(d, src)):
        assert np.all(np.abs(g - r) <= 2e-5 + 2e-5 * np.abs(r)), float(np.abs(g - r).max())


def test_halation_five_bounces_in_rounds(torch_cuda, prepare):
    torch = torch_cuda
    from film_juicer_b200 import runtime
    from oracle import optics

    w, h = 11, 4100  # 65.6 KB per recursion: three at a time
    d = prepare.scatter_halation_record(9.11, strength=(0.1, 0.05, 0.02), bounce_weights=(0.4, 0.25, 0.15, 0.1, 0.1))
    src = planes(w, h, 4)
    dev = [torch.from_numpy(p).cuda() for p in src]
    runtime.scatter_halation(d, dev)
    for t, r in zip(dev, optics.scatter_halation(d, src)):
        g = t.cpu().numpy()
        assert np.all(np.abs(g - r) <= 2e-5 + 2e-5 * np.abs(r)), float(np.abs(g - r).max())


@pytest.mark.parametrize("w,h", [s for s in SIZES if min(s) > 1])
def test_spatial_dir_sizes(torch_cuda, recipes, prepare, w, h):
    torch = torch_cuda
    from film_juicer_b200 import descriptors, runtime
    from oracle import dir as odir

    sd = descriptors.spatial_dir_record(9.11, w, h, diffusion_size_um=20.0, tail_um=60.0, tail_weight=0.3)
    rec = prepare.HostRecord(recipes["print"])
    dr = runtime.DeviceRecipe(rec)
    src = prepare.synthetic_frame(w, h, seed=33)
    filt = [torch.empty((h, w), device="cuda") for _ in range(3)]
    lraw = [torch.empty((h, w), device="cuda") for _ in range(3)]
    dr.spatial_dir_build(sd, filt, lraw, src=torch.from_numpy(src).cuda())
    ref, _, _ = odir.spatial_dir(rec, sd, src=src)
    for t, r in zip(filt, ref):
        g = t.cpu().numpy()
        assert np.all(np.abs(g - r) <= 1e-6 + 1e-5 * np.abs(r)), float(np.abs(g - r).max())
    dr.close()
