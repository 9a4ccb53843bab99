"""Diffusion by tiles at the sizes where its tiling changes: one sample, a frame smaller than
the radius, one sample less, exactly and one more than a tile's inner 128 - 2 r, an odd number
of tiles (the last pair half empty), the smallest and largest radius and the first one beyond
it. Bound as for the other forms: |d| <= 2e-6 max(1, max |input|)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [8, 19, 40, 41])
@pytest.mark.parametrize("dw,dh,stride", [(None, None, 0), (-1, 0, 0), (0, 1, 3), (1, -1, 1), (130, 40, 5)])
def test_tile_sizes(torch_cuda, radius, dw, dh, stride):
    torch = torch_cuda
    from film_juicer_b200 import descriptors, runtime
    from oracle import optics

    inner = 128 - 2 * radius
    w, h = (1, 3) if dw is None else (inner + dw, inner + dh)
    comps = runtime.diffusion_components(descriptors.diffusion_record(9.0, 256))
    rng = np.random.default_rng(radius)
    planes = [rng.uniform(0.0, 4.0, size=(h, w)).astype(np.float32) for _ in range(3)]
    src = torch.zeros((3, h, w + stride), device="cuda")
    src[:, :, :w] = torch.from_numpy(np.stack(planes)).cuda()
    dst = torch.full_like(src, -7.0)
    runtime.diffusion(comps, radius, 0.3, [src[c, :, :w] for c in range(3)], [dst[c, :, :w] for c in range(3)])
    got = dst.cpu().numpy()
    assert np.all(got[:, :, w:] == -7.0)
    for g, r in zip(got[:, :, :w], optics.diffusion(comps, radius, 0.3, planes)):
        assert np.all(np.abs(g - r) <= 2e-6 * 4.0), float(np.abs(g - r).max())
