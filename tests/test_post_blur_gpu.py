"""The post effects' blurs at the edges of their segments (288 outputs of a row, nine rows of
a column, eight of each per CTA) and with radii from one to wider than the frame, against the
oracle's post effects, which sum each output's taps by themselves: the pixel bound
2e-4 + 3e-4 |oracle| of tests/test_scanner_post_gpu.py. A misplaced sample shows: the frames
are noise, which a blur wide enough to hide it would flatten."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    (1, 75, dict(lens_blur_sigma_px=0.6)),
    (75, 1, dict(lens_blur_sigma_px=0.6, unsharp_sigma_px=0.5, unsharp_amount=0.8)),
    (287, 71, dict(lens_blur_sigma_px=0.8)),
    (288, 72, dict(unsharp_sigma_px=0.7, unsharp_amount=0.7)),
    (289, 73, dict(lens_blur_sigma_px=0.8, unsharp_sigma_px=0.7, unsharp_amount=0.7)),
    (577, 145, dict(lens_blur_sigma_px=1.5, unsharp_sigma_px=0.5, unsharp_amount=0.4)),
    (600, 30, dict(glare_percent=0.5, glare_roughness=0.4, glare_blur_sigma_px=6.0, lens_blur_sigma_px=0.7)),
    (310, 40, dict(lens_blur_sigma_px=0.7, lens_blur_radius=2048)),
]


@pytest.mark.parametrize("w,h,kw", CASES, ids=[f"{w}x{h}" for w, h, _ in CASES])
def test_blur_segments_match_oracle(torch_cuda, oracle, recipes, prepare, w, h, kw):
    from film_juicer_b200 import descriptors, runtime

    torch = torch_cuda
    rec = prepare.HostRecord(recipes["direct"])
    post = descriptors.scanner_post_record(**kw)
    rng = np.random.default_rng(w * 1000 + h)
    src = np.ascontiguousarray(rng.uniform(0.02, 0.9, size=(h, w, 3)).astype(np.float32))
    s = torch.from_numpy(src).cuda()
    dr = runtime.DeviceRecipe(rec)
    dens = [torch.empty((h, w), device="cuda") for _ in range(3)]
    dr.capture_density(s, dens)
    seed = oracle.glare_seed(rec.h.recipe_hash, 11, 0, 0)
    got = torch.empty_like(s)
    runtime.render_from_density_post(dr, post, seed, (0, 0), dens, got, src=s)
    want, _ = oracle.render_post(rec, post, seed, 0, 0, [d.cpu().numpy() for d in dens], src=src)
    err = np.abs(got.cpu().numpy() - want) - (2e-4 + 3e-4 * np.abs(want))
    assert float(err.max()) <= 0.0, float(err.max())
    dr.close()
