"""Camera exposure of pixels whose chromaticity quotients leave the FP32 range: components of
both signs up to 4e29 whose XYZ sum is negative, so that X or Y is divided by the floor
1e-10. The table coordinate then clamps at 1; a quotient that turned into NaN would clamp
at 0. The film table is negated, so that the (negative) sum times the table entry is a
positive exposure and the entry read shows. Bound as for the carrier planes in
test_pixel_parity_gpu.py: 1e-6 + 2e-5 |oracle|."""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DIRECTIONS = [(4.0, -1.0, -1.0), (-3.0, 2.0, -1.0), (1.0, -1.0, -1.0)]  # X > 0, Y > 0, all of X, Y, Z <= 0
SCALES = [1.0, 1e10, 1e17, 1e20, 1e26, 1e28, 1e29]


@pytest.mark.parametrize("route", ["direct", "print"])
def test_camera_exposure_at_the_range_ends(torch_cuda, recipes, prepare, oracle, route):
    from film_juicer_b200 import runtime

    torch = torch_cuda
    recipe = copy.deepcopy(recipes[route])
    recipe.arrays["tc_lut"] = -recipe.arrays["tc_lut"]
    rec = prepare.HostRecord(recipe)
    dr = runtime.DeviceRecipe(rec)
    src = np.array([[[np.float32(c * s) for c in d] for s in SCALES] for d in DIRECTIONS], np.float32)
    h, w = src.shape[:2]
    planes = [torch.empty((h, w), device="cuda") for _ in range(3)]
    dr.camera_exposure(torch.from_numpy(src).cuda(), planes)
    ref, _ = oracle.render(rec, src, stage=3)
    dr.close()
    assert all(np.isfinite(r).all() and (r[1:] > 0.0).all() for r in ref)
    for g, r in zip(planes, ref):
        err = np.abs(g.cpu().numpy() - r) - (1e-6 + 2e-5 * np.abs(r))
        assert err.max() <= 0.0, err
