"""The grain sample kernel's per-tile tables (draw offsets, Wang cells, noise lattices, the layer
axis) against the direct evaluation they stand for: the same absolute pixel must get the same
bits whatever tile it falls into. A large frame (64-row tiles) is compared with small crops of
it (8-row tiles at other alignments), with crops that start at negative coordinates (whose
tiles hold no cells, so every hash is evaluated at the pixel) and with the general layer-axis
search. The grain is taken without blurs, so a pixel depends on its own coordinates only and
the comparison is exact.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
W, H = 1250, 790  # enough tiles for the tallest ones


def _record(recipe, extent, pixel_um, frame_time, sublayers):
    from film_juicer_b200 import grain_plan as gp

    a = recipe.arrays
    layers = [[a["density_layers"][:, l, c] for c in range(3)] for l in range(3)]
    inp = gp.GrainInput(render_extent=(0, 0, W, H), full_frame_extent=(0, 0, W, H), pixel_size_um=pixel_um,
                        layer_curves=layers, frame_time=frame_time)
    inp.correlation_sigma_px = 0.0
    inp.dye_cloud_blur_um = 0.0
    if not sublayers:
        inp.sublayers_active = False
        inp.sublayer_count = 4  # one more than the draw tables hold
    rec = gp.visual_grain_record(inp, gp.plan(inp), gp.GrainCoefficients(), curves_cmy=a["density_rgb"])
    # the plan refuses extents outside its frame, the library takes them
    rec.render_extent.x, rec.render_extent.y, rec.render_extent.width, rec.render_extent.height = extent
    return rec


def _noise(pow2):
    from film_juicer_b200 import grain_plan as gp

    rng = np.random.default_rng(3)
    return gp.Noise(rng.integers(0, 256, size=(4, 64, 128) if pow2 else (3, 48, 40), dtype=np.uint8),
                    rng.integers(0, 256, size=(16, 32, 32), dtype=np.uint8), gp.wang_lut_two_colors())


# pixel sizes: cells of many pixels, ordinary ones, a few pixels, and more cells than a tile holds
@pytest.mark.parametrize("pixel_um", [0.5, 9.4, 600.0, 3000.0])
@pytest.mark.parametrize("pow2,frame_time,sublayers", [(True, 3.0, True), (True, 10.375, True), (False, 10.375, True),
                                                       (True, 10.375, False)])
def test_tiles_agree(torch_cuda, recipes, prepare, pixel_um, pow2, frame_time, sublayers):
    from film_juicer_b200 import abi, runtime

    torch = torch_cuda
    recipe = runtime.DeviceRecipe(prepare.HostRecord(recipes["print"]))
    noise_rec = _noise(pow2)
    noise = runtime.DeviceNoise(noise_rec.record)
    rng = np.random.default_rng(8)
    base = torch.from_numpy(rng.uniform(-0.1, 2.2, size=(3, H + 80, W + 80)).astype(np.float32)).cuda()

    def render(x, y, w, h, edit=None):
        rec = _record(recipes["print"], (x, y, w, h), pixel_um, frame_time, sublayers)
        if edit:
            edit(rec)
        # planes of the absolute pixels x .. x + w - 1 (the plane's origin is at -80, -80)
        planes = [base[c, 80 + y:80 + y + h, 80 + x:80 + x + w].contiguous() for c in range(3)]
        runtime.visual_grain(recipe, rec, planes, noise)
        return torch.stack(planes)

    whole = render(0, 0, W, H)
    assert torch.isfinite(whole).all()
    for x, y, w, h in ((37, 21, 100, 90), (31, 63, 33, 65), (W - 97, H - 71, 97, 71), (5, 700, 1, 1)):
        assert torch.equal(render(x, y, w, h), whole[:, y:y + h, x:x + w]), (x, y)
    for x, y, w, h in ((-20, -7, 90, 40), (3, -40, 64, 70)):
        got = render(x, y, w, h)
        x0, y0 = max(x, 0), max(y, 0)
        assert torch.equal(got[:, y0 - y:, x0 - x:], whole[:, y0:y + h, x0:x + w]), (x, y)
    if sublayers:
        def general_axis(rec):
            rec.flags &= ~(abi.FJ_GRAIN_AXIS_FINITE_C | abi.FJ_GRAIN_AXIS_FINITE_C << 1 | abi.FJ_GRAIN_AXIS_FINITE_C << 2)

        assert torch.equal(render(37, 21, 100, 90, general_axis), whole[:, 21:111, 37:137])
    recipe.close()
