"""The interval that a curve lookup selects, on the axes of test_curve_axes_gpu.py with ordinates
that show it: the slope is 0.5 of one sign or the other from cell to cell, so a neighbouring
cell's line misses by up to the cell's width. (On smooth curves a neighbour of a fine axis stays
within the bounds.) Oracle and bounds are those of that file."""
import numpy as np
import pytest

from test_curve_axes_gpu import H, W, _resampled

pytestmark = pytest.mark.gpu


def _zigzag(axis, base):
    y = np.full(len(axis), base)
    for i in range(1, len(axis)):
        step = 0.5 * (float(axis[i]) - float(axis[i - 1]))
        y[i] = y[i - 1] + (-step if y[i - 1] > base else step)
    return y


def _with_zigzag(recipe, kind):
    r = _resampled(recipe, kind)
    a = r.arrays
    for axis_key, key, base in (("log_exposure", "density_rgb", 1.0), ("print_log_exposure", "print_density_cmy", 0.8)):
        if axis_key in a and key in a:
            z = np.stack([_zigzag(a[axis_key], base + 0.1 * c) for c in range(3)], axis=1)
            a[key] = np.ascontiguousarray((z if a[key].shape[0] == len(a[axis_key]) else z.T).astype(np.float32))
    return r


@pytest.mark.parametrize("kind", ["even3", "even257", "alternating", "clustered5", "clustered256", "clustered600",
                                  "clustered1024", "repeated"])
@pytest.mark.parametrize("route", ["direct", "print"])
def test_selected_intervals(torch_cuda, recipes, prepare, oracle, route, kind):
    from film_juicer_b200 import runtime

    torch = torch_cuda
    rec = prepare.HostRecord(_with_zigzag(recipes[route], kind))
    dr = runtime.DeviceRecipe(rec)
    src = np.ascontiguousarray(prepare.synthetic_frame(W, H, seed=20261205))
    s = torch.from_numpy(src).cuda()
    planes = [torch.empty((H, W), device="cuda") for _ in range(3)]
    dr.capture_density(s, planes)
    out = torch.empty_like(s)
    dr.render(s, out)
    density, _ = oracle.render(rec, src, stage=1)
    image, _ = oracle.render(rec, src)
    dr.close()
    for got, ref in zip(planes, density):
        assert np.isfinite(ref).all() and np.ptp(ref) > 0.0
        err = np.abs(got.cpu().numpy() - ref) - (1e-4 + 1e-4 * np.abs(ref))
        assert err.max() <= 0.0, err.max()
    err = np.abs(out.cpu().numpy() - image) - (2e-4 + 3e-4 * np.abs(image))
    assert err.max() <= 0.0, err.max()
