"""Curve lookups on axes of every kind the pixel chain accepts, against the CPU oracle's
binary search: few and many samples, even, uneven and clustered spacing (a lookup table),
a repeated abscissa and curves too long for tables (the search itself).

The prepared curves are resampled on the new axes, so their slopes, and with them the
effect of the FP32 rounding of the logarithm, stay those of the ordinary recipes and the
tolerances are the pixel chain's own: 1e-4 + 1e-4 |oracle| on dye density and
2e-4 + 3e-4 |oracle| on encoded output (tests/test_pixel_parity_gpu.py). A lookup that
selected a wrong interval would extrapolate from it, or fail on the coarse axes, where one
interval spans a stop or more.
"""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
W, H = 123, 67


def _axis(kind):
    """Positions in [0, 1]."""
    if kind.startswith("even"):
        return np.linspace(0.0, 1.0, int(kind[4:]))
    if kind == "alternating":
        steps = np.tile([1.0, 24.0], 120)
        return np.concatenate([[0.0], np.cumsum(steps) / steps.sum()])
    if kind.startswith("clustered"):
        return np.linspace(0.0, 1.0, int(kind[9:])) ** 2
    if kind == "repeated":
        u = np.linspace(0.0, 1.0, 256)
        u[100] = u[99]
        return u
    raise ValueError(kind)


def _resampled(recipe, kind):
    r = copy.deepcopy(recipe)
    a = r.arrays
    u = _axis(kind)

    def move(axis_key, value_keys):
        x = a[axis_key].astype(np.float64)
        new = x[0] + (x[-1] - x[0]) * u
        for key in value_keys:
            if key in a:
                v = a[key].astype(np.float64)
                v = v if v.shape[0] == len(x) else v.T  # (n, channels)
                w = np.stack([np.interp(new, x, v[:, c]) for c in range(v.shape[1])], axis=1)
                a[key] = np.ascontiguousarray((w if a[key].shape[0] == len(x) else w.T).astype(np.float32))
        a[axis_key] = new.astype(np.float32)

    a.pop("density_layers", None)
    move("log_exposure", ["density_rgb", "dir_axes_rgb"])
    if "print_log_exposure" in a:
        move("print_log_exposure", ["print_density_cmy"])
    return r


@pytest.mark.parametrize("kind", ["even2", "even3", "even257", "alternating", "clustered5", "clustered256",
                                  "clustered600", "clustered1024", "repeated"])
@pytest.mark.parametrize("route", ["direct", "print"])
def test_curve_axes_match_oracle(torch_cuda, recipes, prepare, oracle, route, kind):
    from film_juicer_b200 import runtime

    torch = torch_cuda
    rec = prepare.HostRecord(_resampled(recipes[route], kind))
    dr = runtime.DeviceRecipe(rec)
    src = np.ascontiguousarray(prepare.synthetic_frame(W, H, seed=20261207))
    s = torch.from_numpy(src).cuda()
    planes = [torch.empty((H, W), device="cuda") for _ in range(3)]
    dr.capture_density(s, planes)
    out = torch.empty_like(s)
    dr.render(s, out)
    density, _ = oracle.render(rec, src, stage=1)
    image, _ = oracle.render(rec, src)
    dr.close()
    for got, ref in zip(planes, density):
        err = np.abs(got.cpu().numpy() - ref) - (1e-4 + 1e-4 * np.abs(ref))
        assert err.max() <= 0.0, err.max()
    err = np.abs(out.cpu().numpy() - image) - (2e-4 + 3e-4 * np.abs(image))
    assert err.max() <= 0.0, err.max()
