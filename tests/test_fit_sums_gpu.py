"""The adjoint's sum over pixels: on a flat frame with a flat cotangent every pixel adds the
same FP32 term, so the gradient is the pixel count times the one-pixel frame's gradient, and
what differs is the rounding of the sum.

A thread adds 16 equal terms in FP32 before FP64 takes over: step j rounds j / 16 of the
final partial sum by at most 2^-24, together at most 8.5 * 2^-24 = 5.1e-7 of it, and no less
than that is asked of frames of any size. Parameters that a pixel adds one term to (exposure
and gamma of the film layers, print gamma and exposure); the knees get several of both
signs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOUND = 8.5 * 2.0 ** -24
ONE_TERM = [0, 1, 2, 3, 4, 5, 6, 7, 8, 12]


def gradient(torch, fitting, dr, h, w):
    src = torch.tensor([0.31, 0.22, 0.13], device="cuda").expand(h, w, 3).contiguous()
    theta = fitting.default_theta(dr).to(torch.float32).requires_grad_(True)
    cot = torch.tensor([0.7, -0.4, 0.9], device="cuda")[:, None, None].expand(3, h, w).contiguous()
    fitting.chain(theta, dr, src).backward(cot)
    return theta.grad.double().cpu().numpy()


@pytest.mark.parametrize("route", ["direct", "print"])
@pytest.mark.parametrize("w,h", [(1000, 17), (2048, 2048), (4099, 5003)])
def test_gradient_of_a_flat_frame(torch_cuda, recipes, prepare, route, w, h):
    from film_juicer_b200 import fitting, runtime

    dr = runtime.DeviceRecipe(prepare.HostRecord(recipes[route]))
    one = gradient(torch_cuda, fitting, dr, 1, 1)[ONE_TERM]
    got = gradient(torch_cuda, fitting, dr, h, w)[ONE_TERM]
    dr.close()
    want = one * (w * h)
    # the gradient tensor itself is FP32
    assert np.all(np.abs(got - want) <= (BOUND + 2.0 ** -24) * np.abs(want)), (got - want) / np.where(want == 0, 1, want)
