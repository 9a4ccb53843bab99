"""The post effects' blurs at radii whose row segments share their inputs (above 400) and whose
column taps are not staged: at the first such radius, at segment and CTA edges (288 outputs, eight
segments), and where the radius exceeds the frame. Reference and bound are those of
test_post_blur_gpu.py; a small sigma keeps the noise from being flattened."""
import pytest

from test_post_blur_gpu import test_blur_segments_match_oracle as check

pytestmark = pytest.mark.gpu

CASES = [(1, 40, 401), (40, 1, 401), (288, 9, 401), (289, 73, 402), (2304, 5, 500), (2305, 6, 401), (2593, 3, 700),
         (5000, 4, 2048), (12, 900, 450)]


@pytest.mark.parametrize("w,h,radius", CASES)
def test_wide_radii(torch_cuda, oracle, recipes, prepare, w, h, radius):
    check(torch_cuda, oracle, recipes, prepare, w, h,
          dict(lens_blur_sigma_px=0.8, lens_blur_radius=radius, unsharp_sigma_px=0.7, unsharp_radius=radius,
               unsharp_amount=0.7))
