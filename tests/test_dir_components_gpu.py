"""Spatial DIR records beyond those a host derives from the film: a recursion without a factored
form (one real pole, or three), which runs in FP64 in the line form beside factored ones, and taps of
radius 10 to 64, two launches of their own each. Oracle and bounds are those of
test_line_pairs_gpu.py; the launch count shows that the line form ran."""
import pytest

from test_line_rounds_gpu import check_dir, planes

pytestmark = pytest.mark.gpu


def recursion(component, feedback):
    from film_juicer_b200 import abi

    g = component
    g.reference_operator = abi.FJ_DIR_OPERATOR_YVV_REFLECT
    g.sigma_px = max(3.0, g.sigma_px)
    g.radius = int(3.0 * g.sigma_px + 0.5)
    for i in range(3):
        g.feedback[i] = g.feedback_numerators[i] = feedback[i]
    g.feedforward = g.feedforward_numerator = 1.0 - (feedback[0] + feedback[1] + feedback[2])
    g.normalization_denominator = 1.0


# real poles 0.9; 0.8, 0.5, 0.25; and a pair of 0.7 beside a negative one
POLES = {"one": (0.9, 0.0, 0.0), "three": (1.55, -0.725, 0.1), "negative": (1.2, -0.21, -0.098)}


@pytest.mark.parametrize("poles", sorted(POLES))
@pytest.mark.parametrize("w,h,which", [(643, 361, (3,)), (640, 361, (0, 1, 2, 3)), (1600, 3700, (2, 3)), (9, 40, (3,)),
                                       (14600, 9, (3,)), (9, 14600, (1, 3))])
def test_recursions_without_a_factored_form(torch_cuda, w, h, which, poles):
    from film_juicer_b200 import descriptors

    sd = descriptors.spatial_dir_record(5.0, w, h, diffusion_size_um=20.0, tail_um=60.0, tail_weight=0.3)
    for k in which:
        recursion(sd.components[k], POLES[poles])
    check_dir(torch_cuda, sd, planes(w, h, 11), 4)


def taps(component, sigma, radius):
    from film_juicer_b200 import abi

    component.reference_operator = abi.FJ_DIR_OPERATOR_FIR_REFLECT
    component.sigma_px, component.radius = sigma, radius


@pytest.mark.parametrize("w,h", [(643, 361), (40, 3700), (7, 5), (1, 9), (9, 1), (289, 73), (14600, 9)])
@pytest.mark.parametrize("radii", [(10,), (64,), (9, 10), (11, 40, 2, 64)])
def test_wide_taps(torch_cuda, w, h, radii):
    from film_juicer_b200 import descriptors

    sd = descriptors.spatial_dir_record(5.0, w, h, diffusion_size_um=20.0, tail_um=60.0, tail_weight=0.3)
    for k, r in enumerate(radii):
        taps(sd.components[k], 2.9 if r > 2 else 0.7, r)
    wide = sum(r > 9 for r in radii)
    recursive = 3 if len(radii) < 4 else 0  # starts, rows, starts
    check_dir(torch_cuda, sd, planes(w, h, 12), 1 + 2 * wide + recursive + 1)


@pytest.mark.parametrize("w,h,kind", [(643, 361, "taps"), (643, 361, "recursive"), (160, 90, "default"),
                                      (643, 361, "default"), (64, 3700, "recursive"), (643, 361, "only taps")])
def test_outputs_in_other_channels_inputs(torch_cuda, w, h, kind):
    """The corrections of all channels are read before a filtered plane is written."""
    from film_juicer_b200 import descriptors, runtime

    torch = torch_cuda
    if kind == "default":
        sd = descriptors.spatial_dir_record(35000.0 / w, w, h)
    else:
        sd = descriptors.spatial_dir_record(5.0, w, h, diffusion_size_um=20.0, tail_um=60.0, tail_weight=0.3)
    if kind == "taps":
        taps(sd.components[0], 2.9, 12)
    if kind == "only taps":
        for k, r in enumerate((11, 40, 2, 64)):
            taps(sd.components[k], 2.9 if r > 2 else 0.7, r)
    f = runtime.DirFilter(sd, w, h)
    src = [torch.from_numpy(p).cuda() for p in planes(w, h, 13)]
    want = [torch.empty_like(p) for p in src]
    f.apply(src, want)
    work = [p.clone() for p in src]
    f.apply(work, [work[1], work[2], work[0]])
    got = [work[1], work[2], work[0]]
    f.close()
    for g, t in zip(got, want):
        assert torch.equal(g, t)
