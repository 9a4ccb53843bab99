"""The elementary functions of fjb_math.cuh over the ranges they state, against FP64: largest and rms
error in units in the last place at most what the header says (0.5 is correct rounding; the
FP64 result's own rounding is below 1e-4), and no larger than CUDA's function has on the same
arguments. Outside the ranges the `any` forms are CUDA's."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
N = 1 << 22
QUOTIENT, ROOT, LOG10, CBRT, POW, ANGLE = range(6)


@pytest.fixture(scope="module")
def probe(torch_cuda, tmp_path_factory):
    from film_juicer_b200 import build

    torch = torch_cuda
    so = str(tmp_path_factory.mktemp("probe") / "math_probe.so")
    subprocess.run([build.nvcc(), "-std=c++17", *build.ARCH, "-O3", "-shared", "-Xcompiler", "-fPIC", "-cudart=static",
                    "-o", so, os.path.join(HERE, "math_probe.cu")], check=True)
    lib = C.CDLL(so)

    def evaluate(op, library, a, b):
        out = torch.empty_like(a)
        ptr = [C.c_void_p(t.data_ptr()) for t in (a, b, out)]
        assert lib.math_probe(C.c_int(op), C.c_int(int(library)), *ptr, C.c_longlong(a.numel()),
                              C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()
        return out
    return evaluate


def log_uniform(torch, gen, low, high, signed=False):
    u = torch.rand(N, device="cuda", generator=gen, dtype=torch.float64)
    x = torch.exp(np.log(low) + u * (np.log(high) - np.log(low))).float()
    return torch.where(torch.rand(N, device="cuda", generator=gen) < 0.5, -x, x) if signed else x


def errors(torch, got, exact):
    _, exponent = torch.frexp(exact)
    e = (got.double() - exact) * torch.exp2(24.0 - exponent.clamp(min=-125).double())
    return float(e.abs().max()), float(e.square().mean().sqrt())


# function, arguments, exact value, largest and rms error stated
CASES = [
    ("quotient", QUOTIENT, ((1e-15, 1e15, True), (1e-14, 1e14, True)), lambda t, a, b: a / b, 0.5001, 0.2888),
    ("root", ROOT, ((1e-30, 1e30, False), None), lambda t, a, b: a.sqrt(), 0.5001, 0.2888),
    ("log10", LOG10, ((1e-37, 3e38, False), None), lambda t, a, b: a.log10(), 1.4, 0.4),
    ("log10 about 1", LOG10, ((0.4, 2.5, False), None), lambda t, a, b: a.log10(), 1.4, 0.4),
    ("cube root", CBRT, ((1e-30, 1e30, True), None), lambda t, a, b: a.sign() * a.abs().pow(1.0 / 3.0), 0.74, 0.31),
    ("x^(5/12)", POW, ((1e-6, 1e6, False), None), lambda t, a, b: a.pow(5.0 / 12.0), 1.3, 0.35),
    ("angle", ANGLE, ((1e-3, 1.0, True), (1e-3, 1.0, True)), lambda t, a, b: t.atan2(a, b), 1.8, 0.37),
    ("angle near the axes", ANGLE, ((1e-10, 1.0, True), (1e-10, 1.0, True)), lambda t, a, b: t.atan2(a, b), 1.8, 0.37),
]


@pytest.mark.parametrize("name,op,ranges,exact,largest,rms", CASES, ids=[c[0] for c in CASES])
def test_errors_over_the_stated_range(torch_cuda, probe, name, op, ranges, exact, largest, rms):
    torch = torch_cuda
    gen = torch.Generator(device="cuda").manual_seed(20261205 + op)
    a = log_uniform(torch, gen, *ranges[0])
    b = log_uniform(torch, gen, *ranges[1]) if ranges[1] else a
    want = exact(torch, a.double(), b.double())
    own, library = (errors(torch, probe(op, k, a, b), want) for k in (False, True))
    assert own[0] <= largest and own[1] <= rms, own
    assert own[0] <= max(library[0], 0.5001) and own[1] <= library[1] * 1.001, (own, library)


@pytest.mark.parametrize("op", [LOG10, CBRT])
def test_arguments_outside_the_range_go_to_the_library(torch_cuda, probe, op):
    torch = torch_cuda
    tiny = float(np.float32(1e-42))
    x = torch.tensor([0.0, -0.0, tiny, 1e-40, 3.3e38, float("inf"), float("nan")]
                     + ([-1.0, -3e38] if op == LOG10 else [-tiny, 1e-31, -1e31, 3e38, -float("inf")]), device="cuda")
    own, library = (probe(op, k, x, x).cpu().numpy() for k in (False, True))
    np.testing.assert_array_equal(own, library)


def test_angle_on_the_axes_and_diagonals(torch_cuda, probe):
    torch = torch_cuda
    y = torch.tensor([0.0, 0.0, -0.0, -0.0, 1.0, -1.0, 1.0, -1.0, 1.0, -1.0], device="cuda")
    x = torch.tensor([1.0, -1.0, 1.0, -1.0, 0.0, 0.0, 1.0, 1.0, -1.0, -1.0], device="cuda")
    got, want = probe(ANGLE, False, y, x).double(), torch.atan2(y.double(), x.double())
    assert float((got - want).abs().max()) <= 1.8 * 2.0 ** -22  # an ulp of pi
    np.testing.assert_array_equal(torch.signbit(got).cpu().numpy(), torch.signbit(y).cpu().numpy())
