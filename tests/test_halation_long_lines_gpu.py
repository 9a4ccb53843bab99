"""Precision of the back-reflection's recursion in the direct form (legacy records) on lines of
12288 samples, as rows and as columns, against the same recursion in 64 bits.

One bounce of 156 um on a 35 mm gate (sigma 54.8 px), strength 1, so that the output is
(x + G x) / 2. Rounding is amplified by the recursion's DC gain (4e4 here) and grows with the
length that a piece runs in FP32. Restated on the CPU for these planes (FP32 steps, FP64
states between pieces): rms relative error of G 9.4e-5 for pieces of 64 samples, 2.9e-4 for
32 pieces of 385. Bound: 1.5e-4."""
import numpy as np
import pytest

LENGTH, LINES = 12288, 6


def lines(seed):
    """LINES lines of 12 stops: smooth fields with fine texture, (LINES, LENGTH) float32."""
    rng = np.random.default_rng(seed)
    x = np.linspace(0.0, 1.0, LENGTH)
    out = np.empty((LINES, LENGTH))
    for k in range(LINES):
        f = np.zeros(LENGTH)
        for _ in range(8):
            f += rng.uniform(-1, 1) * np.exp(-((x - rng.uniform()) / rng.uniform(0.02, 0.15)) ** 2 / 2)
        f = 0.02 + 0.96 * (f - f.min()) / np.ptp(f) + 0.01 * rng.standard_normal(LENGTH)
        out[k] = 2.0 ** (-8.0 + 12.0 * np.clip(f, 0.0, 1.0))
    return out.astype(np.float32)


def recursion(y, c, ascending):
    """One direction along axis 0 in 64 bits, from a replicate start."""
    b, b1, b2, b3 = (float(v) for v in c)
    order = range(len(y)) if ascending else range(len(y) - 1, -1, -1)
    s = None
    out = np.empty_like(y)
    for i in order:
        if s is None:
            s = (y[i], y[i], y[i])
        v = b * y[i] + b1 * s[0] + b2 * s[1] + b3 * s[2]
        s = (v, s[0], s[1])
        out[i] = v
    return out


def filtered(plane, c):
    """Rows from left to right and back, then columns from the bottom up and back."""
    t = plane.astype(np.float64).T
    t = recursion(recursion(t, c, True), c, False).T
    return recursion(recursion(t, c, False), c, True)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [True, False])
def test_direct_form_keeps_its_precision_on_long_lines(torch_cuda, prepare, rows):
    from film_juicer_b200 import runtime

    torch = torch_cuda
    d = prepare.scatter_halation_record(35000.0 / LENGTH, scatter_amount=0.0, strength=(1.0, 1.0, 1.0),
                                        halation_first_sigma_um=(156.0, 156.0, 156.0), bounce_weights=(1.0,), legacy=True)
    src = [lines(k) if rows else np.ascontiguousarray(lines(k).T) for k in range(3)]
    dev = [torch.from_numpy(p).cuda() for p in src]
    runtime.scatter_halation(d, dev)
    for c in range(3):
        want = filtered(src[c], d.channels[c].bounce[0].yvv[:4])
        got = 2.0 * dev[c].cpu().numpy().astype(np.float64) - src[c]
        rms = float(np.sqrt(np.mean(((got - want) / want) ** 2)))
        assert rms <= 1.5e-4, rms
