"""Rounding of scatter/halation against 64 bits, records with factored recursions: the weighted sum
of the carrier and its Gaussians adds the small terms first, so that the result's error is
that of the last additions. Emulated on random terms with the records' weights, a pass has a
relative rms of 3.6e-8 that way and 5.2e-8 when the carrier comes first; two passes and the
filters' own rounding: 4.8e-8 and 6.3e-8 on frames of 12 stops. Bound: 5.5e-8."""
import numpy as np
import pytest

from film_juicer_b200 import abi

W, H = 900, 500
PIXEL_UM = 35000.0 / 1920


def fields(seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:H, 0:W] / W
    out = np.empty((3, H, W))
    for k in range(3):
        f = np.zeros((H, W))
        for _ in range(8):
            cx, cy, s = rng.uniform(0, 1), rng.uniform(0, H / W), rng.uniform(0.02, 0.15)
            f += rng.uniform(-1, 1) * np.exp(-(((x - cx) / s) ** 2 + ((y - cy) / s) ** 2) / 2)
        f = 0.02 + 0.96 * (f - f.min()) / np.ptp(f) + 0.01 * rng.standard_normal((H, W))
        out[k] = 2.0 ** (-8.0 + 12.0 * np.clip(f, 0.0, 1.0))
    return out.astype(np.float32)


def section(x, h, g, t):
    """Both directions along axis 0, replicate starts."""
    for order in (range(len(x)), range(len(x) - 1, -1, -1)):
        y = np.empty_like(x)
        s1 = s2 = x[order[0]]
        s3 = np.zeros_like(s1)
        for i in order:
            s1 = s1 + h * (x[i] - s1)
            s3 = t * s3 + g * (s1 - s2)
            s2 = s2 + s3
            y[i] = s2
        x = y
    return x


def gaussian(plane, g):
    if g.kind == abi.FJ_HALATION_IDENTITY:
        return plane
    if g.kind == abi.FJ_HALATION_FIR_REFLECT:
        taps, r = list(g.fir_weights)[:2 * g.radius + 1], g.radius
        ext = np.pad(plane, ((0, 0), (r, r)), mode="symmetric")
        plane = sum(float(w) * ext[:, k:k + W] for k, w in enumerate(taps))
        ext = np.pad(plane, ((r, r), (0, 0)), mode="symmetric")
        return sum(float(w) * ext[2 * r - k:2 * r - k + H] for k, w in enumerate(taps))
    k = [float(v) for v in g.yvv[:3]]
    rows = section(np.ascontiguousarray(plane.T), *k).T
    return section(rows[::-1], *k)[::-1]  # from the bottom up first


def exact(d, src):
    amplitudes = [float(np.float32(a)) for a in (0.1633, 0.6496, 0.1870)]
    out = []
    for c in range(3):
        ch, x = d.channels[c], src[c].astype(np.float64)
        a, w, s = float(d.scatter_amount), float(ch.tail_weight), float(ch.total_strength)
        tail = sum(m * gaussian(x, ch.tail[i]) for i, m in enumerate(amplitudes))
        x = (1.0 - a) * x + a * ((1.0 - w) * gaussian(x, ch.core) + w * tail)
        if s:
            x = (x + s * sum(float(d.bounce_weights[b]) * gaussian(x, ch.bounce[b]) for b in range(d.bounce_count))) / (1.0 + s)
        out.append(x)
    return out


@pytest.mark.gpu
def test_rounding_of_the_weighted_sums(torch_cuda, prepare):
    from film_juicer_b200 import runtime

    torch = torch_cuda
    d = prepare.scatter_halation_record(PIXEL_UM, legacy=False)
    src = fields(5)
    dev = [torch.from_numpy(p).cuda() for p in src]
    runtime.scatter_halation(d, dev)
    for t, want in zip(dev, exact(d, src)):
        rms = float(np.sqrt(np.mean((t.cpu().numpy() / want - 1.0) ** 2)))
        assert rms <= 5.5e-8, rms
