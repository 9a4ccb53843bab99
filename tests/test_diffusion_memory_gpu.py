"""Standalone diffusion calls that need more device memory than the library's pool serves (the
transforms of a 5120x2880 frame at radius 41, 475 MB): the values, and that nothing of it is kept.
A flat plane stays flat: FP32 transforms of up to 2^13 points are good to about 1e-6 of the value,
2e-5 is allowed."""
import pytest

pytestmark = pytest.mark.gpu


def test_large_call_gives_its_memory_back(torch_cuda):
    from film_juicer_b200 import descriptors, runtime

    torch = torch_cuda
    comps = runtime.diffusion_components(descriptors.diffusion_record(6.8, 5120))
    src = [torch.full((2880, 5120), v, device="cuda") for v in (0.25, 1.0, 3.0)]
    dst = [torch.empty_like(p) for p in src]
    runtime.diffusion(comps, 3, 0.5, src, dst)  # the pool is there
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        runtime.diffusion(comps, 41, 0.5, src, dst)
    for s, d in zip(src, dst):
        assert float((d - s).abs().max()) <= 2e-5 * float(s.max())
    torch.cuda.synchronize()
    # the comparison's temporaries are torch's; the call's own 475 MB are not among what is gone
    torch.cuda.empty_cache()
    assert before - torch.cuda.mem_get_info()[0] < 128 << 20
