"""Two host threads whose calls need different amounts of shared memory of the same kernels: each
gets its own results, and no launch is refused. A kernel's shared-memory limit belongs to
the function, so a thread that set it to its own call's size would take it away from the other
between that one's setting and launch."""
import threading

import pytest

pytestmark = pytest.mark.gpu
CALLS = 400


def scatter_halation(torch, runtime, prepare, w, h):
    record = prepare.scatter_halation_record(9.11)
    scratch = torch.empty(int(runtime.load_library().fjb_scatter_halation_scratch_bytes(w, h)) // 4, device="cuda")
    src = torch.rand((3, h, w), device="cuda")

    def call(stream):
        out = src.clone()
        runtime.scatter_halation(record, tuple(out), scratch=scratch, stream=stream)
        return out
    return call


def spatial_dir(torch, runtime, prepare, w, h):
    from film_juicer_b200 import descriptors

    f = runtime.DirFilter(descriptors.spatial_dir_record(9.11, w, h), w, h)
    src = torch.rand((3, h, w), device="cuda")

    def call(stream):
        out = torch.empty_like(src)
        f.apply(tuple(src), tuple(out), stream=stream)
        return out
    return call


def post_blur(torch, runtime, prepare, sigma):
    import os

    from conftest import GOLDEN
    from film_juicer_b200 import descriptors

    recipe = prepare.PreparedRecipe.load(os.path.join(GOLDEN, "recipe_print.npz"))
    dr = runtime.DeviceRecipe(prepare.HostRecord(recipe))
    record = descriptors.scanner_post_record(lens_blur_sigma_px=sigma)
    scratch = torch.empty(int(runtime.load_library().fjb_scanner_post_scratch_bytes(64, 16)) // 4, device="cuda")
    density = torch.rand((3, 16, 64), device="cuda")

    def call(stream):
        out = torch.empty((16, 64, 3), device="cuda")
        runtime.render_from_density_post(dr, record, 1, (0, 0), tuple(density), out, scratch=scratch, stream=stream)
        return out
    return call


@pytest.mark.parametrize("stage,large,small", [(scatter_halation, (32, 3000), (32, 1600)),
                                               (scatter_halation, (9000, 8), (5000, 8)),
                                               (spatial_dir, (32, 3000), (32, 1600)),
                                               (spatial_dir, (9000, 8), (5000, 8)),
                                               (post_blur, (200.0,), (30.0,))])
def test_calls_of_two_threads(torch_cuda, prepare, stage, large, small):
    from film_juicer_b200 import runtime

    torch = torch_cuda
    calls = [stage(torch, runtime, prepare, *size) for size in (large, small)]
    streams = [torch.cuda.Stream() for _ in calls]
    torch.cuda.synchronize()
    failures, results = [], [None, None]
    barrier = threading.Barrier(2)

    def work(k):
        try:
            with torch.cuda.stream(streams[k]):
                barrier.wait()
                for _ in range(CALLS):
                    results[k] = calls[k](streams[k])
        except Exception as e:  # reported by the test's own thread
            failures.append(f"{k}: {e}")

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failures, failures
    for k, call in enumerate(calls):
        assert torch.equal(results[k], call(None))
