"""The solve functions on several streams and threads at once: every result has
the bits of the same solve alone."""

import threading

import pytest
import torch

from finitevolx_b200.solvers.spectral import solve_helmholtz_dct, solve_helmholtz_dst

pytestmark = pytest.mark.gpu


def _fields(n, dtype, shape=(320, 264)):
    gen = torch.Generator(device="cuda").manual_seed(5)
    return [torch.randn(*shape, device="cuda", dtype=dtype, generator=gen) for _ in range(n)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("solve", [solve_helmholtz_dst, solve_helmholtz_dct])
def test_streams_at_once(cuda_ok, solve, dtype):
    fs = _fields(24, dtype)
    alone = [solve(f, 0.1, 0.2, 1.5) for f in fs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(4)]
    got = [None] * len(fs)
    for k, f in enumerate(fs):
        with torch.cuda.stream(streams[k % 4]):
            got[k] = solve(f, 0.1, 0.2, 1.5)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(alone, got))


@pytest.mark.parametrize("own_streams", [False, True])
def test_threads_at_once(cuda_ok, own_streams):
    fs = _fields(32, torch.float64)
    alone = [solve_helmholtz_dst(f, 0.1, 0.2, 1.5) for f in fs]
    torch.cuda.synchronize()
    got, errors = [None] * len(fs), []

    def work(t):
        try:
            with torch.cuda.stream(torch.cuda.Stream() if own_streams else torch.cuda.default_stream()):
                for k in range(t, len(fs), 4):
                    got[k] = solve_helmholtz_dst(fs[k], 0.1, 0.2, 1.5)
        except Exception as e:  # reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    assert all(torch.equal(a, b) for a, b in zip(alone, got))


def test_capture_after_use(cuda_ok):
    f, g = _fields(2, torch.float64)
    want = [solve_helmholtz_dst(x, 0.1, 0.2, 1.5) for x in (f, g)]
    x = f.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = solve_helmholtz_dst(x, 0.1, 0.2, 1.5)
    for y, ref in ((g, want[1]), (f, want[0])):
        x.copy_(y)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)


def test_fp64_after_an_fp32_only_plan(cuda_ok):
    from finitevolx_b200.solvers.spectral import get_plan
    f = _fields(1, torch.float64, (24, 40))[0]
    want = solve_helmholtz_dst(f, 0.1, 0.2, 1.5)
    get_plan(24, 40, 0.1, 0.2, (1.75,), 1, fp64=False)
    got = get_plan(24, 40, 0.1, 0.2, (1.75,), 1).solve(f)
    assert torch.equal(got, solve_helmholtz_dst(f, 0.1, 0.2, 1.75)) and not torch.equal(got, want)
