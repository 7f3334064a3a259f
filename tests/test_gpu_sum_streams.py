"""Domain integrals and inner products on several streams at once and in graphs:
the bits of the same sums alone (partial sums and tickets are not shared)."""

import pytest
import torch

from finitevolx_b200 import diagnostics as D

pytestmark = pytest.mark.gpu


def test_integrals_on_streams(cuda_ok):
    gen = torch.Generator(device="cuda").manual_seed(2)
    fs = [torch.randn(700 + 40 * k, 900, device="cuda", dtype=torch.float64, generator=gen) for k in range(8)]
    alone = [float(D.total_enstrophy(f, 0.3, 0.2)) for f in fs]
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    got = [[] for _ in fs]
    for _ in range(20):
        for k, f in enumerate(fs):
            with torch.cuda.stream(streams[k % 4]):
                got[k].append(D.total_enstrophy(f, 0.3, 0.2))
    torch.cuda.synchronize()
    assert all(float(x) == ref for xs, ref in zip(got, alone) for x in xs)


def test_integral_in_a_graph(cuda_ok):
    f, g = (torch.randn(600, 500, device="cuda", dtype=torch.float64) for _ in range(2))
    want = [float(D.total_energy(x, f, 0.3, 0.2)) for x in (f, g)]
    x = f.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = D.total_energy(x, f, 0.3, 0.2)
        out2 = D.total_energy(x, f, 0.3, 0.2)
    side = torch.cuda.Stream()
    for y, ref in ((g, want[1]), (f, want[0]), (g, want[1])):
        x.copy_(y)
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            graph.replay()
        eager = D.total_energy(f, f, 0.3, 0.2)
        torch.cuda.synchronize()
        assert float(out) == float(out2) == ref and float(eager) == want[0]


def test_inner_products_on_streams(cuda_ok):
    from finitevolx_b200.solvers.iterative import _dot
    gen = torch.Generator(device="cuda").manual_seed(3)
    fs = [torch.randn(300 + 200 * k, 700, device="cuda", dtype=torch.float64, generator=gen) for k in range(8)]
    alone = [float(_dot(f, f)) for f in fs]
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    got = [[] for _ in fs]
    for _ in range(20):
        for k, f in enumerate(fs):
            with torch.cuda.stream(streams[k % 4]):
                got[k].append(_dot(f, f))
    torch.cuda.synchronize()
    assert all(float(x) == ref for xs, ref in zip(got, alone) for x in xs)
