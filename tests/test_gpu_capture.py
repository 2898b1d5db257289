"""Products called while the caller captures a CUDA graph of their own: at the
arguments' first, second and later use the launches become part of that graph.
Tolerance 1e-5 relative max-norm: the fold's atomics may add in another order."""
import numpy as np
import pytest

import gmr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plan():
    m = gmr.gen_mosaic(3000, 700, 16, 0.01, 1e-3, 5)
    return gmr.Plan.build(gmr.repair(m), 3000, 700)


@pytest.mark.parametrize("op", ["right", "left"])
@pytest.mark.parametrize("uses", [0, 1, 2, 3])
@pytest.mark.parametrize("B", [1, 5, 32])
def test_product_under_capture(plan, op, uses, B):
    torch = pytest.importorskip("torch")
    eng = gmr.Engine(plan)
    eng.enable_left(plan)
    n, k = (700, 3000) if op == "right" else (3000, 700)
    gen = torch.Generator(device="cuda").manual_seed(B)
    X = torch.rand((n, B), device="cuda", generator=gen) * 2 - 1
    Y = torch.zeros((k, B), device="cuda")
    multiply = eng.multiply_device if op == "right" else eng.multiply_left_device

    def call(x, y):
        multiply(0, x.data_ptr(), y.data_ptr(), B, stream=torch.cuda.current_stream().cuda_stream)

    X0, want = X.clone(), torch.zeros_like(Y)
    call(X0, want)  # other buffers: the engine's scratch is there before the capture
    for _ in range(uses):
        call(X, Y)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(X, Y)
    for _ in range(2):
        Y.fill_(7)
        graph.replay()
        torch.cuda.synchronize()
        assert np.abs((Y - want).cpu().numpy()).max() <= 1e-5 * want.abs().max().item()
    call(X, Y)  # and the engine's own graph after it
    call(X, Y)
    torch.cuda.synchronize()
    assert np.abs((Y - want).cpu().numpy()).max() <= 1e-5 * want.abs().max().item()
