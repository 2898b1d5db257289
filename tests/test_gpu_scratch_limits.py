"""Products on a device that has no memory left for what only makes them faster:
the padded layout of odd and misaligned batches, the one-word lists.  The rest of
the device's memory is held by a tensor meanwhile; the allocations that do not
fit are refused by cudaMalloc and nothing is launched with them."""
import numpy as np
import pytest

import gmr

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _worst(torch, a, b, tmp):
    """max |a - b|, a slice at a time in a buffer that is there already."""
    worst = 0.0
    for i in range(0, a.shape[0], len(tmp)):
        t = tmp[: min(len(tmp), a.shape[0] - i), : a.shape[1]]
        torch.sub(a[i:i + len(t)], b[i:i + len(t)], out=t)
        worst = max(worst, float(t.abs_().max()))
    return worst


class _Held:
    """All of the device's free memory but `leave` bytes."""

    def __init__(self, torch, leave):
        self.torch, self.leave = torch, leave

    def __enter__(self):
        torch = self.torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        self.t = torch.empty(max(0, (free - self.leave) // (2 * MB) * 2 * MB), dtype=torch.uint8, device="cuda")
        assert torch.cuda.mem_get_info()[0] <= self.leave + 4 * MB

    def __exit__(self, *exc):
        self.torch.cuda.synchronize()
        del self.t
        self.torch.cuda.empty_cache()


def test_without_memory_for_the_padded_layout():
    torch = pytest.importorskip("torch")
    rows, cols = 8 << 20, 60  # padded rows of Y: 256 MB and more
    rng = np.random.default_rng(1)
    col = rng.integers(0, cols, rows)
    C = np.zeros(2 * rows, dtype=np.int32)
    C[::2] = col + 1
    plan = gmr.Plan.build(gmr.Grammar.from_arrays(cols + 1, [[1, 2]], C, [2.0]), rows, cols)
    eng = gmr.Engine(plan)
    eng.enable_left(plan)
    at = torch.from_numpy(col).cuda()
    launches = {}
    big, small = torch.empty(rows * 5 + 8, device="cuda"), torch.empty(cols * 5 + 8, device="cuda")
    for hold in (True, False):
        for op in ("right", "left"):
            for B, off in ((5, 0), (4, 1)):  # an odd width; rows off a 16-byte boundary
                X, Y = (small, big) if op == "right" else (big, small)
                n, k = (cols, rows) if op == "right" else (rows, cols)
                x, y = X[off:off + n * B].view(n, B), Y[off:off + k * B].view(k, B)
                x.copy_(torch.rand((n, B), device="cuda") * 2 - 1)
                if op == "right":
                    want = 2 * x[at]
                else:
                    want = torch.zeros((cols, B), dtype=torch.float64, device="cuda").index_add_(0, at, 2 * x.double()).float()
                limit = 1e-5 * float(want.abs().max())
                tmp = torch.empty((min(k, 1 << 20), B), device="cuda")
                multiply = eng.multiply_device if op == "right" else eng.multiply_left_device

                def check():
                    for _ in range(3):  # launched one by one, captured, replayed
                        y.fill_(7)
                        multiply(0, x.data_ptr(), y.data_ptr(), B, stream=torch.cuda.current_stream().cuda_stream)
                        torch.cuda.synchronize()
                        assert _worst(torch, y, want, tmp) <= limit
                    launches[op, B, hold] = eng.last_launches

                if hold:
                    with _Held(torch, 96 * MB):
                        check()
                else:
                    check()
        eng = gmr.Engine(plan)  # memory is there again: a new engine pads
        eng.enable_left(plan)
    for op, extra in (("right", 1), ("left", 2)):  # the padded layout copies Y, and X of the left product
        for B in (5, 4):
            assert launches[op, B, False] == launches[op, B, True] + extra


def test_without_memory_for_the_one_word_list():
    torch = pytest.importorskip("torch")
    rows, cols, B = 20000, 5000, 64
    m = gmr.gen_mosaic(rows, cols, 64, 0.01, 1e-3, 3)
    plan = gmr.Plan.build(gmr.repair(m, device=0), rows, cols, device=0)
    list_bytes = 4 * int(plan.array("em_off")[-1])
    need = (plan.stats["n_ops"] + plan.stats["n_terms"]) * B * 4
    assert list_bytes > 24 * MB and need > 8 * list_bytes
    eng, fresh = gmr.Engine(plan), gmr.Engine(plan)
    X = torch.rand((cols, B), device="cuda") * 2 - 1
    Y, want, y1, want1 = (torch.empty((rows, w), device="cuda") for w in (B, B, 1, 1))
    x1 = X[:, :1].contiguous()
    fresh.multiply_device(0, X.data_ptr(), want.data_ptr(), B)
    fresh.multiply_device(0, x1.data_ptr(), want1.data_ptr(), 1)
    eng.multiply_device(0, x1.data_ptr(), y1.data_ptr(), 1)
    torch.cuda.synchronize()
    fresh.close()
    bytes_before = eng.device_bytes
    tmp, limit = torch.empty_like(Y), 1e-5 * float(want.abs().max())
    with _Held(torch, need - 12 * MB):
        for _ in range(3):
            Y.fill_(7)
            eng.multiply_device(0, X.data_ptr(), Y.data_ptr(), B)
            torch.cuda.synchronize()
            assert _worst(torch, Y, want, tmp) <= limit
    assert eng.device_bytes < bytes_before + need - list_bytes // 2
    y1.fill_(7)
    eng.multiply_device(0, x1.data_ptr(), y1.data_ptr(), 1)  # by the per-level folds
    torch.cuda.synchronize()
    assert float((y1 - want1).abs().max()) <= 1e-5 * float(want1.abs().max())
