"""The one-launch fold of 4-byte values (word_fold.cuh): matrices whose emission
list crosses its edges, against sums over the uncompressed entries.  Tolerance
for (+,x): 1e-5 relative max-norm of FP64, as everywhere; exact otherwise."""
import numpy as np
import pytest

import gmr
from helpers import INF

pytestmark = pytest.mark.gpu

CASES = {
    # more than 65,536 rows (two blocks of rows), many chunks, copies of Y
    "two_row_blocks": lambda: gmr.gen_mosaic(70001, 610, 64, 0.01, 1e-3, 3),
    # few long rows: runs far longer than a warp step
    "long_rows": lambda: gmr.gen_mosaic(41, 30000, 16, 0.02, 0.01, 4),
    # one chunk, short runs, empty rows at the end of the matrix
    "graph": lambda: gmr.gen_copy_graph(21000, 12, 0.7, False, 5),
}


@pytest.mark.parametrize("sr", range(3))
@pytest.mark.parametrize("name", list(CASES))
def test_word_fold(name, sr):
    m = CASES[name]()
    rows, cols, codes, V = m.rows, m.cols, m.codes(), m.values()
    r = np.repeat(np.arange(rows), np.diff(np.r_[-1, np.flatnonzero(codes == 0)]) - 1)
    nz = codes[codes != 0].astype(np.int64) - 1
    c, v = nz % cols, V[nz // cols]
    eng = gmr.Engine(gmr.Plan.build(gmr.repair(m, device=0), rows, cols, device=0))
    rng = np.random.default_rng(7)
    if sr == 0:
        x = rng.uniform(-1, 1, cols).astype(np.float32)
        y = eng.multiply(x, 0)[:, 0]
        ref = np.bincount(r, v * x[c].astype(np.float64), rows)
        assert np.abs(y - ref).max() <= 1e-5 * np.abs(ref).max()
    elif sr == 1:
        B = 17
        X = rng.random((cols, B)) < 3.0 / cols
        y = gmr.unpack_bits(eng.multiply(gmr.pack_bits(X), 1, B=B), B)
        for b in range(B):
            np.testing.assert_array_equal(y[:, b], np.bincount(r, X[c, b], rows) > 0)
    else:
        x = np.where(rng.random(cols) < 0.01, rng.integers(0, 1000, cols), 2**31 - 1).astype(np.int32)
        y = eng.multiply(x, 2)[:, 0]
        ref = np.full(rows, INF, dtype=np.int64)
        np.minimum.at(ref, r, np.where(x[c] >= INF, INF, v.astype(np.int64) + x[c]))
        np.testing.assert_array_equal(y, ref)
    # the same multiply again, and with the per-level folds: the plan's other order of the same emissions
    X1 = np.ones((cols, 1), dtype=np.int32 if sr else np.float32)
    a, b = eng.multiply(X1, sr, B=1), eng.multiply(X1, sr, B=1, push=gmr.PUSH_NEVER)
    if sr:
        np.testing.assert_array_equal(a, b)
    else:
        assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()


# the left product's list starts at 6 M emissions; "graph" stays on the edge lists
LEFT = {"two_chunks_of_x": lambda: gmr.gen_mosaic(70001, 1500, 64, 0.01, 1e-3, 3), "graph": CASES["graph"]}


@pytest.mark.parametrize("sr", range(3))
@pytest.mark.parametrize("name", list(LEFT))
def test_left_word_fold(name, sr):
    """x^T M at one word per value: rows beyond one chunk of x, targets in
    several blocks of 65,536 (rules, then terminals), and an x off the 16-byte
    boundary, which takes the edge lists instead."""
    import torch

    m = LEFT[name]()
    rows, cols, codes, V = m.rows, m.cols, m.codes(), m.values()
    r = np.repeat(np.arange(rows), np.diff(np.r_[-1, np.flatnonzero(codes == 0)]) - 1)
    nz = codes[codes != 0].astype(np.int64) - 1
    c, v = nz % cols, V[nz // cols]
    plan = gmr.Plan.build(gmr.repair(m, device=0), rows, cols, device=0)
    eng = gmr.Engine(plan)
    eng.enable_left(plan)
    rng = np.random.default_rng(8)
    if sr == 0:
        x = rng.uniform(-1, 1, rows).astype(np.float32)
        ref = np.bincount(c, v * x[r].astype(np.float64), cols)
    elif sr == 1:
        x = np.where(rng.random(rows) < 3.0 / rows, rng.integers(1, 2**32, rows, dtype=np.uint64), 0).astype(np.uint32)
        ref = np.zeros(cols, dtype=np.uint32)
        np.bitwise_or.at(ref, c, x[r])
    else:
        x = np.where(rng.random(rows) < 0.01, rng.integers(0, 1000, rows), 2**31 - 1).astype(np.int32)
        ref = np.full(cols, INF, dtype=np.int64)
        np.minimum.at(ref, c, np.where(x[r] >= INF, INF, v.astype(np.int64) + x[r]))
    buf = torch.zeros(rows + 4, dtype=torch.int32, device="cuda")
    for offset in (0, 1):
        buf[offset:offset + rows] = torch.from_numpy(x.view(np.int32)).cuda()
        for _ in range(3):
            dY = torch.full((cols,), 7, dtype=torch.int32, device="cuda")
            eng.multiply_left_device(sr, buf.data_ptr() + 4 * offset, dY.data_ptr(), 32 if sr == 1 else 1)
            torch.cuda.synchronize()
        y = dY.cpu().numpy().view(x.dtype)
        if sr == 0:
            assert np.abs(y - ref).max() <= 1e-5 * np.abs(ref).max()
        else:
            np.testing.assert_array_equal(y, ref)


def test_fixpoint_with_word_fold():
    """The device loop runs the one-launch fold in its body: reachability of 32
    sets against the per-level folds iterated from the host."""
    import torch

    m = CASES["graph"]()
    n = m.rows
    eng = gmr.Engine(gmr.Plan.build(gmr.repair(m, device=0), n, n, device=0))
    x = np.zeros((n, 1), dtype=np.uint32)
    x[np.arange(32) * 600, 0] = np.uint32(1) << np.arange(32, dtype=np.uint32)
    dX = torch.from_numpy(x.view(np.int32)).cuda()
    dY = torch.empty_like(dX)
    iters = eng.fixpoint_device("boolean", dX.data_ptr(), dY.data_ptr(), 32)
    ref, k = x, 0
    while True:
        nxt = ref | eng.multiply(ref, 1, B=32, push=gmr.PUSH_NEVER)
        k += 1
        if (nxt == ref).all():
            break
        ref = nxt
    np.testing.assert_array_equal(dX.cpu().numpy().view(np.uint32), ref)
    assert iters == k
