"""gmr_engine_enable_left called again: with the same plan, and with the plan of
the same rows in another order (equal counts, other edges).  (+,x) within 1e-5
relative max-norm of FP64, the others exact."""
import numpy as np
import pytest

import gmr
from helpers import INF

pytestmark = pytest.mark.gpu


def _plans(rows, cols, founders):
    """A mosaic and the same mosaic with its rows in reverse order."""
    m = gmr.gen_mosaic(rows, cols, founders, 0.01, 1e-3, 3)
    codes, V = m.codes(), m.values()
    ends = np.flatnonzero(codes == 0)
    starts = np.r_[0, ends[:-1] + 1]
    n = ends - starts + 1
    s, n = starts[::-1], n[::-1]
    reverse = np.repeat(s - np.r_[0, np.cumsum(n)[:-1]], n) + np.arange(n.sum())
    m2 = gmr.Csrv.from_codes(rows, cols, codes[reverse], V)
    plans = [gmr.Plan.build(gmr.repair(x, device=0), rows, cols, device=0) for x in (m, m2)]
    r = np.repeat(np.arange(rows), ends - starts)
    nz = codes[codes != 0].astype(np.int64) - 1
    return plans, r, nz % cols, V[nz // cols]


@pytest.fixture(scope="module")
def small():
    return _plans(1200, 300, 16) + (1200, 300)


@pytest.fixture(scope="module")
def large():  # above the 9 Mi emissions from which one-word (+,x) products fold the rows' edges at once
    return _plans(120001, 1500, 64) + (120001, 1500)


@pytest.mark.parametrize("size", ["small", "large"])
@pytest.mark.parametrize("sr", range(3))
@pytest.mark.parametrize("B", [1, 8])
def test_enable_left_again(size, sr, B, request):
    torch = pytest.importorskip("torch")
    plans, r, c, v, rows, cols = request.getfixturevalue(size)
    if size == "large" and B > 1 and sr:
        pytest.skip("the edge lists of the large plan: one semiring")
    assert all(plans[0].stats[k] == plans[1].stats[k] for k in ("n_ops", "depth", "n_terms"))
    eng = gmr.Engine(plans[0])
    rng = np.random.default_rng(sr)
    W = B if sr != 1 else 1
    if sr == 0:
        x = rng.uniform(-1, 1, (rows, W)).astype(np.float32)
    elif sr == 1:
        x = np.where(rng.random((rows, W)) < 3.0 / rows, rng.integers(1, 2**32, (rows, W), dtype=np.uint64), 0).astype(np.uint32)
    else:
        x = np.where(rng.random((rows, W)) < 0.01, rng.integers(0, 1000, (rows, W)), 2**31 - 1).astype(np.int32)
    dX = torch.from_numpy(x.view(np.int32)).cuda()
    dY = torch.zeros((cols, W), dtype=torch.int32, device="cuda")
    for which in (0, 0, 1, 1, 0):
        eng.enable_left(plans[which])
        xr = x if which == 0 else x[::-1]
        for _ in range(3):  # launched one by one, captured, replayed
            dY.fill_(7)
            eng.multiply_left_device(sr, dX.data_ptr(), dY.data_ptr(), 32 if sr == 1 else B)
        torch.cuda.synchronize()
        y = dY.cpu().numpy().view(x.dtype)
        for b in range(W):
            if sr == 0:
                ref = np.bincount(c, v * xr[r, b].astype(np.float64), cols)
                assert np.abs(y[:, b] - ref).max() <= 1e-5 * np.abs(ref).max()
            elif sr == 1:
                ref = np.zeros(cols, dtype=np.uint32)
                np.bitwise_or.at(ref, c, xr[r, b])
                np.testing.assert_array_equal(y[:, b], ref)
            else:
                ref = np.full(cols, INF, dtype=np.int64)
                np.minimum.at(ref, c, np.where(xr[r, b] >= INF, INF, v.astype(np.int64) + xr[r, b]))
                np.testing.assert_array_equal(y[:, b], ref)


def test_a_plan_of_other_sizes_is_refused(small):
    plan = small[0][0]
    g = gmr.Grammar.from_arrays(4, [[1, 2], [4, 3]], [5, 0], [1.0])    # two levels
    flat = gmr.Grammar.from_arrays(4, [[1, 2], [2, 3]], [4, 5, 0], [1.0])  # as many rules in one
    few = gmr.Grammar.from_arrays(4, [[1, 2], [4, 2]], [5, 0], [1.0])  # fewer terminals
    eng = gmr.Engine(gmr.Plan.build(g, 1, 3))
    for other in (plan, gmr.Plan.build(flat, 1, 3)):
        with pytest.raises(gmr.GmrError):
            eng.enable_left(other)
    with pytest.raises(gmr.GmrError):
        gmr.Engine(gmr.Plan.build(few, 1, 3)).enable_left(gmr.Plan.build(g, 1, 3))
    eng.enable_left(gmr.Plan.build(g, 1, 3))
