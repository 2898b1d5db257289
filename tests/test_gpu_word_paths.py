"""The one-launch fold of 4-byte values where its other tests do not take it:
several copies of Y, (+,x) on long and on short rows above its threshold, a list of
one chunk, the left product's list, packs, the fixpoint loop, the timing recorder
and the autotuner.  Each case states
from the plan that the fold applies.  (+,x) within 1e-5 relative max-norm of
FP64, the others exact."""
import re
from pathlib import Path

import numpy as np
import pytest

import gmr
from helpers import load_case
from oracle import oracle as O
from test_gpu_parity import check, engine_inputs, engine_outputs, oracle_columns

pytestmark = pytest.mark.gpu

HEADER = (Path(gmr.__file__).resolve().parent.parent / "csrc" / "word_fold.cuh").read_text()


def _constant(name):
    return eval(re.search(rf"\b{name} = ([^,;]+)[,;]", HEADER).group(1), {})


CHUNK, PER_COPY = _constant("kWordChunk"), _constant("kWordChunksPerCopy")


def _chunks(plan):
    return -(-((plan.stats["n_terms"] + 63) // 64 * 64 + plan.stats["n_ops"]) // CHUNK)


def _folds(plan, rows, least):
    E = int(plan.array("em_off")[-1])
    return (E >= _constant(least) and E >= _constant("kWordMinPerRow") * _chunks(plan) * rows
            and plan.stats["depth"] >= _constant("kWordMinDepth"))


def _build(m):
    rows, cols, codes, V = m.rows, m.cols, m.codes(), m.values()
    r = np.repeat(np.arange(rows), np.diff(np.r_[-1, np.flatnonzero(codes == 0)]) - 1)
    nz = codes[codes != 0].astype(np.int64) - 1
    plan = gmr.Plan.build(gmr.repair(m, device=0), rows, cols, device=0)
    return dict(plan=plan, rows=rows, cols=cols, r=r, c=nz % cols, v=V[nz // cols])


@pytest.fixture(scope="module")
def copies():  # 19 chunks: two copies of Y
    d = _build(gmr.gen_mosaic(70001, 1500, 64, 0.01, 1e-3, 3))
    assert _chunks(d["plan"]) > PER_COPY and _folds(d["plan"], d["rows"], "kWordMinEmissionsPlus")
    return d


CASES = {
    "copies": None,
    "long_rows": lambda: gmr.gen_mosaic(41, 400000, 16, 0.02, 0.01, 4),
    "short_rows": lambda: gmr.gen_mosaic(300000, 300, 64, 0.01, 1e-3, 0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_plus_times_above_its_threshold(name, request):
    d = request.getfixturevalue("copies") if CASES[name] is None else _build(CASES[name]())
    assert _folds(d["plan"], d["rows"], "kWordMinEmissionsPlus")
    eng = gmr.Engine(d["plan"])
    x = np.random.default_rng(7).uniform(-1, 1, d["cols"]).astype(np.float32)
    ref = np.bincount(d["r"], d["v"] * x[d["c"]].astype(np.float64), d["rows"])
    for _ in range(3):  # Y's copies are zeroed again each time
        y = eng.multiply(x, 0)[:, 0]
        launches = eng.last_launches
        assert np.abs(y - ref).max() <= 1e-5 * np.abs(ref).max()
    y = eng.multiply(x, 0, push=gmr.PUSH_NEVER)[:, 0]  # level by level
    assert np.abs(y - ref).max() <= 1e-5 * np.abs(ref).max()
    assert launches == eng.last_launches + (_chunks(d["plan"]) > PER_COPY)  # the sum of the copies


def test_recorder_and_autotuner_with_copies(copies):
    torch = pytest.importorskip("torch")
    eng = gmr.Engine(copies["plan"])
    X = torch.rand((copies["cols"], 1), device="cuda") * 2 - 1
    Y = torch.empty((copies["rows"], 1), device="cuda")
    want = torch.from_numpy(eng.multiply(X.cpu().numpy(), 0)).cuda()
    limit = 1e-5 * float(want.abs().max())
    ms = eng.time_launches(0, X.data_ptr(), Y.data_ptr(), 1)
    assert len(ms) == eng.depth + 2 and (ms > 0).all()
    assert float((Y - want).abs().max()) <= limit
    times = eng.autotune(0, X.data_ptr(), Y.data_ptr(), 1)
    assert times.shape == (eng.depth + 2, eng.N_LEVEL_VARIANTS)
    Y.fill_(7)
    eng.multiply_device(0, X.data_ptr(), Y.data_ptr(), 1)
    torch.cuda.synchronize()
    assert float((Y - want).abs().max()) <= limit


@pytest.mark.parametrize("sr", range(3))
def test_left_list(sr):
    """Rows beyond one chunk of x, targets in several blocks of 65,536; an x off
    the 16-byte boundary takes the edge lists."""
    torch = pytest.importorskip("torch")
    d = _build(gmr.gen_mosaic(120001, 1500, 64, 0.01, 1e-3, 3))
    assert int(d["plan"].array("em_off")[-1]) >= _constant("kLeftWordMinEmissions") and d["rows"] > CHUNK
    eng = gmr.Engine(d["plan"])
    before = eng.device_bytes
    eng.enable_left(d["plan"])
    # both orders are on the device: 8 bytes an edge, and 4 a row's edge in the list
    assert eng.device_bytes - before > 8 * len(d["plan"].array("le_src")) + 4 * int(d["plan"].array("em_off")[-1])
    rng = np.random.default_rng(8)
    r, c, rows, cols = d["r"], d["c"], d["rows"], d["cols"]
    if sr == 0:
        x = rng.uniform(-1, 1, rows).astype(np.float32)
        ref = np.bincount(c, d["v"] * x[r].astype(np.float64), cols)
    elif sr == 1:
        x = np.where(rng.random(rows) < 3.0 / rows, rng.integers(1, 2**32, rows, dtype=np.uint64), 0).astype(np.uint32)
        ref = np.zeros(cols, dtype=np.uint32)
        np.bitwise_or.at(ref, c, x[r])
    else:
        x = np.where(rng.random(rows) < 0.01, rng.integers(0, 1000, rows), 2**31 - 1).astype(np.int32)
        ref = np.full(cols, 10**9, dtype=np.int64)
        np.minimum.at(ref, c, np.where(x[r] >= 10**9, 10**9, d["v"].astype(np.int64) + x[r]))
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


def test_pack_of_one_word_engines(copies):
    """Branches of a pack's graph with the fold, two copies of Y in one of them."""
    torch = pytest.importorskip("torch")
    g = _build(gmr.gen_mosaic(1500, 800, 64, 0.01, 1e-3, 0))
    engs = [gmr.Engine(copies["plan"]), gmr.Engine(g["plan"])]
    assert _folds(g["plan"], 1500, "kWordMinEmissions") and _chunks(g["plan"]) == 1
    rng = np.random.default_rng(3)
    X = [rng.uniform(-1, 1, (copies["cols"], 1)).astype(np.float32),
         rng.integers(0, 2**32, (g["cols"], 1), dtype=np.uint64).astype(np.uint32)]
    want = [engs[0].multiply(X[0], 0), engs[1].multiply(X[1], 1, B=32)]
    dX = [torch.from_numpy(x.view(np.int32)).cuda() for x in X]
    dY = [torch.empty((n, 1), dtype=torch.int32, device="cuda") for n in (copies["rows"], g["rows"])]
    pack = gmr.Pack(engs)
    for _ in range(3):
        for y in dY:
            y.fill_(7)
        pack.multiply_device([0, 1], [x.data_ptr() for x in dX], [y.data_ptr() for y in dY], [1, 32])
        torch.cuda.synchronize()
        y0 = dY[0].cpu().numpy().view(np.float32)
        assert np.abs(y0 - want[0]).max() <= 1e-5 * np.abs(want[0]).max()
        np.testing.assert_array_equal(dY[1].cpu().numpy().view(np.uint32), want[1])


@pytest.mark.parametrize("sr,words", [(1, 5), (1, 7), (2, 5), (2, 9)])
def test_fixpoint_of_padded_batches(sr, words):
    """The device loop with padded X and Y in its body, against the oracle's iteration."""
    torch = pytest.importorskip("torch")
    c = load_case("graph_400" if sr == 1 else "graph_w300")
    n, B = int(c["rows"]), words if sr == 2 else 32 * words - 3
    eng = gmr.Engine(gmr.Plan.build(gmr.Grammar.from_arrays(int(c["alpha"]), c["rules"], c["C"], c["V"]), n, n))
    sched = O.RefSchedule(int(c["alpha"]), c["rules"], c["C"])
    rng = np.random.default_rng(words)
    if sr == 1:
        X = (rng.random((n, B)) < 0.01).astype(np.float32)
    else:
        X = np.where(rng.random((n, B)) < 0.01, 0.0, 1e9).astype(np.float32)
    ref, steps = X.copy(), 0
    while True:
        steps += 1
        Y = oracle_columns(sched, sr, c["V"], ref, n, n)
        new = np.maximum(ref, Y) if sr == 1 else np.minimum(ref, Y)
        if np.array_equal(new, ref):
            break
        ref = new
    Xw = engine_inputs(sr, X) if sr == 1 else X.astype(np.int32)
    assert Xw.shape[1] == words
    for _ in range(2):  # the loop's graph is used again
        dX = torch.from_numpy(Xw.view(np.int32).copy()).cuda()
        dY = torch.empty_like(dX)
        assert eng.fixpoint_device(sr, dX.data_ptr(), dY.data_ptr(), B) == steps
        check(sr, engine_outputs(sr, dX.cpu().numpy().view(np.uint32 if sr == 1 else np.int32), B), ref)


@pytest.fixture(scope="module")
def square():
    d = _build(gmr.gen_mosaic(1500, 1500, 64, 0.01, 1e-3, 0))
    assert _folds(d["plan"], 1500, "kWordMinEmissions")
    return d


@pytest.mark.parametrize("sr,B", [(1, 1), (1, 32), (2, 1)])
def test_few_chunks_and_the_fixpoint_loop(square, sr, B):
    """Idempotent semirings fold in one launch from few emissions on: one product
    and the loop's result against the per-level folds iterated from the host."""
    torch = pytest.importorskip("torch")
    n = square["rows"]
    eng = gmr.Engine(square["plan"])
    rng = np.random.default_rng(B)
    if sr == 1:
        x = np.zeros((n, 1), dtype=np.uint32)
        x[rng.choice(n, B, replace=False), 0] = np.uint32(1) << np.arange(B, dtype=np.uint32)
    else:
        x = np.full((n, 1), 10**9, dtype=np.int32)
        x[rng.choice(n, 3, replace=False)] = 0
    dX = torch.from_numpy(x.view(np.int32).copy()).cuda()
    dY = torch.empty_like(dX)
    np.testing.assert_array_equal(eng.multiply(x, sr, B=B), eng.multiply(x, sr, B=B, push=gmr.PUSH_NEVER))
    steps, ref = 0, x
    while True:
        y = eng.multiply(ref, sr, B=B, push=gmr.PUSH_NEVER)
        new = ref | y if sr == 1 else np.minimum(ref, y)
        steps += 1
        if np.array_equal(new, ref):
            break
        ref = new
    assert eng.fixpoint_device(sr, dX.data_ptr(), dY.data_ptr(), B) == steps
    np.testing.assert_array_equal(dX.cpu().numpy().view(x.dtype), ref)
