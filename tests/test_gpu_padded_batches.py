"""Batches whose rows of X and Y no 16-byte access reaches (odd widths, X and Y
off a 16-byte boundary): the padded layout against the oracle, at widths on
both sides of each edge of the rule (4 words, 8-word rounding, 32-byte lanes
from 32 words, tiles of 128).  Tolerance as in test_gpu_parity: 1e-5 relative
max-norm of FP64 for (+,x), exact for the others."""
import numpy as np
import pytest

import gmr
from oracle import oracle as O
from test_gpu_parity import check, engine_inputs, engine_outputs, oracle_columns, random_X

pytestmark = pytest.mark.gpu


def _grammar(weighted):
    m = gmr.gen_copy_graph(700, 9, 0.6, True, 5) if weighted else gmr.gen_mosaic(900, 150, 16, 0.02, 0.002, 3)
    return m, gmr.repair(m, 2)


@pytest.mark.parametrize("weighted", [False, True])  # True: terminals evaluated in place from the padded X
@pytest.mark.parametrize("sr", range(3))
@pytest.mark.parametrize("words", [1, 3, 5, 7, 9, 31, 33, 40, 100, 127, 130, 257])
def test_odd_widths(weighted, sr, words):
    if sr == 1 and words > 9:
        pytest.skip("bit-packed: the word widths above cover the layout")
    m, g = _grammar(weighted)
    B = words * 32 - 5 if sr == 1 else words
    eng = gmr.Engine(gmr.Plan.build(g, m.rows, m.cols))
    sched = O.RefSchedule(g.alpha, g.rules(), g.C())
    X = random_X(sr, m.cols, B, words)
    ref = oracle_columns(sched, sr, g.values(), X, m.rows, m.cols)
    for cfg in (dict(), dict(variant=gmr.VARIANT_FUSED, ops_per_cta=5), dict(variant=gmr.VARIANT_PLAIN),
                dict(emit_mode=gmr.EMIT_ROWS)):
        check(sr, engine_outputs(sr, eng.multiply(engine_inputs(sr, X), sr, B=B, **cfg), B), ref)


@pytest.mark.parametrize("offset", [1, 2, 4])
@pytest.mark.parametrize("B", [4, 6, 32])
def test_misaligned_pointers(offset, B):
    """X and Y `offset` words past a 256-byte boundary; nothing around Y is written."""
    import torch

    m, g = _grammar(False)
    eng = gmr.Engine(gmr.Plan.build(g, m.rows, m.cols))
    X = random_X(0, m.cols, B, 1)
    xb = torch.zeros(X.size + 8, device="cuda")
    yb = torch.full((m.rows * B + 16,), 7.0, device="cuda")
    xb[offset:offset + X.size] = torch.from_numpy(X.reshape(-1)).cuda()
    for _ in range(2):  # the second call replays the captured graph
        eng.multiply_device("plustimes", xb.data_ptr() + 4 * offset, yb.data_ptr() + 4 * offset, B)
    torch.cuda.synchronize()
    y = yb.cpu().numpy()
    assert (y[:offset] == 7).all() and (y[offset + m.rows * B:] == 7).all()
    sched = O.RefSchedule(g.alpha, g.rules(), g.C())
    check(0, y[offset:offset + m.rows * B].reshape(m.rows, B), oracle_columns(sched, 0, g.values(), X, m.rows, m.cols))


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("sr", range(3))
@pytest.mark.parametrize("words", [1, 2, 3, 4, 5, 8, 12, 31, 32, 33, 96, 130, 1030])
def test_left_widths(weighted, sr, words):
    """The left product at every lane layout: one and two words (warp folds of
    128 edges), odd widths, 32-byte lanes, more lanes than a block's threads."""
    import torch
    from helpers import brute_left

    if sr == 1 and words > 5:
        pytest.skip("bit-packed: the word widths above cover the layout")
    m, g = _grammar(weighted)
    B = words * 32 - 5 if sr == 1 else words
    plan = gmr.Plan.build(g, m.rows, m.cols)
    eng = gmr.Engine(plan)
    eng.enable_left(plan)
    X = random_X(sr, m.rows, B, words)
    dX = torch.from_numpy(engine_inputs(sr, X).view(np.int32)).cuda()
    ref = brute_left(m.codes(), g.values(), X, m.rows, m.cols, sr)
    for _ in range(3):  # launched one by one, captured, replayed
        dY = torch.full((m.cols, dX.shape[1]), 7, dtype=torch.int32, device="cuda")
        eng.multiply_left_device(sr, dX.data_ptr(), dY.data_ptr(), B)
        torch.cuda.synchronize()
    Y = dY.cpu().numpy().view(np.uint32 if sr == 1 else np.float32 if sr == 0 else np.int32)
    check(sr, engine_outputs(sr, Y, B), ref)
