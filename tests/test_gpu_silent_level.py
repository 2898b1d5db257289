"""A deepest level that no row emits (a rule nothing refers to), with the
emissions ending at every remainder of four: the single-kernel sweeps walk
that level too and must leave Y alone.  Tolerances as in test_gpu_parity."""
import numpy as np
import pytest

import gmr
from oracle import oracle as O
from test_gpu_parity import check, engine_inputs, engine_outputs, oracle_columns, random_X


def _silent(rest):
    """A mosaic's grammar with one rule above its deepest one that nothing uses,
    and rows of one terminal until the emissions leave `rest` modulo 4."""
    m = gmr.gen_mosaic(400, 120, 16, 0.02, 0.002, 3)
    g = gmr.repair(m, 2)
    rules, alpha = g.rules().reshape(-1, 2), g.alpha
    level = np.zeros(alpha + len(rules), dtype=int)
    for i, (l, r) in enumerate(rules):
        level[alpha + i] = max(level[l], level[r]) + 1
    top = int(level.argmax())
    C = g.C()
    while (int((C != 0).sum()) - rest) % 4:
        C = np.r_[C, 1, 0]
    rows = int((C == 0).sum())
    with_top = gmr.Grammar.from_arrays(alpha, np.r_[rules, [[top, top]]], C, g.values())
    plan = gmr.Plan.build(with_top, rows, m.cols)
    return plan, O.RefSchedule(alpha, rules.reshape(-1), C), g.values(), rows, m.cols


@pytest.mark.parametrize("rest", range(4))
def test_plan_has_a_silent_level(rest):
    plan, *_ = _silent(rest)
    off = plan.array("em_off")
    assert plan.stats["depth"] == len(off) - 2 and off[-1] == off[-2] and off[-1] % 4 == rest


@pytest.mark.gpu
@pytest.mark.parametrize("sr", range(3))
@pytest.mark.parametrize("rest", range(4))
def test_single_kernel_sweeps(rest, sr):
    torch = pytest.importorskip("torch")
    plan, sched, V, rows, cols = _silent(rest)
    for words in (1, 2, 4, 8, 20, 32):  # one lane per value, two and more, no power of two
        B = 32 * words if sr == 1 else words
        X = random_X(sr, cols, B, words)
        Xw = engine_inputs(sr, X)
        ref = oracle_columns(sched, sr, V, X, rows, cols)
        eng = gmr.Engine(plan)
        for cfg in (dict(variant=gmr.VARIANT_PERSISTENT), dict(variant=gmr.VARIANT_PERSISTENT, lane_bytes=32), dict()):
            check(sr, engine_outputs(sr, eng.multiply(Xw, sr, B=B, **cfg), B), ref)
        dX = torch.from_numpy(Xw.view(np.int32)).cuda()
        pack = gmr.Pack([eng])
        for mode in (gmr.Pack.PERSISTENT, gmr.Pack.LEVELS):
            pack.set_mode(mode)
            dY = torch.full((rows, Xw.shape[1]), 7, dtype=torch.int32, device="cuda")
            pack.multiply_device([sr], [dX.data_ptr()], [dY.data_ptr()], [B])
            torch.cuda.synchronize()
            Y = dY.cpu().numpy().view({0: np.float32, 1: np.uint32, 2: np.int32}[sr])
            check(sr, engine_outputs(sr, Y, B), ref)
