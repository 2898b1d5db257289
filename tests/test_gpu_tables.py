"""Per-launch tables at one lane per value: what a table asks for is what runs,
and what the learned model installs there."""
import numpy as np
import pytest

import gmr
from gmr import learn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mosaic():  # above the 2 Mi emissions from which (+,x) folds them in one launch
    m = gmr.gen_mosaic(12000, 3000, 64, 0.01, 1e-3, 3)
    plan = gmr.Plan.build(gmr.repair(m, device=0), 12000, 3000, device=0)
    assert plan.array("em_off")[-1] > 2 << 20
    return plan


@pytest.mark.parametrize("B", [1, 2, 4])
def test_row_owned_tables_add_in_a_fixed_order(mosaic, B):
    """A table of row-owned folds gives the bits that emit_mode = rows gives, every time."""
    eng = gmr.Engine(mosaic)
    X = np.random.default_rng(B).uniform(-1, 1, (3000, B)).astype(np.float32)
    want = eng.multiply(X, 0, B=B, emit_mode=gmr.EMIT_ROWS)
    default = eng.multiply(X, 0, B=B)
    for v in (3, 8):
        eng.set_level_variants(0, B, [v] * (eng.depth + 2))
        for _ in range(3):
            np.testing.assert_array_equal(eng.multiply(X, 0, B=B), want)
    assert np.abs(default - want).max() <= 1e-5 * np.abs(want).max()
    eng.set_level_variants(0, B, [4] * (eng.depth + 2))
    assert np.abs(eng.multiply(X, 0, B=B) - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("sr,B", [(0, 1), (0, 2), (0, 4), (1, 32), (1, 128), (2, 1), (0, 32)])
def test_learned_tables(mosaic, sr, B):
    """The installed table is the argmin of the returned predictions; plain where
    one launch folds everything, no row-owned or atomic folds at one lane, no
    chunks of 16 at four."""
    eng = gmr.Engine(mosaic)
    pred = learn.choose_learned(eng, mosaic, learn.Mlp.load(learn.MODEL_PATH), sr, B)
    table = eng.level_variants(sr, B)
    np.testing.assert_array_equal(table[1:], pred[1:].argmin(axis=1))
    words = B if sr != 1 else B // 32
    if words == 1:
        assert not table.any()
    elif words <= 4:
        assert not (table % 5).any()
    else:  # four lanes: chunks of 32 in the place of 16
        assert (table[1:] % 5).all()


def test_autotuner_where_one_launch_folds_everything(mosaic):
    """Nothing to choose: the plain table, one set of times, no mode costs."""
    torch = pytest.importorskip("torch")
    eng = gmr.Engine(mosaic)
    X = torch.rand((3000, 1), device="cuda")
    Y = torch.empty((12000, 1), device="cuda")
    times = eng.autotune(0, X.data_ptr(), Y.data_ptr(), 1)
    assert times.shape == (eng.depth + 2, eng.N_LEVEL_VARIANTS) and (times[1:] > 0).all()
    assert (times == times[:, :1]).all()
    assert not eng.level_variants(0, 1).any() and eng.mode_costs(0, 1) is None
