"""A planned batch whose captured graph is run again after other calls have
used the arena: the same counts as the exact batch."""
import pytest

import perft_gpu_2026_b200 as pg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    """A network that predicts a constant: every call of a depth has one plan."""
    with pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30) as eng:
        eng.mlp_init(seed=5, out_bias=[5.5, 11.0, 16.5, 22.0])
        params = eng.mlp_params()
        params[:-4] = 0.0
        eng.mlp_set_params(params)
        yield eng


@pytest.mark.parametrize("n", [1, 500, 3000])
@pytest.mark.parametrize("depth", [2, 3, 4])
def test_graph_runs_again_after_other_calls(engine, n, depth):
    roots = pg.random_playouts(41 + n, n, 4, 20, packed=True)
    other = pg.random_playouts(7, 700, 0, 60, packed=True)
    p = pg.parse_fen(pg.START_FEN)
    want = engine.perft_batch(roots, depth)
    others = engine.perft_batch(other, 3)
    first, st = engine.perft_batch_planned(roots, depth)
    assert first == want and st.graph_batches == 1 and st.retries == 0
    for between in (
        lambda: engine.perft_position(p, 4) == 197281,
        lambda: engine.perft_position(p, 6) == 119060324,
        lambda: engine.perft_batch(other, 3) == others,
        lambda: engine.perft_position(p, 5) == 4865609,
    ):
        assert between()
        again, st = engine.perft_batch_planned(roots, depth)
        assert again == want and st.retries == 0
    # another batch of the same shape through the same graph
    fresh = pg.random_playouts(42 + n, n, 4, 20, packed=True)
    got, _ = engine.perft_batch_planned(fresh, depth)
    assert got == engine.perft_batch(fresh, depth)
    got, _ = engine.perft_batch_planned(fresh, depth)
    assert got == engine.perft_batch(fresh, depth)


def test_graph_runs_again_after_its_plan_was_outgrown(engine):
    """Roots that outgrow the plan run exactly, over the graph's own arrays; the
    next batch of that shape is right again."""
    wide = pg.parse_fen("R6R/3Q4/1Q4Q1/4Q3/2Q4Q/Q4Q2/pp1Q4/kBNN1KB1 w - - 0 1")  # 218 moves
    roots = pg.pack_positions([wide] * 300)
    calm = pg.random_playouts(3, 300, 4, 20, packed=True)
    want = engine.perft_batch(calm, 3)
    assert engine.perft_batch_planned(calm, 3)[0] == want
    got, st = engine.perft_batch_planned(roots, 3)
    assert st.retries == 1 and got == engine.perft_batch(roots, 3)
    got, st = engine.perft_batch_planned(calm, 3)
    assert got == want and st.retries == 0
