"""Small levels and leaves (one warp per position): counts against the oracle
and the host path at the sizes where the driver changes kernels."""
import pytest

import perft_gpu_2026_b200 as pg
from test_fold import FENS, _walk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 5, 64, 273, 274, 8192, 8193])
def test_batches_around_the_small_level_limit(n, oracle):
    """273 roots have about 8,192 moves, 8,192 and 8,193 roots are the last small
    and the first large level; both colours to move."""
    roots = _walk(FENS[0], max(n // 2, 1), 30, seed=n) + _walk(pg.START_FEN, n - max(n // 2, 1), 60, seed=n + 1)
    assert len(roots) == n
    with pg.Engine(device=0, use_tt=False, arena_bytes=2 << 30) as eng:
        for d in (2, 3):
            got = eng.perft_batch(roots, d)
            step = max(1, n // 400)
            for k in range(0, n, step):
                assert got[k] == oracle.perft(pg.to_fen(roots[k]), d), (k, d, pg.to_fen(roots[k]))


@pytest.mark.parametrize("fen", FENS + ["7k/5Q2/8/8/8/8/8/K7 b - - 0 1", "k7/8/1Q6/8/8/8/8/1R2K3 b - - 0 1"])
@pytest.mark.parametrize("strict", [False, True])
def test_small_single_positions(fen, strict, oracle):
    """Depths 3 to 5 around the leaf whose size the host does not read; few or
    no moves (mate, stalemate) among them.  Arenas with and without room for
    whole-level kernels give the same counts."""
    p = pg.parse_fen(fen)
    with pg.Engine(device=0, use_tt=False, strict=strict, arena_bytes=1 << 30) as eng, \
            pg.Engine(device=0, use_tt=False, strict=strict, arena_bytes=4 << 20) as tight:
        for q in [p] + [pg.make_move(p, m) for m in pg.generate_moves(p)][:6]:
            for d in (3, 4):
                want = oracle.perft(pg.to_fen(q), d, strict)
                assert eng.perft_position(q, d) == want
                assert tight.perft_position(q, d) == want
        st = eng.last_stats()
        assert st.leaf_edges == 0 or st.kernels == 3 * st.levels + 1  # no edges: the call ended early
        assert eng.perft_position(p, 5) == tight.perft_position(p, 5)


def test_levels_report_their_sizes():
    p = pg.parse_fen(pg.START_FEN)
    with pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30) as eng:
        assert eng.perft_position(p, 6) == 119060324
        st = eng.last_stats()
        assert list(st.level_sizes[:4]) == [20, 400, 8902, 197281] and st.levels == 3
        assert st.leaf_edges == 197281 and st.leaf_positions == 4865609
        assert eng.perft_position(p, 4) == 197281
        st = eng.last_stats()
        assert list(st.level_sizes[:2]) == [20, 400] and st.leaf_edges == 400 and st.leaf_positions == 8902
