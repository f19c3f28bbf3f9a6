"""The folded leaf's kernels at the sizes where they change: leaves of more than
8,192 edges (smaller ones take one warp per edge) just off multiples of a warp, of
small and of large CTAs, a stage of queued moves that overflows, one sum and one
counter per root, both colours to move.  Against the oracle."""
import pytest

import perft_gpu_2026_b200 as pg

pytestmark = pytest.mark.gpu

QUEENS = "1k6/ppp5/8/1Q1Q1Q1Q/Q1Q1Q1Q1/1Q1Q1Q1Q/Q1Q1Q1Q1/K7 b - - 0 1"
SMALL = 64            # threads of a CTA below one wave of edges
LARGE = 384           # and from there on
WAVE = 148 * 768      # edges of a wave (threads of k_fold on the GPU)


@pytest.fixture(scope="module")
def by_moves():
    """Positions by their number of moves."""
    out = {}
    for p in pg.random_playouts(77, 3000, 4, 90):
        out.setdefault(pg.count_moves(p, True), []).append(p)
    assert 1 in out and all(k in out for k in range(17, 40))
    return out


def roots_with(total, by_moves):
    """Positions with `total` moves together, drawn from 200 of them."""
    pool = [p for k in range(17, 40) for p in by_moves[k][:8]]
    out, left, k = [], total, 0
    while left > 40 + 39:
        out.append(pool[k % len(pool)])
        left -= pg.count_moves(out[-1], True)
        k += 1
    while left:
        n = max(k for k in by_moves if 0 < k <= min(left, 39))
        out.append(by_moves[n][0])
        left -= n
    return out


@pytest.mark.parametrize("total", [8193, 8223, 8224, 8225, 8192 + SMALL - 1, 8192 + SMALL, 8192 + SMALL + 1,
                                   WAVE - 1, WAVE, WAVE + 1, WAVE + 31, WAVE + LARGE - 1, WAVE + LARGE,
                                   WAVE + LARGE + 1])
@pytest.mark.parametrize("strict", [False, True])
def test_batches_of_exact_sizes(total, strict, by_moves, oracle):
    roots = roots_with(total, by_moves)
    want = {}
    for r in roots:
        if r.key() not in want:
            want[r.key()] = oracle.perft(pg.to_fen(r), 3, strict)
    with pg.Engine(device=0, use_tt=False, strict=strict, arena_bytes=1 << 30) as eng:
        got = eng.perft_batch(roots, 3)
        st = eng.last_stats()
    assert st.leaf_edges == total and st.leaf_reruns == 0
    assert got == [want[r.key()] for r in roots]


@pytest.mark.parametrize("fen,depth,edges", [
    ("8/2p5/3p4/KP5r/1R3p1k/8/4P1P1/8 w - - 0 1", 6, 43238),   # white's moves as the leaf's edges
    ("8/2p5/3p4/KP5r/1R3p1k/8/4P1P1/8 w - - 0 1", 7, 674624),  # black's
    ("8/4p1p1/8/1r3P1K/kp5R/3P4/2P5/8 b - - 0 1", 6, 43238),
    ("r3k2r/Pppp1ppp/1b3nbN/nP6/BBP1P3/q4N2/Pp1P2PP/R2Q1RK1 w kq - 0 1", 5, 9467),
])
@pytest.mark.parametrize("strict", [False, True])
def test_single_positions(fen, depth, edges, strict, oracle):
    with pg.Engine(device=0, use_tt=False, strict=strict, arena_bytes=1 << 30) as eng:
        assert eng.perft_position(pg.parse_fen(fen), depth) == oracle.perft(fen, depth, strict)
        st = eng.last_stats()
        assert st.leaf_edges == edges and st.leaf_reruns == 0


@pytest.mark.parametrize("strict", [False, True])
def test_a_stage_that_overflows(strict, by_moves, oracle):
    """Six edges a root that queue 57 moves each, 1,800 a warp where the stage holds
    384; among them roots that queue few."""
    q = pg.parse_fen(QUEENS)
    _, made, bad = pg.selftest_fold([pg.make_move(q, m) for m in pg.generate_moves(q)])
    assert bad == 0 and made > 2 * 6 * 50
    roots = ([q] * 7 + [by_moves[30][0], by_moves[17][0]]) * 150
    want = {r.key(): oracle.perft(pg.to_fen(r), 3, strict) for r in roots[:9]}
    with pg.Engine(device=0, use_tt=False, strict=strict, arena_bytes=1 << 30) as eng:
        assert eng.perft_batch(roots, 3) == [want[r.key()] for r in roots]
        assert eng.last_stats().leaf_edges > 8192 and eng.last_stats().leaf_reruns == 0
        # the same, the other colour to move at the leaf
        assert eng.perft_batch(roots[:270], 4) == [oracle.perft(pg.to_fen(r), 4, strict) for r in roots[:9]] * 30
