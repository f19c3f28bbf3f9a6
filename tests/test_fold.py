"""Folded counting (leaf kernel 6): perft(2) of a position by set arithmetic
against making and counting every move - on the host over playouts and
constructed positions, and on the GPU against the oracle where the kernels'
own edges lie (one edge, a partial warp, a partial CTA, a stage that overflows,
a queue too short for its chunk)."""
import pytest

import perft_gpu_2026_b200 as pg

# pins of every kind, castling paths, double and promotion pushes, en passant
# (pinned along the rank too), piece crowds, 16 pieces onto one square
FENS = [
    "r3k2r/p1ppqpb1/bn2pnp1/3PN3/1p2P3/2N2Q1p/PPPBBPPP/R3K2R w KQkq - 0 1",
    "8/2p5/3p4/KP5r/1R3p1k/8/4P1P1/8 w - - 0 1",
    "r3k2r/Pppp1ppp/1b3nbN/nP6/BBP1P3/q4N2/Pp1P2PP/R2Q1RK1 w kq - 0 1",
    "rnbq1k1r/pp1Pbppp/2p5/8/2B5/8/PPP1NnPP/RNBQK2R w KQ - 1 8",
    "r4rk1/1pp1qppp/p1np1n2/2b1p1B1/2B1P1b1/P1NP1N2/1PP1QPPP/R4RK1 w - - 0 10",
    "R6R/3Q4/1Q4Q1/4Q3/2Q4Q/Q4Q2/pp1Q4/kBNN1KB1 w - - 0 1",
    "2n4k/1P1P4/8/8/8/8/8/4K3 w - - 0 1",
    "k7/8/8/3PpP2/5K2/8/8/8 w - e6 0 1",
    "8/8/8/K2pP2q/8/8/8/7k w - d6 0 1",
    "4k3/8/8/8/8/8/8/QRBNKBRQ w - - 0 1",
    "r3k2r/8/3Q4/8/8/5q2/8/R3K2R b KQkq - 0 1",
    "1n1n4/n3n3/2k5/n3n3/1n1n4/8/8/4K3 b - - 0 1",
    "4k3/pppppppp/8/8/8/8/PPPPPPPP/4K3 w - - 0 1",
    "3qk3/8/8/3p4/8/3Q4/3P4/3RK3 b - - 0 1",
    # 16 white pieces onto d5: eight lines, eight knight jumps
    "7k/2N1N3/1NQQQN2/2Q1Q3/1NQQQN2/2N1N3/8/K7 w - - 0 1",
]


def _walk(fen, n, plies, seed):
    out, st = [], seed
    for _ in range(n):
        p = pg.parse_fen(fen)
        r, st = pg.splitmix64(st)
        for _ in range(r % (plies + 1)):
            m = pg.generate_moves(p)
            if not m:
                break
            r, st = pg.splitmix64(st)
            p = pg.make_move(p, m[r % len(m)])
        out.append(p)
    return out


@pytest.mark.parametrize("fen", FENS)
def test_fold_equals_counting_on_constructed_positions(fen):
    checked, made, bad = pg.selftest_fold(_walk(fen, 3000, 12, seed=7))
    assert bad == 0 and checked > 0


@pytest.mark.parametrize("fen", [
    # double pushes beside pawns: free, pinned on a file and a diagonal, the king
    # and a rook on their rank, two capturers
    "4k3/8/8/8/2p1p3/8/3P4/4K3 w - - 0 1",
    "4k3/8/8/8/4p3/8/3P4/4RK2 w - - 0 1",
    "8/8/6k1/8/4p3/8/2BP4/6K1 w - - 0 1",
    "8/8/8/8/k1p4R/8/1P1P4/4K3 w - - 0 1",
    "5k2/R3p3/8/1p1P1P1q/2P1P1P1/8/1P1P1P1P/4K3 w - - 0 1",
    # sliders that take and are taken along their own lines, with more behind
    "3r3k/3q4/3r4/8/3R4/3Q4/3R4/K7 w - - 0 1",
    "k6b/6q1/5b2/8/3B4/2Q5/1B6/K7 w - - 0 1",
    "7k/8/2b1q3/3P4/2r1b3/1P3P2/8/K7 w - - 0 1",
    "1k6/8/1q1q1q2/2Q1Q3/1b1R1b2/2Q1Q3/1r3r2/K7 w - - 0 1",
    # pawns beside the squares next to the king
    "8/8/3k4/8/1PPPPP2/8/PPP1PPP1/K7 w - - 0 1",
    "8/2p1p3/8/2PkP3/P1p1p1P1/2P1P3/1P1P1P2/K7 w - - 0 1",
])
def test_fold_pawns_beside_and_captured_sliders(fen):
    checked, made, bad = pg.selftest_fold(_walk(fen, 2000, 8, seed=11))
    assert bad == 0 and checked > 0


def test_fold_equals_counting_on_playouts():
    checked, made, bad = pg.selftest_fold(pg.random_playouts(99, 60000, 0, 160, packed=True))
    assert bad == 0
    assert made < 0.45 * checked  # most moves are folded


@pytest.mark.gpu
@pytest.mark.parametrize("fen", FENS)
@pytest.mark.parametrize("strict", [False, True])
def test_folded_leaf_matches_oracle(fen, strict, oracle):
    p = pg.parse_fen(fen)
    with pg.Engine(device=0, use_tt=False, strict=strict, arena_bytes=256 << 20) as eng:
        eng.set_tuning(leaf_kernel=6)
        for d in (3, 4):
            assert eng.perft_position(p, d) == oracle.perft(fen, d, strict), d
        counted = eng.last_stats().leaf_positions
        # both colours to move, and the rooted leaf (a batch of the children)
        kids = [pg.make_move(p, m) for m in pg.generate_moves(p)]
        got = eng.perft_batch(kids, 3)
        assert got == [oracle.perft(pg.to_fen(k), 3, strict) for k in kids]
        # the statistics count every move-count call, folded or not
        eng.set_tuning(leaf_kernel=5)
        eng.perft_position(p, 4)
        assert eng.last_stats().leaf_positions == counted


@pytest.mark.gpu
@pytest.mark.parametrize("arena_mb", [3, 8, 16, 64])
def test_folded_leaf_in_tight_arenas(arena_mb):
    """A leaf in several chunks; chunks whose queue is too short (over 30 queued
    moves per edge here against 16 planned) run again in smaller ones; an arena
    without room for the queue runs the listed leaf.  Same counts as the listed
    leaf with room."""
    p = pg.parse_fen("3qk3/8/8/8/8/8/8/QRBNKBRQ w - - 0 1")
    roots = [pg.make_move(p, m) for m in pg.generate_moves(p)]
    with pg.Engine(device=0, use_tt=False, arena_bytes=2 << 30) as eng:
        eng.set_tuning(leaf_kernel=5)
        want, want_b = eng.perft_position(p, 6), eng.perft_batch(roots, 5)
    with pg.Engine(device=0, use_tt=False, arena_bytes=arena_mb << 20) as eng:
        assert eng.perft_position(p, 6) == want
        assert eng.perft_batch(roots, 5) == want_b


@pytest.mark.gpu
@pytest.mark.parametrize("arena_mb", [48, 192, 2048])
@pytest.mark.parametrize("replace", [1, 2])
def test_folded_table_leaf_is_exact(arena_mb, replace):
    """Table leaf by folding: one chunk, several chunks (192 MB) and an arena
    too small for a chunk (the persistent leaf runs instead); both replacement
    policies; tables full of transpositions, each depth after the others."""
    known = {pg.START_FEN: 119060324, FENS[0]: 8031647685, FENS[1]: 11030083}
    with pg.Engine(device=0, use_tt=True, arena_bytes=arena_mb << 20, device_tt_mb=2048, host_tt_mb=64) as eng:
        eng.set_tuning(tt_replace=replace)
        for fen, want in known.items():
            p = pg.parse_fen(fen)
            for _ in range(2):  # cold and warm tables
                assert eng.perft_position(p, 6) == want
        # a perft-3 call per child: leaves of one partial warp
        kids = [pg.make_move(pg.parse_fen(FENS[0]), m) for m in pg.generate_moves(pg.parse_fen(FENS[0]))]
        assert sum(eng.perft_position(k, 3) for k in kids) == 4085603
