"""En-passant captures that uncover a slider behind the captured pawn.  No game
reaches such a position, but FENs describe it, the generator makes the capture
(as the reference does), the capturing side's king is then in check with the
other side to move, and may be captured: the side without a king has no moves.
Counts against the oracle."""
import random

import pytest

import perft_gpu_2026_b200 as pg

FENS = [
    "1b6/5k2/8/4pP2/5K2/8/8/8 w - e6 0 1",  # the pawn gives check, a bishop stands behind it
    "8/1b3k2/8/3pP3/8/5K2/8/8 w - d6 0 1",  # no check before the capture
    "3r4/5k2/8/3pP3/8/3K4/8/8 w - d6 0 1",  # a rook on the file
    "8/8/5k2/8/3Pp3/8/1B3K2/8 b - d3 0 1",  # black captures
    "q7/5k2/8/3pP1B1/1P6/5K2/2B5/8 w - d6 0 1",
    "r3k2r/1b6/8/3pP3/8/5K2/PP4PP/RN4NR w kq - 0 1",  # the same without the square: nothing uncovered
    "r3k2r/1b6/8/3pP3/8/5K2/PP4PP/RN4NR w kq d6 0 1",
]


def king(p, color):
    occ = p.bb[1] | p.bb[2] | p.bb[3]
    return p.bb[2] & p.bb[3] & ~p.bb[1] & (p.bb[0] if color else occ & ~p.bb[0])


def kingless(p):
    """Positions two moves on whose side to move has lost its king."""
    out = []
    for m in pg.generate_moves(p):
        q = pg.make_move(p, m)
        for r in (pg.make_move(q, k) for k in pg.generate_moves(q)):
            if not king(r, r.color):
                out.append(r)
    return out


def drawn(n, seed):
    """FENs of random placements with such a capture, either colour to move."""
    rng, out = random.Random(seed), []
    while len(out) < n:
        board, c, f = {}, rng.randrange(2), rng.randrange(8)
        g = f + rng.choice((-1, 1))
        if not 0 <= g < 8:
            continue
        victim, taker = (32 + f, 32 + g) if c == 0 else (24 + f, 24 + g)
        board[victim], board[taker] = "pP"[c], "Pp"[c]
        keep = {victim + (8 if c == 0 else -8), victim + (16 if c == 0 else -16)}
        for piece in ["K", "k", rng.choice("bqr" if c == 0 else "BQR")] + rng.sample("NRBQPPnrbqpp", rng.randrange(8)):
            sq = rng.randrange(64)
            if sq not in board and sq not in keep and not (piece in "Pp" and sq // 8 in (0, 7)):
                board[sq] = piece
        rows = []
        for r in range(7, -1, -1):
            rows.append("".join(board.get(8 * r + k, "1") for k in range(8)))
        fen = "/".join(rows) + (" w" if c == 0 else " b") + " - " + "abcdefgh"[f] + ("6" if c == 0 else "3") + " 0 1"
        try:
            p = pg.parse_fen(fen)
        except pg.PerftError:
            continue
        if kingless(p):
            out.append(fen)
    return out


@pytest.mark.parametrize("strict", [False, True])
def test_host_counts_match_oracle(strict, oracle):
    eng = pg.Engine(device=-1, strict=strict)
    for fen in FENS:
        for d in (1, 2, 3, 4):
            assert eng.perft_cpu(pg.parse_fen(fen), d) == oracle.perft(fen, d, strict), (fen, d)
    for fen in drawn(40, seed=3):
        for d in (2, 3):
            assert eng.perft_cpu(pg.parse_fen(fen), d) == oracle.perft(fen, d, strict), (fen, d)


def test_side_without_king_has_no_moves():
    found = 0
    for fen in FENS + drawn(20, seed=4):
        for p in kingless(pg.parse_fen(fen)):
            found += 1
            assert pg.generate_moves(p) == [] and pg.count_moves(p) == 0 and pg.count_moves(p, strict=True) == 0
    assert found > 20


def test_folded_counts_of_a_king_left_in_check():
    """Folding starts from the position with no check on the side that has just
    moved; here it is in check."""
    # perft 2 of the child after f5e6: black to move, the bishop on b8 checks f4
    p = pg.parse_fen(FENS[0])
    child = next(q for q in (pg.make_move(p, m) for m in pg.generate_moves(p))
                 if pg.to_fen(q).startswith("1b6/5k2/4P3/8/5K2"))
    assert sum(pg.count_moves(pg.make_move(child, m)) for m in pg.generate_moves(child)) == 43
    checked, made, bad = pg.selftest_fold([child])
    assert bad == 0 and made == checked
    # such children, what follows them, and their neighbours
    positions = []
    for fen in FENS + drawn(60, seed=5):
        for q in (pg.make_move(pg.parse_fen(fen), m) for m in pg.generate_moves(pg.parse_fen(fen))):
            positions.append(q)
            positions += [pg.make_move(q, m) for m in pg.generate_moves(q)]
    checked, made, bad = pg.selftest_fold(positions)
    assert bad == 0 and checked > 100000


@pytest.mark.gpu
@pytest.mark.parametrize("strict", [False, True])
def test_every_path_matches_oracle(strict, oracle):
    """The same positions through the small kernels, the folded leaf (a batch of
    more than 8,192 leaf edges), the table leaf, the listed leaf and the host."""
    fens = FENS + drawn(24, seed=6)
    roots = [pg.parse_fen(f) for f in fens]
    want = {d: [oracle.perft(f, d, strict) for f in fens] for d in (3, 4)}
    with pg.Engine(device=0, use_tt=False, strict=strict, arena_bytes=1 << 30) as eng:
        for leaf in (6, 5):
            eng.set_tuning(leaf_kernel=leaf)
            for d in (3, 4):
                assert [eng.perft_position(p, d) for p in roots] == want[d], (leaf, d)
                many = roots * 40
                assert eng.perft_batch(many, d) == want[d] * 40, (leaf, d)
                assert eng.last_stats().leaf_edges > 8192
    with pg.Engine(device=0, use_tt=True, strict=strict, arena_bytes=1 << 30, device_tt_mb=1024, host_tt_mb=64) as eng:
        for d in (3, 4):
            for _ in range(2):
                assert [eng.perft_position(p, d) for p in roots] == want[d], d
    deep = [p for p, w in zip(roots, want[4]) if w < 200000]
    assert len(deep) > 3
    with pg.Engine(device=0, use_tt=True, strict=strict, arena_bytes=1 << 30, device_tt_mb=1024, host_tt_mb=64) as eng:
        for p in deep:  # a king captured above the leaf
            assert eng.perft_position(p, 5) == oracle.perft(pg.to_fen(p), 5, strict)
