"""Positions with more than 256 moves (a FEN with two dozen queens): no game has
them, parse_fen takes them, and every list of moves on the default path is long
enough or read in rounds."""
import pytest

import perft_gpu_2026_b200 as pg

QUEENS = "knQQQQQQ/nnQ4Q/QQ5Q/Q6Q/Q6Q/Q6Q/Q6Q/QQQQQQQK"
WHITE = QUEENS + " w - - 0 1"
BLACK = QUEENS + " b - - 0 1"
RAYS = [(1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (1, -1), (-1, 1), (-1, -1)]


def moves_of_white(p):
    """White's moves by walking rays: queens and the king; nothing of White's is
    pinned and the king is not in check."""
    white = (p.bb[1] | p.bb[2] | p.bb[3]) & ~p.bb[0]
    king = p.bb[2] & p.bb[3] & ~p.bb[1] & white
    knights = p.bb[2] & ~p.bb[1] & ~p.bb[3] & p.bb[0]
    guarded = 0
    for s in range(64):
        if knights >> s & 1:
            for dx, dy in ((1, 2), (2, 1), (-1, 2), (-2, 1), (1, -2), (2, -1), (-1, -2), (-2, -1)):
                x, y = s % 8 + dx, s // 8 + dy
                if 0 <= x < 8 and 0 <= y < 8:
                    guarded |= 1 << (8 * y + x)
    out = []
    for s in range(64):
        if not white >> s & 1:
            continue
        for dx, dy in RAYS:
            x, y = s % 8 + dx, s // 8 + dy
            while 0 <= x < 8 and 0 <= y < 8:
                t = 8 * y + x
                if white >> t & 1:
                    break
                if not king >> s & 1 or not guarded >> t & 1:
                    out.append(t << 6 | s)
                if p.bb[0] >> t & 1 or king >> s & 1:
                    break
                x, y = x + dx, y + dy
    return out


def perft2(p):
    return sum(pg.count_moves(pg.make_move(p, m)) for m in moves_of_white(p))


def test_host_path():
    p = pg.parse_fen(WHITE)
    mv = moves_of_white(p)
    assert len(mv) == pg.count_moves(p) > 256
    listed = pg.generate_moves(p)
    assert len(listed) == 256 and set(listed) <= set(mv)  # the buffer's documented size
    eng = pg.Engine(device=-1)
    assert eng.perft_cpu(p, 2) == perft2(p)
    b = pg.parse_fen(BLACK)
    kids = [pg.make_move(b, m) for m in pg.generate_moves(b)]
    assert max(pg.count_moves(k) for k in kids) > 256
    assert eng.perft_cpu(b, 3) == sum(perft2(k) for k in kids)


@pytest.mark.gpu
def test_small_leaf_lists_in_rounds():
    b = pg.parse_fen(BLACK)
    kids = [pg.make_move(b, m) for m in pg.generate_moves(b)]
    want = sum(perft2(k) for k in kids)
    with pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30) as eng:
        assert eng.perft_position(b, 3) == want
        assert eng.last_stats().leaf_positions == sum(pg.count_moves(k) for k in kids)


@pytest.mark.gpu
def test_levels_of_long_lists():
    p = pg.parse_fen(WHITE)
    with pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30) as eng:
        assert eng.perft_batch([p], 2) == [perft2(p)]


@pytest.mark.gpu
@pytest.mark.parametrize("use_tt", [False, True])
def test_every_path(use_tt):
    p, b, start = pg.parse_fen(WHITE), pg.parse_fen(BLACK), pg.parse_fen(pg.START_FEN)
    cpu = pg.Engine(device=-1)
    w3, b3, b4 = cpu.perft_cpu(p, 3), cpu.perft_cpu(b, 3), cpu.perft_cpu(b, 4)
    with pg.Engine(device=0, use_tt=use_tt, arena_bytes=1 << 30, device_tt_mb=512, host_tt_mb=64) as eng:
        assert eng.perft_position(p, 3) == w3  # the root's list
        assert eng.perft_position(b, 4) == b4  # the level whose size the host does not read
        assert eng.perft_batch([p] * 3 + [b] * 3 + [start], 3) == [w3] * 3 + [b3] * 3 + [8902]
        assert eng.perft_batch([b] * 2500, 3) == [b3] * 2500  # more than 8,192 edges: the folded leaf
        assert eng.perft_position(start, 5) == 4865609


@pytest.mark.gpu
@pytest.mark.parametrize("leaf", [1, 2, 3, 4, 5])
def test_leaf_kernels_that_list_moves(leaf):
    """Among other positions, so that warps and CTAs hold both."""
    b, start = pg.parse_fen(BLACK), pg.parse_fen(pg.START_FEN)
    b3 = pg.Engine(device=-1).perft_cpu(b, 3)
    with pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30) as eng:
        eng.set_tuning(leaf_kernel=leaf)
        assert eng.perft_position(b, 3) == b3
        assert eng.perft_batch([b, start] * 200, 3) == [b3, 8902] * 200
        eng.mlp_init(seed=5, out_bias=[5.5, 11.0, 16.5, 22.0])
        params = eng.mlp_params()
        params[:-4] = 0.0
        eng.mlp_set_params(params)
        for planned in (1, 2):
            eng.set_tuning(planned_leaf=planned)
            got, st = eng.perft_batch_planned([b, start] * 200, 3)
            assert got == [b3, 8902] * 200 and st.graph_batches == 1 and st.retries == 0
    for tt_leaf in (1, 2):
        with pg.Engine(device=0, use_tt=True, arena_bytes=1 << 30, device_tt_mb=512, host_tt_mb=64) as eng:
            eng.set_tuning(leaf_kernel=leaf, tt_leaf=tt_leaf)
            for _ in range(2):
                assert eng.perft_position(b, 3) == b3 and eng.perft_position(start, 5) == 4865609
