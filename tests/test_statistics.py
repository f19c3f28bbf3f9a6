"""What last_stats() says was launched and copied."""
import pytest

import perft_gpu_2026_b200 as pg

pytestmark = pytest.mark.gpu


def up(b):
    return (b + 255) // 256 * 256


def test_launches_and_bytes_of_single_positions():
    p = pg.parse_fen(pg.START_FEN)
    uploaded = 3 * 256 + 20 * 4  # board, state and moves at multiples of 256 bytes, parent indices
    with pg.Engine(device=0, use_tt=False, arena_bytes=4 << 30) as eng:
        # whole levels up to 8,192 positions, three kernels for larger ones; the
        # folded leaf is two kernels (this arena's queue takes 8 M edges in one
        # chunk), the small one and the listed one are one
        for depth, launches in ((3, 1), (4, 2), (5, 1 + 1 + 2), (6, 2 + 3 + 2), (7, 2 + 2 * 3 + 2)):
            eng.perft_position(p, depth)
            st = eng.last_stats()
            assert (st.launches, st.kernels, st.leaf_reruns) == (launches, 3 * st.levels + 1, 0), depth
            assert st.h2d_bytes == uploaded and st.d2h_bytes % 256 == 0, depth
        eng.set_tuning(leaf_kernel=5)
        eng.perft_position(p, 6)
        assert eng.last_stats().launches == 2 + 3 + 1


@pytest.mark.parametrize("n", [200, 9000])
def test_launches_and_bytes_of_batches(n):
    roots = pg.random_playouts(5, n, 4, 20, packed=True)
    with pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30) as eng:
        eng.perft_batch(roots, 3)
        st = eng.last_stats()
        small = n <= 8192
        edges = sum(pg.count_moves(r, True) for r in roots)
        assert st.launches == (1 if small else 3) + (1 if edges <= 8192 else 2)
        assert st.h2d_bytes == (up(32 * n) + n if small else 37 * n)
        assert st.d2h_bytes == 8 * n + 2 * 256


def test_launches_of_tables_and_planned_batches():
    p = pg.parse_fen(pg.START_FEN)
    with pg.Engine(device=0, use_tt=True, arena_bytes=1 << 30, device_tt_mb=512, host_tt_mb=64) as eng:
        assert eng.perft_position(p, 5) == 4865609
        # two levels of four kernels and a generation, a chunk of the folded table
        # leaf, two upsweeps of two, the roots' upsweep
        assert eng.last_stats().launches == 2 * 5 + 5 + 2 * 2 + 1
    with pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30) as eng:
        eng.mlp_init(seed=5, out_bias=[5.5, 11.0, 16.5, 22.0])
        params = eng.mlp_params()
        params[:-4] = 0.0
        eng.mlp_set_params(params)
        roots = pg.random_playouts(5, 500, 4, 20, packed=True)
        for _ in range(2):  # captured, then run again
            _, st = eng.perft_batch_planned(roots, 4)
            assert st.graph_batches == 1 and eng.last_stats().launches == 4 + 3 + 2
