"""Calls in arenas that hold only part of their levels: passes that give up and
the smaller passes that follow them."""
import pytest

import perft_gpu_2026_b200 as pg

pytestmark = pytest.mark.gpu

KIWI = "r3k2r/p1ppqpb1/bn2pnp1/3PN3/1p2P3/2N2Q1p/PPPBBPPP/R3K2R w KQkq - 0 1"


@pytest.fixture(scope="module")
def wanted():
    roots = [pg.parse_fen(f) for f in (pg.START_FEN, KIWI, "8/2p5/3p4/KP5r/1R3p1k/8/4P1P1/8 w - - 0 1")]
    batch = pg.random_playouts(17, 300, 0, 60, packed=True)
    with pg.Engine(device=0, use_tt=False, arena_bytes=2 << 30) as eng:
        return roots, [eng.perft_position(p, 5) for p in roots], batch, eng.perft_batch(batch, 4)


@pytest.mark.parametrize("arena_kb", [8, 16, 64, 256, 512, 1024, 1500, 4096, 20000])
def test_passes_that_give_up_and_their_successors(arena_kb, wanted):
    """Each pass that gives up is followed at once by one on other positions."""
    roots, counts, batch, batch_counts = wanted
    with pg.Engine(device=0, use_tt=False, arena_bytes=arena_kb << 10) as eng:
        assert [eng.perft_position(p, 5) for p in roots] == counts
        if arena_kb >= 64:
            assert eng.perft_batch(batch, 4) == batch_counts


def test_leaf_kernels_need_no_memory_after_creation():
    """The cooperative leaf's spill area is there from the start: a call with it
    takes no device memory."""
    import torch

    torch.cuda.set_device(0)
    p = pg.parse_fen(KIWI)
    with pg.Engine(device=0, use_tt=False, arena_bytes=256 << 20) as eng:
        want = eng.perft_position(p, 5)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info(0)[0]
        eng.set_tuning(leaf_kernel=2)
        assert eng.perft_position(p, 5) == want
        assert free - torch.cuda.mem_get_info(0)[0] < 64 << 20


def exact_bytes(edges, positions):
    """Arena bytes of a call whose levels have `edges` edges and materialise
    `positions` positions, every array of the size it needs (multiples of 256)."""
    up = lambda b: (b + 255) // 256 * 256
    total = 2 * 256 + up(2 * edges[0]) + up(4 * edges[0])
    for n, nxt in zip(positions, edges[1:]):
        total += sum(up(n * k) for k in (32, 1, 4, 8)) + up(8 * ((n + 4095) // 4096 + 1)) + up(2 * nxt) + up(4 * nxt)
    return total


def test_an_arena_of_exact_size_is_enough():
    """The whole-level kernels' wider lists do not make a call split that fits
    without them (perft 7: levels of 20, 400, 8,902, 197,281 and 4,865,609 edges)."""
    edges = [20, 400, 8902, 197281, 4865609]
    p = pg.parse_fen(pg.START_FEN)
    with pg.Engine(device=0, use_tt=False, arena_bytes=exact_bytes(edges, edges[:-1]) + 8192) as eng:
        assert eng.perft_position(p, 7) == 3195901860
        st = eng.last_stats()
        assert st.levels == 4 and list(st.level_sizes[:5]) == edges
        assert eng.perft_batch([p], 7) == [3195901860]
    with pg.Engine(device=0, use_tt=False, arena_bytes=exact_bytes(edges, edges[:-1]) - 65536) as eng:
        assert eng.perft_position(p, 7) == 3195901860
        assert eng.last_stats().levels > 4  # a little less, and it is split


ROOKS = "3qk3/8/8/8/8/8/8/QRBNKBRQ w - - 0 1"
CROWD = "4k3/qqqqqqqq/8/8/8/8/QQQQQQQQ/4K3 w - - 0 1"
QUEENS = "1k6/ppp5/8/1Q1Q1Q1Q/Q1Q1Q1Q1/1Q1Q1Q1Q/Q1Q1Q1Q1/K7 b - - 0 1"


@pytest.mark.parametrize("fen,depth", [(KIWI, 5), (ROOKS, 6)])
@pytest.mark.parametrize("room_mb", [1, 4, 8.25, 64])
def test_short_queues_do_not_make_tiny_chunks(fen, depth, room_mb):
    """An arena with `room_mb` left for the folded leaf's queue: chunks of 64 K
    edges at least, or the listed leaf."""
    p = pg.parse_fen(fen)
    with pg.Engine(device=0, use_tt=False, arena_bytes=2 << 30) as eng:
        want = eng.perft_position(p, depth)
        st = eng.last_stats()
        edges = list(st.level_sizes[:st.levels + 1])
    with pg.Engine(device=0, use_tt=False, arena_bytes=exact_bytes(edges, edges[:-1]) + int(room_mb * (1 << 20))) as eng:
        assert eng.perft_position(p, depth) == want
        st = eng.last_stats()
        assert list(st.level_sizes[:st.levels + 1]) == edges
        # levels (twice, where the whole-level kernels' lists left too little
        # room), chunks, and a leaf counted again
        assert st.launches <= 2 * 3 * st.levels + 2 * (2 * (edges[-1] // 65536 + 1) + 1)


def test_queue_too_short_in_a_single_position():
    """Room for 16 to 20 queued moves per edge where a sample of them queues 23:
    the leaf runs again."""
    p = pg.parse_fen(CROWD)
    kids = [pg.make_move(p, m) for m in pg.generate_moves(p)]
    leaves = pg.pack_positions([pg.make_move(k, m) for k in kids for m in pg.generate_moves(k)])
    _, made, bad = pg.selftest_fold(leaves)
    queued, n = made // 2, len(leaves)  # both conventions
    assert bad == 0 and n > 8192 and queued > 21 * n
    with pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30) as eng:
        want = eng.perft_position(p, 4)
        st = eng.last_stats()
        assert st.leaf_edges == n and st.leaf_reruns == 0
        counted = st.leaf_positions
    arena = exact_bytes([len(kids), n], [len(kids)]) + 8 * 18 * n
    with pg.Engine(device=0, use_tt=False, arena_bytes=arena) as eng:
        for _ in range(2):
            assert eng.perft_position(p, 4) == want
            st = eng.last_stats()
            assert st.leaf_reruns == 1 and st.leaf_positions == counted


@pytest.mark.parametrize("n,arena_mb", [
    (2000, 3),      # 350 K items for 12,000 edges that queue 57 each: then the listed leaf
    (175000, 160),  # 17.9 M items for 1.05 M edges: then chunks of 70 K edges that always fit
])
def test_queue_too_short_in_a_batch(n, arena_mb):
    roots = [pg.parse_fen(QUEENS), pg.parse_fen(KIWI)]
    with pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30) as eng:
        want = [eng.perft_position(r, 3) for r in roots]
    batch = pg.pack_positions([roots[0]] * (n - 2) + [roots[1], roots[0]])
    with pg.Engine(device=0, use_tt=False, arena_bytes=arena_mb << 20) as eng:
        assert eng.perft_batch(batch, 3) == [want[0]] * (n - 2) + [want[1], want[0]]
        assert eng.last_stats().leaf_reruns == 1


def test_queue_too_short_in_a_planned_batch():
    """12,000 edges that queue 57 moves each, a planned leaf of 22 K edges at 16
    to 30: the plan counts as outgrown and the batch runs exactly."""
    root = pg.parse_fen(QUEENS)
    with pg.Engine(device=0, use_tt=False, arena_bytes=1 << 30) as eng:
        want = eng.perft_position(root, 3)
    with pg.Engine(device=0, use_tt=False, arena_bytes=5 << 20) as eng:
        eng.mlp_init(seed=5, out_bias=[3.0, 9.0, 13.0, 18.0])
        params = eng.mlp_params()
        params[:-4] = 0.0
        eng.mlp_set_params(params)
        for _ in range(2):
            got, st = eng.perft_batch_planned([root] * 2000, 3)
            assert got == [want] * 2000 and st.graph_batches == 1 and st.retries == 1
