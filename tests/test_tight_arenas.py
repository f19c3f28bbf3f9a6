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
