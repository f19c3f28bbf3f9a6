// pb_wide.cuh - level and leaf kernels for small levels: one warp per position.
//
// With a few thousand positions one thread each leaves the GPU idle and a
// kernel lasts as long as one thread's serial work, whatever the size: make+count
// 13 us, scan 4, generation 19-30, the folded leaf and its queue 33 + 14.  Here a
// warp shares a position: every lane computes what the side's legality needs,
// then takes the pieces on its two squares; a leaf's lanes then count one
// grandchild each.  That costs several times the instructions per position, so
// the driver uses it up to WIDE_MAX positions only.  A level is one kernel with
// no scan, and where the next one is the leaf of a small tree the host does not
// wait in between.  Measured on B200 at perft 4 of a 20-ply playout (29
// positions, 980 edges): level 36 -> 9 us, leaf 47 -> 15 us, the whole call 115
// -> 41 us (with the uploads and readbacks in one copy each).
#pragma once
#include "pb_core.cuh"
#include "pb_kernels.cuh"

namespace pb {

constexpr int WIDE_WARPS = 4;         // warps per CTA
constexpr int WIDE_LEVEL_WARPS = 16;  // of a level of more than WIDE_SMALL positions
constexpr u32 WIDE_SMALL = 1024;

// What the legal moves of side C depend on besides the piece.
template <int C> struct MovePrep {
    Sets s;
    u64 pinned, threat, safe, ep_from, ep_to;  // ep_from: pawns that may take en passant
    int ksq;
    bool check, only_king;
};
template <int C> PB_HD MovePrep<C> move_prep(const Board &b, u32 st)
{
    MovePrep<C> p;
    p.s = derive<C>(b);
    const Sets &s = p.s;
    const u64 king = s.kings & s.us;
    p.ksq = bit_index(king);
    p.pinned = pinned_set(p.ksq, s.bq & s.them, s.rq & s.them, s.occ);
    p.threat = enemy_attacks<C>(s, king, p.ksq);
    p.check = king_in_check(king, p.threat);
    p.only_king = false;
    p.safe = ~0ULL;
    u64 checkers = 0;
    if (p.check) {
        checkers = (cap_west<C>(king) | cap_east<C>(king)) & s.pawns & s.them;
        checkers |= knight_att(p.ksq) & s.knights & s.them;
        checkers |= bishop_att(p.ksq, s.occ) & s.bq & s.them;
        checkers |= rook_att(p.ksq, s.occ) & s.rq & s.them;
        p.only_king = more_than_one(checkers);
        p.safe = checkers | between(p.ksq, bit_index(checkers));
    }
    p.ep_from = 0;
    p.ep_to = ep_target<C>(st);
    if (p.ep_to) {
        const u64 victim = push1<1 - C>(p.ep_to);
        if (!p.check || victim == checkers)
            for (u64 src = (east1(victim) | west1(victim)) & s.pawns & s.us; src; src &= src - 1) {
                const u64 pawn = src & (0 - src);
                bool ok;
                if (p.check)
                    ok = !(pawn & p.pinned);
                else if (pawn & p.pinned)
                    ok = (p.ep_to & line_through(lsb(src), p.ksq)) != 0;
                else
                    ok = !(rook_att(p.ksq, s.occ ^ victim ^ pawn) & s.rq & s.them & (RANK1 << (p.ksq & 56)));
                if (ok) p.ep_from |= pawn;
            }
    }
    return p;
}

// Legal targets of the piece on `sq` (0 if it is not side C's); castling as the
// king's square two files aside, en passant as the pawn's target.
template <int C> PB_HD u64 piece_targets(const MovePrep<C> &p, u32 st, int sq)
{
    const Sets &s = p.s;
    const u64 bit = 1ULL << sq;
    if (!(bit & s.us)) return 0;
    if (bit & s.kings) {
        u64 t = king_att(sq) & ~(p.threat | s.us);
        const u32 castle = C == WHITE ? (st & 3) : ((st >> 2) & 3);
        if (castle && !p.check) {
            constexpr u64 KS = C == WHITE ? 0x60ULL : 0x6000000000000000ULL;
            constexpr u64 QS_EMPTY = C == WHITE ? 0x0EULL : 0x0E00000000000000ULL;
            constexpr u64 QS_SAFE = C == WHITE ? 0x0CULL : 0x0C00000000000000ULL;
            constexpr int K0 = C == WHITE ? 4 : 60;
            if ((castle & 1) && !(KS & (s.occ | p.threat))) t |= 1ULL << (K0 + 2);
            if ((castle & 2) && !(QS_EMPTY & s.occ) && !(QS_SAFE & p.threat)) t |= 1ULL << (K0 - 2);
        }
        return t;
    }
    const bool pin = (bit & p.pinned) != 0;
    if (p.only_king || (pin && p.check)) return 0;
    u64 t;
    if (bit & s.pawns) {
        const u64 d = push1<C>(bit) & ~s.occ;
        t = d | (push1<C>(d & double_push_rank<C>()) & ~s.occ) | ((cap_west<C>(bit) | cap_east<C>(bit)) & s.them);
    } else if (bit & s.knights) {
        t = knight_att(sq);
    } else {
        t = bit & s.bq ? bishop_att(sq, s.occ) : 0;
        if (bit & s.rq) t |= rook_att(sq, s.occ);
    }
    t &= ~s.us & p.safe;
    if (pin) t &= line_through(sq, p.ksq);
    if (bit & p.ep_from) t |= p.ep_to;
    return t;
}

// Moves of a piece with targets t: one per target, four per promotion.
template <int C> PB_HD int move_count(const MovePrep<C> &p, int sq, u64 t)
{
    return popc(t) + ((1ULL << sq) & p.s.pawns ? 3 * popc(t & PROMO_RANKS) : 0);
}
template <int C, class Put> PB_HD void put_moves(const MovePrep<C> &p, int sq, u64 t, Put put)
{
    const u64 bit = 1ULL << sq;
    const bool pawn = (bit & p.s.pawns) != 0, king = (bit & p.s.kings) != 0;
    for (; t; t &= t - 1) {
        const int to = lsb(t);
        const u64 tb = t & (0 - t);
        int flags = MF_QUIET;
        if (pawn) {
            if (tb & PROMO_RANKS) {
                for (int k = 0; k < 4; k++) put(make_move_code(sq, to, MF_PROMO + k));
                continue;
            }
            if (tb == p.ep_to && (bit & p.ep_from))
                flags = MF_EP;
            else if ((to - sq == 16 || sq - to == 16) && ((east1(tb) | west1(tb)) & p.s.pawns & p.s.them))
                flags = MF_DOUBLE_PUSH;
        } else if (king) {
            flags = to - sq == 2 ? MF_KING_CASTLE : sq - to == 2 ? MF_QUEEN_CASTLE : MF_QUIET;
        }
        put(make_move_code(sq, to, flags));
    }
}

// The warp's position `b` (the same in every lane): this lane's two squares'
// targets, its first move's place in the position's list; returns their number.
template <int C>
__device__ __forceinline__ int warp_targets(const MovePrep<C> &p, u32 st, u64 (&t)[2], int *at)
{
    const int lane = threadIdx.x & 31;
    int n = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        t[h] = piece_targets<C>(p, st, lane + 32 * h);
        n += move_count<C>(p, lane + 32 * h, t[h]);
    }
    int x = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    *at = x - n;
    return __shfl_sync(0xffffffffu, x, 31);
}

// A whole small level in one kernel: makes the children of n edges (or, without
// EDGES, takes n positions as they are), stores them and appends their moves to
// the next level's edges.  A CTA's positions take their place from *total in
// one piece, in order; the order of the pieces varies from run to run, and no
// result depends on it.  `cap` edges have room, n * MAX_MOVES; positions past that
// set the error word and the driver takes the kernels with exact sizes.  The
// next kernels read sibling edges in neighbouring threads, so the larger levels
// use pieces of W = 16 positions (200 roots at perft 4: the folded leaf ran 78 us
// on ordered edges, 100 on pieces of one position); the smallest use more CTAs.
template <int C, bool EDGES, bool ROOTED, int W>
__global__ void __launch_bounds__(32 * W)
    k_level_wide(const Board *__restrict__ pboards, const uint8_t *__restrict__ pstates,
                 const u32 *__restrict__ proot, const u32 *__restrict__ pidx, const uint16_t *__restrict__ moves, u32 n,
                 u64 nparents, Board *__restrict__ cboards, uint8_t *__restrict__ cstates, u32 *__restrict__ croot,
                 uint16_t *__restrict__ out_mv, u32 *__restrict__ out_pi, u64 cap, unsigned long long *__restrict__ total,
                 u32 *__restrict__ err)
{
    __shared__ u32 s_cnt[W];
    __shared__ u64 s_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 i = blockIdx.x * W + warp;
    constexpr int D = EDGES ? 1 - C : C;
    const u32 p = i < n ? (EDGES ? pidx[i] : i) : 0u;
    bool valid = i < n;
    if (valid && p >= nparents) {  // only after a generation mismatch upstream
        if (lane == 0) atomicOr(err, DEVERR_CAPACITY);
        valid = false;
    }
    MovePrep<D> prep;
    u64 t[2];
    int at = 0, cnt = 0;
    if (valid) {
        Board b = load_board(pboards + p);
        u32 st = pstates[p];
        if (EDGES) make_move<C>(b, st, moves[i]);
        if (lane == 0) {
            if (EDGES) {
                store_board(cboards + i, b);
                cstates[i] = (uint8_t)st;
            }
            if (ROOTED) croot[i] = EDGES ? proot[p] : i;
        }
        prep = move_prep<D>(b, st);
        cnt = warp_targets<D>(prep, st, t, &at);
    }
    if (lane == 0) s_cnt[warp] = (u32)cnt;
    __syncthreads();
    u32 before = 0, all = 0;
    for (int w = 0; w < W; w++) {
        if (w < warp) before += s_cnt[w];
        all += s_cnt[w];
    }
    if (threadIdx.x == 0) s_base = all ? atomicAdd(total, (unsigned long long)all) : 0;
    __syncthreads();
    if (!valid) return;
    u64 o = s_base + before;
    if (o + cnt > cap) {
        if (lane == 0) atomicOr(err, DEVERR_CAPACITY);
        return;
    }
    o += at;
#pragma unroll
    for (int h = 0; h < 2; h++)
        put_moves<D>(prep, lane + 32 * h, t[h], [&](uint16_t m) {
            out_mv[o] = m;
            out_pi[o] = i;
            o++;
        });
}

// Fused two-ply leaf: a warp per edge, a lane per grandchild.  With n_dev the
// number of edges is on the device.  72 registers for 28 warps per SM: with the
// rounds the compiler took 128 by itself (4,700 edges 31.5 us, 28.6 with 72; up to
// 2,000 edges, less than a wave, 20.4 either way).
template <int C, bool STRICT, bool ROOTED>
__global__ void __launch_bounds__(32 * WIDE_WARPS, 7)
    k_leaf2_wide(const Board *__restrict__ pboards, const uint8_t *__restrict__ pstates, const u32 *__restrict__ proot,
                 const u32 *__restrict__ pidx, const uint16_t *__restrict__ moves, u32 n,
                 const unsigned long long *__restrict__ n_dev, u64 nparents,
                 unsigned long long *__restrict__ root_counts, unsigned long long *__restrict__ counter)
{
    __shared__ uint16_t s_mv[WIDE_WARPS][MAX_MOVES];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (n_dev) n = (u32)min(*n_dev, (unsigned long long)n);  // a level that ran out of room lists fewer
    for (u32 i = blockIdx.x * WIDE_WARPS + warp; i < n; i += gridDim.x * WIDE_WARPS) {
        const u32 p = pidx[i];
        if (p >= nparents) continue;
        Board b = load_board(pboards + p);
        u32 st = pstates[p];
        make_move<C>(b, st, moves[i]);
        int cnt;
        u32 total = 0;
#pragma unroll 1
        for (int done = 0;; done += MAX_MOVES) {  // once: hardly a position has more
            {
                // what legality needs is computed again in each round
                Board c;
                for (int q = 0; q < 4; q++) c.bb[q] = fresh(b.bb[q]);
                const MovePrep<1 - C> prep = move_prep<1 - C>(c, st);
                u64 t[2];
                int at;
                cnt = warp_targets<1 - C>(prep, st, t, &at);
                at -= done;
#pragma unroll
                for (int h = 0; h < 2; h++)
                    put_moves<1 - C>(prep, lane + 32 * h, t[h], [&](uint16_t m) {
                        if ((u32)at < MAX_MOVES) s_mv[warp][at] = m;
                        at++;
                    });
            }
            __syncwarp();
            const int listed = min(cnt - done, (int)MAX_MOVES);
#pragma unroll 1
            for (int k = lane; k < listed; k += 32) {
                Board g = b;
                u32 gs = st;
                make_move<1 - C>(g, gs, s_mv[warp][k]);
                total += count_moves<C, STRICT>(g, gs);
            }
            if (cnt - done <= MAX_MOVES) break;
            __syncwarp();
        }
        total = __reduce_add_sync(0xffffffffu, total);
        if (lane == 0 && cnt) {
            atomicAdd(ROOTED ? root_counts + proot[p] : counter, (unsigned long long)total);
            atomicAdd(counter + 1, (unsigned long long)cnt);
        }
        __syncwarp();  // the list is free again
    }
}

}  // namespace pb
