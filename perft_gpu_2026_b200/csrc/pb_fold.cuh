// pb_fold.cuh - perft(2) of a position without making most of its moves.
//
// The sum over a position's moves of the opponent's move counts is dominated
// by moves after which the opponent's count differs from a common base by a
// few terms that depend only on the squares left and entered.  fold_child
// sums those moves by set arithmetic and hands the rest to a sink, move by
// move, to be made and counted in full (count_moves).
//
// X moves, Y = 1 - X is counted.  The base is Y's move count in the position
// as it stands (no en passant).  Two sets of squares matter: the core, which is
// Y's king and the safe squares of a castling whose path has no Y piece, and
// the ring, the squares next to the king without a Y piece.  A move f -> t of
// a piece p is SIMPLE when it leaves Y's castling, pins and checks alone and
// what it does to the king's moves is plain:
//   - p attacks no core square from f or from t; X-rays through Y's first
//     blocker towards the king count as attacks (a slider there would pin);
//   - f is not an X piece that shields a core or ring square from an X slider,
//     nor one of two blockers with a Y piece between an X slider and the king;
//   - t is not on a line from an X slider to a core or ring square it attacks,
//     nor between a pinned Y piece's pinner and the king;
//   - neither f nor t is on such a castling path;
//   - a piece captured on t is not next to the king, pinned, on a castling
//     corner or a pawn about to promote, is not a pawn that bears on f (unless
//     a pawn takes it, where the overlap is one known move), and is not a
//     slider that the king takes;
//   - no en-passant capture of it is in question: each of Y's pawns beside a
//     double push has one, unless one of them is pinned or the king shares
//     their rank.
// After a simple move
//   - Y's pinned-piece and castling moves are as before; its king moves too,
//     unless p attacks ring squares from f or t: those moves are counted again
//     from the ring squares that X then attacks (one lookup per move);
//   - a captured piece's moves are gone; Y's pieces that guarded t take there;
//   - Y's unpinned pawns change by a weight of f plus a weight of t (pushes
//     unblocked and captures lost on f, pushes blocked and captures gained on
//     t), less one if X slides between the two squares in front of an unmoved
//     pawn;
//   - a Y slider that sees t loses the squares beyond t, and one that sees f
//     gains those beyond f; moves of f along that same line, the slider's own
//     capture included, are corrected one by one.
// Weights of t are summed over all simple moves at once: the number of simple
// moves onto each square is kept in bit-sliced planes (at most 16 pieces can
// reach one square: eight lines and eight knight jumps).
//
// All of this counts Y's moves from a position in which Y is not in check.  Y has
// just moved, so it is not, except after an en-passant capture that uncovered its
// king (pb_core.cuh, Tables); there no move is simple.
//
// Promotions, en passant and castling go to the sink.  On the benchmark's leaves
// 2.5 % of the moves do, on middle-game playouts 11 %, late in a game 17 %; with
// pawns next to the ring, captured sliders and double pushes beside a pawn it was
// 4.2 %, 14 % and 21 %, without the recounted king moves 7.5 %, 21 % and 37 %.
// What is left is mostly checks and pins made or lifted.
#pragma once
#include "pb_core.cuh"

namespace pb {

// Values that the loops over X's pieces read seldom: on the GPU one column of
// shared memory per thread, slots `stride` apart.  Register pressure decides how
// many warps an SM holds; left to itself the compiler kept these and spilled
// what every iteration reads.
enum ShelfSlot {
    SHELF_C3,
    SHELF_C4,
    SHELF_THREAT,
    SHELF_MULTI,
    SHELF_THREAT_Y,
    SHELF_MOVED0,
    SHELF_MOVED1,
    SHELF_MOVED2,
    SHELF_NO_EP,
    SHELF_OK_TO,
    SHELF_RING_B,
    SHELF_RING_R,
    SHELF_CORE_B,
    SHELF_CORE_R,
    SHELF_PINNED_Y,
    SHELF_SLOTS
};
struct Shelf {
    volatile u64 *column;
    int stride;
    PB_HD u64 get(int slot) const { return column[slot * stride]; }
    PB_HD void set(int slot, u64 v) const { column[slot * stride] = v; }
};

// Number of simple moves onto each square, bit-sliced.  Eight or more onto one
// square (c3, c4) are rare, so their terms hide behind one test.
struct TargetPlanes {
    Shelf shelf;
    u64 c0 = 0, c1 = 0, c2 = 0;
    bool rare = false;  // c3 and c4 are set
    PB_HD explicit TargetPlanes(Shelf s) : shelf(s) {}
    PB_HD void add(u64 s)
    {
        u64 k = c0 & s;
        c0 ^= s;
        s = c1 & k;
        c1 ^= k;
        k = c2 & s;
        c2 ^= s;
        if (k) {
            if (!rare) {
                rare = true;
                shelf.set(SHELF_C3, k);
                shelf.set(SHELF_C4, 0);
            } else {
                const u64 c3 = shelf.get(SHELF_C3);
                shelf.set(SHELF_C4, shelf.get(SHELF_C4) | (c3 & k));
                shelf.set(SHELF_C3, c3 ^ k);
            }
        }
    }
    PB_HD u64 c3() const { return shelf.get(SHELF_C3); }
    PB_HD u64 c4() const { return shelf.get(SHELF_C4); }
    PB_HD int sum(u64 m) const
    {
        int n = popc(c0 & m) + 2 * popc(c1 & m) + 4 * popc(c2 & m);
        if (rare) n += 8 * popc(c3() & m) + 16 * popc(c4() & m);
        return n;
    }
    PB_HD u64 any() const { return c0 | c1 | c2 | (rare ? c3() | c4() : 0); }
    PB_HD int at(u64 bit) const
    {
        int n = (c0 & bit ? 1 : 0) + (c1 & bit ? 2 : 0) + (c2 & bit ? 4 : 0);
        if (rare) n += (c3() & bit ? 8 : 0) + (c4() & bit ? 16 : 0);
        return n;
    }
};

PB_HD u64 beyond(int s, int t) { return ldg64(&PB_TAB.beyond[s][t]); }

// What Y's unpinned pawns `fp` add to its count, by square: pushes (p1 single,
// dbl double), captures (cw, cc: squares attacked; on the promotion rank a
// square counts once unless STRICT).  And what an X piece that leaves f gives
// back: m1 a push, m2 the double push behind it too, m3 a double push.
template <int Y, bool STRICT>
struct PawnTerms {
    static constexpr u64 DP = Y == WHITE ? RANK3 : RANK6;
    u64 p1, dbl, cw, cc, m1, m2, m3;
    PB_HD PawnTerms(u64 fp, u64 us, u64 empty)
    {
        const u64 pu = push1<Y>(fp);
        p1 = pu & empty;
        const u64 dreach = push1<Y>(p1 & DP), ce = cap_east<Y>(fp);
        dbl = dreach & empty;
        cw = cap_west<Y>(fp);
        cc = STRICT ? ce : ce & ~(cw & PROMO_RANKS);
        m1 = pu & us;
        m2 = m1 & DP & push1<1 - Y>(empty);
        m3 = dreach & us;
    }
    // weight of leaving the square `fb`
    PB_HD int leave(u64 fb) const
    {
        const int g = (fb & m1 ? 1 : 0) + (fb & m2 ? 1 : 0) + (fb & m3 ? 1 : 0) - (fb & cw ? 1 : 0) - (fb & cc ? 1 : 0);
        return fb & PROMO_RANKS ? 4 * g : g;
    }
};

// Sink: set(from, targets) takes the moves from -> t of one piece (flags 0),
// one(move, promotes) one move, or with `promotes` the four promotions.
// Returns the simple moves' sum of counts; *simple = how many they are.
#ifdef __CUDACC__
#pragma nv_exec_check_disable  // the self-test's sink runs on the host
#endif
template <int X, bool STRICT, class Sink>
PB_HD u32 fold_child(const Board &b, u32 st, Sink &sink, u32 *simple, Shelf shelf)
{
    constexpr int Y = 1 - X;
    constexpr u64 KS_X = X == WHITE ? 0x60ULL : 0x6000000000000000ULL;
    constexpr u64 QE_X = X == WHITE ? 0x0EULL : 0x0E00000000000000ULL;
    constexpr u64 QS_X = X == WHITE ? 0x0CULL : 0x0C00000000000000ULL;
    constexpr u64 KS_Y = Y == WHITE ? 0x60ULL : 0x6000000000000000ULL;
    constexpr u64 QE_Y = Y == WHITE ? 0x0EULL : 0x0E00000000000000ULL;
    constexpr u64 QS_Y = Y == WHITE ? 0x0CULL : 0x0C00000000000000ULL;
    constexpr u64 DP_X = X == WHITE ? RANK3 : RANK6;
    constexpr u64 DP_Y = Y == WHITE ? RANK3 : RANK6;
    constexpr u64 CORNERS_Y = Y == WHITE ? 0x81ULL : 0x8100000000000000ULL;
    constexpr u64 RANK7_Y = Y == WHITE ? 0x00FF000000000000ULL : 0x000000000000FF00ULL;
    const Sets s = derive<X>(b);
    const u64 us = s.us, them = s.them, occ = s.occ, empty = ~occ;
    const u64 xkb = s.kings & us, ykb = s.kings & them;
    const int xk = bit_index(xkb), yk = bit_index(ykb);
    const u64 bqX = s.bq & us, rqX = s.rq & us;

    // ---- Y's zone and what in X's position bears on it
    const u64 ring = king_att(yk) & ~them;
    u64 core = ykb, path = 0;  // the king and the safe squares of an open castling
    const u32 castle_y = Y == WHITE ? (st & 3) : ((st >> 2) & 3);
    if (castle_y) {
        if ((castle_y & 1) && !(KS_Y & them)) path |= KS_Y, core |= KS_Y;
        if ((castle_y & 2) && !(QE_Y & them)) path |= QE_Y, core |= QS_Y;
    }
    u64 core_b, core_r;             // squares from which a diagonal / orthogonal slider bears on the core
    u64 ring_b = 0, ring_r = 0;     // ... on the ring
    u64 keep = path, lines = path;  // squares no simple move leaves / enters
    u64 pinned_y = 0;
    u64 threat, multi;              // squares X attacks / attacks more than once, exact on the zone
    {
        u64 one = cap_west<X>(s.pawns & us), two, q = cap_east<X>(s.pawns & us);
        two = one & q;
        one |= q;
        q = king_att(xk);
        two |= one & q;
        one |= q;
        for (u64 kn = s.knights & us; kn; kn &= kn - 1) {
            q = knight_att(lsb(kn));
            two |= one & q;
            one |= q;
        }
        threat = one;
        multi = two;
    }
    {
        u64 a = bishop_att(yk, occ), checkers_y = (threat & ykb) | (a & bqX);
        core_b = a | bishop_att(yk, occ & ~(a & them));
        a = rook_att(yk, occ);
        checkers_y |= a & rqX;
        core_r = a | rook_att(yk, occ & ~(a & them));
        if (checkers_y) lines = ~0ULL;  // Y in check
    }
    for (u64 sn = (bishop_empty(yk) & bqX) | (rook_empty(yk) & rqX); sn; sn &= sn - 1) {
        const u64 bw = between(lsb(sn), yk), bt = bw & occ, rest = bt & (bt - 1);
        if (!rest) {
            if (bt & them)
                pinned_y |= bt, lines |= bw;
            else
                keep |= bt;
        } else if (!more_than_one(rest) && (bt & them)) {
            keep |= bt & us;
        }
    }
    const u64 occ_k = occ ^ ykb;
    for (u64 z = (ring | core) & ~ykb; z; z &= z - 1) {
        const int q = lsb(z);
        const u64 zb = z & (0 - z);
        const u64 a = bishop_att(q, occ_k), c = rook_att(q, occ_k);
        if (zb & core)
            core_b |= a, core_r |= c;
        else
            ring_b |= a, ring_r |= c;
        const u64 attackers = (a & bqX) | (c & rqX);
        if (attackers) {
            multi |= zb & (more_than_one(attackers) ? ~0ULL : threat);
            threat |= zb;
        }
        for (u64 t = (bishop_empty(q) & bqX) | (rook_empty(q) & rqX); t; t &= t - 1) {
            const u64 bw = between(lsb(t), q), bt = bw & occ_k;
            if (!bt)
                lines |= bw;
            else if (!more_than_one(bt))
                keep |= bt & us;
        }
    }

    // ---- X's legality
    const u64 pinned_x = pinned_set(xk, s.bq & them, s.rq & them, occ);
    const u64 threat_y = enemy_attacks<X>(s, xkb, xk);
    u64 safe = ~0ULL, checkers = 0, mine = us;
    if (king_in_check(xkb, threat_y)) {
        checkers = (cap_west<X>(xkb) | cap_east<X>(xkb)) & s.pawns & them;
        checkers |= knight_att(xk) & s.knights & them;
        checkers |= bishop_att(xk, occ) & s.bq & them;
        checkers |= rook_att(xk, occ) & s.rq & them;
        safe = checkers | between(xk, bit_index(checkers));
        mine = us & ~pinned_x;
        if (more_than_one(checkers)) mine = xkb;
    }

    // ---- Y's base count without its sliders (added with their terms below)
    const int kings = popc(ring & ~threat);
    u32 base = kings;
    if (castle_y) {
        if ((castle_y & 1) && !(KS_Y & (occ | threat))) base++;
        if ((castle_y & 2) && !(QE_Y & occ) && !(QS_Y & threat)) base++;
    }
    const u64 fp = s.pawns & them & ~pinned_y;
    const bool promo = (fp & RANK7_Y) != 0;
    u64 weighted;  // X pieces whose leaving changes a pawn term
    {
        const PawnTerms<Y, STRICT> w(fp, us, empty);
        weighted = w.m1 | w.m3 | ((w.cw | w.cc) & us);
    }
    // captured pieces whose loss is no simple term: next to the king, pinned,
    // a castling rook, a pawn about to promote
    const u64 no_cap = king_att(yk) | pinned_y | (castle_y ? CORNERS_Y : 0ULL) | (promo ? fp & RANK7_Y : 0ULL);
    const u64 bY = s.bq & them & ~pinned_y, rY = s.rq & them & ~pinned_y;
    const u64 stay = lines | (them & no_cap);  // squares no simple move enters
    if (pinned_y & ~s.knights) {
        // pinned pawns and sliders: along the line through the king
        for (u64 q = pinned_y & ~s.knights; q; q &= q - 1) {
            const int sq = lsb(q);
            const u64 bit = q & (0 - q), ln = line_through(sq, yk);
            if (bit & s.pawns) {
                const u64 d = push1<Y>(bit) & ln & empty;
                if (d) base += 1 + ((push1<Y>(d & DP_Y) & empty) ? 1 : 0);
                const u64 c = (cap_west<Y>(bit) | cap_east<Y>(bit)) & ln & us;
                if (c) base += (c & PROMO_RANKS) ? 4 : 1;
            }
            if (bit & s.bq) base += popc(bishop_att(sq, occ) & ~them & ln);
            if (bit & s.rq) base += popc(rook_att(sq, occ) & ~them & ln);
        }
    }

    // ---- X's moves
    TargetPlanes to(shelf);
    shelf.set(SHELF_PINNED_Y, pinned_y);
    shelf.set(SHELF_CORE_B, core_b);
    shelf.set(SHELF_CORE_R, core_r);
    shelf.set(SHELF_RING_B, ring_b);
    shelf.set(SHELF_RING_R, ring_r);
    shelf.set(SHELF_THREAT, threat);
    shelf.set(SHELF_MULTI, multi);
    shelf.set(SHELF_THREAT_Y, threat_y);
    int corr = 0;
    u32 ns = 0;

    // pawns, by sets of target squares: single and double pushes, captures.
    // moved0..2: the number of simple moves of each pawn, bit-sliced.
    u64 moved0 = 0, moved1 = 0, moved2 = 0;
    const u64 pawns = s.pawns & mine;
    // a double push onto `flagged` allows en passant: one move for each pawn
    // beside it, unless one is pinned or the king is on their rank
    const u64 yp = s.pawns & them, flagged = east1(yp) | west1(yp);
    const u64 no_ep = ykb & push1<X>(DP_X) ? flagged : east1(yp & pinned_y) | west1(yp & pinned_y);
    const u64 reach_p = cap_west<Y>(core) | cap_east<Y>(core);
    const u64 ok_to = ~(reach_p | stay | PROMO_RANKS);
    shelf.set(SHELF_NO_EP, no_ep);
    shelf.set(SHELF_OK_TO, ok_to);
    {
        // pinned pawns push along their king's file and capture along its
        // diagonals; all their moves go to the sink
        const u64 free_p = pawns & ~pinned_x, held = pawns & pinned_x, diag = bishop_empty(xk);
        const u64 ok = free_p & ~(reach_p | keep), ok_cap = them & ok_to;
        const u64 d1 = push1<X>(free_p | (held & (FILEA << (xk & 7)))) & empty, d2 = push1<X>(d1 & DP_X) & empty & safe;
        const u64 target = them & safe;
        const u64 xw = (cap_west<X>(free_p) | (cap_west<X>(held & diag) & diag)) & target;
        const u64 xe = (cap_east<X>(free_p) | (cap_east<X>(held & diag) & diag)) & target;
        const u64 s1 = d1 & safe & ok_to & push1<X>(ok);
        const u64 s2 = d2 & ~no_ep & ok_to & push1<X>(push1<X>(ok));
        const u64 sw = cap_west<X>(ok) & xw & ok_cap;
        const u64 se = cap_east<X>(ok) & xe & ok_cap;
        to.add(s1);
        to.add(s2);
        to.add(sw);
        to.add(se);
        ns = popc(s1) + popc(s2) + popc(sw) + popc(se);
        // capture of a pawn that attacks f: its lost capture of f is in both
        // its own loss and f's weight
        if ((sw | se) & fp) corr = popc(sw & fp) + popc(se & fp);
        if (s2 & flagged) corr += popc(s2 & east1(yp)) + popc(s2 & west1(yp));
        // ring squares attacked from f or t: Y's king moves are counted again
        const u64 reach_r = cap_west<Y>(ring) | cap_east<Y>(ring);
        if ((ok | s1 | s2 | sw | se) & reach_r) {
            u64 n1 = s1 & (reach_r | push1<X>(reach_r)), n2 = s2 & (reach_r | push1<X>(push1<X>(reach_r)));
            u64 nw = sw & (reach_r | cap_west<X>(reach_r)), ne = se & (reach_r | cap_east<X>(reach_r));
            while (n1 | n2 | nw | ne) {
                u64 tb, fb;
                if (n1)
                    tb = n1 & (0 - n1), n1 ^= tb, fb = push1<Y>(tb);
                else if (n2)
                    tb = n2 & (0 - n2), n2 ^= tb, fb = push1<Y>(push1<Y>(tb));
                else if (nw)
                    tb = nw & (0 - nw), nw ^= tb, fb = cap_east<Y>(tb);
                else
                    tb = ne & (0 - ne), ne ^= tb, fb = cap_west<Y>(tb);
                const u64 left = (cap_west<X>(fb) | cap_east<X>(fb)) & ~multi;
                corr += popc(ring & ~((threat & ~left) | cap_west<X>(tb) | cap_east<X>(tb))) - kings;
            }
        }
        const u64 f1 = push1<Y>(s1), f2 = push1<Y>(push1<Y>(s2)), fw = cap_east<Y>(sw), fe = cap_west<Y>(se);
        const u64 x = f1 ^ f2 ^ fw, c = (f1 & f2) | (fw & (f1 ^ f2)), c2 = x & fe;
        moved0 = x ^ fe;
        moved1 = c ^ c2;
        moved2 = c & c2;
        shelf.set(SHELF_MOVED0, moved0);
        shelf.set(SHELF_MOVED1, moved1);
        shelf.set(SHELF_MOVED2, moved2);
        if ((moved0 | moved1 | moved2) & weighted) {
            const PawnTerms<Y, STRICT> w(fresh(fp), us, empty);
            const u64 plus[3] = {w.m1, w.m2, w.m3}, minus[2] = {w.cw, w.cc};
#pragma unroll
            for (int k = 0; k < 3; k++)
                corr += popc(moved0 & plus[k]) + 2 * popc(moved1 & plus[k]) + 4 * popc(moved2 & plus[k]);
#pragma unroll
            for (int k = 0; k < 2; k++)
                corr -= popc(moved0 & minus[k]) + 2 * popc(moved1 & minus[k]) + 4 * popc(moved2 & minus[k]);
            corr -= popc(f1 & w.m3);  // from the double-push square of a Y pawn onto its single-push square
        }
        // the rest, move by move: en passant (by source), pushes, captures
        u64 ep_from = 0;
        const u64 ept = ep_target<X>(st);
        if (ept) {
            const u64 victim = push1<Y>(ept);
            if (safe == ~0ULL || victim == checkers) {
                for (u64 src = (east1(victim) | west1(victim)) & pawns; src; src &= src - 1) {
                    const u64 p = src & (0 - src);
                    bool legal = true;
                    if (safe == ~0ULL) {
                        if (p & pinned_x)
                            legal = (ept & line_through(lsb(src), xk)) != 0;
                        else
                            legal = !(rook_att(xk, occ ^ victim ^ p) & s.rq & them & (RANK1 << (xk & 56)));
                    }
                    if (legal) ep_from |= p;
                }
            }
        }
        constexpr int UP = X == WHITE ? 8 : -8;
        constexpr int WEST = X == WHITE ? 7 : -9, EAST = X == WHITE ? 9 : -7;
        u64 r1 = (d1 & safe) ^ s1, r2 = d2 ^ s2, rw = xw ^ sw, re = xe ^ se;
        while (r1 | r2 | rw | re | ep_from) {
            u64 cur, bit;
            int delta;
            u32 flags = 0;
            if (r1) {
                cur = r1, delta = UP, r1 &= r1 - 1;
            } else if (r2) {
                cur = r2, delta = 2 * UP, r2 &= r2 - 1;
            } else if (rw) {
                cur = rw, delta = WEST, rw &= rw - 1;
            } else if (re) {
                cur = re, delta = EAST, re &= re - 1;
            } else {
                cur = ep_from, delta = 0, ep_from &= ep_from - 1;
            }
            bit = cur & (0 - cur);
            const int q = lsb(cur);
            int from = q - delta, dst = q;
            if (delta == 0) dst = lsb(ept), flags = MF_EP;
            if (delta == 2 * UP && (bit & flagged)) flags = MF_DOUBLE_PUSH;
            sink.one(make_move_code(from, dst, flags), (bit & PROMO_RANKS) != 0 && delta != 0);
        }
    }

    if (safe == ~0ULL) {
        const u32 castle_x = X == WHITE ? (st & 3) : ((st >> 2) & 3);
        constexpr int K0 = X == WHITE ? 4 : 60;
        if ((castle_x & 1) && !(KS_X & (occ | threat_y))) sink.one(make_move_code(K0, K0 + 2, MF_KING_CASTLE), false);
        if ((castle_x & 2) && !(QE_X & occ) && !(QS_X & threat_y))
            sink.one(make_move_code(K0, K0 - 2, MF_QUEEN_CASTLE), false);
    }

    // knights, sliders and the king, one by one.  moved: the number of simple
    // moves of each, five bits at five times its rank among them; pieces past
    // the twelfth have none (their moves go to the sink).
    const u64 pieces = us & ~s.pawns;
    u64 moved = 0, movers = moved0 | moved1 | moved2;  // movers: every X piece with a simple move
    // the moves of one piece: `sm` simple ones, the others to the sink
    auto split = [&](int f, u64 fb, u64 t, u64 sm) {
        sink.set(f, t ^ sm);
        if (!sm) return;
        const int n = popc(sm);
        ns += n;
        to.add(sm);
        moved |= (u64)n << (5 * popc(pieces & (fb - 1)));
        movers |= fb;
        if (fb & weighted) {
            const PawnTerms<Y, STRICT> w(fresh(fp), us, empty);
            corr += w.leave(fb) * n;
            // sliding between the two squares in front of an unmoved pawn
            if (fb & w.m2) corr -= popc(sm & push1<Y>(fb));
            if (fb & w.m3) corr -= popc(sm & push1<X>(fb));
        }
    };
    {
        const u64 core_n = knights_bulk(core), ring_n = knights_bulk(ring);
        u64 kn = s.knights & mine & ~pinned_x, cur = xkb;
        for (;;) {
            const int f = lsb(cur);
            const u64 fb = cur & (0 - cur);
            const bool king = cur == xkb;
            const u64 a = king ? king_att(f) : knight_att(f);
            const u64 t = a & ~us & (king ? ~shelf.get(SHELF_THREAT_Y) : safe);
            if (t) {
                u64 core_f = core_n, ring_f = ring_n, no = stay;
                if (king) {
                    core_f = core | east1(core) | west1(core);
                    core_f |= north(core_f) | south(core_f);
                    ring_f = ring | east1(ring) | west1(ring);
                    ring_f |= north(ring_f) | south(ring_f);
                    no |= bY | rY | (fp & (a | push1<X>(push1<X>(fb))));
                }
                const u64 sm = ((fb & (keep | core_f)) || popc(pieces & (fb - 1)) >= 12) ? 0 : t & ~(no | core_f);
                const u64 near = sm & ring_f;
                const u64 left = fb & ring_f ? a & ring & shelf.get(SHELF_THREAT) & ~shelf.get(SHELF_MULTI) : 0;
                if (near | left) {
                    // the ring squares attacked change: Y's king moves do
                    const u64 other = shelf.get(SHELF_THREAT) & ~left;
                    if (left) corr += (popc(ring & ~other) - kings) * popc(sm & ~near);
                    for (u64 q = near; q; q &= q - 1) {
                        const u64 att = king ? king_att(lsb(q)) : knight_att(lsb(q));
                        corr += popc(ring & ~(other | att)) - kings;
                    }
                }
                split(f, fb, t, sm);
            }
            if (!kn) break;
            cur = kn;
            kn &= kn - 1;
        }
    }
    for (u64 sl = (bqX | rqX) & mine; sl; sl &= sl - 1) {
        const int f = lsb(sl);
        const u64 fb = sl & (0 - sl);
        const bool diag = (fb & bqX) != 0;
        u64 a = magic_lookup((diag ? PB_TAB.bishop : PB_TAB.rook) + f, occ), core_f = 0, ring_f = 0;
        if (diag) {
            core_f = shelf.get(SHELF_CORE_B);
            ring_f = shelf.get(SHELF_RING_B);
        }
        if (fb & rqX) {
            core_f |= shelf.get(SHELF_CORE_R);
            ring_f |= shelf.get(SHELF_RING_R);
            if (diag) {
                const u64 c = rook_att(f, occ);
                a |= c;
            }
        }
        u64 t = a & safe & ~us;
        if (fb & pinned_x) t &= line_through(f, xk);
        if (!t) continue;
        const u64 no = stay | core_f | (fp & (king_att(f) | push1<X>(push1<X>(fb))));
        const u64 sm = ((fb & (keep | core_f)) || popc(pieces & (fb - 1)) >= 12) ? 0 : t & ~no;
        u64 near = sm & ring_f, left = 0;
        if (fb & ring_f) {
            left = a & ring & shelf.get(SHELF_THREAT) & ~shelf.get(SHELF_MULTI);
            // a slider that moves away along its line keeps its attack
            for (u64 z = a & ring; z; z &= z - 1) near |= sm & line_through(f, lsb(z));
        }
        if (near | left) {
            const u64 other = shelf.get(SHELF_THREAT) & ~left;
            if (left) corr += (popc(ring & ~other) - kings) * popc(sm & ~near);
            for (u64 q = near; q; q &= q - 1) {
                const int to_sq = lsb(q);
                const u64 occ2 = (occ ^ fb) | (q & (0 - q));
                u64 att = fb & bqX ? bishop_att(to_sq, occ2) : 0;
                if (fb & rqX) att |= rook_att(to_sq, occ2);
                corr += popc(ring & ~(other | att)) - kings;
            }
        }
        split(f, fb, t, sm);
    }

    // ---- weights of the squares entered: Y's pawns, then its pieces
    const u64 any = to.any();
    {
        const u64 mine_y = fresh(fp);
        const PawnTerms<Y, STRICT> w(mine_y, us, empty);
        base += popc(w.p1) + popc(w.dbl) + popc(w.cw & us) + popc(w.cc & us);
        // weight of t: captures gained (cw, cc) less pushes lost (p1, the
        // double push behind it, dbl), plus 2 so that it is never negative,
        // in three bit planes
        const u64 p1d = w.p1 & DP_Y & push1<X>(w.dbl), n0 = (w.p1 ^ p1d) | w.dbl;
        const u64 q0 = w.cw ^ w.cc, q1 = w.cw & w.cc, r1 = ~(n0 | p1d), k0 = q0 & n0;
        const u64 b0 = q0 ^ n0, b1 = q1 ^ r1 ^ k0, b2 = (q1 & r1) | (k0 & (q1 ^ r1));
        corr += to.sum(b0) + 2 * to.sum(b1) - 2 * (int)ns;
        if (any & b2) corr += 4 * to.sum(b2);
        if (promo) {  // on the promotion rank a move counts 4
            base += 3 * (popc(w.p1 & PROMO_RANKS) + popc(w.cw & us & PROMO_RANKS) + popc(w.cc & us & PROMO_RANKS));
            corr += 3 * (to.sum(w.cw & PROMO_RANKS) + to.sum(w.cc & PROMO_RANKS) - to.sum(w.p1 & PROMO_RANKS));
        }
        if (any & mine_y)  // captured pawns take their moves along
            corr -= to.sum(push1<X>(w.p1)) + to.sum(push1<X>(push1<X>(w.dbl))) + to.sum(mine_y & cap_east<X>(us)) +
                    to.sum(mine_y & cap_west<X>(us));
    }
    for (u64 kn = s.knights & them & ~shelf.get(SHELF_PINNED_Y); kn; kn &= kn - 1) {
        const u64 a = knight_att(lsb(kn)), bit = kn & (0 - kn);
        const int mob = popc(a & ~them);
        base += mob;
        if (any & a & them) corr += to.sum(a & them);
        if (any & bit) corr -= to.at(bit) * mob;
    }
    // Y's sliders, diagonal movers first (a loop per kind: 1.3 % faster than one
    // that selects)
#pragma unroll 1
    for (int kind = 0; kind < 2; kind++) {
        const bool diag = kind == 0;
        const Magic *table = diag ? PB_TAB.bishop : PB_TAB.rook;
        const u64 alike = diag ? bqX : rqX, y_alike = diag ? bY : rY;
        for (u64 set = y_alike; set; set &= set - 1) {
            // one slider: its own moves, the squares of simple moves it sees, and
            // the pieces with simple moves it sees
            const u64 bit = set & (0 - set);
            const int sq = lsb(set);
            const Magic *e = table + sq;
            const u64 a = magic_lookup(e, occ);
            const int mob = popc(a & ~them);
            base += mob;
            if (any & ((a & them) | bit)) corr += to.sum(a & them) - to.at(bit) * mob;
            // the squares it gains when the pieces with simple moves leave; one
            // lookup for all, as a ray holds at most one of them
            u64 g = a & movers;
            const u64 opened = magic_lookup(e, occ ^ g);
            // the nearest such square of each ray at once: a lookup with them
            // occupied loses what is beyond them (two planes in flight at a
            // time: 1 % faster than one; three lose it again)
            const u64 view = a & empty;
            if (any & view) {
                for (u64 h0 = to.c0 & view, h1 = to.c1 & view; h0 | h1;) {
                    const u64 cut0 = magic_lookup(e, occ | h0), cut1 = magic_lookup(e, occ | h1);
                    corr -= 3 * mob - popc(cut0 & ~them) - 2 * popc(cut1 & ~them);
                    h0 &= ~cut0;
                    h1 &= ~cut1;
                }
                for (u64 h = to.c2 & view; h;) {
                    const u64 cut = magic_lookup(e, occ | h);
                    corr -= 4 * (mob - popc(cut & ~them));
                    h &= ~cut;
                }
                if (to.rare) {
#pragma unroll 1
                    for (int k = 0; k < 2; k++) {
                        for (u64 h = (k ? to.c4() : to.c3()) & view; h;) {
                            const u64 cut = magic_lookup(e, occ | h);
                            corr -= (8 << k) * (mob - popc(cut & ~them));
                            h &= ~cut;
                        }
                    }
                }
            }
            for (; g; g &= g - 1) {
                const u64 fb = g & (0 - g);
                int n;
                if (fb & s.pawns) {
                    n = (fb & shelf.get(SHELF_MOVED0) ? 1 : 0) + (fb & shelf.get(SHELF_MOVED1) ? 2 : 0) +
                        (fb & shelf.get(SHELF_MOVED2) ? 4 : 0);
                } else {
                    n = (int)(moved >> (5 * popc(pieces & (fb - 1)))) & 31;
                }
                const int f = lsb(g);
                const u64 past = opened & beyond(sq, f);
                const int ext = popc(past & ~them);
                corr += ext * n;
                // moves of f along the same line, up to the capture of the slider
                if (!(fb & (s.pawns | alike))) continue;
                u64 line = 0;
                if (fb & s.pawns) {
                    if (diag) {
                        line = (cap_west<X>(fb) | cap_east<X>(fb)) & (past | bit) & them;
                    } else if (((sq ^ f) & 7) == 0) {
                        const u64 d = push1<X>(fb) & empty;
                        line = d | (push1<X>(d & DP_X) & empty & ~shelf.get(SHELF_NO_EP));
                    }
                    line &= safe & shelf.get(SHELF_OK_TO);
                } else {
                    u64 no = stay | us | (fp & (king_att(f) | push1<X>(push1<X>(fb))));
                    if (fb & bqX) no |= shelf.get(SHELF_CORE_B);
                    if (fb & rqX) no |= shelf.get(SHELF_CORE_R);
                    line = (between(sq, f) | past | bit) & safe & ~no;
                    if (fb & pinned_x) line &= line_through(f, xk);
                }
                if (line) {
                    corr -= ext * popc(line & ~past);
                    corr += popc(line & past & them);
                    for (u64 t = line & past & empty; t; t &= t - 1) corr -= popc(past & beyond(sq, lsb(t)) & ~them);
                }
            }
        }
    }
    *simple = ns;
    return ns * base + (u32)corr;
}

}  // namespace pb
