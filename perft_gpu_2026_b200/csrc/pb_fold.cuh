// pb_fold.cuh - perft(2) of a position without making most of its moves.
//
// The sum over a position's moves of the opponent's move counts is dominated
// by moves after which the opponent's count differs from a common base by a
// few terms that depend only on the squares left and entered.  fold_child
// sums those moves by set arithmetic and hands the rest to a sink, move by
// move, to be made and counted in full (count_moves).
//
// X moves, Y = 1 - X is counted.  The base is Y's move count in the position
// as it stands (no en passant).  A move f -> t of a piece p is SIMPLE when it
// leaves Y's king moves, castling, pins and checks alone:
//   - p attacks no square of Y's zone from f or from t.  The zone is the king,
//     the squares next to it without a Y piece, and the safe squares of a
//     castling whose path has no Y piece; X-rays through Y's first blocker
//     towards the king count as attacks (a slider there would pin);
//   - f is not an X piece that shields a zone square from an X slider, nor
//     one of two blockers with a Y piece between an X slider and the king;
//   - t is not on a line from an X slider to a zone square it attacks, nor
//     between a pinned Y piece's pinner and the king;
//   - neither f nor t is on such a castling path;
//   - a piece captured on t is not next to the king, pinned, on a castling
//     corner or a pawn about to promote, is not a slider that sees f along
//     the line of the capture, and is not a pawn that bears on f (unless a
//     pawn takes it, where the overlap is one known move).
// After a simple move
//   - Y's king, pinned-piece and castling moves are as before;
//   - a captured piece's moves are gone; Y's pieces that guarded t take there;
//   - Y's unpinned pawns change by a weight of f plus a weight of t (pushes
//     unblocked and captures lost on f, pushes blocked and captures gained on
//     t), less one if X slides between the two squares in front of an unmoved
//     pawn;
//   - a Y slider that sees t loses the squares beyond t, and one that sees f
//     gains those beyond f; moves of f along that same line are corrected one
//     by one.
// Weights of t are summed over all simple moves at once: the number of simple
// moves onto each square is kept in bit-sliced planes (at most 16 pieces can
// reach one square: eight lines and eight knight jumps).
//
// Promotions, en passant, castling and double pushes that allow an en-passant
// capture go to the sink.  On the benchmark's leaves 7.5 % of the moves do, on
// middle-game playouts 21 %, in endgames of pieces alone two thirds.
#pragma once
#include "pb_core.cuh"

namespace pb {

// Number of simple moves onto each square, bit-sliced.  Eight or more onto one
// square (c3, c4) are rare, so their terms hide behind one test.
struct TargetPlanes {
    u64 c0 = 0, c1 = 0, c2 = 0, c3 = 0, c4 = 0;
    PB_HD void add(u64 s)
    {
        u64 k = c0 & s;
        c0 ^= s;
        s = c1 & k;
        c1 ^= k;
        k = c2 & s;
        c2 ^= s;
        if (k) {
            c4 |= c3 & k;
            c3 ^= k;
        }
    }
    PB_HD bool rare() const { return c3 != 0 || c4 != 0; }
    PB_HD int sum(u64 m) const
    {
        int n = popc(c0 & m) + 2 * popc(c1 & m) + 4 * popc(c2 & m);
        if (rare()) n += 8 * popc(c3 & m) + 16 * popc(c4 & m);
        return n;
    }
    PB_HD u64 any() const { return c0 | c1 | c2 | c3 | c4; }
    PB_HD int at(u64 bit) const
    {
        int n = (c0 & bit ? 1 : 0) + (c1 & bit ? 2 : 0) + (c2 & bit ? 4 : 0);
        if (rare()) n += (c3 & bit ? 8 : 0) + (c4 & bit ? 16 : 0);
        return n;
    }
};

PB_HD u64 beyond(int s, int t) { return ldg64(&PB_TAB.beyond[s][t]); }

// Sink: set(from, targets) takes the moves from -> t of one piece (flags 0),
// one(move, promotes) one move, or with `promotes` the four promotions.
// Returns the simple moves' sum of counts; *simple = how many they are.
template <int X, bool STRICT, class Sink>
PB_HD u32 fold_child(const Board &b, u32 st, Sink &sink, u32 *simple)
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
    u64 zone = ring | ykb, path = 0;
    const u32 castle_y = Y == WHITE ? (st & 3) : ((st >> 2) & 3);
    if (castle_y) {
        if ((castle_y & 1) && !(KS_Y & them)) path |= KS_Y, zone |= KS_Y;
        if ((castle_y & 2) && !(QE_Y & them)) path |= QE_Y, zone |= QS_Y;
    }
    u64 reach_b, reach_r;           // squares from which a diagonal / orthogonal slider bears on the zone
    u64 keep = path, lines = path;  // squares no simple move leaves / enters
    u64 pinned_y = 0;
    u64 threat = knights_bulk(s.knights & us) | cap_west<X>(s.pawns & us) | cap_east<X>(s.pawns & us) | king_att(xk);
    {
        u64 a = bishop_att(yk, occ);
        reach_b = a | bishop_att(yk, occ & ~(a & them));
        a = rook_att(yk, occ);
        reach_r = a | rook_att(yk, occ & ~(a & them));
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
    for (u64 z = zone & ~ykb; z; z &= z - 1) {
        const int q = lsb(z);
        const u64 a = bishop_att(q, occ_k), c = rook_att(q, occ_k);
        reach_b |= a;
        reach_r |= c;
        if ((a & bqX) | (c & rqX)) threat |= 1ULL << q;
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
    if (threat_y & xkb) {
        checkers = (cap_west<X>(xkb) | cap_east<X>(xkb)) & s.pawns & them;
        checkers |= knight_att(xk) & s.knights & them;
        checkers |= bishop_att(xk, occ) & s.bq & them;
        checkers |= rook_att(xk, occ) & s.rq & them;
        safe = checkers | between(xk, bit_index(checkers));
        mine = us & ~pinned_x;
        if (more_than_one(checkers)) mine = xkb;
    }

    // ---- Y's base count without its sliders (added with their terms below)
    u32 base = popc(ring & ~threat);
    if (castle_y) {
        if ((castle_y & 1) && !(KS_Y & (occ | threat))) base++;
        if ((castle_y & 2) && !(QE_Y & occ) && !(QS_Y & threat)) base++;
    }
    const u64 fp = s.pawns & them & ~pinned_y;
    const u64 pu = push1<Y>(fp), p1 = pu & empty;
    const u64 dreach = push1<Y>(p1 & DP_Y), dbl = dreach & empty;
    const u64 cw = cap_west<Y>(fp), ce = cap_east<Y>(fp);
    // on the promotion rank a square counts 4, and captures onto it once
    // unless STRICT
    const u64 cc = STRICT ? ce : ce & ~(cw & PROMO_RANKS);
    base += popc(p1) + popc(dbl) + popc(cw & us) + popc(cc & us);
    const bool promo = (fp & RANK7_Y) != 0;
    if (promo) base += 3 * (popc(p1 & PROMO_RANKS) + popc(cw & us & PROMO_RANKS) + popc(cc & us & PROMO_RANKS));
    // weights of a square left: f unblocks a push (m1), the double push
    // behind it too (m2), a double push (m3); captures lost are cw, cc
    const u64 m1 = pu & us, m2 = pu & DP_Y & us & push1<X>(empty), m3 = dreach & us;
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
    TargetPlanes to;
    int corr = 0;
    u32 ns = 0;

    // pawns, by sets of target squares: single and double pushes, captures.
    // moved0..2: the number of simple moves of each pawn, bit-sliced.
    u64 moved0 = 0, moved1 = 0, moved2 = 0;
    const u64 pawns = s.pawns & mine;
    const u64 flagged = east1(s.pawns & them) | west1(s.pawns & them);  // a double push here allows en passant
    const u64 reach_p = cap_west<Y>(zone) | cap_east<Y>(zone);
    const u64 ok_to = ~(reach_p | stay | PROMO_RANKS);
    {
        // pinned pawns push along their king's file and capture along its
        // diagonals; all their moves go to the sink
        const u64 free_p = pawns & ~pinned_x, held = pawns & pinned_x, diag = bishop_empty(xk);
        const u64 ok = free_p & ~(reach_p | keep), ok_cap = them & ~bY & ok_to;
        const u64 d1 = push1<X>(free_p | (held & (FILEA << (xk & 7)))) & empty, d2 = push1<X>(d1 & DP_X) & empty & safe;
        const u64 target = them & safe;
        const u64 xw = (cap_west<X>(free_p) | (cap_west<X>(held & diag) & diag)) & target;
        const u64 xe = (cap_east<X>(free_p) | (cap_east<X>(held & diag) & diag)) & target;
        const u64 s1 = d1 & safe & ok_to & push1<X>(ok);
        const u64 s2 = d2 & ~flagged & ok_to & push1<X>(push1<X>(ok));
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
        const u64 f1 = push1<Y>(s1), f2 = push1<Y>(push1<Y>(s2)), fw = cap_east<Y>(sw), fe = cap_west<Y>(se);
        const u64 x = f1 ^ f2 ^ fw, c = (f1 & f2) | (fw & (f1 ^ f2)), c2 = x & fe;
        moved0 = x ^ fe;
        moved1 = c ^ c2;
        moved2 = c & c2;
        if ((moved0 | moved1 | moved2) & (m1 | m3 | cw | cc)) {
            corr += popc(moved0 & m1) + 2 * popc(moved1 & m1) + 4 * popc(moved2 & m1);
            corr += popc(moved0 & m2) + 2 * popc(moved1 & m2) + 4 * popc(moved2 & m2);
            corr += popc(moved0 & m3) + 2 * popc(moved1 & m3) + 4 * popc(moved2 & m3);
            corr -= popc(moved0 & cw) + 2 * popc(moved1 & cw) + 4 * popc(moved2 & cw);
            corr -= popc(moved0 & cc) + 2 * popc(moved1 & cc) + 4 * popc(moved2 & cc);
            corr -= popc(f1 & m3);  // from the double-push square of a Y pawn onto its single-push square
        }
        // the rest, move by move: en passant (by source), pushes, captures
        u64 ep_from = 0;
        const u64 ept = ep_target<X>(st);
        if (ept) {
            const u64 victim = push1<Y>(ept);
            if (!checkers || victim == checkers) {
                for (u64 src = (east1(victim) | west1(victim)) & pawns; src; src &= src - 1) {
                    const u64 p = src & (0 - src);
                    bool legal = true;
                    if (!checkers) {
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

    // knights, sliders and the king, one by one.  moved: the number of simple
    // moves of each, five bits at five times its rank among them; pieces past
    // the twelfth have none (their moves go to the sink).
    const u64 pieces = us & ~s.pawns;
    u64 moved = 0;
    {
        const u64 reach_n = knights_bulk(zone);
        u64 reach_k = zone | east1(zone) | west1(zone);
        reach_k |= north(reach_k) | south(reach_k);
        u64 kn = s.knights & mine & ~pinned_x, sl = (bqX | rqX) & mine, cur = xkb;
        for (;;) {
            const int f = lsb(cur);
            const u64 fb = cur & (0 - cur);
            u64 t, no = stay;
            if (cur == xkb) {
                t = king_att(f) & ~threat_y;
                no |= reach_k | bY | rY | (fp & (king_att(f) | push1<X>(push1<X>(fb))));
                if (fb & reach_k) no = ~0ULL;
            } else if (fb & s.knights) {
                t = knight_att(f) & safe;
                no |= reach_n;
                if (fb & reach_n) no = ~0ULL;
            } else {
                t = 0;
                if (fb & bqX) {
                    t = bishop_att(f, occ);
                    no |= reach_b | (t & bY);
                    if (fb & reach_b) no = ~0ULL;
                }
                if (fb & rqX) {
                    const u64 a = rook_att(f, occ);
                    no |= reach_r | (a & rY);
                    if (fb & reach_r) no = ~0ULL;
                    t |= a;
                }
                no |= fp & (king_att(f) | push1<X>(push1<X>(fb)));
                t &= safe;
                if (fb & pinned_x) t &= line_through(f, xk);
            }
            t &= ~us;
            const int rank = popc(pieces & (fb - 1));
            u64 sm = ((fb & keep) || rank >= 12) ? 0 : t & ~no;
            sink.set(f, t ^ sm);
            if (sm) {
                const int n = popc(sm);
                ns += n;
                to.add(sm);
                moved |= (u64)n << (5 * rank);
                if (fb & (m1 | m3 | cw | cc)) {
                    int g = (fb & m1 ? 1 : 0) + (fb & m2 ? 1 : 0) + (fb & m3 ? 1 : 0) - (fb & cw ? 1 : 0) -
                            (fb & cc ? 1 : 0);
                    if (fb & PROMO_RANKS) g *= 4;
                    corr += g * n;
                    // sliding between the two squares in front of an unmoved pawn
                    if (fb & m2) corr -= popc(sm & push1<Y>(fb));
                    if (fb & m3) corr -= popc(sm & push1<X>(fb));
                }
            }
            if (kn) {
                cur = kn;
                kn &= kn - 1;
            } else if (sl) {
                cur = sl;
                sl &= sl - 1;
            } else {
                break;
            }
        }
    }
    if (!checkers) {
        const u32 castle_x = X == WHITE ? (st & 3) : ((st >> 2) & 3);
        constexpr int K0 = X == WHITE ? 4 : 60;
        if ((castle_x & 1) && !(KS_X & (occ | threat_y))) sink.one(make_move_code(K0, K0 + 2, MF_KING_CASTLE), false);
        if ((castle_x & 2) && !(QE_X & occ) && !(QS_X & threat_y))
            sink.one(make_move_code(K0, K0 - 2, MF_QUEEN_CASTLE), false);
    }

    // ---- weights of the squares entered: Y's pawns, then its pieces
    const u64 any = to.any();
    {
        // weight of t: captures gained (cw, cc) less pushes lost (p1, the
        // double push behind it, dbl), plus 2 so that it is never negative,
        // in three bit planes
        const u64 p1d = p1 & DP_Y & push1<X>(dbl), n0 = (p1 ^ p1d) | dbl;
        const u64 q0 = cw ^ cc, q1 = cw & cc, r1 = ~(n0 | p1d), k0 = q0 & n0;
        const u64 b0 = q0 ^ n0, b1 = q1 ^ r1 ^ k0, b2 = (q1 & r1) | (k0 & (q1 ^ r1));
        corr += to.sum(b0) + 2 * to.sum(b1) - 2 * (int)ns;
        if (any & b2) corr += 4 * to.sum(b2);
        if (promo) corr += 3 * (to.sum(cw & PROMO_RANKS) + to.sum(cc & PROMO_RANKS) - to.sum(p1 & PROMO_RANKS));
    }
    if (any & fp)  // captured pawns take their moves along
        corr -= to.sum(push1<X>(p1)) + to.sum(push1<X>(push1<X>(dbl))) + to.sum(fp & cap_east<X>(us)) +
                to.sum(fp & cap_west<X>(us));
    for (u64 kn = s.knights & them & ~pinned_y; kn; kn &= kn - 1) {
        const u64 a = knight_att(lsb(kn)), bit = kn & (0 - kn);
        const int mob = popc(a & ~them);
        base += mob;
        if (any & a & them) corr += to.sum(a & them);
        if (any & bit) corr -= to.at(bit) * mob;
    }
    u64 bs = bY, rs = rY;
    while (bs | rs) {
        // one slider: its own moves, the squares of simple moves it sees, and
        // the pieces with simple moves it sees
        const bool diag = bs != 0;
        const u64 bit = diag ? bs & (0 - bs) : rs & (0 - rs);
        const int sq = diag ? lsb(bs) : lsb(rs);
        const Magic *e = diag ? &PB_TAB.bishop[sq] : &PB_TAB.rook[sq];
        if (diag)
            bs ^= bit;
        else
            rs ^= bit;
        const u64 a = magic_lookup(e, occ);
        const int mob = popc(a & ~them);
        base += mob;
        if (any & bit) corr -= to.at(bit) * mob;
        if (any & a & them) corr += to.sum(a & them);
        // the nearest such square of each ray at once: a lookup with them
        // occupied loses what is beyond them
        const u64 view = a & empty;
        for (u64 h = to.c0 & view; h;) {
            const u64 cut = magic_lookup(e, occ | h);
            corr -= mob - popc(cut & ~them);
            h &= ~cut;
        }
        for (u64 h = to.c1 & view; h;) {
            const u64 cut = magic_lookup(e, occ | h);
            corr -= 2 * (mob - popc(cut & ~them));
            h &= ~cut;
        }
        for (u64 h = to.c2 & view; h;) {
            const u64 cut = magic_lookup(e, occ | h);
            corr -= 4 * (mob - popc(cut & ~them));
            h &= ~cut;
        }
        if (to.rare()) {
#pragma unroll 1
            for (int k = 0; k < 2; k++)
                for (u64 h = (k ? to.c4 : to.c3) & view; h;) {
                    const u64 cut = magic_lookup(e, occ | h);
                    corr -= (8 << k) * (mob - popc(cut & ~them));
                    h &= ~cut;
                }
        }
        for (u64 g = a & us; g; g &= g - 1) {
            const u64 fb = g & (0 - g);
            int n;
            if (fb & s.pawns) {
                n = (fb & moved0 ? 1 : 0) + (fb & moved1 ? 2 : 0) + (fb & moved2 ? 4 : 0);
            } else {
                const int rank = popc(pieces & (fb - 1));
                n = rank < 12 ? (int)(moved >> (5 * rank)) & 31 : 0;
            }
            if (!n) continue;
            const int f = lsb(g);
            const u64 past = magic_lookup(e, occ ^ fb) & beyond(sq, f);
            const int ext = popc(past & ~them);
            corr += ext * n;
            // moves of f along the same line
            u64 line = 0;
            if (fb & s.pawns) {
                if (diag) {
                    line = (cap_west<X>(fb) | cap_east<X>(fb)) & past & them & ~bY & safe & ok_to;
                } else if (((sq ^ f) & 7) == 0) {
                    const u64 d = push1<X>(fb) & empty;
                    line = (d | (push1<X>(d & DP_X) & empty & ~flagged)) & safe & ok_to;
                }
            } else if (fb & (diag ? bqX : rqX)) {
                u64 no = stay | us | (past & (diag ? bY : rY)) | (fp & (king_att(f) | push1<X>(push1<X>(fb))));
                if (fb & bqX) no |= reach_b;
                if (fb & rqX) no |= reach_r;
                line = (between(sq, f) | past) & safe & ~no;
                if (fb & pinned_x) line &= line_through(f, xk);
            }
            if (line) {
                corr -= ext * popc(line & ~past);
                corr += popc(line & them);
                for (u64 t = line & past & empty; t; t &= t - 1) corr -= popc(past & beyond(sq, lsb(t)) & ~them);
            }
        }
    }
    *simple = ns;
    return ns * base + (u32)corr;
}

}  // namespace pb
