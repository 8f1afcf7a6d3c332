// pg_reply.cuh -- the last two plies of a position without making most of
// its moves.
//
// perft(2) of a position is the sum, over the legal moves of the side to move
// (the mover), of the number of replies.  Most moves change few of the
// replies: the opponent's reply count after such a move is its count on the
// unmoved board (the mover passes) plus a correction that depends on the
// square left and the square reached alone.  reply_sum splits the moves:
//
//  * plain moves are counted in sets: per moving piece the popcount of its
//    plain targets times (passed count + correction for the square left), and
//    over all pieces the corrections for the squares reached, as popcounts of
//    bit planes (a square's correction in binary, one 64-bit mask per digit);
//  * after some of them only the opponent king's own moves change otherwise:
//    they are counted as plain less the king's part, and the emitter gets them
//    for a recount of the king's moves alone (king_replies);
//  * every other move (a check, a discovered line, castling, promotion, en
//    passant, ...) goes to the emitter, and is made and counted as before.
//
// A move from f to t by piece X is plain when, with K the opponent's king:
//  1. K is not attacked on the unmoved board (else no move is plain);
//  2. f and t change no pin and no check: f is not a blocker whose leaving
//     opens a line of another mover's slider to K or pins a piece, nor a
//     pinner; t is not on a line X itself then looks along to K through at most
//     one opposing piece; t does not unpin or capture a pinned piece; a pinned
//     slider sees neither f nor t;
//  3. f and t do not share a line of an opposing slider that sees f, and t is
//     not a pawn whose own count the square left has already corrected;
// and the king's replies change too unless
//  4. the squares K may enter (and cross when castling) are attacked or not
//     as before: X attacks none of the attacked ones from f alone and none of
//     the free ones from t, no slider's line through f or t reaches one, and
//     neither f nor t is next to K (nor on a castling path: such a move is made).
// Then the replies change only by
//  * the opponent's sliders: the rays that ended on f run on, the rays that
//    passed t end there;
//  * its pawns: pushes onto f and t, captures on f and t;
//  * a captured piece: its own moves go, and the pieces that defend t (sliders,
//    knights, pawns) gain the recapture.
// The legality rules enter only through the passed count, whose terms are
// count_moves_ks1's outside check.
//
// What bounds it: integer-ALU issue (78-79% busy over the leaf; the rest is the
// latency of dependent instructions and table loads with 16 warps an SM, and
// loops over a node's pieces of different length in a warp's lanes), as the
// count of a made child (about 900 instructions).  Of a node's 34 moves 73% are
// counted in sets, 10.3% are a king recount (about 150 instructions), 16.9% are
// made; every 16th of 4,096 positions at depths 3..6 spends 16.7 ms of leaf time
// here, 10.7 on made children, 3.1 on king recounts.
// Measured (GB300): those 4,096 positions in 519 ms, 1,203 ms with every child
// made and counted.  What it gives hangs on the position: two at depth 7 took 19.0
// against 44.1 ms (whole call) and 29.3 against 92.5 ms (leaf time).
#pragma once
#include "pg_movegen.cuh"

namespace pg {

// sum and carry of three bit planes
__device__ __forceinline__ u64 plane_sum(u64 a, u64 b, u64 c) { return a ^ b ^ c; }
__device__ __forceinline__ u64 plane_carry(u64 a, u64 b, u64 c) { return (a & b) | (c & (a | b)); }

// a three-digit number per square
struct Planes3 {
    u64 c0, c1, c2;
};

// How many targets an opposing slider's ray has beyond each square, 0..7: where
// it passes, what a piece arriving cuts off; at the slider, its moves along the
// ray; at the other side's piece it ends on, what that piece leaving opens.
// s: the sliders' attack fill along one direction (blockers included), x: the
// same from the squares of `blockers` it ends on, own: the sliders' side (not a
// target), sl: the sliders.  Runs of targets go through empty squares only; the
// opened squares themselves hold nothing.
template <int SH, bool LEFT>
__device__ __forceinline__ Planes3 targets_beyond(u64 s, u64 x, u64 empty, u64 own, u64 sl, u64 blockers)
{
    const u64 through = (s | x) & empty, at = through | sl | (s & blockers), keep = ~(x & empty);
    auto back = [](u64 y, int k) { return LEFT ? (y >> (k * SH)) : (y << (k * SH)); };
    // r_k: a run of k or more targets; by doubling, a run of k from the k-th
    // square of a run of j is one of j + k
    const u64 r1 = back((s | x) & ~own, 1) & at, e1 = r1 & through;
    const u64 r2 = r1 & back(e1, 1), e2 = r2 & through;
    const u64 r3 = r2 & back(e1, 2), e3 = r3 & through;
    const u64 r4 = r2 & back(e2, 2);
    const u64 r5 = r4 & back(e1, 4), r6 = r4 & back(e2, 4), r7 = r4 & back(e3, 4);
    return Planes3{((r1 & ~r2) | (r3 & ~r4) | (r5 & ~r6) | r7) & keep, ((r2 & ~r4) | r6) & keep, r4 & keep};
}

// A queued move: bits 0-15 the move, 16-24 the node's index in its CTA, 25-28
// the landing piece (PC_*, with PC_EP_FLAG), 29 only the king's replies are
// recounted.  A set of moves is a mask and the entry of its square 0, each
// square t adding t x mul: a piece's mask holds target squares (mul 64), a pawn
// set's the lower of the two squares of each move (mul 65).
constexpr u32 Q_PIECE_SHIFT = 25;
constexpr u32 Q_EP = PC_EP_FLAG << Q_PIECE_SHIFT, Q_KING = 1u << 29;
// a set of pawn moves over the squares of `to`, step = to - from
template <int STEP> __device__ __forceinline__ u64 pawn_set(u64 to) { return STEP > 0 ? to >> (STEP > 0 ? STEP : 0) : to; }
template <int STEP> __device__ __forceinline__ constexpr u32 pawn_entry(int flags = 0)
{
    return ((u32)flags << 12) | (u32)(STEP > 0 ? STEP * 64 : -STEP);
}

// the four promotions to each square of m, from `step` below it
template <class E> __device__ __forceinline__ void put_promotions(E& emit, u64 m, int step)
{
    if (!m) return;
    auto put = [&](u16 mv, u32 piece) { emit.put((u32)mv | (piece << Q_PIECE_SHIFT)); };
    each_square(m, [&](int t) { emit_pawn_sq(put, t - step, t, 0); });
}

// The king's moves of the side to move next (1 - S) after S's move mv on b,
// when that king is neither checked before nor after it.  piece: as make_child
template <int S> __device__ __forceinline__ u32 king_replies(const Pos& b, u16 mv, u32 piece)
{
    const int from = mv & 63, to = (mv >> 6) & 63;
    const u64 src = bit64((u32)from), dst = bit64((u32)to);
    const u32 pc = piece & 7u;
    const u64 pawns = b.p & INNER;
    const u64 occ0 = b.k | pawns | b.n | b.bq | b.rq;
    const u64 mine = (S ? occ0 & ~b.w : b.w) & ~src, own = (S ? b.w : occ0 & ~b.w) & ~dst;
    const u64 occ = (occ0 & ~src) | dst;
    const u64 mrq = (b.rq & mine) | ((pc == PC_ROOK || pc == PC_QUEEN) ? dst : 0ull);
    const u64 mbq = (b.bq & mine) | ((pc == PC_BISHOP || pc == PC_QUEEN) ? dst : 0ull);
    const u64 mp = (pawns & mine) | (pc == PC_PAWN ? dst : 0ull);
    const u64 mn = (b.n & mine) | (pc == PC_KNIGHT ? dst : 0ull);
    const u64 mk = pc == PC_KING ? dst : b.k & mine;
    const u64 empty = ~occ;
    const VPro v(empty);
    u64 thr = v.up(mrq) | v.down(mrq);
    const RankPro h(occ);
    thr |= h.east(mrq) | h.west(mrq);
    const u64 pass = empty & NOT_A & NOT_H;
    const DPro<9> d9(pass);
    thr |= d9.up(mbq) | d9.down(mbq);
    const DPro<7> d7(pass);
    thr |= d7.up(mbq) | d7.down(mbq);
    thr |= pawn_attacks<S>(mp) | knight_set(mn) | __ldg(&g_king[sq_of(mk)]);
    return popc(__ldg(&g_king[sq_of(b.k & own)]) & ~(own | thr));
}

// The replies to the plain moves of b (S to move), summed, less the king's part
// where only that is recounted; the other moves go to emit.sets(moves to make,
// king recounts, entry of square 0, mul) or, one at a time, to emit.put(entry)
// and emit.put_ep(entry).  emit.kings counts the king recounts.
template <int S, class E> __device__ __forceinline__ u64 reply_sum(const Pos& b, E& emit)
{
    constexpr int T = 1 - S;
    KsFacts<S> f;
    f.pawns = b.p & INNER;
    f.occ = b.k | f.pawns | b.n | b.bq | b.rq;
    {
        const u64 black = f.occ & ~b.w;
        f.mine = S ? black : b.w;
        f.theirs = S ? b.w : black;
    }
    f.empty = ~f.occ;
    const u64 mine = f.mine, own = f.theirs, occ = f.occ, empty = f.empty, pawns = f.pawns;
    const u64 mrq = b.rq & mine, mbq = b.bq & mine, mp = pawns & mine, mn = b.n & mine, mk = b.k & mine;
    const u64 orq = b.rq & own, obq = b.bq & own;

    // one propagator chain per line kind for every fill below
    const VPro v(empty);
    const RankPro h(occ);
    const u64 pass = empty & NOT_A & NOT_H;
    const DPro<9> d9(pass);
    const DPro<7> d7(pass);
    // the opponent's sliders, per direction
    const u64 s0 = v.up(orq), s1 = v.down(orq), s2 = h.east(orq), s3 = h.west(orq);
    const u64 s4 = d9.up(obq), s5 = d9.down(obq), s6 = d7.up(obq), s7 = d7.down(obq);

    // the mover's side, as in count_moves_ks1: its king is opaque to the fills,
    // so the square behind it on a checking line is added to the threats
    {
        const int ksq = sq_of(mk);
        f.ksq = ksq;
        const u64 kr = SlFancy::rook(ksq, occ), kb = SlFancy::bishop(ksq, occ);
        const u64 kf = kr & file_of(ksq), kd = kb & __ldg(&g_diag[ksq]);
        const u64 kh = kr ^ kf, ka = kb ^ kd;
        f.pf = kf & (s0 | s1) & mine;
        f.pr = kh & (s2 | s3) & mine;
        f.pd = kd & (s4 | s5) & mine;
        f.pa = ka & (s6 | s7) & mine;
        f.pinned = f.pf | f.pr | f.pd | f.pa;
        const u64 cr = kr & orq, csl = cr | (kb & obq);
        f.checkers = csl | (__ldg(&g_knight[ksq]) & b.n & own) | (__ldg(&g_pawn_checks[S][ksq]) & pawns & own);
        u64 cray = 0, behind = 0;
        if (csl) {
            const int csq = lsb(csl);
            cray = __ldg(&g_between[ksq][csq]);
            for (u64 s = csl; s; s &= s - 1) behind |= __ldg(&g_behind[ksq][lsb(s)]);
        }
        f.safe = cray | f.checkers;
        f.threat = s0 | s1 | s2 | s3 | s4 | s5 | s6 | s7 | behind | pawn_attacks<T>(pawns & own) | knight_set(b.n & own) |
                   __ldg(&g_king[sq_of(b.k & own)]);
        const bool in_check = f.checkers != 0;
        f.chk_all = in_check ? ~0ull : 0ull;
        f.tgt = several(f.checkers) ? 0ull : (in_check ? f.safe : ~mine);
    }

    const u64 king = b.k & own;
    const int kq = sq_of(king);
    const u64 kr = SlFancy::rook(kq, occ), kb = SlFancy::bishop(kq, occ);
    const u64 ring = __ldg(&g_king[kq]);

    // squares a plain move may not leave / reach, whatever the piece; and
    // those where only the king's own moves change (from / to next to it, a
    // line opened to or closed from a square it may enter)
    u64 no_f = 0, no_t = 0, king_f = ring, king_t = ring;
    // the opponent's king attacked with the mover to move: nothing is plain
    if ((kr & mrq) | (kb & mbq) | (__ldg(&g_knight[kq]) & mn) | (__ldg(&g_pawn_checks[T][kq]) & mp) | (ring & mk)) {
        no_f = ~0ull;
        no_t = ~0ull;
    }

    // the mover's sliders on K's lines: the opponent's pins, and the blockers
    // that may not leave
    u64 pf = 0, pr = 0, pd = 0, pa = 0;
    {
        const u64 lf = file_of(kq), lr = rank_of(kq), ld = __ldg(&g_diag[kq]), la = anti_of(kq);
        for (u64 s = ((lf | lr) & mrq) | ((ld | la) & mbq); s; s &= s - 1) {
            const int q = lsb(s);
            const u64 sb = lowbit(s);
            const u64 between = __ldg(&g_between[kq][q]);
            const u64 in = between & occ;
            const int n = popc(in);
            if (n == 1) {
                if (in & own) {
                    pf |= (lf & sb) ? in : 0ull;
                    pr |= (lr & sb) ? in : 0ull;
                    pd |= (ld & sb) ? in : 0ull;
                    pa |= (la & sb) ? in : 0ull;
                    no_t |= between;
                    no_f |= sb;
                } else {
                    no_f |= in;
                }
            } else if (n == 2) {
                const u64 m = in & mine;
                no_f |= (m != in) ? m : 0ull;
            }
        }
    }
    const u64 pinned = pf | pr | pd | pa;

    // castling squares of the opponent that its own pieces leave open
    u64 path = 0, cross = 0;
    if (b.p & (T ? 0xCull : 0x3ull)) {
        const int rights = T ? st_bc(b) : st_wc(b);
        constexpr u64 kp = T ? B_KS_PATH : W_KS_PATH, qp = T ? B_QS_PATH : W_QS_PATH, qs = T ? B_QS_SAFE : W_QS_SAFE;
        if ((rights & 1) && !(kp & own)) { path |= kp; cross |= kp; }
        if ((rights & 2) && !(qp & own)) { path |= qp; cross |= qs; }
        no_f |= path;
        no_t |= path | (path ? (T ? 0x81ull << 56 : 0x81ull) : 0ull);  // a captured corner rook takes the right
    }

    // the squares K may enter or cross: free (u0) or attacked, and those attacked once
    u64 u0, u_once, thr, tr, tb;
    {
        const u64 a0 = v.up(mrq), a1 = v.down(mrq), a2 = h.east(mrq), a3 = h.west(mrq);
        const u64 a4 = d9.up(mbq), a5 = d9.down(mbq), a6 = d7.up(mbq), a7 = d7.down(mbq);
        u64 once = a0, twice = 0;
        auto add = [&](u64 x) { twice |= once & x; once |= x; };
        add(a1); add(a2); add(a3); add(a4); add(a5); add(a6); add(a7);
        add(cap_w<S>(mp));
        add(cap_e<S>(mp));
        for (u64 s = mn; s; s &= s - 1) add(__ldg(&g_knight[lsb(s)]));
        add(__ldg(&g_king[sq_of(mk)]));
        thr = once;
        const u64 u = (ring & ~own) | cross;
        u0 = u & ~thr;
        const u64 u1 = u & thr;
        u_once = u1 & ~twice;
        // from where a slider reaches them: fills backward from the squares
        // (on ranks through a board where they are blockers, as the rank fill
        // needs its sources occupied); a slider's own fill along the same
        // direction meets them on the lines that a blocker leaving (free
        // squares) or a piece arriving (attacked ones) changes
        {
            const RankPro g(occ | u0);
            const u64 b0 = v.down(u0), b1 = v.up(u0), b2 = g.west(u0), b3 = g.east(u0);
            const u64 b4 = d9.down(u0), b5 = d9.up(u0), b6 = d7.down(u0), b7 = d7.up(u0);
            tr = b0 | b1 | b2 | b3;
            tb = b4 | b5 | b6 | b7;
            king_f |= (a0 & b0) | (a1 & b1) | (a2 & b2) | (a3 & b3) | (a4 & b4) | (a5 & b5) | (a6 & b6) | (a7 & b7);
        }
        {
            const RankPro g(occ | u1);
            king_t |= ((a0 & v.down(u1)) | (a1 & v.up(u1)) | (a2 & g.west(u1)) | (a3 & g.east(u1)) | (a4 & d9.down(u1)) |
                     (a5 & d9.up(u1)) | (a6 & d7.down(u1)) | (a7 & d7.up(u1))) & empty;
        }
    }
    // where a slider checks, or pins the one piece between
    const u64 xr = SlFancy::rook(kq, occ ^ (kr & own)), xb = SlFancy::bishop(kq, occ ^ (kb & own));
    const u64 tn = knight_set(u0), tk = king_set(u0);
    // with a castling path open, a change near the king may change castling too
    const u64 strict = path ? ~0ull : 0ull;
    const u32 k0 = popc(u0 & ring);

    // ---- the opponent's moves on the unmoved board ----
    const u64 free_ = own & ~pinned;
    const u64 op = pawns & free_;
    u32 n0 = k0;
    // a pinned slider is filled as if it were free: its moves off the pin line
    // are taken back, and nothing it sees is plain
    for (u64 s = pinned & (orq | obq); s; s &= s - 1) {
        const int q = lsb(s);
        const u64 bit = lowbit(s);
        u64 m = (orq & bit) ? SlFancy::rook(q, occ) : 0ull;
        if (obq & bit) m |= SlFancy::bishop(q, occ);
        n0 -= popc(m & ~own & ~((pf & bit) ? file_of(kq) : (pr & bit) ? rank_of(kq) : (pd & bit) ? __ldg(&g_diag[kq]) : anti_of(kq)));
        no_f |= m;
        no_t |= m;
    }
    constexpr u64 back_rank = T ? RANK_1 : RANK_8, last_rank = T ? RANK_1 << 8 : RANK_8 >> 8;
    const u64 d1 = push1<T>(op) & empty;
    const u64 mid = d1 & double_rank<T>();
    const u64 dd = push1<T>(mid) & empty;
    const u64 cw = cap_w<T>(op), ce = cap_e<T>(op);
    {
        const u64 opn = pawns & own;
        const u64 x1 = push1<T>(op | (opn & pf)) & empty;
        n0 += popc(x1) + popc(push1<T>(x1 & double_rank<T>()) & empty);
        const u64 xw = cap_w<T>(op | (opn & (T ? pd : pa))) & mine;
        const u64 xe = cap_e<T>(op | (opn & (T ? pa : pd))) & mine;
        n0 += popc(xw) + popc(xe);
        n0 += 3 * (popc(x1 & back_rank) + popc(xw & back_rank) + popc(xe & back_rank));
        if (path) n0 += can_castle_k<T>(b, occ, thr) + can_castle_q<T>(b, occ, thr);
    }
    // pieces of the mover that stand in front of an opposing pawn, and (open2) two
    // squares in front of one that could step twice; promotion squares count four
    // times: not plain
    const u64 fronts = push1<T>(op) & mine, open2 = push1<T>(mid) & mine;
    {
        const u64 pr8 = (push1<T>(op) | cw | ce) & back_rank;
        no_t |= pr8;
        no_f |= pr8;
    }

    // w: per square the replies lost when a piece arrives, plus 2: on an empty
    // square the rays cut off, the pushes blocked and (as 1 - x) the pawn
    // captures gained; on an opposing piece its moves and (as 1 - x) the pawn
    // recaptures gained.  On a square of the mover's own, the replies gained when
    // its piece leaves, plus 2: the rays opened and (as 1 - x) the pawn captures
    // lost.  The two 2s cancel.  g: the sliders and knights that recapture.
    u64 w0, w1, w2, w3, g0, g1, g2;
    {
        n0 += popc(s0 & ~own) + popc(s1 & ~own) + popc(s2 & ~own) + popc(s3 & ~own) + popc(s4 & ~own) + popc(s5 & ~own) +
              popc(s6 & ~own) + popc(s7 & ~own);
        // knights: their moves at their squares, and the first two's attacks
        u64 kc0 = 0, kc1 = 0, kc2 = 0, kc3 = 0, k1 = 0, k2 = 0;
        for (u64 s = b.n & free_; s; s &= s - 1) {
            const u64 bit = lowbit(s), m = __ldg(&g_knight[lsb(s)]);
            const u32 c = popc(m & ~own);
            n0 += c;
            const u32 c7 = c - (c >> 3);  // 8 as 7 + 1
            kc0 |= (c7 & 1) ? bit : 0ull;
            kc1 |= (c7 & 2) ? bit : 0ull;
            kc2 |= (c7 & 4) ? bit : 0ull;
            kc3 |= (c & 8) ? bit : 0ull;
            no_t |= k2 & m & own;  // three knights recapture: not plain
            k2 |= k1 & m;
            k1 |= m;
        }
        // k1: attacked by a knight, k2: by two or more
        {
            const u64 x0 = plane_sum(s0, s1, s2), y0 = plane_carry(s0, s1, s2);
            const u64 x1 = plane_sum(s3, s4, s5), y1 = plane_carry(s3, s4, s5);
            const u64 kk = k1 & ~k2;
            const u64 x2 = plane_sum(s6, s7, kk), y2 = plane_carry(s6, s7, kk);
            g0 = plane_sum(x0, x1, x2);
            const u64 y3 = plane_carry(x0, x1, x2);
            const u64 z0 = plane_sum(y0, y1, y2), c0 = plane_carry(y0, y1, y2);
            g1 = plane_sum(z0, y3, k2);
            const u64 c1 = plane_carry(z0, y3, k2);
            g2 = c0 ^ c1;
            no_t |= c0 & c1 & own;  // eight or more: not plain
            g0 &= own;
            g1 &= own;
            g2 &= own;
        }
        Planes3 q0 = targets_beyond<8, true>(s0, v.up(s0 & mine), empty, own, orq, mine);
        Planes3 q1 = targets_beyond<8, false>(s1, v.down(s1 & mine), empty, own, orq, mine);
        Planes3 q2 = targets_beyond<1, true>(s2, h.east(s2 & mine), empty, own, orq, mine);
        const Planes3 q3 = targets_beyond<1, false>(s3, h.west(s3 & mine), empty, own, orq, mine);
        Planes3 q4 = targets_beyond<9, true>(s4, d9.up(s4 & mine), empty, own, obq, mine);
        const Planes3 q5 = targets_beyond<9, false>(s5, d9.down(s5 & mine), empty, own, obq, mine);
        const Planes3 q6 = targets_beyond<7, true>(s6, d7.up(s6 & mine), empty, own, obq, mine);
        const Planes3 q7 = targets_beyond<7, false>(s7, d7.down(s7 & mine), empty, own, obq, mine);
        // knights' and pawns' moves at their own squares, where the slider
        // planes are zero
        q0.c0 |= kc0;
        q0.c1 |= kc1;
        q0.c2 |= kc2;
        q2.c0 |= kc3;
        {
            const u64 m1 = push1<S>(d1), m2 = push1<S>(push1<S>(dd));
            const u64 mw = T ? (cw & mine) << 9 : (cw & mine) >> 7, me = T ? (ce & mine) << 7 : (ce & mine) >> 9;
            q0.c0 |= m1 & ~last_rank;
            q0.c2 |= m1 & last_rank;
            q1.c0 |= m2;
            q2.c0 |= mw & ~last_rank;
            q2.c2 |= mw & last_rank;
            q4.c0 |= me & ~last_rank;
            q4.c2 |= me & last_rank;
        }
        // per line at most 7 (on an empty square at most 6, so the push planes
        // fit as carries), then the four lines and the capture planes
        u64 c;
        const u64 pd2 = dd | push1<S>(dd);
        const u64 f0 = plane_sum(q0.c0, q1.c0, d1);
        c = plane_carry(q0.c0, q1.c0, d1);
        const u64 f1 = plane_sum(q0.c1, q1.c1, c), f2 = q0.c2 ^ q1.c2 ^ plane_carry(q0.c1, q1.c1, c);
        const u64 r0 = plane_sum(q2.c0, q3.c0, pd2);
        c = plane_carry(q2.c0, q3.c0, pd2);
        const u64 r1 = plane_sum(q2.c1, q3.c1, c), r2 = q2.c2 ^ q3.c2 ^ plane_carry(q2.c1, q3.c1, c);
        const u64 e0 = q4.c0 ^ q5.c0;
        c = q4.c0 & q5.c0;
        const u64 e1 = plane_sum(q4.c1, q5.c1, c), e2 = q4.c2 ^ q5.c2 ^ plane_carry(q4.c1, q5.c1, c);
        const u64 i0 = q6.c0 ^ q7.c0;
        c = q6.c0 & q7.c0;
        const u64 i1 = plane_sum(q6.c1, q7.c1, c), i2 = q6.c2 ^ q7.c2 ^ plane_carry(q6.c1, q7.c1, c);
        const u64 a0 = plane_sum(f0, r0, ~cw);
        c = plane_carry(f0, r0, ~cw);
        const u64 a1 = plane_sum(f1, r1, c);
        c = plane_carry(f1, r1, c);
        const u64 a2 = plane_sum(f2, r2, c), a3 = plane_carry(f2, r2, c);
        const u64 b0 = plane_sum(e0, i0, ~ce);
        c = plane_carry(e0, i0, ~ce);
        const u64 b1 = plane_sum(e1, i1, c);
        c = plane_carry(e1, i1, c);
        const u64 b2 = plane_sum(e2, i2, c), b3 = plane_carry(e2, i2, c);
        w0 = a0 ^ b0;
        c = a0 & b0;
        w1 = plane_sum(a1, b1, c);
        c = plane_carry(a1, b1, c);
        w2 = plane_sum(a2, b2, c);
        c = plane_carry(a2, b2, c);
        w3 = plane_sum(a3, b3, c);
        const u64 w4 = plane_carry(a3, b3, c);  // 16 or more: not plain
        no_t |= w4;
        no_f |= w4;
    }

    // ---- the mover's moves ----
    // m: how many plain moves reach each square (0..7; a square already
    // reached by seven is not plain for the next piece)
    u64 m0 = 0, m1 = 0, m2 = 0;
    u32 sum = 0;
    auto reach = [&](u64 s) {
        const u64 k0 = m0 & s;
        m0 ^= s;
        const u64 k1 = m1 & k0;
        m1 ^= k0;
        m2 ^= k1;
    };
    auto full = [&]() { return m0 & m1 & m2; };

    // pawns, by target square
    constexpr int PUSH = S ? -8 : 8, CW = S ? -9 : 7, CE = S ? -7 : 9;
    {
        const u64 tgt = f.tgt;
        const u64 fp = mp & ~f.pinned;
        const u64 pin_ok = ~f.chk_all;
        const u64 x1 = push1<S>(fp | (mp & f.pf & pin_ok)) & empty;
        const u64 one = x1 & tgt;
        const u64 two = push1<S>(x1 & double_rank<S>() & ~f.safe) & empty & tgt;
        const u64 xw = cap_w<S>(fp | (mp & (S ? f.pd : f.pa) & pin_ok)) & own & tgt;
        const u64 xe = cap_e<S>(fp | (mp & (S ? f.pa : f.pd) & pin_ok)) & own & tgt;
        // squares a pawn may not leave (fronts: a push stays in an opposing pawn's way), may
        // not leave along the file or a diagonal an opposing slider sees it on
        // (t on that line), and may not reach; near: only the king's moves change
        const u64 near_f = king_f | cap_w<T>(u_once) | cap_e<T>(u_once);
        const u64 near_t = king_t | pawn_attackers_of<T>(u0);
        const u64 no = no_t | pawn_attackers_of<T>(king) | BACK_RANKS | (near_t & strict);
        const u64 stay_x = no_f | (near_f & strict), stay = stay_x | fronts | open2;
        // the replies that leaving the squares of x gives, plus 2 a square
        // the pushes a capturing pawn leaves open behind it
        auto pushes = [&](u64 x) { return popc(x & (fronts | open2)) + popc(push1<T>(x & fronts & double_rank<T>()) & empty); };
        auto leave = [&](u64 x) { return popc(x & w0) + 2 * popc(x & w1) + 4 * popc(x & w2) + 8 * popc(x & w3); };
        {
            const u64 ok = one & ~no & ~push1<S>(stay | s0 | s1);
            const u64 from = push1<T>(ok), by_king = ok & (near_t | push1<S>(near_f));
            reach(ok);
            sum += popc(ok) * n0 + leave(from);
            const u64 rest = one & ~ok & ~BACK_RANKS;
            emit.sets(pawn_set<PUSH>(rest), pawn_set<PUSH>(by_king), pawn_entry<PUSH>(), 65u);
            put_promotions(emit, one & BACK_RANKS, PUSH);
        }
        {
            const u64 ep = (pawns & own);
            const u64 epf = two & (east1(ep) | west1(ep));
            const u64 ok = two & ~(no | epf) & ~push1<S>(push1<S>(stay | s0 | s1));
            const u64 from = push1<T>(push1<T>(ok)), by_king = ok & (near_t | push1<S>(push1<S>(near_f)));
            reach(ok);
            sum += popc(ok) * n0 + leave(from);
            const u64 rest = two & ~ok & ~epf;
            emit.sets(pawn_set<2 * PUSH>(rest), pawn_set<2 * PUSH>(by_king), pawn_entry<2 * PUSH>(MF_DOUBLE), 65u);
            each_square(epf, [&](int t) { emit.put_ep(cmove(t - 2 * PUSH, t, MF_DOUBLE) | Q_EP); });
        }
        // captures: a pawn captured there attacks the capturing pawn itself,
        // which its own moves (w at its square) already hold
        {
            const u64 ok = xw & ~no & ~cap_w<S>(stay_x | (S ? s4 | s5 : s6 | s7));
            const u64 from = S ? ok << 9 : ok >> 7, by_king = ok & (near_t | cap_w<S>(near_f));
            reach(ok);
            sum += popc(ok) * n0 + leave(from) + popc(from & ce) + pushes(from);
            const u64 rest = xw & ~ok & ~BACK_RANKS;
            emit.sets(pawn_set<CW>(rest), pawn_set<CW>(by_king), pawn_entry<CW>(), 65u);
            put_promotions(emit, xw & BACK_RANKS, CW);
        }
        {
            const u64 ok = xe & ~no & ~cap_e<S>(stay_x | (S ? s6 | s7 : s4 | s5));
            const u64 from = S ? ok << 7 : ok >> 9, by_king = ok & (near_t | cap_e<S>(near_f));
            reach(ok);
            sum += popc(ok) * n0 + leave(from) + popc(from & cw) + pushes(from);
            const u64 rest = xe & ~ok & ~BACK_RANKS;
            emit.sets(pawn_set<CE>(rest), pawn_set<CE>(by_king), pawn_entry<CE>(), 65u);
            put_promotions(emit, xe & BACK_RANKS, CE);
        }
    }
    emit_castles_ep<S>(b, f, [&](u16 mv, u32 pc) { emit.put((u32)mv | (pc << Q_PIECE_SHIFT)); });

    // one piece's moves to the squares of `to`: no / near: the squares where they
    // are not plain / only the king's moves change
    auto piece = [&](int q, u64 bit, u64 to, u64 att, u64 no, u64 near, u32 pc) {
        const bool hi = q >= 32;
        const u32 sq = q & 31;
        auto at = [&](u64 x) { return ((hi ? (u32)(x >> 32) : (u32)x) >> sq) & 1u; };
        // pawns that could capture it, the pawn it blocks and that pawn's second
        // step, the pawn whose second step it blocks and that one's first: t there
        // is not plain
        const u64 pawn_att = __ldg(&g_pawn_checks[S][q]) & op, in_front = fronts & bit, front = push1<S>(in_front);
        const u64 second = push1<T>(in_front & double_rank<T>()), back2 = push1<S>(open2 & bit);
        no |= no_t | full() | pawn_att | front | second | back2 | push1<S>(back2);
        near |= king_t;
        if ((bit & king_f) | (att & u_once)) near = ~0ull;
        no |= near & strict;
        if (bit & no_f) no = ~0ull;
        const u64 plain = to & ~no, by_king = plain & near, rest = to & no;
        reach(plain);
        sum += popc(plain) * (n0 + (front != 0) + ((second & empty) != 0) + (back2 != 0) + at(w0) + 2 * at(w1) + 4 * at(w2) + 8 * at(w3));
        emit.sets(rest, by_king, (u32)q | (pc << Q_PIECE_SHIFT), 64u);
    };
    const u64 sv = s0 | s1, sh = s2 | s3, sd = s4 | s5, sa = s6 | s7;
    // the king and the knights
    for (u64 s = mk | (mn & ~f.pinned); s; s &= s - 1) {
        const int q = lsb(s);
        const u64 bit = lowbit(s);
        const bool is_k = (mk & bit) != 0;
        const u64 att = is_k ? __ldg(&g_king[q]) : __ldg(&g_knight[q]);
        // a king that an opposing slider sees (in check) may stay on its line
        const u64 no = is_k ? ((bit & (sv | sh | sd | sa)) ? ~0ull : 0ull) : __ldg(&g_knight[kq]);
        piece(q, bit, att & (is_k ? ~(f.threat | mine) : f.tgt), att, no, is_k ? tk : tn, is_k ? PC_KING : PC_KNIGHT);
    }
    for (u64 s = (mrq | mbq) & ~(f.pinned & f.chk_all); s; s &= s - 1) {
        const int q = lsb(s);
        const u64 bit = lowbit(s);
        const bool is_r = (mrq & bit) != 0, is_b = (mbq & bit) != 0;
        const u64 fl = file_of(q), rk = rank_of(q), dg = __ldg(&g_diag[q]), an = anti_of(q);
        const u64 att = (is_r ? SlFancy::rook(q, occ) : 0ull) | (is_b ? SlFancy::bishop(q, occ) : 0ull);
        u64 to = att & f.tgt;
        if (f.pinned & bit) to &= (f.pf & bit) ? fl : (f.pr & bit) ? rk : (f.pd & bit) ? dg : an;
        // along a line on which an opposing slider sees it
        const u64 no = (is_r ? xr : 0ull) | (is_b ? xb : 0ull) | ((sv & bit) ? fl : 0ull) | ((sh & bit) ? rk : 0ull) |
                       ((sd & bit) ? dg : 0ull) | ((sa & bit) ? an : 0ull);
        piece(q, bit, to, att, no, (is_r ? tr : 0ull) | (is_b ? tb : 0ull), is_r ? (is_b ? PC_QUEEN : PC_ROOK) : PC_BISHOP);
    }

    // the corrections of the squares reached
    auto planes = [&](u64 x, u32 unit) {
        sum += unit * (popc(x & g0) - popc(x & w0)) + (2 * unit) * (popc(x & g1) - popc(x & w1)) +
               (4 * unit) * (popc(x & g2) - popc(x & w2)) - (8 * unit) * popc(x & w3);
    };
    planes(m0, 1);
    planes(m1, 2);
    planes(m2, 4);
    return (u64)(sum - emit.kings * k0);
}

}  // namespace pg
