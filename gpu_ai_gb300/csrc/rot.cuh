// rot.cuh -- the playout kernels' plies on rotated bitboards, seen from the side to move.
//
// Layout.  rules.cuh keeps dark square s = row*4 + c on bit s, where a
// diagonal step shifts even and odd rows by different amounts (two masked
// shifts).  Here square (row, c) sits on bit
//
//     26 + 8*(row/2) + row%2 + 6*c   (mod 32),
//
// which makes every step one rotation: (+1,+1) rotates left by 7, (+1,-1)
// left by 1, (-1,+1) right by 1, (-1,-1) right by 7 for all rows, and a mask
// drops the squares that leave the board.  A jump source mask is then one
// 3-input logic operation on two rotated words (rules.cuh: nine operations),
// and the kernel that runs these plies is bound by its integer pipe.  A row's
// four squares are 6 bits apart, so per-square move counts (0..8) of a row
// are already spread out for a multiply that takes their prefix sums.
//
// Orientation.  Boards are kept from the side to move: its pieces move up the
// board (men: directions 0 and 1).  Turning the board by 180 degrees maps bit
// b to bit 31 - b (the offset 26 is chosen for that), so passing the turn is
// three bit reversals and a swap, and no ply selects masks by the player.
// Under that turn PLAYER_2's move list (rules.cuh) is exactly reversed -- its
// squares descend, and so do the directions of a square -- so move i of its n
// moves is move n-1-i of the list in this orientation.
#pragma once

#include "rules.cuh"

namespace ga {
namespace rot {

GA_HD constexpr uint32_t rotl_c(uint32_t x, uint32_t s) { return (s & 31u) ? (x << (s & 31u)) | (x >> (32u - (s & 31u))) : x; }

GA_HD uint32_t rotl(uint32_t x, uint32_t s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(x, x, s);
#else
  return rotl_c(x, s);
#endif
}
GA_HD uint32_t rotr(uint32_t x, uint32_t s) {
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(x, x, s);
#else
  return rotl_c(x, 32u - (s & 31u));
#endif
}

GA_HD uint32_t reverse(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __brev(x);
#else
  uint32_t r = 0;
  for (int i = 0; i < 32; i++) r |= ((x >> i) & 1u) << (31 - i);
  return r;
#endif
}

constexpr uint32_t kOffset = 26u;
GA_HD constexpr uint32_t bit_of(uint32_t row, uint32_t c) { return (kOffset + 8u * (row >> 1) + (row & 1u) + 6u * c) & 31u; }

// Squares of the rows and columns (c = 0..3) whose bits are set.
GA_HD constexpr uint32_t squares(uint32_t rows, uint32_t even_cols, uint32_t odd_cols) {
  uint32_t m = 0;
  for (uint32_t r = 0; r < 8; r++)
    for (uint32_t c = 0; c < 4; c++)
      if (((rows >> r) & 1u) && ((((r & 1u) ? odd_cols : even_cols) >> c) & 1u)) m |= 1u << bit_of(r, c);
  return m;
}
// Squares from which a step (kStep) or a jump (kJump) in direction d stays on the board.
constexpr uint32_t kStep0 = squares(0x7fu, 0x7u, 0xfu), kStep1 = squares(0x7fu, 0xfu, 0xeu);
constexpr uint32_t kStep2 = squares(0xfeu, 0x7u, 0xfu), kStep3 = squares(0xfeu, 0xfu, 0xeu);
constexpr uint32_t kHop0 = squares(0x3fu, 0x7u, 0x7u), kHop1 = squares(0x3fu, 0xeu, 0xeu);
constexpr uint32_t kHop2 = squares(0xfcu, 0x7u, 0x7u), kHop3 = squares(0xfcu, 0xeu, 0xeu);
constexpr uint32_t kRows03 = squares(0x0fu, 0xfu, 0xfu), kRows01 = squares(0x03u, 0xfu, 0xfu),
                   kRows45 = squares(0x30u, 0xfu, 0xfu), kFirstRow = squares(0x01u, 0xfu, 0xfu),
                   kFarRow = squares(0x80u, 0xfu, 0xfu);
static_assert(rotl_c(kRows01, 16) == kRows45, "rows two apart are 8 bits apart");
static_assert(kFirstRow == rotl_c(0x00041041u, kOffset), "the squares of a row are 6 bits apart");

// Left rotation of a step in direction 0..3, a byte each.
constexpr uint32_t kTurns = 7u | (1u << 8) | (31u << 16) | (25u << 24);

// Conversion of a square set: the squares of one column and row parity all
// rotate alike.
GA_HD uint32_t to_rot(uint32_t x) {
  uint32_t r = 0;
GA_UNROLL
  for (uint32_t c = 0; c < 4; c++) {
    r |= rotl(x, kOffset + 5u * c) & rotl_c(0x01010101u, kOffset + 6u * c);
    r |= rotl(x, kOffset + 5u * c - 3u) & rotl_c(0x01010101u, kOffset + 6u * c + 1u);
  }
  return r;
}
GA_HD uint32_t from_rot(uint32_t x) {
  uint32_t r = 0;
GA_UNROLL
  for (uint32_t c = 0; c < 4; c++) {
    r |= rotr(x, kOffset + 5u * c) & (0x01010101u << c);
    r |= rotr(x, kOffset + 5u * c - 3u) & (0x10101010u << c);
  }
  return r;
}

// A board from the side to move; meta as in Board.
struct RotBoard {
  uint32_t own, opp, kings, meta;
};

GA_HD RotBoard from_board(const Board &b) {
  const uint32_t p1 = to_rot(b.p1), p2 = to_rot(b.p2), k = to_rot(b.kings);
  if (b.meta & 1u) return RotBoard{reverse(p2), reverse(p1), reverse(k), b.meta};
  return RotBoard{p1, p2, k, b.meta};
}
GA_HD Board to_board(const RotBoard &b) {
  if (b.meta & 1u) return Board{from_rot(reverse(b.opp)), from_rot(reverse(b.own)), from_rot(reverse(b.kings)), b.meta};
  return Board{from_rot(b.own), from_rot(b.opp), from_rot(b.kings), b.meta};
}

// The piece on `from` (one bit) goes to `to`, capturing `removed`; the turn passes.
GA_HD void apply(RotBoard &b, uint32_t from, uint32_t to, uint32_t removed) {
  const uint32_t own = (b.own & ~from) | to, opp = b.opp & ~removed;
  const uint32_t crowned = (b.kings & from) ? to : (to & kFarRow);
  const uint32_t kings = (b.kings & ~(removed | from)) | crowned;
  b.own = reverse(opp);
  b.opp = reverse(own);
  b.kings = reverse(kings);
  // the turn passes; the plies since a capture (from bit 8 on) restart after one
  b.meta = (removed ? b.meta & 1u : b.meta + 256u) ^ 1u;
}

// A position's jump sources by direction, its first jumps by kind of piece, and
// whether some capture can continue.
struct View {
  uint32_t empty, king, man;      // king, man: pieces of the side to move
  uint32_t j0, j1, j2, j3;        // squares with an opponent next to them and an empty square behind it
  uint32_t m0, m1;                // men's first jumps
  uint32_t k0, k1, k2, k3;        // kings' first jumps
  uint32_t cont_king, cont_man;   // landing squares from which a king / a man can jump on
  bool capture;
};

GA_HD View view(const RotBoard &b) {
  View v;
  v.empty = ~(b.own | b.opp);
  v.king = b.own & b.kings;
  v.man = b.own & ~b.kings;
  v.j0 = rotr(b.opp, 7) & rotr(v.empty, 14) & kHop0;
  v.j1 = rotr(b.opp, 1) & rotr(v.empty, 2) & kHop1;
  v.j2 = rotl(b.opp, 1) & rotl(v.empty, 2) & kHop2;
  v.j3 = rotl(b.opp, 7) & rotl(v.empty, 14) & kHop3;
  v.m0 = v.man & v.j0;
  v.m1 = v.man & v.j1;
  v.k0 = v.king & v.j0;
  v.k1 = v.king & v.j1;
  v.k2 = v.king & v.j2;
  v.k3 = v.king & v.j3;
  const uint32_t ahead = v.j0 | v.j1;
  v.cont_man = (rotl(v.m0, 14) | rotl(v.m1, 2)) & ahead;
  v.cont_king = (rotl(v.k0, 14) | rotl(v.k1, 2) | rotr(v.k2, 2) | rotr(v.k3, 14)) & (ahead | v.j2 | v.j3);
  v.capture = ((b.own & ahead) | v.k2 | v.k3) != 0;
  return v;
}

// The move masks of a position, the masks of the directions in list order per
// square: a man's captures list direction 1 before direction 0, so the men
// that capture have the first two masks swapped.
struct Masks {
  uint32_t m0, m1, m2, m3;
};

GA_HD Masks masks(const RotBoard &b, const View &v) {
  Masks m;
  m.m0 = v.capture ? v.k0 | v.m1 : b.own & rotr(v.empty, 7) & kStep0;
  m.m1 = v.capture ? v.k1 | v.m0 : b.own & rotr(v.empty, 1) & kStep1;
  m.m2 = v.capture ? v.k2 : v.king & rotl(v.empty, 1) & kStep2;
  m.m3 = v.capture ? v.k3 : v.king & rotl(v.empty, 7) & kStep3;
  return m;
}

// Move masks packed two to a word by half of the board: `lo` rows 0-3, `hi`
// rows 4-7, each word with the first mask's half in place and the second
// mask's half turned by 16 (four rows) into the free half.
struct Packed {
  uint32_t lo_a, lo_b, hi_a, hi_b;  // a: masks 0 and 2, b: masks 1 and 3
  uint32_t low, n;                  // moves in the low half, in all
};

// The two quarters (rows 0-1 and 4-5) whose moves come first in their half.
constexpr uint32_t kQuarters = kRows01 | kRows45;

GA_HD Packed pack(const Masks &m) {
  const uint32_t r2 = rotl(m.m2, 16), r3 = rotl(m.m3, 16);
  Packed p;
  p.lo_a = (m.m0 & kRows03) | (r2 & ~kRows03);
  p.hi_a = (m.m0 & ~kRows03) | (r2 & kRows03);
  p.lo_b = (m.m1 & kRows03) | (r3 & ~kRows03);
  p.hi_b = (m.m1 & ~kRows03) | (r3 & kRows03);
  p.low = (uint32_t)(popc(p.lo_a) + popc(p.lo_b));
  p.n = p.low + (uint32_t)(popc(p.hi_a) + popc(p.hi_b));
  return p;
}

// Move i of the list: its source (one bit) and the place 0..3 of its
// direction's mask.  Halvings that count with POPC (the XU pipe, not the busy
// integer pipe): the half of the board; the quarter (two rows), whose four
// masks of eight squares are packed into one word, turned to a fixed place:
// the even row's squares on the even bits, column c and mask d on bit
// 8d + 6c; then the row, the pair of columns and the column.  That leaves one
// bit per mask, 8 apart: one multiply takes their prefix sums, one
// subtraction compares them with the index left (bytes of 128 + i - prefix).
GA_HD void nth(const Packed &p, uint32_t i, uint32_t &from, uint32_t &place) {
  // (conditional assignments, which compile to predicated instructions, where
  // selects would be: 2.10 -> 2.05 ms on 20,011 positions with 4.0 M playouts)
  uint32_t a = p.lo_a, b = p.lo_b, at = kOffset, sel = kQuarters;
  if (i >= p.low) {
    i -= p.low;
    a = p.hi_a;
    b = p.hi_b;
    at = kOffset + 16u;
  }
  uint32_t c = (uint32_t)(popc(a & kQuarters) + popc(b & kQuarters));
  if (i >= c) {
    i -= c;
    at += 8u;
    sel = ~kQuarters;
  }
  uint32_t z = rotr((a & sel) | (rotl(b, 8) & ~sel), at);
  c = (uint32_t)popc(z & 0x55555555u);
  if (i >= c) {
    i -= c;
    at += 1u;
    z >>= 1;
  }
  c = (uint32_t)popc(z & 0x41414141u);
  if (i >= c) {
    i -= c;
    at += 12u;
    z = rotr(z, 12);
  }
  c = (uint32_t)popc(z & 0x01010101u);
  if (i >= c) {
    i -= c;
    at += 6u;
    z = rotr(z, 6);
  }
  const uint32_t t = i * 0x01010101u + 0x80808080u - (z & 0x01010101u) * 0x01010101u;
  place = (uint32_t)popc(t & 0x00808080u);
  from = rotl(1u, at);
}

// Left rotation of the step of a move: the place is the direction, but for a
// man's captures, whose first two masks were swapped.
GA_HD uint32_t turn_of(const View &v, uint32_t from, uint32_t place) {
  const uint32_t swap = v.capture && (v.man & from) ? 1u : 0u;
  return kTurns >> (8u * (place ^ swap));
}

// Per-square counts (0..8) of a men's multi-jump ply as bit planes.
struct Planes {
  uint32_t s0, s1, s2, s3;
};

GA_HD uint32_t count_in(const Planes &p, uint32_t m) {
  return (uint32_t)(popc(p.s0 & m) + 2 * popc(p.s1 & m) + 4 * popc(p.s2 & m) + 8 * popc(p.s3 & m));
}

// The square that holds entry i of the list whose per-square counts are p
// (squares ascending), as a bit position; i becomes the entry's index within
// the square.  Three halvings over the rows, as in nth; within the row the four
// counts sit 6 bits apart, one multiply sums them up, one subtraction compares
// every prefix with i (fields of 6 bits: 32 + i - prefix, i <= 31 and the
// prefix <= 32, so no field borrows).
GA_HD uint32_t square_of(const Planes &p, uint32_t &i) {
  constexpr uint32_t F = 0x00041041u, H = 0x00820820u;
  const uint32_t c1 = count_in(p, kRows03);
  const bool u1 = i >= c1;
  i -= u1 ? c1 : 0u;
  const uint32_t c2 = count_in(p, u1 ? kRows45 : kRows01);
  const bool u2 = i >= c2;
  i -= u2 ? c2 : 0u;
  uint32_t at = (u1 ? kOffset + 16u : kOffset) + (u2 ? 8u : 0u);
  const uint32_t c3 = count_in(p, rotl(F, at));
  const bool u3 = i >= c3;
  i -= u3 ? c3 : 0u;
  at += u3 ? 1u : 0u;
  const uint32_t q =
      (rotr(p.s0, at) & F) + 2u * (rotr(p.s1, at) & F) + 4u * (rotr(p.s2, at) & F) + 8u * (rotr(p.s3, at) & F);
  const uint32_t d = i * F + H - q * F;  // field k: 32 + i - (counts of squares 0..k of the row)
  const uint32_t sq = 6u * (uint32_t)popc(d & 0x00020820u);
  i = ((d * 64u + i) >> sq) & 31u;
  return at + sq;
}

// A capture ply with one first jump whose chain never forks has one legal
// move: the chain is followed here (captured pieces stay on the board) and
// played; no draw is taken.  Returns false, the board untouched, when the
// chain forks or reaches the depth limit.  A man only goes forward, at most
// three jumps, so its chain needs no visited squares and no backward
// directions; it has its own loop because it is four times as common (one loop
// for both: 2.20 against 2.15 ms on 20,011 positions with 4.0 M playouts).
GA_HD bool play_man_chain(RotBoard &b, const View &v) {
  const uint32_t from = v.m0 | v.m1;  // one bit
  uint32_t removed = rotl(v.m0, 7) | rotl(v.m1, 1), to = rotl(v.m0, 14) | rotl(v.m1, 2);
GA_UNROLL
  for (int k = 0; k < 3; k++) {
    const uint32_t l0 = rotl(to & v.j0, 14), l1 = rotl(to & v.j1, 2);
    if (l0 && l1) return false;
    const uint32_t land = l0 | l1;
    if (!land) break;
    removed |= rotr(l0, 7) | rotr(l1, 1);
    to = land;
  }
  apply(b, from, to, removed);
  return true;
}

// A king's chain never lands twice on a square.
GA_HD bool play_king_chain(RotBoard &b, const View &v) {
  const uint32_t from = v.k0 | v.k1 | v.k2 | v.k3;  // one bit
  uint32_t removed = rotl(v.k0, 7) | rotl(v.k1, 1) | rotr(v.k2, 1) | rotr(v.k3, 7);
  uint32_t to = rotl(v.k0, 14) | rotl(v.k1, 2) | rotr(v.k2, 2) | rotr(v.k3, 14), visited = to;
  for (int depth = 1;; depth++) {  // ends: each jump lands on a square not yet visited
    const uint32_t l0 = rotl(to & v.j0, 14) & ~visited, l1 = rotl(to & v.j1, 2) & ~visited;
    const uint32_t l2 = rotr(to & v.j2, 2) & ~visited, l3 = rotr(to & v.j3, 14) & ~visited;
    const uint32_t land = l0 | l1 | l2 | l3;
    if (land == 0) break;
    if ((land & (land - 1u)) != 0 || depth >= kMaxDepth) return false;
    removed |= rotr(l0, 7) | rotr(l1, 1) | rotl(l2, 1) | rotl(l3, 7);
    to = land;
    visited |= land;
  }
  apply(b, from, to, removed);
  return true;
}

GA_HD bool play_chain(RotBoard &b, const View &v) {
  return v.cont_king ? play_king_chain(b, v) : play_man_chain(b, v);
}

// A capture ply where some man can jump on but no king can.  The number of
// ways a man that landed on a square can go on (1..4; 1: it stops) depends on
// the board alone (men only go forward), so it is computed for every square at
// once as bit planes, twice (a man jumps at most three times); a source
// square's count is the sum over its first jumps.  Move i is found by
// square_of on those counts and by descending: direction 1 comes first.
template <class Pick>
GA_HD int play_men(RotBoard &b, const View &v, Pick &&pick) {
  const uint32_t fork = v.j0 & v.j1, none = ~(v.j0 | v.j1);
  const uint32_t p0 = ~fork, p1 = fork;  // after one more jump
  const uint32_t a0 = rotr(p0, 14) & v.j0, a1 = rotr(p1, 14) & v.j0;
  const uint32_t e0 = rotr(p0, 2) & v.j1, e1 = rotr(p1, 2) & v.j1;
  const uint32_t k0 = a0 & e0;
  const uint32_t c0 = (a0 ^ e0) | none, c1 = a1 ^ e1 ^ k0, c2 = (a1 & e1) | (k0 & (a1 ^ e1));
  // ways of each first jump, on its source square
  const uint32_t x0 = rotr(c0, 14) & v.m0, x1 = rotr(c1, 14) & v.m0, x2 = rotr(c2, 14) & v.m0;
  const uint32_t y0 = rotr(c0, 2) & v.m1, y1 = rotr(c1, 2) & v.m1, y2 = rotr(c2, 2) & v.m1;
  // kings: single jumps
  const uint32_t kx = v.k0 ^ v.k1 ^ v.k2, kc = (v.k0 & v.k1) | (v.k0 & v.k2) | (v.k1 & v.k2);
  const uint32_t g0 = x0 & y0, h1 = x1 ^ y1, g1 = (x1 & y1) | (g0 & h1), h2 = x2 ^ y2;
  Planes p;
  p.s0 = (x0 ^ y0) | (kx ^ v.k3);
  p.s1 = (h1 ^ g0) | (kc ^ (kx & v.k3));
  p.s2 = (h2 ^ g1) | (kc & kx & v.k3);
  p.s3 = (x2 & y2) | (g1 & h2);
  const uint32_t n = count_in(p, ~0u);
  uint32_t i = pick(n);
  i = (b.meta & 1u) ? n - 1u - i : i;
  const uint32_t from = rotl(1u, square_of(p, i));
  uint32_t to, removed;
  if (v.king & from) {
    // a king's single jump: the i-th direction present
    const uint32_t q0 = (v.k0 & from) ? 1u : 0u, q1 = q0 + ((v.k1 & from) ? 1u : 0u),
                   q2 = q1 + ((v.k2 & from) ? 1u : 0u);
    const uint32_t d = (i >= q0 ? 8u : 0u) + (i >= q1 ? 8u : 0u) + (i >= q2 ? 8u : 0u);
    removed = rotl(from, kTurns >> d);
    to = rotl(removed, kTurns >> d);
  } else {
    removed = 0;
    to = from;
    uint32_t t1 = from & v.m1, t0 = from & v.m0;
    while (t0 | t1) {
      const uint32_t l = rotl(t1, 2);  // 0 when direction 1 is not possible
      const uint32_t w = ((c0 & l) ? 1u : 0u) + ((c1 & l) ? 2u : 0u) + ((c2 & l) ? 4u : 0u);
      const bool second = i >= w;
      i -= second ? w : 0u;
      const uint32_t t = second ? 7u : 1u;
      const uint32_t mid = rotl(to, t);
      removed |= mid;
      to = rotl(mid, t);
      t1 = to & v.j1;
      t0 = to & v.j0;
    }
  }
  apply(b, from, to, removed);
  return (int)n;
}

// One uniformly random ply, the move and draws of play_ply_sched: returns the
// number of legal moves (0: the side to move has lost), -1 on a limit, or
// kNeedMen / kNeedKing when a ply of that kind is not allowed now.  King
// captures that go on and fork take the depth-first search of rules.cuh.
template <class Pick>
GA_HD int play_ply_random(RotBoard &b, Pick &&pick, bool men_now, bool king_now) {
  const View v = view(b);
  const Packed p = pack(masks(b, v));
  const uint32_t n = p.n;
  if (v.cont_king | v.cont_man) {
    if (n == 1u && play_chain(b, v)) return 1;
    if (v.cont_king) {
      if (!king_now) return kNeedKing;
      Board s = to_board(b);
      const int c = play_ply(s, pick);
      b = from_board(s);
      return c;
    }
    if (!men_now) return kNeedMen;
    return play_men(b, v, pick);
  }
  if (n == 0) return 0;
  uint32_t i = pick(n), from, place;
  i = (b.meta & 1u) ? n - 1u - i : i;
  nth(p, i, from, place);
  const uint32_t turn = turn_of(v, from, place), next = rotl(from, turn);
  apply(b, from, v.capture ? rotl(next, turn) : next, v.capture ? next : 0u);
  return (int)n;
}

// ---- eps-greedy

// Bit plane q of the value c - row.
GA_HD constexpr uint32_t row_plane(uint32_t q, uint32_t c) {
  uint32_t rows = 0;
  for (uint32_t r = 0; r < 8; r++) rows |= (((c - r) >> q) & 1u) << r;
  return squares(rows, 0xfu, 0xfu);
}

// The gains (eps_delta + 1, at most 13) of the jumps m of one direction as
// four bit planes, on the jumping squares: a captured king 8, a captured man 4
// + its advancement (C - row: C = 10 for a jump up the board, 12 for one down
// it), plus 1 for a king's jump, 3 for a man's, 0 for one that promotes.
template <uint32_t C>
GA_HD void jump_gains(uint32_t m, uint32_t king_taken, uint32_t king, uint32_t man, uint32_t y[4]) {
  constexpr uint32_t crowning = squares(0x20u, 0xfu, 0xfu);
  constexpr uint32_t w0 = row_plane(0, C), w1 = row_plane(1, C), w2 = row_plane(2, C), w3 = row_plane(3, C);
  const uint32_t ck = m & king_taken;
  const uint32_t x0 = w0 & ~ck, x1 = w1 & ~ck, x2 = w2 & ~ck, x3 = w3 | ck;
  const uint32_t a1 = m & man & ~crowning, a0 = (m & king) | a1;
  const uint32_t c0 = x0 & a0, c1 = (x1 & a1) | (c0 & (x1 ^ a1)), c2 = x2 & c1;
  y[0] = x0 ^ a0;
  y[1] = x1 ^ a1 ^ c0;
  y[2] = x2 ^ c1;
  y[3] = x3 ^ c2;
}

// One eps-greedy ply, the move and draws of play_ply_eps_sched (rules.cuh
// explains the values): the moves of largest gain are a subset of the move
// masks, found from the top bit plane down.
template <class Rng>
GA_HD int play_ply_eps(RotBoard &b, Rng &rs, bool men_now, bool king_now) {
  const View v = view(b);
  Masks m = masks(b, v);
  Packed p = pack(m);
  const uint32_t n = p.n;
  if (v.cont_king | v.cont_man) {
    if (n == 1u && play_chain(b, v)) return 1;
    if (v.cont_king ? !king_now : !men_now) return v.cont_king ? kNeedKing : kNeedMen;
    Board s = to_board(b);
    const int c = ply_eps_greedy(s, rs);
    b = from_board(s);
    return c;
  }
  if (n == 0) return 0;
  uint32_t i = 0;
  if (n >= 2u) {
    // by direction (the swap of a man's captures undone)
    uint32_t b0 = m.m0, b1 = m.m1, b2 = m.m2, b3 = m.m3;
    if (v.capture) {
      b0 = v.k0 | v.m0;
      b1 = v.k1 | v.m1;
      const uint32_t oppk = b.opp & b.kings;
      uint32_t y0[4], y1[4], y2[4], y3[4];
      jump_gains<10>(b0, rotr(oppk, 7), v.king, v.man, y0);
      jump_gains<10>(b1, rotr(oppk, 1), v.king, v.man, y1);
      jump_gains<12>(b2, rotl(oppk, 1), v.king, v.man, y2);
      jump_gains<12>(b3, rotl(oppk, 7), v.king, v.man, y3);
GA_UNROLL
      for (int q = 3; q >= 0; q--) {
        const uint32_t t0 = b0 & y0[q], t1 = b1 & y1[q], t2 = b2 & y2[q], t3 = b3 & y3[q];
        const bool any = (t0 | t1 | t2 | t3) != 0;
        b0 = any ? t0 : b0;
        b1 = any ? t1 : b1;
        b2 = any ? t2 : b2;
        b3 = any ? t3 : b3;
      }
      const uint32_t s0 = (b0 & v.king) | (b1 & v.man), s1 = (b1 & v.king) | (b0 & v.man);
      b0 = s0;
      b1 = s1;
    } else {
      // a man's step 1, a king's 0, a promoting step -2
      constexpr uint32_t crowning = squares(0x40u, 0xfu, 0xfu);
      const uint32_t plain = v.man & ~crowning;
      const bool some = ((b0 | b1) & plain) != 0, kings = ((b0 | b1 | b2 | b3) & v.king) != 0;
      const uint32_t pick = some ? plain : (kings ? v.king : v.man);
      b0 &= pick;
      b1 &= pick;
      b2 &= pick;
      b3 &= pick;
    }
    if (rs.next() >= kEpsThreshold) p = pack(Masks{b0, b1, b2, b3});
    const uint32_t cnt = p.n;
    if (cnt >= 2u) {
      i = mulhi_index(rs.next(), cnt);
      i = (b.meta & 1u) ? cnt - 1u - i : i;
    }
  }
  uint32_t from, place;
  nth(p, i, from, place);
  const uint32_t turn = turn_of(v, from, place), next = rotl(from, turn);
  apply(b, from, v.capture ? rotl(next, turn) : next, v.capture ? next : 0u);
  return (int)n;
}

// ---- reference heuristic

// Draws by their number, for a policy that takes many of them in a row: block
// b of four is generated where it is needed.
struct BlockDraws {
  uint32_t k0, k1, id0, id1, k;  // k: draws consumed

  GA_HD void start(uint64_t seed, uint64_t id) {
    k0 = (uint32_t)seed;
    k1 = (uint32_t)(seed >> 32);
    id0 = (uint32_t)id;
    id1 = (uint32_t)(id >> 32);
    k = 0;
  }
  GA_HD void block(uint32_t b, uint32_t c[4]) const {
    c[0] = b;
    c[1] = id0;
    c[2] = id1;
    c[3] = 0u;
    philox4x32_10(c, k0, k1);
  }
  GA_HD uint32_t next() {
    uint32_t c[4];
    block(k >> 2, c);
    const uint32_t w = k++ & 3u;
    return w == 0 ? c[0] : (w == 1 ? c[1] : (w == 2 ? c[2] : c[3]));
  }
};

// heur_noise_q16 (rules.cuh); |sum - 131070| * kHeurNoiseK stays below 2^31.
GA_HD int32_t noise(uint32_t x, uint32_t y) {
#if defined(__CUDA_ARCH__)
  const int32_t sum = (int32_t)__dp2a_lo(x, 0x0101u, __dp2a_lo(y, 0x0101u, 0u));
#else
  const int32_t sum = (int32_t)((x & 0xffffu) + (x >> 16) + (y & 0xffffu) + (y >> 16));
#endif
  return ((sum - 131070) * kHeurNoiseK) >> 16;
}
static_assert((int64_t)131070 * kHeurNoiseK < (int64_t(1) << 31), "the noise product outgrows 32 bits");

// One reference-heuristic ply, the move and draws of play_ply_heur_sched: the
// first maximum of weight + noise over the list, two draws per move.  A move's
// weight is one of four (it promotes or not, takes a king or not), so a ply
// whose moves are all alike needs no weights, only the largest noise; else two
// bits per move, in list order, tell the weights apart.  The loop takes one
// Philox block, two moves, per step and runs loop_n(steps) >= steps, one
// common count for a warp's lanes; only the chosen move is looked up.
template <class LoopN>
GA_HD int play_ply_heuristic(RotBoard &b, BlockDraws &rs, bool men_now, bool king_now, LoopN &&loop_n) {
  const View v = view(b);
  const Packed p = pack(masks(b, v));
  const uint32_t n = p.n;
  const bool cont = (v.cont_king | v.cont_man) != 0;
  if (cont || n > 32u) {
    if (cont && n == 1u && play_chain(b, v)) return 1;
    if (cont && (v.cont_king ? !king_now : !men_now)) return v.cont_king ? kNeedKing : kNeedMen;
    Board s = to_board(b);
    const int c = ply_ref_heuristic(s, rs);
    b = from_board(s);
    return c;
  }
  if (n == 0) return 0;
  const bool second = (b.meta & 1u) != 0;
  // moves that promote (bits of `up`) or take a king (`big`), by place in this orientation's list
  uint32_t up = 0, big = 0;
  int32_t w00 = 0, w01 = 0, w10 = 0, w11 = 0;  // [promotes][takes a king]
  const uint32_t oppk = b.opp & b.kings;
  const uint32_t ready = v.man & (v.capture ? squares(0x20u, 0xfu, 0xfu) : squares(0x40u, 0xfu, 0xfu));
  uint32_t ups, bigs = 0;
  if (v.capture) {
    ups = (uint32_t)(popc(v.m0 & ready) + popc(v.m1 & ready));
    bigs = (uint32_t)(popc((v.m0 | v.k0) & rotr(oppk, 7)) + popc((v.m1 | v.k1) & rotr(oppk, 1)) +
                      popc(v.k2 & rotl(oppk, 1)) + popc(v.k3 & rotl(oppk, 7)));
  } else {
    ups = (uint32_t)(popc(ready & rotr(v.empty, 7) & kStep0) + popc(ready & rotr(v.empty, 1) & kStep1));
  }
  if ((ups != 0u && ups != n) || (bigs != 0u && bigs != n)) {
    const int own = popc(b.own) + 3 * popc(v.king), opp = popc(b.opp) + 3 * popc(oppk);
    w00 = heur_weight_q16(own, opp - (v.capture ? 1 : 0));
    w10 = heur_weight_q16(own + 3, opp - (v.capture ? 1 : 0));
    if (v.capture) {
      w01 = heur_weight_q16(own, opp - 4);
      w11 = heur_weight_q16(own + 3, opp - 4);
      for (uint32_t c = 0; c < n; c++) {
        uint32_t from, place;
        nth(p, c, from, place);
        up |= (ready & from) ? 1u << c : 0u;
        big |= (rotl(from, turn_of(v, from, place)) & oppk) ? 1u << c : 0u;
      }
    } else {
      // the four squares of the row before the last, whose moves are the first of
      // the last two rows'
      constexpr uint32_t F = 0x00041041u, at = kOffset + 24u;
      const Masks m = masks(b, v);
      const uint32_t q = (rotr(m.m0, at) & F) + (rotr(m.m1, at) & F) + (rotr(m.m2, at) & F) + (rotr(m.m3, at) & F);
      const uint32_t t = rotr(ready, at) & F;
      uint32_t pos = n - (uint32_t)(popc(p.hi_a & ~kQuarters) + popc(p.hi_b & ~kQuarters));  // the last two rows'
GA_UNROLL
      for (uint32_t c = 0; c < 4; c++) {
        const uint32_t cnt = (q >> (6u * c)) & 7u;
        up |= ((t >> (6u * c)) & 1u) ? ((1u << cnt) - 1u) << (pos & 31u) : 0u;
        pos += cnt;
      }
    }
    if (second) {  // list order is the reverse
      up = reverse(up) >> (32u - n);
      big = reverse(big) >> (32u - n);
    }
  }
  uint32_t best = 0;
  if (n >= 2u) {
    const uint32_t pair = rs.k >> 1, skip = pair & 1u;  // two draws per move: k is even
    const uint32_t steps = loop_n((skip + n + 1u) >> 1);
    int32_t bw = INT32_MIN;
#if defined(__CUDACC__)
#pragma unroll 2  // two blocks in flight: 841 -> 814 us on the benchmark batch (four: 873)
#endif
    for (uint32_t t = 0; t < steps; t++) {
      uint32_t c[4];
      rs.block((pair >> 1) + t, c);
      const uint32_t m = 2u * t - skip;  // the move of the block's first two draws (none: wraps)
GA_UNROLL
      for (uint32_t h = 0; h < 2; h++) {
        const uint32_t x = m + h;
        const bool u = (up >> (x & 31u)) & 1u, g = (big >> (x & 31u)) & 1u;
        const int32_t w = (u ? (g ? w11 : w10) : (g ? w01 : w00)) + noise(c[2 * h], c[2 * h + 1]);
        const bool more = x < n && w > bw;
        bw = more ? w : bw;
        best = more ? x : best;
      }
    }
    rs.k += 2u * n;
  }
  uint32_t from, place;
  nth(p, second ? n - 1u - best : best, from, place);
  const uint32_t turn = turn_of(v, from, place), next = rotl(from, turn);
  apply(b, from, v.capture ? rotl(next, turn) : next, v.capture ? next : 0u);
  return (int)n;
}

}  // namespace rot
}  // namespace ga
