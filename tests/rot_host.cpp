// rot_host.cpp -- host build of the rotated-bitboard plies (rot.cuh), for CPU
// tests only: each is compared with the ply of rules.cuh it stands for, on
// pseudo-random boards and along games.
#include "../gpu_ai_gb300/csrc/rot.cuh"

using namespace ga;

namespace {

struct Rng {
  uint64_t x;
  uint64_t operator()() {
    uint64_t z = (x += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  }
};

// Any occupancy, sparse to crowded, few to many kings, either side to move.
Board random_board(Rng &next) {
  Board b;
  uint32_t occ = (uint32_t)next();
  if (next() & 1) occ &= (uint32_t)next();
  if ((next() & 3) == 0) occ |= (uint32_t)next();
  const uint32_t mine = (uint32_t)next();
  b.p1 = occ & mine;
  b.p2 = occ & ~mine;
  b.kings = occ & (uint32_t)next() & ((next() & 1) ? ~0u : (uint32_t)next());
  b.kings |= (b.p1 & kRow7) | (b.p2 & kRow0);
  b.meta = (uint32_t)(next() & 1) | ((uint32_t)(next() % 50) << 8);
  return b;
}

bool same(const Board &a, const Board &b) {
  return a.p1 == b.p1 && a.p2 == b.p2 && a.kings == b.kings && a.meta == b.meta;
}

// One ply of `s` both ways with the same draws; kind counts {no moves, forced
// multi-jumps, men's multi-jumps, king searches}.  Boards after, or false.
bool ply_matches(Board &s, uint64_t draws, int policy, uint64_t kind[4]) {
  const uint32_t d[2] = {(uint32_t)draws, (uint32_t)(draws >> 32)};
  struct Draws {
    const uint32_t *d;
    uint32_t k = 0;
    uint32_t next() { return d[k++ & 1u]; }
  };
  Board a = s;
  rot::RotBoard r = rot::from_board(s);
  if (!same(rot::to_board(r), s)) return false;
  Draws da{d}, dr{d};
  int na, nr, sched;
  Board t = s;
  Draws dt{d};
  auto pick = [](Draws &x) { return [&x](uint32_t n) { return n >= 2 ? mulhi_index(x.next(), n) : 0u; }; };
  rot::RotBoard u = r;
  Draws du{d};
  int held;
  if (policy == 1) {  // many draws: streams, from any even draw on
    Stream a1, t1;
    a1.init(draws, draws >> 7, 0);
    for (uint32_t q = 0; q < (uint32_t)(draws >> 60) * 2u; q++) a1.next();
    t1 = a1;
    rot::BlockDraws r1, u1;
    r1.start(draws, draws >> 7);
    r1.k = a1.k;
    u1 = r1;
    struct Refilled {  // play_ply_heur_sched refills a ring
      Stream &s;
      uint32_t next() { return s.next(); }
    } ring{t1};
    auto longer = [](uint32_t m) { return m + m % 3u; };
    na = ply_ref_heuristic(a, a1);
    nr = rot::play_ply_heuristic(r, r1, true, true, longer);
    sched = play_ply_heur_sched(t, ring, t1, false, false, longer, [] {});
    held = rot::play_ply_heuristic(u, u1, false, false, longer);
    da.k = a1.k;
    dr.k = r1.k;
    dt.k = t1.k;
    du.k = u1.k;
  } else if (policy == 2) {
    na = ply_eps_greedy(a, da);
    nr = rot::play_ply_eps(r, dr, true, true);
    sched = play_ply_eps_sched(t, dt, false, false);
    held = rot::play_ply_eps(u, du, false, false);
  } else {
    na = play_ply(a, pick(da));
    nr = rot::play_ply_random(r, pick(dr), true, true);
    sched = play_ply_sched(t, pick(dt), false, false);
    held = rot::play_ply_random(u, pick(du), false, false);
  }
  if (na != nr || da.k != dr.k) return false;
  if (na > 0 && !same(a, rot::to_board(r))) return false;
  if (sched != held || dt.k != du.k || !same(t, rot::to_board(u))) return false;
  if (na == 0) kind[0]++;
  if (sched == 1 && na == 1 && (s.meta >> 8) != 0 && (a.meta >> 8) == 0) kind[1]++;
  if (sched == kNeedMen) kind[2]++;
  if (sched == kNeedKing) kind[3]++;
  s = a;
  return na >= 0;
}

}  // namespace

extern "C" {

// n random boards; returns the number that differ.
long rot_boards(uint64_t n, uint64_t seed, int policy, uint64_t kind[4]) {
  Rng next{seed};
  long bad = 0;
  for (uint64_t i = 0; i < n; i++) {
    Board b = random_board(next);
    if (!ply_matches(b, next(), policy, kind)) bad++;
  }
  return bad;
}

// n games from the start position; returns the number with a ply that differs.
long rot_games(uint64_t n, uint64_t seed, int policy, uint64_t kind[4]) {
  Rng next{seed};
  long bad = 0;
  for (uint64_t i = 0; i < n; i++) {
    Board b{0x00000FFFu, 0xFFF00000u, 0u, 0u};
    for (int p = 0; p < 2000 && ((b.meta >> 8) & 0xffu) < (uint32_t)kDrawPlies; p++) {
      const uint64_t over = kind[0];
      if (!ply_matches(b, next(), policy, kind)) {
        bad++;
        break;
      }
      if (kind[0] != over) break;
    }
  }
  return bad;
}

// Seeded positions by the enumerating plies of rules.cuh, one at a time.
void rot_positions(uint64_t seed, uint32_t n, uint32_t min_plies, uint32_t max_plies, int policy, uint32_t *out) {
  for (uint32_t p = 0; p < n; p++) {
    Stream rs;
    rs.init(seed, p, 1);
    Board b{0x00000FFFu, 0xFFF00000u, 0u, 0u};
    const uint32_t np = min_plies + mulhi_index(rs.next(), max_plies - min_plies + 1u);
    for (uint32_t q = 0; q < np && ((b.meta >> 8) & 0xffu) < (uint32_t)kDrawPlies; q++)
      if ((policy == 1 ? ply<1>(b, rs) : (policy == 2 ? ply<2>(b, rs) : ply<0>(b, rs))) <= 0) break;
    out[4 * p] = b.p1;
    out[4 * p + 1] = b.p2;
    out[4 * p + 2] = b.kings;
    out[4 * p + 3] = b.meta;
  }
}

}  // extern "C"
