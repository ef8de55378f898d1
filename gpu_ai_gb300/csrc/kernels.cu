// kernels.cu -- playout, move-list and position kernels for sm_103a.
//
// Thread-per-playout: each thread keeps its board as four 32-bit words in
// registers (rotated bitboards seen from the side to move, rot.cuh) and plays
// one ply per loop iteration.  The loop is warp-uniform:
// a lane whose game ends writes its int8 outcome and, at the next refill
// iteration (every fourth), takes the next playout index from a
// warp-aggregated claim on a global work counter, so the warp never waits for
// its longest game (the reference's coarsePlayoutKernel work queue,
// src/coarsePlayout.cu:73-86, done with one atomicAdd per warp claim instead
// of a per-thread atomicCAS spin).
#include "detmath.cuh"
#include "launch.h"
#include "rot.cuh"
#include "rules.cuh"

namespace ga {

constexpr uint32_t kFull = 0xffffffffu;

__device__ __forceinline__ uint32_t position_of(const PlayoutArgs &a, uint32_t j) {
  if (a.offsets == nullptr) return j / a.uniform_reps;
  uint32_t lo = 0, hi = a.npos;  // largest p < npos with offsets[p] <= j
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&a.offsets[mid]) <= j) lo = mid; else hi = mid;
  }
  return lo;
}

// Random-stream id of playout j, which plays position p.
__device__ __forceinline__ uint64_t stream_of(const PlayoutArgs &a, uint32_t p, uint32_t j) {
  if (a.pos_stream == nullptr) return a.stream_base + j;
  const uint32_t first = a.offsets ? __ldg(&a.offsets[p]) : p * a.uniform_reps;
  return __ldg(&a.pos_stream[p]) + (j - first);
}

__device__ __forceinline__ Board load_board(const Board *p) {
  uint4 v = __ldg(reinterpret_cast<const uint4 *>(p));
  Board b;
  b.p1 = v.x; b.p2 = v.y; b.kings = v.z; b.meta = v.w;
  return b;
}

__device__ __forceinline__ void store_board(Board *p, const Board &b) {
  *reinterpret_cast<uint4 *>(p) = make_uint4(b.p1, b.p2, b.kings, b.meta);
}

// ---- the playout kernel

// Resident blocks per SM that the register budget is sized for: 64 registers
// a thread for blocks of 256 or more threads (80 for the reference heuristic
// at 256: 3 blocks), 72 (96 for the reference heuristic) for smaller blocks.
template <int POLICY, int BLOCK>
constexpr int playout_min_blocks() {
  constexpr int regs = BLOCK >= 256 ? (POLICY == 1 && BLOCK == 256 ? 80 : 64) : (POLICY == 1 ? 96 : 72);
  return 65536 / (regs * BLOCK);
}

// Block pool of the pooled layout: a shared-memory lock that lane 0 tries to
// take once (a warp that does not get it carries on as the unpooled kernel
// does and tries again on a later iteration: nothing ever waits for it), and
// the two pools' capacity.
constexpr uint32_t kPoolCap = 64;

__device__ __forceinline__ bool pool_lock(uint32_t *lock, uint32_t lane) {
  uint32_t got = 0;
  if (lane == 0) got = atomicCAS(lock, 0u, 1u) == 0u ? 1u : 0u;
  got = __shfl_sync(kFull, got, 0);
  __threadfence_block();
  __syncwarp();
  return got != 0;
}

__device__ __forceinline__ void pool_unlock(uint32_t *lock, uint32_t lane) {
  __threadfence_block();
  __syncwarp();
  if (lane == 0) atomicExch(lock, 0u);
}

__device__ __forceinline__ uint32_t vload(const uint32_t *p) { return *reinterpret_cast<const volatile uint32_t *>(p); }

// The random draws of a game whose ring of eight buffered draws is a column of
// shared memory: draw k is word k % 8 of the column (consecutive threads,
// consecutive banks), one load at a changing index (eight registers would need
// a select among them).  refill() keeps at least four draws buffered.
template <uint32_t TAG>
struct SharedRing {
  uint32_t *ring;   // word 0 of column 0
  uint32_t stride;  // columns
  uint32_t col, k, avail, k0, k1, id0, id1;

  __device__ __forceinline__ void start(uint64_t seed, uint64_t id) {
    k0 = (uint32_t)seed;
    k1 = (uint32_t)(seed >> 32);
    id0 = (uint32_t)id;
    id1 = (uint32_t)(id >> 32);
    k = 0;
    avail = 0;
  }
  __device__ __forceinline__ void refill() {
    if (avail >= 4) return;
    const uint32_t pos = k + avail;  // multiple of 4
    uint32_t c[4] = {pos >> 2, id0, id1, TAG};
    philox4x32_10(c, k0, k1);
    uint32_t *w = ring + (pos & 4u) * stride + col;
#pragma unroll
    for (uint32_t q = 0; q < 4; q++) w[q * stride] = c[q];
    avail += 4;
  }
  __device__ __forceinline__ uint32_t peek() const { return ring[(k & 7u) * stride + col]; }
  // Move index in [0, n) for n >= 1; a draw is consumed only when n >= 2.
  __device__ __forceinline__ uint32_t pick(uint32_t n) {
    const uint32_t i = mulhi_index(peek(), n);  // 0 for n = 1
    const uint32_t use = n >= 2 ? 1u : 0u;
    k += use;
    avail -= use;
    return i;
  }
  __device__ __forceinline__ uint32_t next() {
    const uint32_t r = peek();
    k++;
    avail--;
    return r;
  }
};

// A game as the playout loop holds it: the board and its random draws.  Its
// words are what moves when a game changes lanes (for a SharedRing the column
// moves by its number, the draws stay in place).
template <uint32_t TAG>
struct RotGame {  // uniform random and eps-greedy policies
  rot::RotBoard b;
  SharedRing<TAG> rs;
  static constexpr int kWords = 8, kCol = 7;  // kCol: the word holding the column
  // the start position as four words, and a game begun from them
  __device__ static __forceinline__ uint4 prepare(const Board &at) {
    const rot::RotBoard r = rot::from_board(Board{at.p1, at.p2, at.kings, at.meta & 0xff01u});
    return make_uint4(r.own, r.opp, r.kings, r.meta);
  }
  __device__ __forceinline__ void start(const uint4 &at, uint64_t seed, uint64_t id) {
    b = rot::RotBoard{at.x, at.y, at.z, at.w};
    rs.start(seed, id);
  }
  __device__ __forceinline__ bool drawn() const { return b.meta >= ((uint32_t)kDrawPlies << 8); }
  __device__ __forceinline__ void refill() { rs.refill(); }
  template <int POLICY>
  __device__ __forceinline__ int play(bool men_ok, bool king_ok) {
    if constexpr (POLICY == 2) return rot::play_ply_eps(b, rs, men_ok, king_ok);
    else return rot::play_ply_random(b, [&](uint32_t n) { return rs.pick(n); }, men_ok, king_ok);
  }
  __device__ __forceinline__ void save(uint32_t (&v)[kWords]) const {
    v[0] = b.own; v[1] = b.opp; v[2] = b.kings; v[3] = b.meta | (rs.avail << 16);
    v[4] = rs.k; v[5] = rs.id0; v[6] = rs.id1; v[7] = rs.col;
  }
  __device__ __forceinline__ void load(const uint32_t (&v)[kWords]) {
    b.own = v[0]; b.opp = v[1]; b.kings = v[2]; b.meta = v[3] & 0xffffu; rs.avail = v[3] >> 16;
    rs.k = v[4]; rs.id0 = v[5]; rs.id1 = v[6]; rs.col = v[7];
  }
};

struct HeurGame {  // reference heuristic: two draws per move, generated where they are used
  rot::RotBoard b;
  rot::BlockDraws rs;
  static constexpr int kWords = 7, kCol = -1;
  __device__ static __forceinline__ uint4 prepare(const Board &at) { return RotGame<0>::prepare(at); }
  __device__ __forceinline__ void start(const uint4 &at, uint64_t seed, uint64_t id) {
    b = rot::RotBoard{at.x, at.y, at.z, at.w};
    rs.start(seed, id);
  }
  __device__ __forceinline__ bool drawn() const { return b.meta >= ((uint32_t)kDrawPlies << 8); }
  __device__ __forceinline__ void refill() {}
  template <int POLICY>
  __device__ __forceinline__ int play(bool men_ok, bool king_ok) {
    return rot::play_ply_heuristic(b, rs, men_ok, king_ok,
                                   [](uint32_t m) { return __reduce_max_sync(__activemask(), m); });
  }
  __device__ __forceinline__ void save(uint32_t (&v)[kWords]) const {
    v[0] = b.own; v[1] = b.opp; v[2] = b.kings; v[3] = b.meta; v[4] = rs.k; v[5] = rs.id0; v[6] = rs.id1;
  }
  __device__ __forceinline__ void load(const uint32_t (&v)[kWords]) {
    b.own = v[0]; b.opp = v[1]; b.kings = v[2]; b.meta = v[3]; rs.k = v[4]; rs.id0 = v[5]; rs.id1 = v[6];
  }
};

template <int POLICY, bool POSITIONS> struct GameOf { using type = RotGame<POSITIONS ? 1u : 0u>; };
template <> struct GameOf<1, false> { using type = HeurGame; };

// Bound by the integer (ALU) pipe while every lane has a game (84 % of its
// peak on 20,011 positions with 4.0 M playouts, 65 % of the lanes active: the
// rest is the code of the multi-jump plies, which few lanes of a warp run at a
// time), and by the length of the last games once the work runs out.  Plies on
// rotated bitboards from the side to move instead of rules.cuh's, draws in
// shared memory: 372 -> 297 us on the benchmark batch (262,144 playouts; 287
// with the inner loop), 2.95 -> 2.43 ms on the 4.0 M (2.15 with claims in bulk,
// 2.05 with the inner loop), 1.60 -> 0.86 ms for the reference heuristic's
// benchmark batch (it no longer walks a cursor per move), 443 -> 368 us for
// 65,536 eps-greedy playouts through the host call.
//
// POSITIONS: the loop makes seeded positions instead (gpuai_selfplay_positions):
// game j is a game from the standard start on stream (seed, j, 1), whose first
// draw says how many plies it is played, and its board is the result.  A block
// takes a fixed range of them through a counter in its shared memory (their
// lengths are alike everywhere, and calls on several streams share nothing).
// A thread per position without this loop waited for its warp's longest game
// and enumerated eps-greedy moves: 500,000 eps-greedy positions of 0..90 plies 2.67 -> 0.95 ms.
template <int POLICY, int BLOCK, bool POOL, bool POSITIONS = false>
__global__ void __launch_bounds__(BLOCK, (playout_min_blocks<POLICY, BLOCK>()))
    playout_kernel(PlayoutArgs a, PositionArgs pa = PositionArgs{}) {
  if (a.dev_sizes != nullptr) {
    a.npos = __ldg(&a.dev_sizes[0]);
    a.total = __ldg(&a.dev_sizes[1]);
  }
  using Game = typename GameOf<POLICY, POSITIONS>::type;
  uint32_t first = 0, left = 0;  // POSITIONS: the block's first game, plies left to play
  if constexpr (POSITIONS) {
    __shared__ uint32_t s_counter;
    if (threadIdx.x == 0) s_counter = 0;
    __syncthreads();
    first = (uint32_t)((uint64_t)a.total * blockIdx.x / gridDim.x);
    a.total = (uint32_t)((uint64_t)a.total * (blockIdx.x + 1u) / gridDim.x) - first;
    a.counter = &s_counter;
  }
  constexpr bool kRing = Game::kCol >= 0;  // draws buffered in shared memory
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t j = 0, plies_here = 0;
  bool have = false, exhausted = false;

  // No ply counter stops a game here: 50 plies without a capture end it, and
  // a capture takes at least one of at most 64 piece bits off the board.
  static_assert(64u * kDrawPlies <= kMaxPlies, "the 50-ply rule ends a game within kMaxPlies");
  static_assert(POLICY >= 0 && POLICY <= 2, "policies: 0 random, 1 reference heuristic, 2 eps-greedy");
  {
    // Uniform random policy: at most one draw per ply, so Philox blocks are
    // generated for the whole warp every fourth iteration (SharedRing keeps
    // four or more draws buffered) and new games start on those iterations
    // too.  eps-greedy (policy 2, rot::play_ply_eps) takes at most two draws
    // per ply and refills every second iteration.  The reference heuristic
    // (policy 1, rot::play_ply_heuristic) takes two draws per legal move: its
    // ply loops over Philox blocks, two moves each, for the warp's longest move
    // list, so Philox still runs for the whole warp at once.
    // Plies whose capture can be extended take longer code.  Those with one
    // legal move (about two thirds) follow their chain at once; the others,
    // men's multi-jumps (about 1% of plies) and plies where a king's capture
    // can continue (about 0.2%, the costlier depth-first search), are deferred
    // to every kMenPeriod-th (eps-greedy and reference heuristic only:
    // defer_men) and every king_period(POLICY)-th iteration, so that the lanes
    // needing that code run it together and the other iterations stay
    // branch-free.
    // Once the work counter is exhausted, a warp with sparse_lanes(POLICY) or fewer
    // games defers nothing: its few games are latency-bound.
    //
    // Once the work counter is exhausted, every compact_period(POLICY)-th iteration the
    // block packs its unfinished games (board, random-stream state, counters)
    // into its lowest threads through shared memory; warps left without games
    // wait at the next barrier instead of issuing empty iterations.  The loop
    // ends for the whole block when it has no game left.
    //
    // Pooled layout (POOL): while work remains, a lane whose ply must wait for
    // a men's multi-jump or king capture search hands its game to the block's
    // pending pool and takes a new one; once the pool holds 32 such games, the
    // warp that sees it moves its own games to the block's ready pool, takes
    // the 32 and plays their deferred plies at once with every lane busy.
    // Free lanes take ready games before new ones (and pending ones once the
    // work ran out); compaction packs the pools' games too.  A game keeps its
    // whole state (board, stream, ring of draws) wherever it is played, so
    // the outcomes are the same as without the pools.  Every pool entry owns a
    // ring column, and a game that moves in or out trades columns with it.
    // ... and the playout index with the pending kind (POSITIONS: and the plies left)
    constexpr int kWords = Game::kWords + (POSITIONS ? 2 : 1);
    static_assert(kWords >= 7, "a stock entry takes seven words");
    constexpr uint32_t kCap = POOL ? kPoolCap : 1u;
    constexpr uint32_t kColumns = kRing ? BLOCK + (POOL ? 2u * kCap : 0u) : 1u;
    __shared__ uint32_t s_ring[kRing ? 8u * kColumns : 1u];
    __shared__ uint32_t s_slot[kWords][BLOCK];
    __shared__ uint32_t s_cnt[BLOCK / 32];
    __shared__ uint32_t s_pend[kWords][kCap];   // games waiting for a deferred ply
    __shared__ uint32_t s_ready[kWords][kCap];  // games a swap moved out of their lane
    __shared__ uint32_t s_pool[4];              // lock, pending games, ready games
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    Game g;
    g.start(make_uint4(0, 0, 0, 0), a.seed, 0);
    if constexpr (kRing) {
      g.rs.ring = s_ring;
      g.rs.stride = kColumns;
      g.rs.col = threadIdx.x;
    }
    if constexpr (POOL) {
      if (threadIdx.x < 4) s_pool[threadIdx.x] = 0;
      if constexpr (kRing) {
        for (uint32_t q = threadIdx.x; q < kCap; q += BLOCK) {
          s_pend[Game::kCol][q] = BLOCK + q;
          s_ready[Game::kCol][q] = BLOCK + kCap + q;
        }
      }
      __syncthreads();
    }
    uint32_t pend = 0;    // deferred ply: 0 none, 1 men's multi-jump, 2 king capture search
    bool sparse = false;  // warp-uniform: the work ran out and the warp holds sparse_lanes(POLICY) games or fewer
    constexpr uint32_t kCompactPeriod = compact_period(POLICY);
    constexpr uint32_t kSparseLanes = sparse_lanes(POLICY);
    // a game's state in word q of column idx of a [kWords][stride] area; with
    // `trade`, the lane gives its ring column for the entry's
    auto put = [&](uint32_t *area, uint32_t stride, uint32_t idx, bool trade) {
      uint32_t v[Game::kWords];
      g.save(v);
      if constexpr (kRing) {
        if (trade) g.rs.col = area[Game::kCol * stride + idx];
      }
#pragma unroll
      for (int q = 0; q < Game::kWords; q++) area[q * stride + idx] = v[q];
      area[Game::kWords * stride + idx] = j | (pend == 2u ? 0x80000000u : 0u);  // a pending men's ply is found again
      if constexpr (POSITIONS) area[(Game::kWords + 1) * stride + idx] = left;
    };
    auto take = [&](uint32_t *area, uint32_t stride, uint32_t idx, bool trade) {
      uint32_t v[Game::kWords];
#pragma unroll
      for (int q = 0; q < Game::kWords; q++) v[q] = area[q * stride + idx];
      if constexpr (kRing) {
        if (trade) area[Game::kCol * stride + idx] = g.rs.col;
      }
      g.load(v);
      j = area[Game::kWords * stride + idx] & 0x7fffffffu;
      pend = (area[Game::kWords * stride + idx] >> 31) * 2u;
      if constexpr (POSITIONS) left = area[(Game::kWords + 1) * stride + idx];
    };
    // Claim order (equal repetitions, at most BLOCK positions): lanes take
    // the playouts of positions with more pieces first.  Their games are
    // longer on average, so the last claims of the batch are the shorter
    // games and less of the batch tail waits on a game that started late.
    // Playout j keeps its index (its outcome slot and random stream); only the
    // order in which lanes take the playouts changes.
    __shared__ uint16_t s_order[BLOCK];
    __shared__ uint8_t s_key[BLOCK];
    const bool ordered = !POSITIONS && a.offsets == nullptr && a.npos > 1 && a.npos <= (uint32_t)BLOCK;
    if (ordered) {  // uniform over the block
      const uint32_t t = threadIdx.x;
      if (t < a.npos) {
        const Board pb = load_board(a.pos + t);
        s_key[t] = (uint8_t)popc(pb.p1 | pb.p2);
      }
      __syncthreads();
      if (t < a.npos) {
        const uint32_t kt = s_key[t];
        uint32_t rank = 0;
        for (uint32_t u = 0; u < a.npos; u++) {
          const uint32_t ku = s_key[u];
          rank += (ku > kt || (ku == kt && u < t)) ? 1u : 0u;
        }
        s_order[rank] = (uint16_t)t;
      }
      __syncthreads();
    }
    // Lanes without a game claim playouts with one atomicAdd per warp.  While
    // much work remains a warp claims up to 32 at once and keeps them as its
    // stock: all its lanes look up and convert the positions together (with
    // uneven repetitions a binary search of the offsets), once per 32 games,
    // instead of the two or three lanes that need one.  A claim is at most a
    // quarter of the warp's share of what remains, so a stock is empty again
    // before the counter runs out; a small batch claims what it needs.  The
    // stock lives in the warp's part of s_slot, which is free until the block's
    // stocks are empty (compaction starts after that).
    // 20,011 positions with 4.0 M uneven playouts: 2.43 -> 2.15 ms; labels of
    // 16,384 positions by 1,024 playouts each: 7.65 -> 6.47 ms.
    constexpr uint32_t kBulkClaim = 8;  // the benchmark batch (3 at most) is 1 % slower with bulk claims of any size
    // A batch smaller than the grid's lanes is dealt out evenly over the blocks
    // at the start, each block's share over as few warps as hold it: the host
    // launches a block per playout up to the resident ones, so a small batch has
    // few games per SM and per warp, each at a lone game's latency (256 playouts
    // of one position, host call: 146-153 -> 116-126 us on two GPUs; 65,536
    // eps-greedy ones: 355 -> 337 us).  More warps with fewer games each, here or after packing, are
    // slower once an SM holds more than a few (2, 4, 8 warps per block at least:
    // 1-5 % on the benchmark batch, 3-39 % on 65,536 playouts).
    const uint32_t share = POSITIONS ? a.total : (a.total + gridDim.x - 1u) / gridDim.x;
    const uint32_t holding = (share + 31u) / 32u;  // warps that claim
    const uint32_t lanes =  // ... and their lanes that do
        share >= BLOCK ? kFull : (warp < holding ? kFull >> (32u - (share + holding - 1u) / holding) : 0u);
    uint32_t stock = 0, stock_end = 0, chunk = 0;  // games left, entries, next claim: warp-uniform
    bool dry = false;                              // the counter ran out: warp-uniform
    const uint32_t chunk_shift = 32u - __clz((POSITIONS ? 1u : gridDim.x) * (BLOCK / 32u) * 4u - 1u);
    constexpr uint32_t kRefillMask = POLICY == 2 ? 1u : 3u;
    for (uint32_t it = 0;; ++it) {
      bool swapped = false;  // warp-uniform: this iteration's games came from the pending pool
      if constexpr (POOL) {
        // 32 games wait for their deferred ply and the ready pool has room for
        // this warp's games: play the 32 in this warp now (checked on the men's
        // phase iterations only)
        if (!exhausted && (it & (kMenPeriod - 1u)) == kMenPhase) {
          uint32_t ok = 0;
          if (lane == 0) ok = vload(&s_pool[1]) >= 32u && vload(&s_pool[2]) + 32u <= kCap;
          if (__shfl_sync(kFull, ok, 0) && pool_lock(&s_pool[0], lane)) {
            const uint32_t npend = vload(&s_pool[1]), nready = vload(&s_pool[2]);
            const uint32_t hm = __ballot_sync(kFull, have);
            if (npend >= 32u && nready + (uint32_t)__popc(hm) <= kCap) {
              if (have) put(&s_ready[0][0], kCap, nready + __popc(hm & lt), true);
              take(&s_pend[0][0], kCap, npend - 32u + lane, true);
              have = true;
              if (lane == 0) {
                s_pool[1] = npend - 32u;
                s_pool[2] = nready + __popc(hm);
              }
              swapped = true;
            }
            pool_unlock(&s_pool[0], lane);
            if (swapped) g.refill();
          }
        }
      }
      if ((it & kRefillMask) == 0) {
        if constexpr (POOL) {
          // free lanes take ready games (and, once the work ran out, pending ones)
          const uint32_t fm = __ballot_sync(kFull, !have);
          if (fm) {
            uint32_t avail = 0;
            if (lane == 0) avail = vload(&s_pool[2]) + (exhausted ? vload(&s_pool[1]) : 0u);
            if (__shfl_sync(kFull, avail, 0) && pool_lock(&s_pool[0], lane)) {
              const uint32_t nr = vload(&s_pool[2]), np = exhausted ? vload(&s_pool[1]) : 0u;
              const uint32_t rank = __popc(fm & lt), k = min((uint32_t)__popc(fm), nr + np);
              if (!have && rank < k) {
                if (rank < nr) take(&s_ready[0][0], kCap, nr - 1u - rank, true);
                else take(&s_pend[0][0], kCap, np - 1u - (rank - nr), true);
                have = true;
              }
              if (lane == 0) {
                const uint32_t from_r = min(k, nr);
                s_pool[2] = nr - from_r;
                if (exhausted) s_pool[1] = np - (k - from_r);
              }
              pool_unlock(&s_pool[0], lane);
            }
          }
        }
        if (!exhausted) {
          uint32_t need = __ballot_sync(kFull, !have) & lanes;
          bool fresh = false;
          if (need && stock == 0 && !dry) {
            const uint32_t cnt = __popc(need), rank = __popc(need & lt);
            const bool bulk = chunk >= kBulkClaim;  // warp-uniform
            const uint32_t m = bulk ? min(32u, chunk) : cnt;
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(a.counter, m);
            base = __shfl_sync(kFull, base, 0);
            const uint32_t got = base < a.total ? min(m, a.total - base) : 0u;
            dry = base + m >= a.total;
            chunk = dry ? 0u : (a.total - base - m) >> chunk_shift;
            const uint32_t e = bulk ? lane : rank;
            if (e < got && (bulk || ((need >> lane) & 1u))) {
              uint32_t q = base + e;
              if (ordered) {  // claim index -> playout index
                const uint32_t k = q / a.uniform_reps;
                q = (uint32_t)s_order[k] * a.uniform_reps + (q - k * a.uniform_reps);
              }
              Board at = {0x00000FFFu, 0xFFF00000u, 0u, 0u};
              uint64_t id;
              uint32_t plies = 0;
              if constexpr (POSITIONS) {
                id = first + q;
                uint32_t c[4] = {0u, (uint32_t)id, 0u, 1u};
                philox4x32_10(c, (uint32_t)a.seed, (uint32_t)(a.seed >> 32));
                plies = pa.min_plies + mulhi_index(c[0], pa.max_plies - pa.min_plies + 1u);
              } else {
                const uint32_t p = position_of(a, q);
                at = Board{0, 0, 0, 0};
                if (GA_IN_BOUNDS(p < a.npos, a.status)) at = load_board(a.pos + p);
                id = stream_of(a, p, q);
              }
              const uint4 v = Game::prepare(at);
              if (bulk) {
                const uint32_t t = warp * 32u + lane;
                s_slot[0][t] = v.x; s_slot[1][t] = v.y; s_slot[2][t] = v.z; s_slot[3][t] = v.w;
                s_slot[4][t] = q; s_slot[5][t] = (uint32_t)id; s_slot[6][t] = POSITIONS ? plies : (uint32_t)(id >> 32);
              } else {
                j = q;
                g.start(v, a.seed, id);
                left = plies;
                have = fresh = true;
              }
            }
            stock = bulk ? got : 0u;
            stock_end = stock;
            __syncwarp();
          }
          if (need && stock) {  // the warp's stock serves its free lanes
            need = __ballot_sync(kFull, !have) & lanes;
            const uint32_t rank = __popc(need & lt), k = min((uint32_t)__popc(need), stock);
            if (((need >> lane) & 1u) && rank < k) {
              const uint32_t t = warp * 32u + stock_end - stock + rank;
              j = s_slot[4][t];
              left = s_slot[6][t];
              g.start(make_uint4(s_slot[0][t], s_slot[1][t], s_slot[2][t], s_slot[3][t]), a.seed,
                      (POSITIONS ? 0ull : (uint64_t)left << 32) | s_slot[5][t]);
              have = fresh = true;
            }
            __syncwarp();
            stock -= k;
          }
          exhausted = dry && stock == 0;
          if constexpr (POSITIONS) {
            if (fresh) {  // the first draw is used up
              g.refill();
              g.rs.k = 1;
              g.rs.avail = 3;
            }
          }
        }
        if (have) g.refill();
      }
      // The plies up to the next iteration that may start games, without the
      // checks in between that only matter there (308 -> 297 us on the benchmark
      // batch, 2.16 -> 2.13 ms on 4.0 M uneven playouts); in the pooled layout one
      // ply, its pools are looked at after each.
      bool deferred_now = false;  // this iteration's ply was deferred (a candidate for the pending pool)
      for (;; ++it) {
        const bool men_ok = !defer_men(POLICY) || sparse || swapped || (it & (kMenPeriod - 1u)) == kMenPhase;
        const bool king_ok = sparse || swapped || (it & (king_period(POLICY) - 1u)) == kKingPhase;
        do {
          if (!have) break;
          if ((pend == 1u && !men_ok) || (pend == 2u && !king_ok)) break;  // still deferred
          if constexpr (POSITIONS) {
            if (left == 0 || g.drawn()) {
              store_board(pa.out + first + j, rot::to_board(g.b));
              have = false;
              break;
            }
          } else if (g.drawn()) {
            if (GA_IN_BOUNDS(j < a.total, a.status)) a.out[j] = 0;
            have = false;
            break;
          }
          const int n = g.template play<POLICY>(men_ok, king_ok);
          if (n == kNeedMen || n == kNeedKing) {
            pend = n == kNeedMen ? 1u : 2u;
            deferred_now = true;
            break;
          }
          pend = 0;
          if (n > 0) {
            if constexpr (POSITIONS) left--;
            else plies_here++;
            break;
          }
          if constexpr (POSITIONS) {
            left = 0;  // the game is over: its board is stored at its next turn
            break;
          }
          if (n < 0) atomicOr(a.status, kStatusDepth);
          if (GA_IN_BOUNDS(j < a.total, a.status))
            a.out[j] = (int8_t)(n == 0 ? ((g.b.meta & 1u) ? 1 : -1) : 0);  // side to move cannot move: loses
          have = false;
        } while (false);
        if (POOL || (it & kRefillMask) == kRefillMask) break;
      }
      if constexpr (POOL) {
        // hand deferred games to the pending pool while work remains
        if (!exhausted && !sparse) {
          const uint32_t pm = __ballot_sync(kFull, deferred_now);
          uint32_t room = 0;
          if (pm && lane == 0) room = vload(&s_pool[1]) < kCap;
          if (pm && __shfl_sync(kFull, room, 0) && pool_lock(&s_pool[0], lane)) {
            const uint32_t np = vload(&s_pool[1]);
            const uint32_t k = min((uint32_t)__popc(pm), kCap - np), rank = __popc(pm & lt);
            if (deferred_now && rank < k) {
              put(&s_pend[0][0], kCap, np + rank, true);
              have = false;
              pend = 0;
            }
            if (lane == 0) s_pool[1] = np + k;
            pool_unlock(&s_pool[0], lane);
          }
        }
      }

      if ((it & (kCompactPeriod - 1u)) != kCompactPeriod - 1u) {
        if (exhausted) {
          const uint32_t live = __ballot_sync(kFull, have);
          sparse = __popc(live) <= kSparseLanes;
          // a warp with no game left skips ahead to the block's next compaction point
          if (!live) it = (it | (kCompactPeriod - 1u)) - 1u;
        }
        continue;
      }
      if (!exhausted) {
        // A warp whose lanes are all busy makes no claims: it reads the work
        // counter itself (with games in stock it is not done either way).  Counter values only grow, and a warp waits at the
        // barrier below only after it saw the counter at or past the total, so
        // every other warp of the block sees that too at its next compaction
        // point and joins it: no barrier is needed while work remains.
        uint32_t c = 0;
        if (lane == 0) c = *reinterpret_cast<volatile const uint32_t *>(a.counter);
        if (__shfl_sync(kFull, c, 0) < a.total || stock != 0) continue;  // warp-uniform
        exhausted = true;
      }
      // Only warps that know the work is exhausted get here; they all pass the
      // same sequence of compaction points (it % compact_period equal, absolute
      // iteration counts may differ).  This barrier also keeps a fast warp from
      // writing s_cnt for the next point while a slow one still reads it.
      __syncthreads();
      const uint32_t m = __ballot_sync(kFull, have);
      if (lane == 0) s_cnt[warp] = __popc(m);
      __syncthreads();
      uint32_t total = 0, before = 0, busy_warps = 0;
#pragma unroll
      for (uint32_t w = 0; w < BLOCK / 32; w++) {
        const uint32_t c = s_cnt[w];
        before += w < warp ? c : 0u;
        total += c;
        busy_warps += c ? 1u : 0u;
      }
      // games still in the pools (stable here: every warp knows the work ran
      // out, so none pushes, and all are between the two barriers)
      const uint32_t nr = POOL ? vload(&s_pool[2]) : 0u, np = POOL ? vload(&s_pool[1]) : 0u;
      if (total + nr + np == 0) break;
      sparse = __popc(m) <= kSparseLanes;
      if (nr + np == 0 && (total + 31u) / 32u >= busy_warps) continue;  // packing would free no warp
      const uint32_t n_all = min((uint32_t)BLOCK, total + nr + np);  // games the block's lanes hold after packing
      if (have) put(&s_slot[0][0], BLOCK, before + __popc(m & lt), false);
      if constexpr (POOL) {
        // pool games fill the lanes after the live ones: ready games first
        const uint32_t t = threadIdx.x;
        if (t >= total && t < n_all) {
          const uint32_t e = t - total;
          uint32_t v[kWords];
          if (e < nr) {
#pragma unroll
            for (int q = 0; q < kWords; q++) v[q] = s_ready[q][nr - 1u - e];
          } else {
#pragma unroll
            for (int q = 0; q < kWords; q++) v[q] = s_pend[q][np - 1u - (e - nr)];
          }
#pragma unroll
          for (int q = 0; q < kWords; q++) s_slot[q][t] = v[q];
        }
      }
      __syncthreads();
      if constexpr (POOL) {
        // every thread has read the counts (before the barrier above); a
        // second barrier publishes the new ones before any lane pops again
        if (threadIdx.x == 0) {
          const uint32_t moved = n_all - total, from_r = min(moved, nr);
          s_pool[2] = nr - from_r;
          s_pool[1] = np - (moved - from_r);
        }
        __syncthreads();
      }
      // the games go round the warps that keep any, so that each holds as few as can be
      const uint32_t keep = (n_all + 31u) / 32u, e = lane * keep + warp;
      have = warp < keep && e < n_all;
      sparse = __popc(__ballot_sync(kFull, have)) <= kSparseLanes;
      if (have) take(&s_slot[0][0], BLOCK, e, false);
    }
  }
  if (a.plies != nullptr) {
    unsigned long long my_plies = plies_here;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) my_plies += __shfl_xor_sync(kFull, my_plies, o);
    if (lane == 0) atomicAdd(a.plies, my_plies);
  }
}

// ---- warp per playout (uniform random policy)

// Warp-cooperative layout, the shape of the reference's playoutKernel
// (src/multiplePlayout.cu:14-52: one block of threads per playout, one thread
// per square), kept as the alternative the autotuner measures against thread
// per playout.  Lane s owns dark square s.  Each ply every lane counts the
// legal moves that start on its square (only captures when the side to move
// has one); a warp prefix sum over the lanes puts them in the reference's
// move-list order (squares ascending, each square's moves in its DFS /
// direction order).  Lane 0 draws the move index from the playout's stream
// exactly as the thread-per-playout kernel does (one draw per ply with two or
// more moves), the lane owning that index applies its move, and the board is
// broadcast.  Outcomes equal the thread-per-playout kernel's bit for bit.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) warp_playout_kernel(PlayoutArgs a) {
  if (a.dev_sizes != nullptr) {
    a.npos = __ldg(&a.dev_sizes[0]);
    a.total = __ldg(&a.dev_sizes[1]);
  }
  const uint32_t lane = threadIdx.x & 31u;
  const int sq = (int)lane;
  unsigned long long plies_here = 0;
  for (;;) {
    uint32_t j = 0;
    if (lane == 0) j = atomicAdd(a.counter, 1u);
    j = __shfl_sync(kFull, j, 0);
    if (j >= a.total) break;
    const uint32_t p = position_of(a, j);
    Board b = load_board(a.pos + p);
    Stream rs;  // drawn by lane 0 only
    rs.init(a.seed, stream_of(a, p, j), 0);
    uint32_t game_plies = 0;
    int outcome = 0;
    for (;;) {
      if (((b.meta >> 8) & 0xffu) >= (uint32_t)kDrawPlies) break;  // draw
      Side s;
      make_side(b, s);
      const uint32_t J = jumpers(s);
      uint32_t md[4];
      direct_masks(s, md);
      int cnt = 0;
      if (J) {
        if ((J >> sq) & 1u) cnt = capture_walk(s, sq, [](int, uint32_t, int, uint32_t) { return false; });
      } else {
        cnt = (int)(((md[0] >> sq) & 1u) + ((md[1] >> sq) & 1u) + ((md[2] >> sq) & 1u) + ((md[3] >> sq) & 1u));
      }
      if (__any_sync(kFull, cnt < 0)) {  // capture deeper than kMaxDepth
        if (lane == 0) atomicOr(a.status, kStatusDepth);
        outcome = 0;
        break;
      }
      uint32_t incl = (uint32_t)cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= (uint32_t)o) incl += t;
      }
      const uint32_t n = __shfl_sync(kFull, incl, 31);
      if (n == 0) {
        outcome = (b.meta & 1u) ? 1 : -1;  // side to move cannot move: loses
        break;
      }
      uint32_t idx = 0;
      if (lane == 0 && n >= 2) idx = mulhi_index(rs.next(), n);
      idx = __shfl_sync(kFull, idx, 0);
      const uint32_t excl = incl - (uint32_t)cnt;
      const bool mine = idx >= excl && idx < incl;
      const int owner = __ffs(__ballot_sync(kFull, mine)) - 1;
      if (mine) {
        uint32_t want = idx - excl;
        if (J) {
          capture_walk(s, sq, [&](int t, uint32_t removed, int, uint32_t) {
            if (want-- != 0) return false;
            apply_move(b, sq, t, removed);
            return true;
          });
        } else {
          for (int d = 0; d < 4; d++)
            if ((md[d] >> sq) & 1u) {
              if (want == 0) {
                apply_move(b, sq, sq + step_off(sq, d), 0u);
                break;
              }
              want--;
            }
        }
      }
      b.p1 = __shfl_sync(kFull, b.p1, owner);
      b.p2 = __shfl_sync(kFull, b.p2, owner);
      b.kings = __shfl_sync(kFull, b.kings, owner);
      b.meta = __shfl_sync(kFull, b.meta, owner);
      if (++game_plies > kMaxPlies) {
        if (lane == 0) atomicOr(a.status, kStatusPlyCap);
        outcome = 0;
        break;
      }
      plies_here++;
    }
    if (lane == 0) a.out[j] = (int8_t)outcome;
  }
  if (a.plies != nullptr && lane == 0) atomicAdd(a.plies, plies_here);
}

// ---- learned-proposal plies (thread per playout)

// One guided ply: the legal moves of playout j's board are weighted by the
// network's policy -- the softmax at temperature T of each move's (from, to)
// logit over the legal pairs, a pair's share split equally among the moves
// that have it -- as integers w = max(1, floor(2^24 e^((l - lmax) / T)) / mult),
// and the move taken is the first whose running weight sum exceeds
// mulhi(draw, sum of w).  The draw is draw number `ply` of the playout's
// stream under tag kTagProposal (the playout's own random moves use tag 0).
// The float steps are detmath.cuh's, so a CPU replay fed the same logits and
// draws picks the same move.  A finished game keeps its board.
__global__ void __launch_bounds__(128) proposal_ply_kernel(ProposalArgs a) {
  if (a.dev_sizes != nullptr) {
    a.npos = __ldg(&a.dev_sizes[0]);
    a.total = __ldg(&a.dev_sizes[1]);
  }
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j == 0 && a.out_sizes != nullptr) {
    a.out_sizes[0] = a.total;
    a.out_sizes[1] = a.total;
  }
  if (j >= a.total) return;
  uint32_t row = j;
  uint64_t sid = a.stream_base + j;
  if (a.per_position) {
    PlayoutArgs pa{};
    pa.offsets = a.offsets;
    pa.npos = a.npos;
    pa.uniform_reps = a.uniform_reps;
    pa.stream_base = a.stream_base;
    pa.pos_stream = a.pos_stream;
    row = position_of(pa, j);
    sid = stream_of(pa, row, j);
  } else if (a.play_stream != nullptr) {
    sid = a.play_stream[j];
  }
  Board b = load_board(a.in + row);
  const uint16_t *lg = a.logits + (size_t)row * 1024u;
  if (a.trace_boards) a.trace_boards[j] = b;
  if (a.trace_logits) {
    const uint4 *src = reinterpret_cast<const uint4 *>(lg);
    uint4 *dst = reinterpret_cast<uint4 *>(a.trace_logits + (size_t)j * 1024u);
    for (int q = 0; q < 128; q++) dst[q] = src[q];
  }
  if (a.out_stream) a.out_stream[j] = sid;
  if (((b.meta >> 8) & 0xffu) < (uint32_t)kDrawPlies) {
    Side sd;
    make_side(b, sd);
    const uint32_t J = jumpers(sd);
    uint32_t c[4] = {a.ply >> 2, (uint32_t)sid, (uint32_t)(sid >> 32), kTagProposal};
    philox4x32_10(c, (uint32_t)a.seed, (uint32_t)(a.seed >> 32));
    const uint32_t w = a.ply & 3u;
    const uint32_t draw = w == 0 ? c[0] : (w == 1 ? c[1] : (w == 2 ? c[2] : c[3]));
    uint16_t pair[kProposalMaxMoves];
    int k = 0;
    float lmax = -3.0e38f;
    const int n = for_each_move(sd, J, [&](int from, int to, uint32_t, int, uint32_t) {
      if (k < kProposalMaxMoves) {
        pair[k] = (uint16_t)(from * 32 + to);
        lmax = fmaxf(lmax, __uint_as_float((uint32_t)lg[pair[k]] << 16));
      }
      k++;
      return false;
    });
    if (n > 0) {
      uint32_t pick = 0;
      if (n > kProposalMaxMoves) {
        pick = mulhi_index(draw, (uint32_t)n);
      } else if (n >= 2) {
        uint32_t wt[kProposalMaxMoves];
        uint32_t sum = 0;
        for (int m = 0; m < n; m++) {
          uint32_t mult = 0;
          for (int q = 0; q < n; q++) mult += pair[q] == pair[m];
          const float l = __uint_as_float((uint32_t)lg[pair[m]] << 16);
          const float e = dm::det_exp(dm::mul(dm::sub(l, lmax), a.inv_temperature));
          const uint32_t v = __float2uint_rz(dm::mul(e, 16777216.0f)) / mult;
          wt[m] = v > 0u ? v : 1u;
          sum += wt[m];
        }
        const uint32_t r = mulhi_index(draw, sum);
        uint32_t acc = 0;
        for (int m = 0; m < n; m++) {
          acc += wt[m];
          if (acc > r) {
            pick = (uint32_t)m;
            break;
          }
        }
      }
      uint32_t at = 0;
      const Board before = b;
      for_each_move(sd, J, [&](int from, int to, uint32_t removed, int, uint32_t) {
        if (at++ != pick) return false;
        b = before;
        apply_move(b, from, to, removed);
        return true;
      });
    }
  }
  store_board(a.out + j, b);
}

// ---- move lists (thread per board)

__global__ void genmoves_kernel(const Board *pos, uint32_t n, uint8_t *out, uint32_t max_moves,
                                uint8_t *counts, uint32_t *status) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Board b = load_board(pos + i);
  Side s;
  make_side(b, s);
  const uint32_t J = jumpers(s);
  uint32_t k = 0;
  const int c = for_each_move(s, J, [&](int from, int to, uint32_t removed, int jumps,
                                        uint32_t dirs) {
    if (k < max_moves) {
      uint32_t w[8];
      pack_move(b, from, to, jumps, dirs, w);
      uint4 *dst = reinterpret_cast<uint4 *>(out + 32 * ((size_t)i * max_moves + k));
      dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
      dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
    k++;
    return false;
  });
  if (c < 0) atomicOr(status, kStatusDepth);
  if (k > max_moves) atomicOr(status, kStatusOverflow);
  counts[i] = (uint8_t)(k > 255u ? 255u : k);
}

// ---- seeded positions of the reference heuristic (thread per position, stream tag 1)

// Position p: U{min_plies..max_plies} plies from the standard start (random
// stream (seed, p, 1)), stopping early at a finished game.  The other policies
// run in playout_kernel; this one's plies take draws in pairs from an even one
// on there, and the first draw here is the length's.
__global__ void heuristic_positions_kernel(uint64_t seed, uint32_t n, PositionArgs pa) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  Stream rs;
  rs.init(seed, p, 1);
  Board b = {0x00000FFFu, 0xFFF00000u, 0u, 0u};
  const uint32_t np = pa.min_plies + mulhi_index(rs.next(), pa.max_plies - pa.min_plies + 1u);
  for (uint32_t q = 0; q < np; q++) {
    if (((b.meta >> 8) & 0xffu) >= (uint32_t)kDrawPlies) break;
    if (ply<1>(b, rs) <= 0) break;
  }
  store_board(pa.out + p, b);
}

// ---- launchers

template <int POLICY, bool POOL>
static const void *kernel_for(int block) {
  switch (block) {
    case 64: return (const void *)playout_kernel<POLICY, 64, POOL>;
    case 128: return (const void *)playout_kernel<POLICY, 128, POOL>;
    case 512: return (const void *)playout_kernel<POLICY, 512, POOL>;
    default: return (const void *)playout_kernel<POLICY, 256, POOL>;
  }
}

static const void *warp_kernel_for(int block) {
  switch (block) {
    case 64: return (const void *)warp_playout_kernel<64>;
    case 128: return (const void *)warp_playout_kernel<128>;
    case 512: return (const void *)warp_playout_kernel<512>;
    default: return (const void *)warp_playout_kernel<256>;
  }
}

static const void *playout_fn(int policy, int block, int layout) {
  if (layout == kLayoutWarp) return warp_kernel_for(block);
  if (layout == kLayoutPooled) {
    if (policy == 1) return kernel_for<1, true>(block);
    if (policy == 2) return kernel_for<2, true>(block);
    return kernel_for<0, true>(block);
  }
  if (policy == 1) return kernel_for<1, false>(block);
  if (policy == 2) return kernel_for<2, false>(block);
  return kernel_for<0, false>(block);
}

bool valid_block(int block) { return block == 64 || block == 128 || block == 256 || block == 512; }

cudaError_t playout_occupancy(int policy, int block, int *blocks_per_sm, int layout) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, playout_fn(policy, block, layout), block, 0);
}

cudaError_t launch_playouts(const PlayoutArgs &a, int policy, int block, int grid, cudaStream_t s, int layout) {
  if (layout == kLayoutWarp && policy != 0) return cudaErrorInvalidValue;
  PositionArgs none{};
  void *args[] = {const_cast<PlayoutArgs *>(&a), &none};  // (the warp layout takes the first alone)
  return cudaLaunchKernel(playout_fn(policy, block, layout), dim3(grid), dim3(block), args, 0, s);
}

cudaError_t launch_proposal_ply(const ProposalArgs &a, cudaStream_t s) {
  const uint32_t grid = (a.total + 127u) / 128u;  // a.total: upper bound when dev_sizes is set
  if (grid == 0) return cudaSuccess;
  proposal_ply_kernel<<<grid, 128, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_genmoves(const Board *pos, uint32_t n, void *out, uint32_t max_moves,
                            uint8_t *counts, uint32_t *status, cudaStream_t s) {
  const int block = 128;
  genmoves_kernel<<<(n + block - 1) / block, block, 0, s>>>(pos, n, (uint8_t *)out, max_moves,
                                                           counts, status);
  return cudaGetLastError();
}

cudaError_t launch_random_positions(uint64_t seed, uint32_t n, uint32_t min_plies,
                                    uint32_t max_plies, Board *out, cudaStream_t s, int sms, int policy) {
  const PositionArgs pa{min_plies, max_plies, out};
  if (policy == 1) {
    heuristic_positions_kernel<<<(n + 127) / 128, 128, 0, s>>>(seed, n, pa);
    return cudaGetLastError();
  }
  constexpr int block = 256;
  const uint32_t resident = (uint32_t)sms * playout_min_blocks<0, block>(), grid = n < resident ? n : resident;
  PlayoutArgs a{};
  a.npos = 1;
  a.uniform_reps = n;
  a.total = n;
  a.seed = seed;
  if (policy == 2) playout_kernel<2, block, false, true><<<grid, block, 0, s>>>(a, pa);
  else playout_kernel<0, block, false, true><<<grid, block, 0, s>>>(a, pa);
  return cudaGetLastError();
}

}  // namespace ga
