// search.cu -- many MCTS searches at once, with their trees in device memory.
//
// The reference runs one search per MCTSPlayer on the host and sends each leaf
// batch to the GPU (src/player.cpp:134-150, src/mcts.cpp:63-191).  Here all
// searches' trees live in one node pool in HBM (structure of arrays, one
// contiguous node range per search) and one step advances every active
// search:
//
//   quota_kernel     leaf slots per search this step (min(Q, remaining
//                    budget)), prefix sums, total leaves / playouts
//   select_kernel    a block per search: the step's Q leaf slots are split
//                    over the tree level by level the way the reference's
//                    GameTree::select splits a batch (src/mcts.cpp:63-157):
//                    untried children share the slots equally, otherwise in
//                    proportion to UCB1, remainders to the heaviest children;
//                    a leaf given more than one slot is expanded; a group of
//                    lanes takes a frontier node, a child per lane
//   playout_kernel   the playout kernel on the leaf boards (sizes and stream
//                    ids read from device memory)
//   backprop_kernel  one thread per leaf: visits and score up the path
//
// Learned searches (a policy/value network attached) add, between the
// playouts and the backpropagation, the network's forward pass on the leaf
// boards (net.cu) and leaf_eval_kernel, which turns a leaf's move logits into
// priors of its moves and its value head into the leaf value.  Their selection
// splits a node's slots by PUCT with virtual visits (split_puct) and expands a
// node once it has been evaluated; backprop blends the network value with the
// playout results.
//
// The launches of a step are replayed as one CUDA graph.  Because each
// search is selected by one block in a fixed order and its playouts use
// its own stream ids, a search's tree and result do not depend on which other
// searches share the steps.
//
// Node record (one uint4 per node, read with one load): x = first child (-1
// before expansion), y = number of children | state << 16, z = playouts through
// the node, w = score in half points of the player who moved into the node.
#include "../../include/gpuai.h"
#include "host/state.hpp"
#include "detmath.cuh"
#include "launch.h"
#include "net.h"
#include "rules.cuh"

#include <cuda_fp16.h>

#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <iterator>
#include <map>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

namespace ga {
namespace {

constexpr uint32_t kExpanded = 1u, kTerminal = 2u, kEvaluated = 4u;  // node state bits (info.y >> 16)
constexpr uint32_t kFull = 0xffffffffu;  // all lanes of a warp
// Levels a selection descends at most (tests compile a smaller limit in)
#ifndef GPUAI_MAX_SELECT_DEPTH
#define GPUAI_MAX_SELECT_DEPTH 512
#endif
constexpr int kMaxSelectDepth = GPUAI_MAX_SELECT_DEPTH;
constexpr uint32_t kStatusSelectDepth = 8u;
// Frontier entries whose expansions take nodes together in a step with Q leaves
// per search (select_kernel).
inline uint32_t select_round(uint32_t Q) { return Q < 128 ? 32u : (Q < 256 ? 128u : (Q < 512 ? 256u : 512u)); }
constexpr uint32_t kMaxLeavesPerStep = 512;  // threads and frontier capacity of the widest select block
constexpr float kUcbC = 1.41421356f;
constexpr int kMaxChildren = 64;  // moves per position handled by split_slots
constexpr uint32_t kUnits = 64;   // learned searches: visit units per leaf slot (score2 = units * (1 + value))
constexpr uint32_t kPriors = 32;  // stored priors per node (more moves: uniform priors)
constexpr uint32_t kAhead = 4;    // slots whose exploration terms split_puct prepares together (2 and 8: slower)
constexpr float kFpuReduction = 0.1f;  // unvisited child's Q = parent's Q - this
constexpr float kTerminalLeaf = 2.0f;  // leaf value marking a finished game

struct Pool {  // one entry per node
  uint32_t nodes;  // capacity (bounds checks of the checked build)
  uint4 *info;   // {first child, nchild | state << 16, visits, score2}
  uint4 *board;
  int32_t *parent;
  uint32_t *move, *removed;
  __half *prior;  // learned searches: kPriors per node, the node's moves' priors
};

struct Table {  // one entry per search slot
  int32_t *root, *node_next, *node_end;
  unsigned long long *stream_next, *budget, *done;
  uint32_t *quota_off;  // slots + 1
};

struct Leaves {
  uint4 *board;
  int32_t *node, *search;
  unsigned long long *stream;
  int8_t *out;
  uint32_t *sizes;  // {leaves, playouts}
  float *value;     // learned searches: network value for the side to move at the leaf
};

struct Learned {
  float c_puct;
  float value_weight;
  uint32_t max_leaves;  // leaf slots per search and step at most (bounds checks of the checked build)
};

__device__ __forceinline__ bool board_terminal(const Board &b) {
  if (((b.meta >> 8) & 0xffu) >= (uint32_t)kDrawPlies) return true;
  Side s;
  make_side(b, s);
  return count_moves(s, jumpers(s)) == 0;
}

// Leaf slots per search and their prefix sums (one block).
__global__ void __launch_bounds__(1024) quota_kernel(Table t, uint32_t slots, uint32_t Q, uint32_t ppl, Leaves l) {
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t carry;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (uint32_t base = 0; base < slots; base += 1024) {
    const uint32_t s = base + tid;
    uint32_t q = 0;
    if (s < slots && t.root[s] >= 0) {
      const unsigned long long b = t.budget[s], d = t.done[s];
      if (d < b) {
        const unsigned long long need = (b - d + ppl - 1) / ppl;
        q = need < Q ? (uint32_t)need : Q;
      }
    }
    uint32_t v = q;
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t n = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += n;
    }
    if (lane == 31) warp_sum[warp] = v;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = warp_sum[lane];
      for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += n;
      }
      warp_sum[lane] = w;
    }
    __syncthreads();
    const uint32_t excl = v - q + (warp ? warp_sum[warp - 1] : 0u);
    if (s < slots) t.quota_off[s] = carry + excl;
    __syncthreads();
    if (tid == 0) carry += warp_sum[31];
    __syncthreads();
  }
  if (tid == 0) {
    t.quota_off[slots] = carry;
    l.sizes[0] = carry;
    l.sizes[1] = carry * ppl;
  }
}

// Number of children a node with board b would get (its legal moves), 0 for none or when
// the game is over (a node's terminal flag is set only for roots; a finished
// game below the root is found here, when it is first to be expanded).
__device__ int child_count(const Board &b) {
  if (((b.meta >> 8) & 0xffu) >= (uint32_t)kDrawPlies) return 0;
  Side sd;
  make_side(b, sd);
  uint32_t M[4];
  bool capture;
  const int k = simple_move_masks(sd, M, capture) ? popc(M[0]) + popc(M[1]) + popc(M[2]) + popc(M[3])
                                                  : count_moves(sd, jumpers(sd));
  return (k > 0 && k <= kMaxChildren) ? k : 0;
}

// Writes child c, reached by the move (from, to, removed), of node n.
__device__ __forceinline__ void write_child(const Pool &p, const Board &b, int32_t n, int32_t c, int from, int to,
                                            uint32_t removed, int jumps) {
  Board cb = b;
  apply_move(cb, from, to, removed);
  p.board[c] = make_uint4(cb.p1, cb.p2, cb.kings, cb.meta);
  p.parent[c] = n;
  p.info[c] = make_uint4(0xffffffffu, 0u, 0u, 0u);
  p.move[c] = (uint32_t)from | ((uint32_t)to << 8) | ((uint32_t)jumps << 16) |
              ((promotes(b, from, to) ? 1u : 0u) << 24);
  p.removed[c] = removed;
}

// Writes the k children of node n at node indices base.. with G lanes (gl =
// 0..G-1), a child each: where no capture can continue a lane takes its move
// straight from the move masks, else it walks the list and writes its share.
// (The node's own record is its thread's to update.)
template <uint32_t G>
__device__ __forceinline__ void expand_group(const Pool &p, const Board &b, int32_t n, int32_t base, int k,
                                             uint32_t gl) {
  Side sd;
  make_side(b, sd);
  uint32_t M[4];
  bool capture;
  if (simple_move_masks(sd, M, capture)) {
    for (int c = (int)gl; c < k; c += (int)G) {
      int from, to;
      uint32_t removed;
      nth_move(M[0], M[1], M[2], M[3], (uint32_t)c, capture, sd.own & ~sd.ownK, from, to, removed);
      write_child(p, b, n, base + c, from, to, removed, capture ? 1 : 0);
    }
  } else {
    int c = 0;
    for_each_move(sd, jumpers(sd), [&](int from, int to, uint32_t removed, int jumps, uint32_t) {
      if ((uint32_t)c % G == gl) write_child(p, b, n, base + c, from, to, removed, jumps);
      c++;
      return false;
    });
  }
}

// Splits T slots over the children of node n (the reference's rule,
// src/mcts.cpp:95-136): untried children share them equally; otherwise in
// proportion to UCB1 weights rounded down; the remainder goes one each to the
// heaviest children (first on ties).  Weights that sum to zero count as
// equal.
// The weights use the correctly rounded operations of detmath.cuh in a fixed
// order, so the CPU restatement (oracle/search.py) reproduces every split.
// A quotient with a zero numerator takes the division's slow path, and its
// whole warp with it (330 against 58 cycles): where there is nothing to divide,
// here and in split_puct, lanes divide 1 and drop the result.
__device__ __forceinline__ float ucb_weight(uint32_t visits, uint32_t score2, float lnN) {
  const float n = (float)(visits ? visits : 1u);
  const float mean = dm::div(score2 ? dm::mul(0.5f, (float)score2) : 1.0f, n);
  return dm::add(score2 ? mean : 0.0f, dm::mul(kUcbC, dm::sqrt_(dm::div(lnN, n))));
}

// The children of a node on a group of G lanes, child c on lane c % G as its
// (c / G)-th of J: what a split reads of them, and the slots it
// gives.  The k children of a node just expanded (fresh) are not read: none has
// been visited.  `own` takes a lane's first child from v0 and h0.
template <int J, uint32_t G>
struct Children {
  static constexpr int kPerLane = J;
  static constexpr uint32_t kLanes = G;
  uint32_t link[J], state[J], visits[J], score2[J], give[J];
  float prior[J];
  __device__ __forceinline__ void load(const Pool &p, int32_t first, int k, bool fresh, uint32_t gl,
                                       const __half *priors, bool own, const uint4 &v0, __half h0) {
#pragma unroll
    for (int j = 0; j < J; j++) {
      const int c = (int)gl + (int)G * j;
      uint4 v = make_uint4(0xffffffffu, 0u, 0u, 0u);
      __half h = __float2half(0.0f);
      if (j == 0 && own) {
        v = v0;
        h = h0;
      } else {
        if (c < k && !fresh) v = p.info[first + c];
        if (c < k && priors) h = priors[c];
      }
      link[j] = v.x;
      state[j] = v.y;
      visits[j] = v.z;
      score2[j] = v.w;
      prior[j] = __half2float(h);
      give[j] = 0;
    }
  }
  // The children given slots, in child order, to entries at.. of the level's slots.
  __device__ __forceinline__ void put(int32_t first, int32_t *t_node, uint32_t *t_cnt, uint4 *t_info, uint32_t at,
                                      uint32_t gl, uint32_t group) const {
    const uint32_t lower = group & ((1u << (threadIdx.x & 31u)) - 1u);
#pragma unroll
    for (int j = 0; j < J; j++) {
      const uint32_t got = __ballot_sync(kFull, give[j] != 0) & group;
      if (give[j]) {
        const uint32_t w = at + __popc(got & lower);
        t_node[w] = first + (int32_t)(gl + G * j);
        t_cnt[w] = give[j];
        t_info[w] = make_uint4(link[j], state[j], visits[j], score2[j]);
      }
      at += __popc(got);
    }
  }
};

// Splits T slots over the k children of a node; `lane0` is the group's first
// lane of the warp.  Every lane of the warp calls it, a group without a node
// with k = T = 0: an operation of the warp with a mask per group runs once for
// each mask (four groups of eight lanes: a shuffle 131 against 50 cycles, a
// vote 395 against 56, a reduction 516 against 56).
template <int J, uint32_t G>
__device__ __forceinline__ void split_slots(Children<J, G> &ch, int k, uint32_t parent_visits, uint32_t T, uint32_t gl,
                                            uint32_t lane0, uint32_t group) {
  const float lnN = dm::det_log((float)(parent_visits > 0 ? parent_visits : 1u));
  float w[J], wsum = 0.0f;
  uint32_t untried = 0;
#pragma unroll
  for (int j = 0; j < J; j++) {
    const bool child = (int)(gl + G * j) < k, fresh = child && ch.visits[j] == 0;
    w[j] = ucb_weight(ch.visits[j], ch.score2[j], lnN);
    if (!child || fresh) w[j] = child ? 3.0e38f : -2.0f;  // no child: below every weight
    untried += __popc(__ballot_sync(kFull, fresh) & group);
  }
  // the sum in child order, and how many children are heavier (first on ties)
  uint32_t heavier[J];
#pragma unroll
  for (int j = 0; j < J; j++) heavier[j] = 0;
#pragma unroll
  for (int i = 0; i < J; i++) {
    const int here = k - (int)G * i;  // k is the warp's where G is 32
#pragma unroll (G < 32u ? (int)G : 4)
    for (int c = 0; c < (G < 32u ? (int)G : here); c++) {
      const float x = __shfl_sync(kFull, w[i], lane0 + c);
      wsum = dm::add(wsum, c < here ? x : 0.0f);
#pragma unroll
      for (int j = 0; j < J; j++)
        heavier[j] += (uint32_t)((x > w[j]) | ((x == w[j]) & (c + (int)G * i < (int)(gl + G * j))));
    }
  }
  const bool equal = untried == 0 && !(wsum > 0.0f);
  const float whole = untried || k == 0 ? 1.0f : (equal ? (float)k : wsum);
  const uint32_t each = untried ? T / untried : 0u;
  uint32_t assigned = 0;
#pragma unroll
  for (int j = 0; j < J; j++) {
    const bool child = (int)(gl + G * j) < k;
    if (equal && child) {
      w[j] = 1.0f;
      heavier[j] = gl + G * j;
    }
    const uint32_t share = (uint32_t)dm::mul((float)T, dm::div(child && !untried ? w[j] : 1.0f, whole));
    if (child) ch.give[j] = untried ? (ch.visits[j] == 0 ? each : 0u) : share;
    assigned += ch.give[j];
  }
#pragma unroll
  for (uint32_t o = 1; o < G; o <<= 1) assigned += __shfl_xor_sync(kFull, assigned, o);
  const uint32_t rest = assigned < T ? T - assigned : 0u;  // fewer than k: one each to the heaviest
#pragma unroll
  for (int j = 0; j < J; j++)
    if ((int)(gl + G * j) < k && heavier[j] < rest) ch.give[j]++;
}

// Learned searches: splits T slots over the k children of node n one slot at
// a time, each to the child with the largest Q + c_puct * P * sqrt(N + t + 1)
// / (1 + n + slots already given) (first on ties), where Q is the child's mean
// score for the player to move at n (an unvisited child: n's own Q minus
// kFpuReduction), P its prior (uniform when n has more than kPriors moves or
// has not been evaluated), N = n's visits and n the child's, in leaf slots.
// A warp takes a node, a child per lane (two for more than 32).  A slot is a
// chain of a few operations: the square roots of 32 slots are taken at once, a
// lane each, the exploration terms that the next kAhead slots can need together,
// a child's next score, chosen or not, is ready before one is chosen, and the
// scores (never negative) are compared as whole numbers by one reduction.  300
// cycles a slot with a division after each choice, 200 now.
template <int J>
__device__ __forceinline__ void split_puct(Children<J, 32> &ch, int k, bool priors, uint32_t parent_visits,
                                           uint32_t parent_score2, uint32_t T, float c_puct, uint32_t lane) {
  if (k == 1) {
    if (lane == 0) ch.give[0] = T;
    return;
  }
  const float half1 = dm::mul(0.5f, (float)parent_score2), all1 = (float)(parent_visits ? parent_visits : 1u);
  float q[J], pr[J], nv[J];
#pragma unroll
  for (int j = 0; j < J; j++) {  // the parent's mean on lane 31, where it has no child, else apart
    const bool parent = J == 1 && (int)lane >= k, tried = ch.visits[j] != 0;
    q[j] = dm::div(parent ? half1 : (tried ? dm::mul(0.5f, (float)ch.score2[j]) : 1.0f),
                   parent ? all1 : (tried ? (float)ch.visits[j] : 1.0f));
  }
  const float mean = J == 1 && k < 32 ? __shfl_sync(kFull, q[0], 31) : dm::div(half1, all1);
  const float fpu = parent_visits ? fmaxf(0.0f, dm::sub(dm::sub(1.0f, mean), kFpuReduction)) : 0.5f;
  const float uniform = priors ? 0.0f : dm::div(1.0f, (float)k);
#pragma unroll
  for (int j = 0; j < J; j++) {
    if (ch.visits[j] == 0) q[j] = fpu;
    if ((int)lane + 32 * j >= k) q[j] = -4.0e18f;  // no child: below every score
    nv[j] = dm::add(1.0f, (float)(ch.visits[j] / kUnits));
    pr[j] = (int)lane + 32 * j < k ? dm::mul(c_puct, priors ? ch.prior[j] : uniform) : 1.0f;
  }
  const float N = (float)(parent_visits / kUnits);
  float roots = 0.0f;
  const uint32_t lower = (1u << lane) - 1u;
  for (uint32_t t = 0; t < T;) {
    // the children's exploration terms, without the sqrt(N) factor, for as many slots as the next kAhead can give one
    const uint32_t ahead = min(T - t, kAhead);
    float u[J][kAhead + 1], sq[kAhead];
    if (J == 1 && k <= 16 && ahead > 1) {
      // few children: the lanes beyond them take later terms of the same quotient
      const uint32_t width = k <= 8 ? 8u : 16u, c = lane & (width - 1u), later = lane / width;
      const float p0 = __shfl_sync(kFull, pr[0], c);
      const float n0 = __shfl_sync(kFull, nv[0], c), n1 = dm::add(n0, 1.0f), n2 = dm::add(n1, 1.0f),
                  n3 = dm::add(n2, 1.0f);
      if (k <= 8) {
        const float d = dm::div(p0, later & 2u ? (later & 1u ? n3 : n2) : (later & 1u ? n1 : n0));
#pragma unroll
        for (uint32_t i = 0; i < kAhead; i++) u[0][i] = __shfl_sync(kFull, d, c + 8u * i);
      } else {
        const float a = dm::div(p0, later ? n1 : n0), b = dm::div(p0, later ? n3 : n2);
#pragma unroll
        for (uint32_t i = 0; i < kAhead; i++) u[0][i] = __shfl_sync(kFull, i < 2 ? a : b, c + 16u * (i & 1u));
      }
      u[0][kAhead] = 0.0f;
    } else {
#pragma unroll
      for (int j = 0; j < J; j++) {
        float n = nv[j];
#pragma unroll
        for (uint32_t i = 0; i < kAhead; i++) {
          u[j][i] = i < ahead ? dm::div(pr[j], n) : 0.0f;
          n = dm::add(n, 1.0f);
        }
        u[j][kAhead] = 0.0f;
      }
    }
    if (t % 32u == 0) roots = dm::sqrt_(dm::add(dm::add(N, (float)(t + lane)), 1.0f));
#pragma unroll
    for (uint32_t i = 0; i < kAhead; i++) sq[i] = __shfl_sync(kFull, roots, (t + i) % 32u);
    int key[J];
#pragma unroll
    for (int j = 0; j < J; j++) key[j] = __float_as_int(dm::add(dm::mul(sq[0], u[j][0]), q[j]));
#pragma unroll
    for (uint32_t i = 0; i < kAhead; i++) {
      if (i >= ahead) break;
      int top = key[0];
#pragma unroll
      for (int j = 1; j < J; j++) top = max(top, key[j]);
      top = __reduce_max_sync(kFull, top);
      uint32_t before = 0;  // children of lower index with the same score
#pragma unroll
      for (int j = 0; j < J; j++) {
        const float next = i + 1 < kAhead ? sq[i + 1 < kAhead ? i + 1 : i] : 0.0f;
        const int passed = __float_as_int(dm::add(dm::mul(next, u[j][0]), q[j])),
                  taken = __float_as_int(dm::add(dm::mul(next, u[j][1]), q[j]));
        const uint32_t same = __ballot_sync(kFull, key[j] == top);
        const bool mine = (key[j] == top) & ((before | (same & lower)) == 0);
        before |= same;
        ch.give[j] += mine ? 1u : 0u;
        nv[j] = mine ? dm::add(nv[j], 1.0f) : nv[j];
        key[j] = mine ? taken : passed;
#pragma unroll
        for (uint32_t a = 0; a < kAhead; a++) u[j][a] = mine ? u[j][a + 1] : u[j][a];
      }
    }
    t += ahead;
  }
}

// A block of T threads per search (T >= the step's leaves per search).  The
// frontier holds (node, slots) pairs, a thread each; a level expands or splits
// them, and its leaf slots and the children given slots go, in entry order, to
// the search's leaf list and the next frontier, with the records the split has
// read.  The slots of an entry are a range of the level's slots (their prefix
// sums), which holds the entry's children or leaf slots in between; a
// compaction over the slots makes the next frontier.
//
// What bounds it is the latency of a level, so each level's serial stretches
// are shared out: a group of lanes (eight, a warp for learned searches and for
// nodes of more than 16 children) expands or splits a node, a child per lane,
// whose record is loaded while the node before is split.  A thread per entry
// that enumerated, loaded and split one child after the other took 152 us for a
// step of 64 searches x 512 leaves, and 205 us for one of 200 learned searches
// x 64 leaves; groups that used masks of their own and divided zeros 97 and
// 70 us; as it stands 56 and 55 us.
//
// Node ranges run out by rounds of `round` entries (a warp's below 128 leaves
// per search, else 128, 256 or 512): an expansion that does not fit what its
// round's earlier expansions leave plays out instead, and so do the round's
// later ones; the next round starts from what was used.
template <bool LEARNED, int T>
__global__ void __launch_bounds__(T, 1024 / T)
    select_kernel(Pool p, Table t, Leaves l, uint32_t slots, uint32_t ppl, uint32_t round, Learned lrn,
                  uint32_t *status) {
  constexpr int kWarps = T / 32;
  constexpr uint32_t G = LEARNED ? 32u : 8u, kGroups = 32u / G;  // lanes that take a node, nodes a warp takes
  constexpr uint32_t kLeafSlot = 0x80000000u;
  __shared__ int32_t f_node[T];   // the frontier: node, slots, the node's record
  __shared__ uint32_t f_cnt[T];
  __shared__ uint4 f_info[T];
  __shared__ int32_t t_node[T];   // the level's slots: a child and its slots, or a leaf slot, or nothing
  __shared__ uint32_t t_cnt[T];
  __shared__ uint4 t_info[T];
  __shared__ int32_t s_leaf[T];   // the leaf slots' nodes
  __shared__ uint4 s_board[T];    // boards of the nodes to expand
  __shared__ __align__(16) uint32_t s_scan[2][kWarps];
  // the entries that expand or split, for their groups: first child, children | state << 8 | fresh << 31 (0:
  // none), first slot
  __shared__ int32_t s_first[T];
  __shared__ uint32_t s_k[T], s_at[T];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t gl = tid % G, gi = tid / G, lane0 = lane & ~(G - 1u), group = (0xffffffffu >> (32u - G)) << lane0;
  const uint32_t s = blockIdx.x;
  const int32_t root = t.root[s];
  if (root < 0) return;  // uniform over the block
  const uint32_t off = t.quota_off[s], q = t.quota_off[s + 1] - off;
  if (q == 0 || !GA_IN_BOUNDS(q <= (uint32_t)T, status)) return;
  // Entries and slots are at most q, a thread each: the warps beyond them take
  // no part in the scans.  Two sums go in one word (slots, at most 512, below
  // children, at most 512 * kMaxChildren), and the warps' totals alternate
  // between two buffers, so that a scan is one barrier.
  const uint32_t qw = (q + 31u) / 32u;
  uint32_t buf = 0;
  if (tid < 2 * kWarps) s_scan[tid / kWarps][tid % kWarps] = 0;
  // v: the inclusive sums within the warp; returns those over the block
  auto over_warps = [&](uint32_t v, uint32_t &total) -> uint32_t {
    if (lane == 31 && warp < qw) s_scan[buf][warp] = v;
    __syncthreads();
    uint32_t before = 0, sum = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w += 4) {
      if ((uint32_t)w >= qw) break;
      const uint4 x = *reinterpret_cast<const uint4 *>(&s_scan[buf][w]);
      before += ((uint32_t)w < warp ? x.x : 0u) + (w + 1u < warp ? x.y : 0u) + (w + 2u < warp ? x.z : 0u) +
                (w + 3u < warp ? x.w : 0u);
      sum += (x.x + x.y) + (x.z + x.w);
    }
    buf ^= 1u;
    total = sum;
    return v + before;
  };
  auto scan = [&](uint32_t v, uint32_t &total) -> uint32_t {
    if (warp < qw) {
#pragma unroll
      for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += x;
      }
    }
    return over_warps(v, total);
  };
  auto block_max = [&](uint32_t x) -> uint32_t {
    x = __reduce_max_sync(0xffffffffu, x);
    if (lane == 31 && warp < qw) s_scan[buf][warp] = x;
    __syncthreads();
    uint32_t m = 0;
    for (uint32_t w = 0; w < qw; w++) m = max(m, s_scan[buf][w]);
    buf ^= 1u;
    return m;
  };
  uint32_t nf = 1, emitted = 0;
  int32_t node_next = t.node_next[s];
  const int32_t node_end = t.node_end[s];
  t_cnt[tid] = 0;
  if (tid == 0) {
    f_node[0] = root;
    f_cnt[0] = q;
    f_info[0] = p.info[root];
  }
  __syncthreads();
  for (int depth = 0; nf > 0; depth++) {
    if (depth >= kMaxSelectDepth) {
      if (tid == 0) atomicOr(status, kStatusSelectDepth);
      break;
    }
    // what each thread's entry does: leaf slots, an expansion (grow), a split
    int32_t n = -1, first = 0, k = 0;
    uint32_t slots_here = 0, visits = 0, score2 = 0, st = 0;
    int grow = 0;  // children the node gets if it is expanded now
    bool leaf = false;
    if (tid < nf) {
      n = f_node[tid];
      slots_here = f_cnt[tid];
      const uint4 inf = f_info[tid];
      st = inf.y >> 16;
      visits = inf.z;
      score2 = inf.w;
      first = (int32_t)inf.x;
      k = (int32_t)(inf.y & 0xffffu);
      if (st & kTerminal) {
        leaf = true;
      } else if (!(st & kExpanded)) {
        // a learned node is expanded once the network has evaluated it, a
        // plain one when it is given more than one slot
        if (LEARNED ? (st & kEvaluated) != 0 : slots_here > 1) {
          const uint4 bv = p.board[n];
          s_board[tid] = bv;
          grow = child_count(Board{bv.x, bv.y, bv.z, bv.w});
        }
        leaf = grow == 0;
      }
    }
    uint32_t tot;
    const uint32_t sums = scan(slots_here | ((uint32_t)grow << 16), tot);
    const uint32_t gx = sums >> 16, stot = tot & 0xffffu, gtot = tot >> 16;
    const uint32_t at = (sums & 0xffffu) - slots_here;  // the entry's first slot of the level's
    bool fresh = false;
    if (gtot != 0) {  // uniform over the block
      if (node_next + (int64_t)gtot <= node_end) {
        fresh = grow > 0;
        first = fresh ? node_next + (int32_t)gx - grow : first;
        node_next += (int32_t)gtot;
      } else {
        s_at[tid] = gx;
        __syncthreads();
        for (uint32_t r = 0; r < nf; r += round) {  // fitting is a prefix of a round's entries: its sums grow
          const uint32_t in_round = gx - (r ? s_at[r - 1u] : 0u);
          const bool fits = grow > 0 && tid >= r && tid < r + round && node_next + (int64_t)in_round <= node_end;
          if (fits) {
            fresh = true;
            first = node_next + (int32_t)in_round - grow;
          }
          node_next += (int32_t)block_max(fits ? in_round : 0u);
        }
        leaf = leaf || (grow > 0 && !fresh);
      }
      if (fresh) {
        k = grow;
        if (!GA_IN_BOUNDS(first + k <= node_end && (uint32_t)node_end <= p.nodes, status)) {
          fresh = false;
          leaf = true;
        }
      }
      if (fresh) p.info[n] = make_uint4((uint32_t)first, (uint32_t)k | ((st | kExpanded) << 16), visits, score2);
    }
    if (tid < nf && leaf) {
      for (uint32_t r = 0; r < slots_here; r++) {
        t_node[at + r] = n;
        t_cnt[at + r] = kLeafSlot;
      }
    }
    s_first[tid] = first;
    s_k[tid] = tid < nf && !leaf ? (uint32_t)k | (st << 8) | (fresh ? 0x80000000u : 0u) : 0u;
    s_at[tid] = at;
    __syncthreads();
    // a lane's child of an entry, loaded while the entry before it is split
    uint4 next_v = make_uint4(0u, 0u, 0u, 0u);
    __half next_h = __float2half(0.0f);
    auto fetch = [&](uint32_t e) {
      const uint32_t ke = e < nf ? s_k[e] : 0u;
      next_v = make_uint4(0xffffffffu, 0u, 0u, 0u);
      if (gl < (ke & 0xffu)) {
        if (!(ke & 0x80000000u)) next_v = p.info[s_first[e] + (int32_t)gl];
        if (LEARNED && ((ke >> 8) & kEvaluated)) next_h = p.prior[(size_t)f_node[e] * kPriors + gl];
      }
    };
    fetch(gi);
    for (uint32_t e0 = warp * kGroups; e0 < nf; e0 += T / G) {  // uniform over the warp
      const uint32_t e = e0 + gi % kGroups, ke = e < nf ? s_k[e] : 0u;
      const uint4 v0 = next_v;
      const __half h0 = next_h;
      fetch(e + T / G);
      const int kk = (int)(ke & 0xffu);
      const bool fr = (ke & 0x80000000u) != 0;
      // the groups' nodes (no children and no slots where a group has none here)
      auto split = [&](auto &&ch, uint32_t at, int k, uint32_t ke, uint32_t gl, uint32_t lane0, uint32_t group) {
        using C = std::remove_reference_t<decltype(ch)>;
        const int32_t first = s_first[at];
        const uint32_t cnt = k ? f_cnt[at] : 0u;
        const __half *pri = nullptr;
        if (LEARNED && ((ke >> 8) & kEvaluated) && k <= (int)kPriors) pri = p.prior + (size_t)f_node[at] * kPriors;
        ch.load(p, first, k, (ke & 0x80000000u) != 0, gl, pri, C::kLanes == G, v0, h0);
        if constexpr (LEARNED)
          split_puct<C::kPerLane>(ch, k, pri != nullptr, f_info[at].z, f_info[at].w, cnt, lrn.c_puct, lane);
        else split_slots(ch, k, f_info[at].z, cnt, gl, lane0, group);
        ch.put(first, t_node, t_cnt, t_info, s_at[at], gl, group);
      };
      const bool many = kk > 2 * (int)G;
      const int ks = many ? 0 : kk;
      const uint32_t at_e = ks ? e : 0u;
      if (__any_sync(kFull, ks > (int)G)) split(Children<2, G>{}, at_e, ks, ke, gl, lane0, group);
      else if (__any_sync(kFull, ks != 0)) split(Children<1, G>{}, at_e, ks, ke, gl, lane0, group);
      if constexpr (!LEARNED) {  // nodes of more than 16 children take the warp
        for (uint32_t left = __ballot_sync(kFull, many && gl == 0); left; left &= left - 1u) {
          const uint32_t b = e0 + (__ffs(left) - 1u) / G, kb = s_k[b];
          split(Children<2, 32u>{}, b, (int)(kb & 0xffu), kb, lane, 0u, kFull);
        }
      }
      if (fr) {
        const uint4 bv = s_board[e];
        expand_group<G>(p, Board{bv.x, bv.y, bv.z, bv.w}, f_node[e], s_first[e], kk, gl);
      }
    }
    __syncthreads();
    // compaction of the level's slots: the next frontier and the leaf slots
    const uint32_t have = tid < stot ? t_cnt[tid] : 0u;
    const int32_t node = tid < stot ? t_node[tid] : 0;
    const bool is_leaf = have == kLeafSlot;
    const uint32_t upto = 0xffffffffu >> (31u - lane);
    const uint32_t kept = __popc(__ballot_sync(0xffffffffu, have != 0 && !is_leaf) & upto),
                   left = __popc(__ballot_sync(0xffffffffu, is_leaf) & upto);
    const uint32_t places = over_warps(kept | (left << 16), tot);
    const uint32_t kx = places & 0xffffu, lx = places >> 16;
    t_cnt[tid] = 0;
    if (is_leaf) {
      if (GA_IN_BOUNDS(emitted + lx <= q && (uint32_t)node < p.nodes, status)) s_leaf[emitted + lx - 1u] = node;
    } else if (have && GA_IN_BOUNDS((uint32_t)node < p.nodes, status)) {
      f_node[kx - 1u] = node;
      f_cnt[kx - 1u] = have;
      f_info[kx - 1u] = t_info[tid];
    }
    nf = tot & 0xffffu;
    emitted += tot >> 16;
    __syncthreads();
  }
  // the leaf slots, with their random streams in slot order; the slots of a
  // selection that stopped at the depth limit play out the root, so that no
  // kernel of the step meets an earlier step's entry (whose search may be gone)
  const unsigned long long sbase = t.stream_next[s];
  if (tid < q && GA_IN_BOUNDS(off + tid < slots * lrn.max_leaves, status)) {
    const int32_t n = tid < emitted ? s_leaf[tid] : root;
    l.board[off + tid] = p.board[n];
    l.node[off + tid] = n;
    l.search[off + tid] = (int32_t)s;
  }
  if (tid < q) l.stream[off + tid] = sbase + (unsigned long long)tid * ppl;
  __syncthreads();
  if (tid == 0) {
    t.node_next[s] = node_next;
    t.stream_next[s] = sbase + (unsigned long long)q * ppl;
  }
}

// Adds a leaf's result up its path, one thread per leaf: `visits` to every node
// and, to a node that PLAYER_1 moved into, s1 half points, else s2 (the players
// alternate along the path).  The root and the search's count take the same
// addition from every leaf of the search: a warp whose leaves are all of one
// search adds its sum there once.  A path that does not end at the root adds
// nothing there.  (With an addition per leaf, and each node's
// board loaded for its mover, 16.5 against 8 us a step of 64 searches x 512
// leaves.)
__device__ __forceinline__ void add_up(const Pool &p, const Table &t, bool on, int32_t s, int32_t leaf,
                                       uint32_t leaf_turn, uint32_t visits, uint32_t s1, uint32_t s2, uint32_t ppl,
                                       uint32_t *status) {
  const int32_t root = on ? t.root[s] : -1;
  bool first = (leaf_turn & 1u) != 0;  // PLAYER_1 moved into the leaf
  int32_t n = leaf;
  if (on) {
    while (n != root && n >= 0) {
      if (!GA_IN_BOUNDS((uint32_t)n < p.nodes, status)) break;
      atomicAdd(&p.info[n].z, visits);
      atomicAdd(&p.info[n].w, first ? s1 : s2);
      first = !first;
      n = p.parent[n];
    }
  }
  const bool ends = on && n >= 0 && n == root;
  const uint32_t score = on ? (first ? s1 : s2) : 0u;
  const int32_t s0 = __shfl_sync(kFull, s, 0);  // every lane takes part, also those without a leaf
  if (__all_sync(kFull, ends && s == s0)) {
    const uint32_t sum = __reduce_add_sync(kFull, score);
    if ((threadIdx.x & 31u) == 0) {
      atomicAdd(&p.info[root].z, 32u * visits);
      atomicAdd(&p.info[root].w, sum);
      atomicAdd(&t.done[s], 32ull * ppl);
    }
  } else if (on) {
    if (ends) {
      atomicAdd(&p.info[root].z, visits);
      atomicAdd(&p.info[root].w, score);
    }
    atomicAdd(&t.done[s], (unsigned long long)ppl);
  }
}

// Outcomes up the path (score in half points for the player who made the move
// into each node).
__global__ void backprop_kernel(Pool p, Table t, Leaves l, uint32_t ppl, uint32_t max_leaves, uint32_t *status) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = i < max_leaves && i < l.sizes[0];
  uint32_t w1 = 0, w2 = 0, dr = 0, turn = 0;
  int32_t s = -1, leaf = -1;
  if (on) {
    s = l.search[i];
    leaf = l.node[i];
    turn = l.board[i].w;
    for (uint32_t k = 0; k < ppl; k++) {
      const int8_t o = l.out[(size_t)i * ppl + k];
      w1 += o > 0;
      w2 += o < 0;
      dr += o == 0;
    }
  }
  add_up(p, t, on, s, leaf, turn, ppl, 2u * w1 + dr, 2u * w2 + dr, ppl, status);
}

// Learned searches: the leaf's result for PLAYER_1 is value_weight * network
// value + (1 - value_weight) * playout mean (terminal leaves: the playouts,
// which end at once with the exact result), added as kUnits visits.
__global__ void backprop_learned_kernel(Pool p, Table t, Leaves l, uint32_t ppl, uint32_t max_leaves,
                                        Learned lrn, uint32_t *status) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = i < max_leaves && i < l.sizes[0];
  int32_t s = -1, leaf = -1;
  uint32_t turn = 0, s1 = 0;
  if (on) {
    s = l.search[i];
    leaf = l.node[i];
    turn = l.board[i].w;
    int sum = 0;  // outcomes for PLAYER_1
    for (uint32_t k = 0; k < ppl; k++) sum += l.out[(size_t)i * ppl + k];
    const float pm = dm::div((float)sum, (float)ppl);
    float x1 = pm;
    const float v = l.value[i];
    if (v <= 1.0f) {  // kTerminalLeaf (> 1): a finished game, whose playouts give the exact result
      const float v1 = (turn & 1u) ? -v : v;  // the value is for the side to move
      x1 = dm::add(dm::mul(lrn.value_weight, v1), dm::mul(dm::sub(1.0f, lrn.value_weight), pm));
    }
    x1 = fminf(1.0f, fmaxf(-1.0f, x1));
    s1 = (uint32_t)__float2int_rn(dm::mul((float)kUnits, dm::add(1.0f, x1)));  // half points of PLAYER_1
  }
  add_up(p, t, on, s, leaf, turn, kUnits, s1, 2u * kUnits - s1, ppl, status);
}

// Learned searches: kEvalLanes lanes per leaf.  The leaf value (tanh of the value
// head, for the side to move; kTerminalLeaf for a finished game) and, the
// first time a node is a leaf, its moves' priors: the softmax of the move
// logits over its legal (from, to) pairs, a pair's probability shared equally
// by the moves that have it.
// Where no capture can continue the pairs are the moves, and a lane takes every
// eighth of them straight from the move masks; else one lane walks the list.
// The sum is in move order in both.  A thread per leaf was bound by the walks of
// 32 different boards in a warp and by its chain of dependent loads: 34 us for
// 12,800 leaves, 11 us now (a step of 200 searches x 64 leaves 213 -> 191 us, with
// one guided ply 272 -> 249 us).
constexpr uint32_t kEvalLanes = 8, kEvalThreads = 128;
__global__ void __launch_bounds__(kEvalThreads)
    leaf_eval_kernel(Pool p, Leaves l, const __nv_bfloat16 *logits, const float *vraw, uint32_t max_leaves) {
  constexpr int G = (int)kEvalLanes, J = (int)kPriors / G;
  const uint32_t i = blockIdx.x * (kEvalThreads / kEvalLanes) + threadIdx.x / kEvalLanes;
  const int gl = (int)(threadIdx.x % kEvalLanes), lane0 = (int)(threadIdx.x & 31u) - gl;
  const bool on = i < max_leaves && i < l.sizes[0];
  const uint4 bv = on ? l.board[i] : make_uint4(0u, 0u, 0u, 0u);
  const Board b{bv.x, bv.y, bv.z, bv.w};
  Side sd;
  make_side(b, sd);
  uint32_t M[4];
  bool capture;
  const bool simple = simple_move_masks(sd, M, capture);
  const int k = !on ? 0
                    : (simple ? popc(M[0]) + popc(M[1]) + popc(M[2]) + popc(M[3]) : count_moves(sd, jumpers(sd)));
  const bool over = k == 0 || ((b.meta >> 8) & 0xffu) >= (uint32_t)kDrawPlies;
  if (on && gl == 0) l.value[i] = over ? kTerminalLeaf : dm::det_tanh(vraw[i]);
  const int32_t n = on ? l.node[i] : 0;
  // One lane reads the node's state for its group: other groups with the same
  // node set kEvaluated meanwhile, and the group's maximum and sum need all its
  // lanes or none.  (A group that finds it set leaves the priors to the others,
  // which write the whole list, the same one.)
  const uint32_t state = __shfl_sync(kFull, on && gl == 0 ? p.info[n].y >> 16 : 0u, lane0);
  const bool fresh = on && !over && !(state & (kEvaluated | kTerminal));
  const __nv_bfloat16 *lr = logits + (size_t)i * net::kOut;
  const bool shared = fresh && simple && k <= (int)kPriors;
  if (__any_sync(kFull, shared)) {
    float x[J], lmax = -3.0e38f, sum = 0.0f;
#pragma unroll
    for (int j = 0; j < J; j++) {
      const int c = gl + G * j;
      x[j] = -3.0e38f;
      if (shared && c < k) {
        int from, to;
        uint32_t removed;
        nth_move(M[0], M[1], M[2], M[3], (uint32_t)c, capture, sd.own & ~sd.ownK, from, to, removed);
        x[j] = __bfloat162float(lr[from * 32 + to]);
        lmax = fmaxf(lmax, x[j]);
      }
    }
#pragma unroll
    for (int o = 1; o < G; o <<= 1) lmax = fmaxf(lmax, __shfl_xor_sync(kFull, lmax, o));
#pragma unroll
    for (int j = 0; j < J; j++) {
      const bool child = shared && gl + G * j < k;
      x[j] = dm::det_exp(dm::sub(x[j], lmax));
      if (!__any_sync(kFull, shared && k > G * j)) break;
#pragma unroll
      for (int c = 0; c < G; c++) sum = dm::add(sum, __shfl_sync(kFull, child ? x[j] : 0.0f, lane0 + c));
    }
#pragma unroll
    for (int j = 0; j < J; j++)
      if (shared)
        p.prior[(size_t)n * kPriors + gl + G * j] = __float2half_rn(gl + G * j < k ? dm::div(x[j], sum) : 0.0f);
  }
  if (!fresh || gl != 0) return;
  int written = shared ? (int)kPriors : 0;  // the rest of the node's priors are zero
  if (!simple && k >= 1 && k <= (int)kPriors) {  // (k is -1 where a capture passes the depth limit)
    uint16_t pair[kPriors] = {};
    uint8_t of[kPriors];
    uint8_t mult[kPriors];
    int np = 0, m = 0;
    for_each_move(sd, jumpers(sd), [&](int from, int to, uint32_t, int, uint32_t) {
      const uint16_t pi = (uint16_t)(from * 32 + to);
      int u = 0;
      while (u < np && pair[u] != pi) u++;
      if (u == np) {
        pair[np] = pi;
        mult[np] = 0;
        np++;
      }
      mult[u]++;
      of[m++] = (uint8_t)u;
      return false;
    });
    float e[kPriors];
    float lmax = -3.0e38f;
    for (int u = 0; u < np; u++) {
      e[u] = __bfloat162float(lr[pair[u]]);
      lmax = fmaxf(lmax, e[u]);
    }
    float sum = 0.0f;
    for (int u = 0; u < np; u++) {
      e[u] = dm::det_exp(dm::sub(e[u], lmax));
      sum = dm::add(sum, e[u]);
    }
    for (int j = 0; j < k; j++) {
      const int u = of[j];
      p.prior[(size_t)n * kPriors + j] = __float2half_rn(dm::div(dm::div(e[u], sum), (float)mult[u]));
    }
    written = k;
  }
  for (int j = written; j < (int)kPriors; j++) p.prior[(size_t)n * kPriors + j] = __float2half_rn(0.0f);
  atomicOr(&p.info[n].y, kEvaluated << 16);
}

__global__ void init_search_kernel(Pool p, Table t, int32_t slot, int32_t start, int32_t cap, uint4 board,
                                   unsigned long long budget, unsigned long long stream_base) {
  p.board[start] = board;
  p.parent[start] = -1;
  const Board b{board.x, board.y, board.z, board.w};
  p.info[start] = make_uint4(0xffffffffu, (board_terminal(b) ? kTerminal : 0u) << 16, 0u, 0u);
  p.move[start] = 0;
  p.removed[start] = 0;
  t.root[slot] = start;
  t.node_next[slot] = start + 1;
  t.node_end[slot] = start + cap;
  t.stream_next[slot] = stream_base;
  t.budget[slot] = budget;
  t.done[slot] = 0;
}

__global__ void remove_search_kernel(Table t, int32_t slot) { t.root[slot] = -1; }

// A search's root and its children, as gpuai_searches_children reports them.
struct RootReport {
  uint4 board, info;
  int32_t nodes_used;
  uint32_t pad[3];
  uint2 child[kMaxChildren];  // visits, score2
};

// Gathers the report into pinned host memory (one block of kMaxChildren
// threads).  One launch and one wait in place of four copies and two waits, the
// second pair of which needed the first's result: 47 -> 18 us for Searches.best.
__global__ void root_report_kernel(Pool p, Table t, int32_t slot, int32_t root, RootReport *out) {
  const uint4 info = p.info[root];
  const uint32_t k = ((info.y >> 16) & kExpanded) ? info.y & 0xffffu : 0u, c = threadIdx.x;
  if (c < k) {
    const uint4 ci = p.info[info.x + c];
    out->child[c] = make_uint2(ci.z, ci.w);
  }
  if (c == 0) {
    out->board = p.board[root];
    out->info = info;
    out->nodes_used = t.node_next[slot] - root;
  }
}

}  // namespace
}  // namespace ga

using namespace ga;

struct gpuai_searches {
  int device = 0;
  cudaStream_t stream = nullptr;
  uint32_t slots = 0, pool_nodes = 0, qmax = 0, ppl = 1;
  int32_t policy = 0;
  uint64_t seed = 0;
  int sms = 0, blocks_per_sm = 1;
  Pool pool{};
  Table tab{};
  Leaves leaves{};
  uint32_t *ctl = nullptr;  // counter, status, plies (2 words)
  RootReport *report = nullptr;  // pinned host memory, written by root_report_kernel
  std::map<uint32_t, uint32_t> free_ranges;  // start -> length
  std::vector<int32_t> start, cap;           // per slot; start -1 = free slot
  cudaGraphExec_t graph = nullptr;
  uint32_t graph_q = 0;
  std::mutex mu;
  std::vector<void *> allocations;
  // learned searches
  gpuai_net *net = nullptr;
  Learned lrn{1.5f, 1.0f, 0u};
  ga::net::Fwd fw;
  cudaStream_t side = nullptr;  // the network's branch of a learned step
  cudaEvent_t fork = nullptr, join = nullptr;
  // learned-proposal playouts: the first `guided` plies of each playout are
  // drawn from the network's policy
  uint32_t guided = 0;
  float inv_temperature = 1.0f;
  ga::net::Fwd pfw;               // forward on the playouts' boards (later guided plies)
  ga::Board *pcur = nullptr;      // each playout's board
  unsigned long long *pstream = nullptr;  // each playout's stream id
  uint32_t *psizes = nullptr;     // {playouts, playouts}
};

namespace {

int err(int code, const std::string &m) { return ga::record_error(code, m.c_str()); }
int cuda_err(cudaError_t e, const char *what) {
  return err(e == cudaErrorMemoryAllocation ? GPUAI_ERR_OOM : GPUAI_ERR_CUDA,
             std::string("searches: ") + what + ": " + cudaGetErrorString(e));
}

#define SCK(call, what)                                   \
  do {                                                    \
    cudaError_t e_ = (call);                              \
    if (e_ != cudaSuccess) return cuda_err(e_, what);     \
  } while (0)

template <class T>
cudaError_t dalloc(gpuai_searches *s, T **p, size_t n) {
  void *q = nullptr;
  cudaError_t e = cudaMalloc(&q, n * sizeof(T) + 16);
  if (e == cudaSuccess) {
    s->allocations.push_back(q);
    *p = static_cast<T *>(q);
  }
  return e;
}

int enqueue_step(gpuai_searches *s, uint32_t q) {
  const cudaStream_t st = s->stream;
  // work counter and ply count restart every step; status bits accumulate
  // until poll reads them
  SCK(cudaMemsetAsync(s->ctl, 0, sizeof(uint32_t), st), "reset work counter");
  quota_kernel<<<1, 1024, 0, st>>>(s->tab, s->slots, q, s->ppl, s->leaves);
  // a block per search with a thread per leaf
  auto sel = [&](auto kernel, uint32_t threads) {
    kernel<<<s->slots, threads, 0, st>>>(s->pool, s->tab, s->leaves, s->slots, s->ppl, select_round(q), s->lrn,
                                         s->ctl + 1);
  };
  if (s->net) {
    // 16 warps, a node each, while two blocks per SM hold all searches: 1 to 4 %
    // of a step (1 search x 64 leaves 120.6 -> 117.0 us, 200 x 64 194.8 -> 192.3,
    // 300 x 256 461 -> 451); 16 leaves have no work for them (200 x 16: 136.5
    // against 137.6 us)
    const bool wide = q > 256 || (q > 16 && s->slots <= 2u * (uint32_t)s->sms);
    if (!wide) sel(select_kernel<true, 256>, 256);
    else sel(select_kernel<true, 512>, 512);
  } else {
    if (q <= 128) sel(select_kernel<false, 128>, 128);
    else if (q <= 256) sel(select_kernel<false, 256>, 256);
    else sel(select_kernel<false, 512>, 512);
  }
  // The playouts' number is known on the device alone when a step is enqueued
  // (and a captured step is replayed as the searches finish), so every step
  // launches 256-thread blocks: us a step with 256 / 128 threads, one search of 64
  // leaves x 2 93.6 / 91.8, 4 searches 114 / 106, 16 of 64 x 8 132 / 131, 64 of
  // 128 x 8 185 / 187.
  PlayoutArgs a;
  a.pos = reinterpret_cast<const Board *>(s->leaves.board);
  a.offsets = nullptr;
  a.npos = 0;
  a.uniform_reps = s->ppl;
  a.total = 0;
  a.seed = s->seed;
  a.stream_base = 0;
  a.out = s->leaves.out;
  a.counter = s->ctl;
  a.status = s->ctl + 1;
  a.plies = nullptr;
  a.pos_stream = reinterpret_cast<const uint64_t *>(s->leaves.stream);
  a.dev_sizes = s->leaves.sizes;
  const uint32_t max_leaves = s->slots * s->qmax;
  const uint32_t eval_blocks = (uint32_t)(((uint64_t)max_leaves * kEvalLanes + kEvalThreads - 1) / kEvalThreads);
  if (s->net && s->guided > 0) {
    // learned-proposal step: the network's forward on the leaves gives the
    // priors, the leaf values and the first guided ply of every playout;
    // later guided plies run the network on the playouts' boards; then the
    // uniformly random rest of each game
    SCK(ga::net::forward(s->net, s->fw, reinterpret_cast<const gpuai_board *>(s->leaves.board), 0, s->leaves.sizes,
                         s->ctl + 1, st),
        "network forward on the leaves");
    leaf_eval_kernel<<<eval_blocks, kEvalThreads, 0, st>>>(s->pool, s->leaves, s->fw.logits_b, s->fw.vraw,
                                                               max_leaves);
    SCK(cudaGetLastError(), "leaf evaluation launch");
    ProposalArgs pa{};
    pa.in = reinterpret_cast<const Board *>(s->leaves.board);
    pa.uniform_reps = s->ppl;
    pa.total = max_leaves * s->ppl;  // grid bound; the sizes come from device memory
    pa.dev_sizes = s->leaves.sizes;
    pa.per_position = true;
    pa.logits = reinterpret_cast<const uint16_t *>(s->fw.logits_b);
    pa.seed = s->seed;
    pa.pos_stream = reinterpret_cast<const uint64_t *>(s->leaves.stream);
    pa.inv_temperature = s->inv_temperature;
    pa.out = s->pcur;
    pa.out_stream = reinterpret_cast<uint64_t *>(s->pstream);
    pa.out_sizes = s->psizes;
    for (uint32_t g = 0; g < s->guided; g++) {
      if (g > 0) {
        SCK(ga::net::forward(s->net, s->pfw, reinterpret_cast<const gpuai_board *>(s->pcur), 0, s->psizes,
                             s->ctl + 1, st),
            "network forward on the playouts");
        pa.in = s->pcur;
        pa.per_position = false;
        pa.dev_sizes = s->psizes;
        pa.logits = reinterpret_cast<const uint16_t *>(s->pfw.logits_b);
        pa.pos_stream = nullptr;
        pa.play_stream = reinterpret_cast<const uint64_t *>(s->pstream);
        pa.out_stream = nullptr;
        pa.out_sizes = nullptr;
      }
      pa.ply = g;
      SCK(ga::launch_proposal_ply(pa, st), "guided ply launch");
    }
    PlayoutArgs b = a;
    b.pos = s->pcur;
    b.uniform_reps = 1;
    b.pos_stream = reinterpret_cast<const uint64_t *>(s->pstream);
    b.dev_sizes = s->psizes;
    SCK(launch_playouts(b, s->policy, kPlayoutBlock, s->sms * s->blocks_per_sm, st), "playout kernel launch");
    backprop_learned_kernel<<<(max_leaves + 255) / 256, 256, 0, st>>>(s->pool, s->tab, s->leaves, s->ppl,
                                                                      max_leaves, s->lrn, s->ctl + 1);
    SCK(cudaGetLastError(), "search kernel launch");
    return GPUAI_OK;
  }
  if (s->net) {
    // the network's forward pass and the leaf evaluation do not depend on the
    // playouts: they run on a second stream and fill the SMs that the playout
    // kernel's last games leave idle; backprop waits for both
    SCK(cudaEventRecord(s->fork, st), "fork");
    SCK(cudaStreamWaitEvent(s->side, s->fork, 0), "fork");
    SCK(ga::net::forward(s->net, s->fw, reinterpret_cast<const gpuai_board *>(s->leaves.board), 0, s->leaves.sizes,
                         s->ctl + 1, s->side),
        "network forward on the leaves");
    leaf_eval_kernel<<<eval_blocks, kEvalThreads, 0, s->side>>>(s->pool, s->leaves, s->fw.logits_b,
                                                                    s->fw.vraw, max_leaves);
    SCK(cudaGetLastError(), "leaf evaluation launch");
    SCK(cudaEventRecord(s->join, s->side), "join");
  }
  SCK(launch_playouts(a, s->policy, kPlayoutBlock, s->sms * s->blocks_per_sm, st), "playout kernel launch");
  if (s->net) {
    SCK(cudaStreamWaitEvent(st, s->join, 0), "join");
    backprop_learned_kernel<<<(max_leaves + 255) / 256, 256, 0, st>>>(s->pool, s->tab, s->leaves, s->ppl,
                                                                      max_leaves, s->lrn, s->ctl + 1);
  } else {
    backprop_kernel<<<(max_leaves + 255) / 256, 256, 0, st>>>(s->pool, s->tab, s->leaves, s->ppl, max_leaves,
                                                              s->ctl + 1);
  }
  SCK(cudaGetLastError(), "search kernel launch");
  return GPUAI_OK;
}

}  // namespace

extern "C" {

int gpuai_searches_create(int device, uint32_t max_searches, uint32_t pool_nodes, uint32_t max_leaves_per_step,
                          uint32_t playouts_per_leaf, int32_t policy, uint64_t seed, gpuai_searches **out) {
  if (!out) return err(GPUAI_ERR_INVALID, "gpuai_searches_create: out is NULL");
  *out = nullptr;
  if (max_searches == 0 || pool_nodes == 0 || max_leaves_per_step == 0 || playouts_per_leaf == 0)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_create: zero size");
  if (policy < 0 || policy > 2) return err(GPUAI_ERR_INVALID, "gpuai_searches_create: unknown policy");
  if (max_leaves_per_step > kMaxLeavesPerStep)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_create: max_leaves_per_step above 512");
  if ((uint64_t)max_searches * max_leaves_per_step * playouts_per_leaf > 0x7fffffffull || pool_nodes > 0x7fffffffu)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_create: sizes exceed 2^31");
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count)
    return err(GPUAI_ERR_NO_DEVICE, "gpuai_searches_create: no such CUDA device");
  gpuai_searches *s = new gpuai_searches;
  s->device = device;
  s->slots = max_searches;
  s->pool_nodes = pool_nodes;
  s->qmax = max_leaves_per_step;
  s->ppl = playouts_per_leaf;
  s->policy = policy;
  s->seed = seed;
  s->pool.nodes = pool_nodes;
  s->lrn.max_leaves = max_leaves_per_step;
  auto fail = [&](int rc) {
    gpuai_searches_destroy(s);
    return rc;
  };
  if (cudaSetDevice(device) != cudaSuccess) return fail(err(GPUAI_ERR_CUDA, "cudaSetDevice failed"));
  cudaError_t e = cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) e = playout_occupancy(policy, kPlayoutBlock, &s->blocks_per_sm);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
  const size_t P = pool_nodes, S = max_searches, L = (size_t)max_searches * max_leaves_per_step;
  if (e == cudaSuccess) e = dalloc(s, &s->pool.info, P);
  if (e == cudaSuccess) e = dalloc(s, &s->pool.board, P);
  if (e == cudaSuccess) e = dalloc(s, &s->pool.parent, P);
  if (e == cudaSuccess) e = dalloc(s, &s->pool.move, P);
  if (e == cudaSuccess) e = dalloc(s, &s->pool.removed, P);
  if (e == cudaSuccess) e = dalloc(s, &s->tab.root, S);
  if (e == cudaSuccess) e = dalloc(s, &s->tab.node_next, S);
  if (e == cudaSuccess) e = dalloc(s, &s->tab.node_end, S);
  if (e == cudaSuccess) e = dalloc(s, &s->tab.stream_next, S);
  if (e == cudaSuccess) e = dalloc(s, &s->tab.budget, S);
  if (e == cudaSuccess) e = dalloc(s, &s->tab.done, S);
  if (e == cudaSuccess) e = dalloc(s, &s->tab.quota_off, S + 1);
  if (e == cudaSuccess) e = dalloc(s, &s->leaves.board, L);
  if (e == cudaSuccess) e = dalloc(s, &s->leaves.node, L);
  if (e == cudaSuccess) e = dalloc(s, &s->leaves.search, L);
  if (e == cudaSuccess) e = dalloc(s, &s->leaves.stream, L);
  if (e == cudaSuccess) e = dalloc(s, &s->leaves.out, L * playouts_per_leaf);
  if (e == cudaSuccess) e = dalloc(s, &s->leaves.sizes, 2);
  if (e == cudaSuccess) e = dalloc(s, &s->ctl, 4);
  if (e == cudaSuccess)
    e = cudaHostAlloc(reinterpret_cast<void **>(&s->report), sizeof(RootReport), cudaHostAllocMapped);
  if (e == cudaSuccess) e = cudaMemsetAsync(s->tab.root, 0xff, S * sizeof(int32_t), s->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(s->leaves.sizes, 0, 2 * sizeof(uint32_t), s->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(s->ctl, 0, 4 * sizeof(uint32_t), s->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  if (e != cudaSuccess) return fail(cuda_err(e, "gpuai_searches_create"));
  s->free_ranges[0] = pool_nodes;
  s->start.assign(S, -1);
  s->cap.assign(S, 0);
  *out = s;
  return GPUAI_OK;
}

void gpuai_searches_destroy(gpuai_searches *s) {
  if (!s) return;
  cudaSetDevice(s->device);
  if (s->stream) cudaStreamSynchronize(s->stream);
  if (s->side) cudaStreamSynchronize(s->side);
  if (s->graph) cudaGraphExecDestroy(s->graph);
  for (void *p : s->allocations) cudaFree(p);
  if (s->report) cudaFreeHost(s->report);
  if (s->fork) cudaEventDestroy(s->fork);
  if (s->join) cudaEventDestroy(s->join);
  if (s->side) cudaStreamDestroy(s->side);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
}

int gpuai_searches_add(gpuai_searches *s, const gpuai_board *root, uint64_t playout_budget, uint32_t node_capacity,
                       uint64_t stream_base, int32_t *slot) {
  if (!s || !root || !slot) return err(GPUAI_ERR_INVALID, "gpuai_searches_add: NULL argument");
  if (node_capacity < 1) return err(GPUAI_ERR_INVALID, "gpuai_searches_add: node_capacity must be >= 1");
  if ((root->p1 & root->p2) || (root->kings & ~(root->p1 | root->p2)) || (root->meta & ~0xff01u))
    return err(GPUAI_ERR_INVALID, "gpuai_searches_add: malformed board");
  std::lock_guard<std::mutex> lock(s->mu);
  int32_t free_slot = -1;
  for (uint32_t i = 0; i < s->slots; i++)
    if (s->start[i] < 0) {
      free_slot = (int32_t)i;
      break;
    }
  if (free_slot < 0) return err(GPUAI_ERR_OOM, "gpuai_searches_add: admission refused: all search slots busy");
  auto it = s->free_ranges.begin();
  for (; it != s->free_ranges.end(); ++it)
    if (it->second >= node_capacity) break;
  if (it == s->free_ranges.end())
    return err(GPUAI_ERR_OOM, "gpuai_searches_add: admission refused: no free node range of that size");
  const uint32_t start = it->first, len = it->second;
  s->free_ranges.erase(it);
  if (len > node_capacity) s->free_ranges[start + node_capacity] = len - node_capacity;
  s->start[free_slot] = (int32_t)start;
  s->cap[free_slot] = (int32_t)node_capacity;
  SCK(cudaSetDevice(s->device), "cudaSetDevice");
  init_search_kernel<<<1, 1, 0, s->stream>>>(s->pool, s->tab, free_slot, (int32_t)start, (int32_t)node_capacity,
                                              make_uint4(root->p1, root->p2, root->kings, root->meta),
                                              playout_budget, stream_base);
  SCK(cudaGetLastError(), "init_search_kernel");
  *slot = free_slot;
  return GPUAI_OK;
}

int gpuai_searches_remove(gpuai_searches *s, int32_t slot) {
  if (!s) return err(GPUAI_ERR_INVALID, "gpuai_searches_remove: NULL");
  std::lock_guard<std::mutex> lock(s->mu);
  if (slot < 0 || (uint32_t)slot >= s->slots || s->start[slot] < 0)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_remove: no such search");
  SCK(cudaSetDevice(s->device), "cudaSetDevice");
  remove_search_kernel<<<1, 1, 0, s->stream>>>(s->tab, slot);
  SCK(cudaGetLastError(), "remove_search_kernel");
  // return the node range, merging with free neighbours
  uint32_t start = (uint32_t)s->start[slot], len = (uint32_t)s->cap[slot];
  auto next = s->free_ranges.lower_bound(start);
  if (next != s->free_ranges.end() && next->first == start + len) {
    len += next->second;
    next = s->free_ranges.erase(next);
  }
  if (next != s->free_ranges.begin()) {
    auto prev = std::prev(next);
    if (prev->first + prev->second == start) {
      start = prev->first;
      len += prev->second;
      s->free_ranges.erase(prev);
    }
  }
  s->free_ranges[start] = len;
  s->start[slot] = -1;
  s->cap[slot] = 0;
  return GPUAI_OK;
}

int gpuai_searches_step(gpuai_searches *s, uint32_t steps, uint32_t leaves_per_search, int32_t use_graph) {
  GPUAI_RANGE("gpuai_searches_step");
  if (!s) return err(GPUAI_ERR_INVALID, "gpuai_searches_step: NULL");
  if (leaves_per_search == 0 || leaves_per_search > s->qmax)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_step: leaves_per_search outside 1..max_leaves_per_step");
  std::lock_guard<std::mutex> lock(s->mu);
  SCK(cudaSetDevice(s->device), "cudaSetDevice");
  if (!use_graph) {
    for (uint32_t k = 0; k < steps; k++) {
      const int rc = enqueue_step(s, leaves_per_search);
      if (rc) return rc;
    }
    return GPUAI_OK;
  }
  if (!s->graph || s->graph_q != leaves_per_search) {
    if (s->graph) cudaGraphExecDestroy(s->graph);
    s->graph = nullptr;
    cudaGraph_t g = nullptr;
    SCK(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal), "begin capture");
    const int rc = enqueue_step(s, leaves_per_search);
    const cudaError_t e = cudaStreamEndCapture(s->stream, &g);
    if (rc) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    SCK(e, "end capture");
    const cudaError_t ei = cudaGraphInstantiate(&s->graph, g, 0);
    cudaGraphDestroy(g);
    SCK(ei, "graph instantiate");
    s->graph_q = leaves_per_search;
  }
  for (uint32_t k = 0; k < steps; k++) SCK(cudaGraphLaunch(s->graph, s->stream), "graph launch");
  return GPUAI_OK;
}

int gpuai_searches_poll(gpuai_searches *s, uint64_t *done, uint64_t *budget, uint32_t n, uint32_t *status) {
  GPUAI_RANGE("gpuai_searches_poll");
  if (!s || !done || !budget) return err(GPUAI_ERR_INVALID, "gpuai_searches_poll: NULL");
  if (n > s->slots) return err(GPUAI_ERR_INVALID, "gpuai_searches_poll: n exceeds max_searches");
  std::lock_guard<std::mutex> lock(s->mu);
  SCK(cudaSetDevice(s->device), "cudaSetDevice");
  uint32_t st = 0;
  SCK(cudaMemcpyAsync(done, s->tab.done, n * sizeof(uint64_t), cudaMemcpyDeviceToHost, s->stream), "poll");
  SCK(cudaMemcpyAsync(budget, s->tab.budget, n * sizeof(uint64_t), cudaMemcpyDeviceToHost, s->stream), "poll");
  SCK(cudaMemcpyAsync(&st, s->ctl + 1, sizeof st, cudaMemcpyDeviceToHost, s->stream), "poll");
  SCK(cudaStreamSynchronize(s->stream), "search steps");
  if (st) SCK(cudaMemsetAsync(s->ctl + 1, 0, sizeof(uint32_t), s->stream), "clear status");  // reported once
  for (uint32_t i = 0; i < n; i++)
    if (s->start[i] < 0) done[i] = budget[i] = 0;
  if (status) *status = st;
  if (st) return err(GPUAI_ERR_LIMIT, "gpuai_searches_poll: a kernel reported a limit");
  return GPUAI_OK;
}

int gpuai_searches_set_net(gpuai_searches *s, gpuai_net *net, float value_weight, float c_puct) {
  if (!s) return err(GPUAI_ERR_INVALID, "gpuai_searches_set_net: NULL");
  if (!(value_weight >= 0.0f && value_weight <= 1.0f) || !(c_puct > 0.0f && c_puct < 1.0e6f))
    return err(GPUAI_ERR_INVALID, "gpuai_searches_set_net: value_weight must be in [0, 1] and c_puct > 0");
  std::lock_guard<std::mutex> lock(s->mu);
  for (uint32_t i = 0; i < s->slots; i++)
    if (s->start[i] >= 0) return err(GPUAI_ERR_INVALID, "gpuai_searches_set_net: searches are admitted");
  if (net && ga::net::device_of(net) != s->device)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_set_net: network and searches are on different devices");
  SCK(cudaSetDevice(s->device), "cudaSetDevice");
  if (net && !s->pool.prior) {
    const size_t L = (size_t)s->slots * s->qmax;
    SCK(cudaStreamCreateWithFlags(&s->side, cudaStreamNonBlocking), "network stream");
    SCK(cudaEventCreateWithFlags(&s->fork, cudaEventDisableTiming), "event");
    SCK(cudaEventCreateWithFlags(&s->join, cudaEventDisableTiming), "event");
    SCK(dalloc(s, &s->pool.prior, (size_t)s->pool_nodes * kPriors), "prior pool");
    SCK(dalloc(s, &s->leaves.value, L), "leaf values");
    SCK(ga::net::fwd_alloc(s->fw, (uint32_t)L, s->allocations, true), "network workspace");
  }
  s->net = net;
  s->lrn.c_puct = c_puct;
  s->lrn.value_weight = value_weight;
  if (s->graph) cudaGraphExecDestroy(s->graph);  // the step's launches change
  s->graph = nullptr;
  return GPUAI_OK;
}

int gpuai_searches_set_proposal(gpuai_searches *s, uint32_t guided_plies, float temperature) {
  if (!s) return err(GPUAI_ERR_INVALID, "gpuai_searches_set_proposal: NULL");
  if (guided_plies > ga::net::kMaxGuidedPlies)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_set_proposal: guided_plies above 32");
  if (!(temperature > 0.0f && temperature < 1.0e6f))
    return err(GPUAI_ERR_INVALID, "gpuai_searches_set_proposal: temperature must be positive");
  std::lock_guard<std::mutex> lock(s->mu);
  if (guided_plies > 0 && !s->net)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_set_proposal: attach a network first (gpuai_searches_set_net)");
  for (uint32_t i = 0; i < s->slots; i++)
    if (s->start[i] >= 0) return err(GPUAI_ERR_INVALID, "gpuai_searches_set_proposal: searches are admitted");
  SCK(cudaSetDevice(s->device), "cudaSetDevice");
  const size_t P = (size_t)s->slots * s->qmax * s->ppl;
  if (guided_plies > 0 && !s->pcur) {
    SCK(dalloc(s, &s->pcur, P), "proposal boards");
    SCK(dalloc(s, &s->pstream, P), "proposal streams");
    SCK(dalloc(s, &s->psizes, 2), "proposal sizes");
  }
  if (guided_plies > 1 && !s->pfw.rows) SCK(ga::net::fwd_alloc(s->pfw, (uint32_t)P, s->allocations, true), "network workspace");
  s->guided = guided_plies;
  s->inv_temperature = 1.0f / temperature;
  if (s->graph) cudaGraphExecDestroy(s->graph);  // the step's launches change
  s->graph = nullptr;
  return GPUAI_OK;
}

int gpuai_searches_children(gpuai_searches *s, int32_t slot, gpuai_move *moves, uint32_t *visits,
                            uint32_t *score2, uint32_t max_children, uint32_t *nchildren, uint32_t *nodes_used) {
  if (!s || !nchildren) return err(GPUAI_ERR_INVALID, "gpuai_searches_children: NULL");
  std::lock_guard<std::mutex> lock(s->mu);
  if (slot < 0 || (uint32_t)slot >= s->slots || s->start[slot] < 0)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_children: no such search");
  SCK(cudaSetDevice(s->device), "cudaSetDevice");
  root_report_kernel<<<1, kMaxChildren, 0, s->stream>>>(s->pool, s->tab, slot, s->start[slot], s->report);
  SCK(cudaGetLastError(), "children");
  SCK(cudaStreamSynchronize(s->stream), "children");
  const RootReport &rep = *s->report;
  if (nodes_used) *nodes_used = (uint32_t)rep.nodes_used;
  const int32_t k = ((rep.info.y >> 16) & kExpanded) ? (int32_t)(rep.info.y & 0xffffu) : 0;
  *nchildren = (uint32_t)k;
  if (k <= 0) return GPUAI_OK;
  // full move records from the root's move list (same order as the children)
  gpuai::State root_state;
  root_state.b = gpuai_board{rep.board.x, rep.board.y, rep.board.z, rep.board.w};
  const std::vector<gpuai::Move> all = moves ? root_state.getMoves() : std::vector<gpuai::Move>();
  for (uint32_t i = 0; i < (uint32_t)k && i < max_children; i++) {
    if (visits) visits[i] = rep.child[i].x;
    if (score2) score2[i] = rep.child[i].y;
    if (moves && i < all.size()) moves[i] = all[i].m;
  }
  return GPUAI_OK;
}

int gpuai_searches_nodes(gpuai_searches *s, int32_t slot, uint32_t max_nodes, uint32_t *info, gpuai_board *boards,
                         int32_t *parent, uint16_t *priors, uint32_t *nnodes) {
  if (!s || !nnodes) return err(GPUAI_ERR_INVALID, "gpuai_searches_nodes: NULL");
  std::lock_guard<std::mutex> lock(s->mu);
  if (slot < 0 || (uint32_t)slot >= s->slots || s->start[slot] < 0)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_nodes: no such search");
  if (priors && !s->pool.prior) return err(GPUAI_ERR_INVALID, "gpuai_searches_nodes: the searches keep no priors");
  SCK(cudaSetDevice(s->device), "cudaSetDevice");
  const int32_t r = s->start[slot];
  int32_t next = 0;
  SCK(cudaMemcpyAsync(&next, s->tab.node_next + slot, 4, cudaMemcpyDeviceToHost, s->stream), "nodes");
  SCK(cudaStreamSynchronize(s->stream), "nodes");
  const uint32_t used = (uint32_t)(next - r);
  *nnodes = used;
  const uint32_t n = used < max_nodes ? used : max_nodes;
  if (n == 0) return GPUAI_OK;
  std::vector<uint4> inf(n);
  std::vector<int32_t> par(n);
  SCK(cudaMemcpyAsync(inf.data(), s->pool.info + r, 16 * (size_t)n, cudaMemcpyDeviceToHost, s->stream), "nodes");
  SCK(cudaMemcpyAsync(par.data(), s->pool.parent + r, 4 * (size_t)n, cudaMemcpyDeviceToHost, s->stream), "nodes");
  if (boards)
    SCK(cudaMemcpyAsync(boards, s->pool.board + r, 16 * (size_t)n, cudaMemcpyDeviceToHost, s->stream), "nodes");
  if (priors)
    SCK(cudaMemcpyAsync(priors, s->pool.prior + (size_t)r * kPriors, 2 * kPriors * (size_t)n,
                        cudaMemcpyDeviceToHost, s->stream),
        "nodes");
  SCK(cudaStreamSynchronize(s->stream), "nodes");
  for (uint32_t i = 0; i < n; i++) {
    if (info) {
      info[4 * i] = inf[i].x == 0xffffffffu ? 0xffffffffu : inf[i].x - (uint32_t)r;
      info[4 * i + 1] = inf[i].y;
      info[4 * i + 2] = inf[i].z;
      info[4 * i + 3] = inf[i].w;
    }
    if (parent) parent[i] = par[i] < 0 ? -1 : par[i] - r;
    // a node that was not evaluated has no priors (the range may have been another search's)
    if (priors && !((inf[i].y >> 16) & kEvaluated)) std::memset(priors + (size_t)i * kPriors, 0, 2 * kPriors);
  }
  return GPUAI_OK;
}

int gpuai_searches_leaves(gpuai_searches *s, uint32_t max_leaves, uint32_t *nleaves, int32_t *search, int32_t *node,
                          gpuai_board *boards, uint64_t *streams, int8_t *outcomes, float *net_value,
                          uint16_t *net_logits) {
  if (!s || !nleaves) return err(GPUAI_ERR_INVALID, "gpuai_searches_leaves: NULL");
  std::lock_guard<std::mutex> lock(s->mu);
  if ((net_value || net_logits) && !s->net)
    return err(GPUAI_ERR_INVALID, "gpuai_searches_leaves: no network is attached");
  SCK(cudaSetDevice(s->device), "cudaSetDevice");
  uint32_t sizes[2] = {0, 0};
  SCK(cudaMemcpyAsync(sizes, s->leaves.sizes, 8, cudaMemcpyDeviceToHost, s->stream), "leaves");
  SCK(cudaStreamSynchronize(s->stream), "leaves");
  *nleaves = sizes[0];
  const uint32_t n = sizes[0] < max_leaves ? sizes[0] : max_leaves;
  if (n == 0) return GPUAI_OK;
  std::vector<int32_t> srch(n), nd(n);
  SCK(cudaMemcpyAsync(srch.data(), s->leaves.search, 4 * (size_t)n, cudaMemcpyDeviceToHost, s->stream), "leaves");
  SCK(cudaMemcpyAsync(nd.data(), s->leaves.node, 4 * (size_t)n, cudaMemcpyDeviceToHost, s->stream), "leaves");
  if (boards)
    SCK(cudaMemcpyAsync(boards, s->leaves.board, 16 * (size_t)n, cudaMemcpyDeviceToHost, s->stream), "leaves");
  if (streams)
    SCK(cudaMemcpyAsync(streams, s->leaves.stream, 8 * (size_t)n, cudaMemcpyDeviceToHost, s->stream), "leaves");
  if (outcomes)
    SCK(cudaMemcpyAsync(outcomes, s->leaves.out, (size_t)n * s->ppl, cudaMemcpyDeviceToHost, s->stream), "leaves");
  if (net_value)
    SCK(cudaMemcpyAsync(net_value, s->fw.vraw, 4 * (size_t)n, cudaMemcpyDeviceToHost, s->stream), "leaves");
  if (net_logits)
    SCK(cudaMemcpyAsync(net_logits, s->fw.logits_b, 2 * (size_t)n * ga::net::kOut, cudaMemcpyDeviceToHost,
                        s->stream),
        "leaves");
  SCK(cudaStreamSynchronize(s->stream), "leaves");
  for (uint32_t i = 0; i < n; i++) {
    if (search) search[i] = srch[i];
    const int32_t st = (srch[i] >= 0 && (uint32_t)srch[i] < s->slots) ? s->start[srch[i]] : -1;
    if (node) node[i] = st < 0 ? -1 : nd[i] - st;
  }
  return GPUAI_OK;
}

}  // extern "C"
