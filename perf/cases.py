"""The calls whose speed this repository keeps an eye on, with their sizes.

Each case is a dict of plain values; `prepare` makes from it what a program
has in hand before the call (boards, an engine, a network, a search pool),
`run` is one pass through the public entry points, `work` what a pass cannot do
without, and `exact` the computed numbers in 64 bits.  `listed` are the sizes
that the repository's own configurations, tests and benchmark use (or generic
ones near them); `draw` gives more of the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gpu_ai_gb300 import POLICY_EPS_GREEDY, POLICY_RANDOM, POLICY_REF_HEURISTIC, Engine, Net, Searches

MAX_CHILDREN = 64
PLIES = {POLICY_RANDOM: 52.0, POLICY_REF_HEURISTIC: 70.0, POLICY_EPS_GREEDY: 50.0}  # a game's length, roughly
OPS_PER_PLY = 260  # integer operations of one bitboard ply
FORWARD_FLOPS = 2 * (192 * 256 + 256 * 256 + 256 * 1024)
TRAIN_FLOPS = 3 * FORWARD_FLOPS - 2 * 192 * 256


def listed():
    return [
        # the smallest call: one position's value from a few hundred playouts, host buffers (a player's quick look)
        {"name": "one position", "kind": "playouts", "policy": POLICY_RANDOM, "npos": 1, "reps": 256, "ragged": False,
         "host": True},
        # the repository's benchmark batch, device buffers
        {"name": "benchmark batch", "kind": "playouts", "policy": POLICY_RANDOM, "npos": 64, "reps": 4096,
         "ragged": False, "host": False},
        # many positions with uneven repetitions (a tree's leaves by their slots), device buffers, several waves
        {"name": "uneven repetitions", "kind": "playouts", "policy": POLICY_RANDOM, "npos": 20011, "reps": 200,
         "ragged": True, "host": False},
        # the reference's heuristic playouts on the benchmark batch
        {"name": "reference heuristic", "kind": "playouts", "policy": POLICY_REF_HEURISTIC, "npos": 64, "reps": 4096,
         "ragged": False, "host": False},
        # a host tree's leaf batch with the eps-greedy playout policy: 16K leaves, 4 playouts each, host buffers
        {"name": "leaf batch", "kind": "playouts", "policy": POLICY_EPS_GREEDY, "npos": 16384, "reps": 4,
         "ragged": False, "host": True},
        # training labels: each position's legal moves valued by playouts
        {"name": "labels", "kind": "labels", "n": 16384, "playouts": 1024},
        # self-play positions for training, eps-greedy games cut after 0..90 plies
        {"name": "self-play", "kind": "selfplay", "policy": POLICY_EPS_GREEDY, "n": 500000, "max_plies": 90},
        # move lists of a set of games (which are over, which moves there are), host buffers
        {"name": "move lists", "kind": "genmoves", "n": 3001, "max_moves": 64},
        # a move's worth of searches as the server runs them: wide steps, plain playouts; then every search's move
        # and its root's statistics, and one search's tree
        {"name": "searches", "kind": "search", "n": 64, "leaves": 512, "ppl": 8, "steps": 32, "learned": False,
         "policy": POLICY_RANDOM, "guided": 0},
        # a match's learned searches: network priors and leaf values, narrow steps
        {"name": "learned searches", "kind": "search", "n": 200, "leaves": 64, "ppl": 2, "steps": 48, "learned": True,
         "policy": POLICY_RANDOM, "guided": 0},
        # training steps on consecutive minibatches, then the weights
        {"name": "training", "kind": "train", "batch": 8192, "steps": 8},
        # the network's values and move logits of a set of positions, host buffers
        {"name": "forward", "kind": "forward", "n": 1000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["playouts", "playouts", "playouts", "playouts", "labels", "selfplay", "genmoves", "search",
                       "search", "train", "forward"])
    if kind == "playouts":
        policy = rng.choice([POLICY_RANDOM, POLICY_RANDOM, POLICY_REF_HEURISTIC, POLICY_EPS_GREEDY])
        total = _log_int(rng, 64, {POLICY_RANDOM: 1 << 22, POLICY_REF_HEURISTIC: 1 << 19, POLICY_EPS_GREEDY: 1 << 20}[policy])
        npos = _log_int(rng, 1, min(total, 100000))
        reps = max(1, total // npos)
        return {"kind": kind, "policy": policy, "npos": npos, "reps": reps, "ragged": reps > 1 and rng.random() < 0.4,
                "host": npos * reps <= (1 << 20) and rng.random() < 0.5}
    if kind == "labels":
        playouts = _log_int(rng, 33, 4096)
        return {"kind": kind, "n": _log_int(rng, 16, (1 << 24) // playouts), "playouts": playouts}
    if kind == "selfplay":
        return {"kind": kind, "policy": rng.choice([POLICY_RANDOM, POLICY_EPS_GREEDY]), "n": _log_int(rng, 1000, 500000),
                "max_plies": rng.randint(20, 90)}
    if kind == "genmoves":
        return {"kind": kind, "n": _log_int(rng, 1, 20000), "max_moves": rng.choice([48, 64])}
    if kind == "search":
        learned = rng.random() < 0.5
        leaves = rng.choice([32, 64, 100]) if learned else _log_int(rng, 16, 512)
        return {"kind": kind, "n": _log_int(rng, 1, 200 if leaves <= 100 else 64), "leaves": leaves,
                "ppl": rng.choice([1, 2, 4]) if learned else rng.choice([1, 4, 8]), "steps": rng.randint(8, 32),
                "learned": learned, "policy": POLICY_RANDOM if learned or rng.random() < 0.7 else POLICY_REF_HEURISTIC,
                "guided": rng.choice([0, 0, 2]) if learned else 0}
    if kind == "train":
        return {"kind": kind, "batch": _log_int(rng, 128, 32768), "steps": 2}
    return {"kind": kind, "n": _log_int(rng, 1, 8192)}


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    eng = Engine(0)
    rng = np.random.default_rng(seed)
    s = {"case": case, "eng": eng, "seed": seed}
    if kind == "playouts":
        pos = eng.random_positions(seed, case["npos"], 0, 30 if case["npos"] <= 64 else 60)
        reps = np.full(case["npos"], case["reps"], np.uint32)
        if case["ragged"]:  # a few positions get most of the playouts, some get none
            w = rng.lognormal(0.0, 1.2, case["npos"])
            reps = np.floor(w / w.sum() * case["npos"] * case["reps"]).astype(np.uint32)
            reps[int(np.argmax(reps))] += np.uint32(case["npos"] * case["reps"] - int(reps.sum(dtype=np.uint64)))
        total = int(reps.sum(dtype=np.uint64))
        s["total"] = total
        if case["host"]:
            s.update(pos=pos, reps=reps, out=np.empty(total, np.int8))
        else:
            off = None
            if case["ragged"]:
                off = _device(np.concatenate([[0], np.cumsum(reps, dtype=np.uint64)]).astype(np.uint32))
            s.update(pos=_device(pos), off=off, out=torch.empty(total, dtype=torch.int8, device="cuda"))
    elif kind == "labels":
        n = case["n"]
        s.update(pos=_positions_on_device(eng, seed, n, 90), value=torch.empty(n, device="cuda"),
                 q=torch.empty(n, 32, device="cuda"), k=torch.empty(n, dtype=torch.uint8, device="cuda"))
    elif kind == "selfplay":
        s.update(boards=torch.empty(case["n"], 4, dtype=torch.int32, device="cuda"))
    elif kind == "genmoves":
        s.update(pos=eng.random_positions(seed, case["n"], 0, 90))
    elif kind == "search":
        cap = 4 + case["leaves"] * case["steps"] * 12
        s["cap"] = cap
        s["roots"] = eng.random_positions(seed, case["n"], 0, 60)
        s["searches"] = Searches(case["n"], case["n"] * cap, case["leaves"], case["ppl"], case["policy"], seed=seed)
        if case["learned"]:
            s["searches"].set_net(Net(0, max_batch=256, seed=seed), 0.5, 1.5)
            if case["guided"]:
                s["searches"].set_proposal(case["guided"], 0.5)
    elif kind == "train":
        n = case["batch"] * case["steps"]
        pos = _positions_on_device(eng, seed, n, 60)
        value, q = torch.empty(n, device="cuda"), torch.empty(n, 32, device="cuda")
        k = torch.empty(n, dtype=torch.uint8, device="cuda")
        eng.label_positions(pos.data_ptr(), n, 64, seed, 0, POLICY_RANDOM, value.data_ptr(), q.data_ptr(), k.data_ptr(),
                            torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        s.update(pos=pos, value=value, q=q, net=Net(0, max_batch=case["batch"], seed=seed))
    else:
        s.update(pos=eng.random_positions(seed, case["n"], 0, 60), net=Net(0, max_batch=8192, seed=seed))
    return s


def _positions_on_device(eng, seed, n, max_plies):
    boards = torch.empty(n, 4, dtype=torch.int32, device="cuda")
    eng.selfplay_positions(seed, n, 0, max_plies, POLICY_RANDOM, boards.data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
    return boards


def run(s):
    case, eng, seed = s["case"], s["eng"], s["seed"]
    kind = case["kind"]
    if kind == "playouts":
        if case["host"]:
            return eng.playouts(s["pos"], s["reps"], seed=seed, stream_base=7, policy=case["policy"], out=s["out"])
        off = s["off"]
        eng.playouts_device(s["pos"].data_ptr(), None if off is None else off.data_ptr(), case["npos"],
                            case["reps"] if off is None else 0, s["total"], seed, 7, case["policy"],
                            s["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return s["out"]
    if kind == "labels":
        eng.label_positions(s["pos"].data_ptr(), case["n"], case["playouts"], seed, 0, POLICY_RANDOM,
                            s["value"].data_ptr(), s["q"].data_ptr(), s["k"].data_ptr(),
                            torch.cuda.current_stream().cuda_stream)
        return {"value": s["value"], "move values": s["q"], "moves": s["k"]}
    if kind == "selfplay":
        eng.selfplay_positions(seed, case["n"], 0, case["max_plies"], case["policy"], s["boards"].data_ptr(),
                               torch.cuda.current_stream().cuda_stream)
        return s["boards"]
    if kind == "genmoves":
        moves, counts = eng.genmoves(s["pos"], case["max_moves"])
        return {"moves": moves, "counts": counts}
    if kind == "search":
        pool, n = s["searches"], case["n"]
        slots = [pool.add(r, 1 << 40, s["cap"], i << 40) for i, r in enumerate(s["roots"])]
        pool.step(case["steps"], case["leaves"])
        done, _ = pool.poll()
        visits = np.zeros((n, MAX_CHILDREN), np.int64)
        score2 = np.zeros((n, MAX_CHILDREN), np.int64)
        moves = np.zeros((n, 32), np.uint8)
        for i, slot in enumerate(slots):
            move, c = pool.best(slot)
            visits[i, :len(c["visits"])] = c["visits"]
            score2[i, :len(c["score2"])] = c["score2"]
            if move is not None:
                moves[i] = move
        info = pool.nodes(slots[0])["info"]
        tree = np.zeros((s["cap"], 4), np.int32)  # trees of other roots have other sizes
        tree[:len(info)] = info.view(np.int32)
        for slot in slots:
            pool.remove(slot)
        return {"playouts": done.astype(np.int64), "visits": visits, "score2": score2, "moves": moves, "tree": tree}
    if kind == "train":
        net, b = s["net"], case["batch"]
        for k in range(case["steps"]):
            net.train_step(s["pos"].data_ptr() + 16 * b * k, s["value"].data_ptr() + 4 * b * k,
                           s["q"].data_ptr() + 128 * b * k, b, 1e-3)
        return net.params()
    value, logits = s["net"].forward(s["pos"])
    return {"value": value, "logits": logits}


def work(case):
    kind = case["kind"]
    if kind == "playouts":
        total = case["npos"] * case["reps"]
        return {"bytes": 16 * case["npos"] + total, "flops": total * PLIES[case["policy"]] * OPS_PER_PLY}
    if kind == "labels":
        return {"bytes": case["n"] * (16 + 128 + 4 + 1), "flops": case["n"] * case["playouts"] * 35.0 * OPS_PER_PLY}
    if kind == "selfplay":
        return {"bytes": 16 * case["n"], "flops": case["n"] * 0.45 * case["max_plies"] * OPS_PER_PLY}
    if kind == "genmoves":
        return {"bytes": case["n"] * (16 + 1 + 32 * case["max_moves"]), "flops": case["n"] * OPS_PER_PLY}
    if kind == "search":
        leaves = case["n"] * case["leaves"] * case["steps"]
        flops = leaves * case["ppl"] * PLIES[case["policy"]] * OPS_PER_PLY
        if case["learned"]:
            flops += leaves * FORWARD_FLOPS * (1 + max(0, case["guided"] - 1) * case["ppl"])
        return {"bytes": leaves * (16 + case["ppl"]), "flops": flops}
    if kind == "train":
        rows = case["batch"] * case["steps"]
        return {"bytes": rows * (16 + 4 + 128) + case["steps"] * 378625 * 6 * 4, "flops": rows * TRAIN_FLOPS}
    return {"bytes": case["n"] * (16 + 4 + 4096), "flops": case["n"] * FORWARD_FLOPS}


# ---- the computed numbers in 64 bits

_SIZES = (("W1", (256, 192)), ("b1", (256,)), ("W2", (256, 256)), ("b2", (256,)), ("W3", (1024, 256)), ("b3", (1024,)),
          ("wv", (256,)), ("bv", (1,)))


def _unpack(flat):
    out, at = {}, 0
    for name, shape in _SIZES:
        n = int(np.prod(shape))
        out[name] = flat[at:at + n].reshape(shape)
        at += n
    return out


def _features(boards):
    b = boards.view(np.uint32)
    side = (b[:, 3] & 1).astype(bool)
    own, opp, kings = np.where(side, b[:, 1], b[:, 0]), np.where(side, b[:, 0], b[:, 1]), b[:, 2]
    x = np.zeros((len(b), 192))
    for i, plane in enumerate((own & ~kings, own & kings, opp & ~kings, opp & kings)):
        x[:, 32 * i:32 * i + 32] = (plane[:, None] >> np.arange(32, dtype=np.uint32)) & 1
    x[:, 128] = side
    return torch.from_numpy(x).cuda()


def _forward(p, x):
    h = torch.relu(torch.relu(x @ p["W1"].T + p["b1"]) @ p["W2"].T + p["b2"])
    return torch.tanh(h @ p["wv"] + p["bv"]), h @ p["W3"].T + p["b3"]


def _neighbours():
    """Per square, its diagonal neighbour in the four directions (+1,+1), (+1,-1), (-1,+1), (-1,-1), or -1."""
    table = []
    for s in range(32):
        r, c = s // 4, 2 * (s % 4) + (1 if (s // 4) % 2 == 0 else 0)
        row = []
        for dr, dc in ((1, 1), (1, -1), (-1, 1), (-1, -1)):
            rr, cc = r + dr, c + dc
            row.append(rr * 4 + cc // 2 if 0 <= rr < 8 and 0 <= cc < 8 else -1)
        table.append(row)
    return table


_NEXT = _neighbours()


def _pairs(board):
    """from * 32 + to of each legal move in list order: captures are forced and go on as far as they can, captured
    pieces stay on the board meanwhile, no square is landed on twice; squares ascending."""
    p1, p2, kings, meta = (int(v) for v in board)
    turn = meta & 1
    own, opp = (p2, p1) if turn else (p1, p2)
    taken = own | opp
    captures, steps = [], []

    def jumps(at, dirs, seen):
        for d in dirs:
            over = _NEXT[at][d]
            to = _NEXT[over][d] if over >= 0 and (opp >> over) & 1 else -1
            if to >= 0 and not (taken >> to) & 1 and not (seen >> to) & 1:
                yield to

    def follow(start, at, dirs, seen):
        more = False
        for to in jumps(at, dirs, seen):
            more = True
            follow(start, to, dirs, seen | (1 << to))
        if not more and seen:
            captures.append(start * 32 + at)

    for sq in range(32):
        if (own >> sq) & 1:
            king = (kings >> sq) & 1
            follow(sq, sq, (0, 1, 2, 3) if king else ((3, 2) if turn else (1, 0)), 0)
            if not captures:
                for d in (0, 1, 2, 3) if king else ((2, 3) if turn else (0, 1)):
                    to = _NEXT[sq][d]
                    if to >= 0 and not (taken >> to) & 1:
                        steps.append(sq * 32 + to)
    return captures or steps


def _exact_training(case, s):
    b, steps = case["batch"], case["steps"]
    flat = torch.from_numpy(s["net"].params()).double().cuda()
    m, v = torch.zeros_like(flat), torch.zeros_like(flat)
    boards = s["pos"].cpu().numpy()
    for k in range(steps):
        rows = boards[b * k:b * (k + 1)]
        lists = [_pairs(r) for r in rows.view(np.uint32)]
        of = np.full((b, 32), -1, np.int64)
        for i, pairs in enumerate(lists):
            if 1 <= len(pairs) <= 32:
                of[i, :len(pairs)] = pairs
        of = torch.from_numpy(of).cuda()
        x, z, q = _features(rows), s["value"][b * k:b * (k + 1)].double(), s["q"][b * k:b * (k + 1)].double()
        p = flat.clone().requires_grad_(True)
        value, logits = _forward(_unpack(p), x)
        legal = of >= 0
        some = legal.any(1)
        w = torch.softmax(torch.where(legal, q / float(np.float32(0.1)), -torch.inf)[some], 1)
        at = torch.where(legal, of, torch.zeros_like(of))[some]
        target = torch.zeros_like(logits[some]).scatter_add_(1, at, torch.where(legal[some], w, torch.zeros_like(w)))
        mask = torch.zeros_like(logits[some]).scatter_add_(1, at, legal[some].double()) > 0
        lp = torch.log_softmax(torch.where(mask, logits[some], torch.full_like(logits[some], -torch.inf)), 1)
        ce = -(target * torch.where(mask, lp, torch.zeros_like(lp))).sum()
        loss = (ce + ((value - z) ** 2).sum()) / b
        (g,) = torch.autograd.grad(loss, p)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        lr = float(np.float32(1e-3))
        flat = flat - lr * (m / (1 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
    return flat.cpu().numpy()


def exact(case, seed):
    if case["kind"] == "forward":
        s = prepare(case, seed)
        p = _unpack(torch.from_numpy(s["net"].params()).double().cuda())
        value, logits = _forward(p, _features(s["pos"]))
        return {"value": value, "logits": logits}
    if case["kind"] == "train":
        return _exact_training(case, prepare(case, seed))
    return None  # whole numbers, or means of whole numbers
