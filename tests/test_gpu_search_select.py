"""The block-per-search selection at the sizes where it can go wrong, node for
node against the CPU restatement: steps on either side of each block width,
node ranges that run out in the first, a middle and the last round of a
frontier, and roots whose nodes have more children than a group of lanes holds
at once (8), than two do (16), or one child (a forced line)."""
import numpy as np
import pytest

import oracle_lib as L
from golden_boards import random_boards
from oracle import search as S
from test_gpu_search_oracle import _compare_step, _compare_trees, _peaky_params, _replay, _run

pytestmark = pytest.mark.gpu


def _roots(lo, hi, n, seed):
    """n live positions with lo..hi legal moves (many kings: long lists)."""
    pos = random_boards(np.random.default_rng(seed), 60000)
    pos[:, 3] &= np.uint32(1)
    _, counts = L.genmoves(pos)
    pos = pos[(counts >= lo) & (counts <= hi)]
    assert len(pos) >= n
    return list(pos[:n])


def _king_roots(lo, hi, n, seed):
    """n positions of twelve kings against one with lo..hi moves, more than random boards have."""
    rng = np.random.default_rng(seed)
    pos = np.zeros((40000, 4), np.uint32)
    for b in pos:
        at = rng.permutation(32)[:13]
        b[0] = sum(1 << int(i) for i in at[:12])
        b[1] = 1 << int(at[12])
        b[2] = b[0] | b[1]
    _, counts = L.genmoves(pos)
    pos = pos[(counts >= lo) & (counts <= hi)]
    assert len(pos) >= n
    return list(pos[:n])


@pytest.mark.parametrize("q", [1, 31, 33, 127, 129, 200, 257, 300, 511])
def test_every_block_width_and_a_range_that_runs_out(q):
    roots = list(L.random_positions(300 + q, 4, 0, 40))
    steps = 4 + 1200 // q if q < 32 else 12
    _run(policy=0, ppl=1, q=q, budgets=[6000] * 4, caps=[12000, 60 + q // 2, 200 + 2 * q, 9 + q], roots=roots,
         graph=q % 2 == 0, steps=steps)


@pytest.mark.parametrize("lo,hi", [(1, 1), (9, 12), (17, 40)])
def test_nodes_with_few_and_many_children(lo, hi):
    roots = _roots(lo, hi, 4, lo)
    _run(policy=0, ppl=2, q=100, budgets=[3000] * 4, caps=[20000] * 4, roots=roots, graph=True, steps=14)


@pytest.mark.parametrize("lo,hi,q", [(2, 8, 43), (9, 16, 43), (17, 32, 43), (33, 45, 43), (9, 16, 15)])
def test_learned_splits_by_number_of_children(lo, hi, q):
    """The slots of a learned node are handed out in fours, with the terms of up
    to 8, up to 16, up to 32 and more children laid out differently; 43 leaves
    leave a remainder and a partly filled warp, 15 take the narrower block."""
    from gpu_ai_gb300 import Net, Searches
    net = Net(0, max_batch=256, seed=1)
    net.set_params(_peaky_params(5))
    gpu = Searches(3, 60000, q, playouts_per_leaf=1, policy=0, seed=3)
    gpu.set_net(net, value_weight=0.5, c_puct=1.5)
    learned = {"value_weight": 0.5, "c_puct": 1.5}
    o = S.SearchesOracle(3, 1, 0, 3, children=L.children, playouts=_replay, learned=learned)
    slots = []
    for i, r in enumerate(_roots(lo, hi, 3, lo) if lo <= 32 else _king_roots(lo, hi, 3, lo)):
        slots.append(gpu.add(r, 400, 15000, (i + 7) << 36))
        assert o.add(r, 400, 15000, (i + 7) << 36) == slots[-1]
    for step in range(10):
        gpu.step(1, q, True)
        gpu.poll()
        lv = gpu.leaves(net=True)
        o.step(q, net_value=lv["net_value"], net_logits=lv["net_logits"])
        _compare_step(gpu, o, step, net=True)
        _compare_trees(gpu, o, slots, step, priors=True)
    gpu.close()
    net.close()
