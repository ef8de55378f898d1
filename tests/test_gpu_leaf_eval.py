"""The priors of a node that is the leaf of many slots at once: every group of
lanes that evaluates it, in whichever warp and block, finds it not yet
evaluated or done, and the node's priors are the ones of a single evaluation
(the softmax over all its moves)."""
import numpy as np
import pytest

import oracle_lib as L
from oracle import search as S
from test_gpu_search_oracle import _peaky_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(2, 8), (9, 16), (17, 32)])
@pytest.mark.parametrize("graph", [False, True])
def test_one_node_in_every_slot(lo, hi, graph):
    """The first step of a learned search gives all its leaf slots to the root:
    512 slots of each of 16 roots, in 512 blocks of the evaluation kernel."""
    from gpu_ai_gb300 import Net, Searches
    from test_gpu_search_select import _roots
    q, n = 512, 16
    net = Net(0, max_batch=256, seed=1)
    net.set_params(_peaky_params(5))
    learned = {"value_weight": 0.5, "c_puct": 1.5}
    for seed in range(2):
        roots = _roots(lo, hi, n, 100 * seed + lo)
        gpu = Searches(n, 4000, q, playouts_per_leaf=1, policy=0, seed=3)
        gpu.set_net(net, **learned)
        o = S.SearchesOracle(n, 1, 0, 3, children=L.children, playouts=None, learned=learned)
        for i, r in enumerate(roots):
            assert gpu.add(r, 600, 60, (i + 7) << 36) == o.add(r, 600, 60, (i + 7) << 36)
        gpu.step(1, q, graph)
        gpu.poll()
        lv = gpu.leaves(net=True)
        assert (lv["node"] == 0).all() and len(lv["node"]) == q * n
        o.step(q, net_value=lv["net_value"], net_logits=lv["net_logits"], outcomes=lv["outcomes"])
        for slot in range(n):
            g = gpu.nodes(slot, priors=True)
            np.testing.assert_array_equal(g["priors"].view(np.uint16), o.priors(slot).view(np.uint16))
            np.testing.assert_array_equal(g["info"], o.tree(slot)["info"])
        gpu.close()
    net.close()


@pytest.mark.parametrize("lo,hi,lo2,hi2", [(17, 32, 2, 3), (9, 16, 1, 1), (17, 32, 9, 12)])
def test_priors_of_a_reused_node_range(lo, hi, lo2, hi2):
    """A search in the node range of a removed one whose nodes had more moves:
    the priors past a node's moves, and those of nodes that are not evaluated,
    are zero."""
    from gpu_ai_gb300 import Net, Searches
    from test_gpu_search_oracle import _compare_step, _compare_trees
    from test_gpu_search_select import _roots
    net = Net(0, max_batch=256, seed=1)
    net.set_params(_peaky_params(5))
    learned = {"value_weight": 0.5, "c_puct": 1.5}
    gpu = Searches(1, 3000, 33, playouts_per_leaf=1, policy=0, seed=3)
    gpu.set_net(net, **learned)
    o = S.SearchesOracle(1, 1, 0, 3, children=L.children, playouts=None, learned=learned)
    for root in _roots(lo, hi, 1, lo) + _roots(lo2, hi2, 2, lo2):
        assert gpu.add(root, 400, 3000, 1 << 36) == o.add(root, 400, 3000, 1 << 36) == 0
        for step in range(12):
            gpu.step(1, 33, False)
            gpu.poll()
            lv = gpu.leaves(net=True)
            o.step(33, net_value=lv["net_value"], net_logits=lv["net_logits"], outcomes=lv["outcomes"])
            _compare_step(gpu, o, step, net=True)
            _compare_trees(gpu, o, [0], step, priors=True)
        gpu.remove(0)
        o.remove(0)
    gpu.close()
    net.close()
