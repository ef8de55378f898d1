"""Learned selection on both sides of the rule that chooses its block: 512
threads above 16 leaves per search while the pool has at most two searches per
SM and above 256 leaves in any pool, else 256.  Node for node against the CPU
restatement, with searches in the first, a middle and the last slots of a pool
whose other slots are free."""
import pytest

import oracle_lib as L
from oracle import search as S
from test_gpu_search_oracle import _compare_step, _compare_trees, _peaky_params, _replay

pytestmark = pytest.mark.gpu


# pool: searches per SM (0: three searches in all), and `extra` more
@pytest.mark.parametrize("pool,extra,q,steps", [
    (2, 1, 17, 12), (2, 1, 33, 10), (2, 1, 43, 10), (2, 1, 128, 8), (2, 1, 255, 6), (2, 1, 256, 6),  # 256 threads
    (2, 1, 257, 6), (2, 0, 33, 10), (2, 0, 256, 6),  # 512
    (0, 0, 16, 12),  # 256
    (0, 0, 17, 12), (0, 0, 256, 6), (0, 0, 257, 6), (0, 0, 512, 5)])  # 512
def test_learned_selection_by_pool_and_step(engine, pool, extra, q, steps):
    from gpu_ai_gb300 import Net, Searches
    n = pool * engine.device_info()["sms"] + extra if pool else 3
    net = Net(0, max_batch=256, seed=1)
    net.set_params(_peaky_params(5))
    learned = {"value_weight": 0.5, "c_puct": 1.5}
    gpu = Searches(n, 60000, q, playouts_per_leaf=1, policy=0, seed=3)
    gpu.set_net(net, **learned)
    o = S.SearchesOracle(n, 1, 0, 3, children=L.children, playouts=_replay, learned=learned)
    roots = L.random_positions(60 + q, n, 0, 40)
    keep = sorted({0, n // 2, n - 1})
    for i in range(n):  # fill the pool, then leave three searches in it
        cap = (12000, 60 + q, 12000)[keep.index(i)] if i in keep else 1
        assert gpu.add(roots[i], 50 * q + 7, cap, (i + 7) << 36) == o.add(roots[i], 50 * q + 7, cap, (i + 7) << 36)
    for i in range(n):
        if i not in keep:
            gpu.remove(i)
            o.remove(i)
    for step in range(steps):
        gpu.step(1, q, step % 2 == 0)
        gpu.poll()
        lv = gpu.leaves(net=True)
        o.step(q, net_value=lv["net_value"], net_logits=lv["net_logits"])
        _compare_step(gpu, o, step, net=True)
        _compare_trees(gpu, o, keep, step, priors=True)
    gpu.close()
    net.close()
