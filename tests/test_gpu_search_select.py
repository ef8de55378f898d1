"""The block-per-search selection at the sizes where it can go wrong, node for
node against the CPU restatement: steps on either side of each block width,
node ranges that run out in the first, a middle and the last round of a
frontier, and roots whose nodes have more children than a group of lanes holds
at once (8), than two do (16), or one child (a forced line)."""
import numpy as np
import pytest

import oracle_lib as L
from golden_boards import random_boards
from test_gpu_search_oracle import _run

pytestmark = pytest.mark.gpu


def _roots(lo, hi, n, seed):
    """n live positions with lo..hi legal moves (many kings: long lists)."""
    pos = random_boards(np.random.default_rng(seed), 60000)
    pos[:, 3] &= np.uint32(1)
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
