"""The playout kernel's launch shape by batch size, on contexts of their own:
outcomes equal the oracle replay on either side of the two limits (8 playouts
per SM, the resident lanes) for every policy, with equal and with uneven
repetitions, and the shape that is launched, read from a captured launch, is by
size again once a shape or layout was set back to a new context's."""
import ctypes

import numpy as np
import pytest

import oracle_lib as L

pytestmark = pytest.mark.gpu


class _KernelParams(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS (v2)
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("shared", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def _launched(eng, policy, total):
    """(blocks, threads) of the playout kernel that a call of `total` playouts launches (captured, not run)."""
    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    d_pos = torch.from_numpy(L.start_board().reshape(1, 4).view(np.int32).copy()).cuda()
    d_out = torch.empty(total, dtype=torch.int8, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    handle, graph = ctypes.c_void_p(s.cuda_stream), ctypes.c_void_p()
    assert cu.cuStreamBeginCapture_v2(handle, 2) == 0  # relaxed mode
    try:
        eng.playouts_device(d_pos.data_ptr(), None, 1, total, total, 1, 0, policy, d_out.data_ptr(), s.cuda_stream)
    finally:
        assert cu.cuStreamEndCapture(handle, ctypes.byref(graph)) == 0
    n = ctypes.c_size_t()
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    found = []
    for node in nodes:
        kind = ctypes.c_int()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value == 0:  # a kernel
            p = _KernelParams()
            assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(p)) == 0
            found.append((p.grid[0], p.block[0]))
    assert cu.cuGraphDestroy(graph) == 0
    assert len(found) == 1
    return found[0]


@pytest.fixture()
def fresh(lib_built):
    from gpu_ai_gb300 import Engine
    e = Engine(0)
    yield e
    e.close()


def _limits(eng, policy):
    shape, sms = eng.get_launch(policy), eng.device_info()["sms"]
    return 8 * sms, sms * shape["blocks_per_sm"] * shape["block_threads"]


@pytest.mark.parametrize("policy", [0, 1, 2])
def test_shape_by_size_and_back(fresh, policy):
    from gpu_ai_gb300 import LAYOUT_POOLED, LAYOUT_THREAD
    few, lanes = _limits(fresh, policy)
    start = fresh.get_launch(policy)
    sizes = (1, few - 1, few, few + 1, lanes, lanes + 1, 4 * lanes)
    want = [_launched(fresh, policy, n) for n in sizes]
    assert [t for _, t in want] == [128, 128, 128, 256, 256, start["block_threads"], start["block_threads"]]
    fresh.set_launch(policy, 128, 0)  # a block per playout up to the resident ones
    resident = fresh.device_info()["sms"] * fresh.get_launch(policy)["max_blocks_per_sm"]
    assert [b for b, _ in want[:3]] == [min(n, resident) for n in sizes[:3]]
    assert want[-1][0] * want[-1][1] == lanes
    # another shape holds for every size
    other = 512 if start["block_threads"] == 256 else 256
    fresh.set_launch(policy, other, 1)
    assert [_launched(fresh, policy, n)[1] for n in sizes] == [other] * len(sizes)
    fresh.set_launch(policy, start["block_threads"], start["blocks_per_sm"])
    assert [_launched(fresh, policy, n) for n in sizes] == want
    # ... and so does another layout
    fresh.set_layout(policy, LAYOUT_POOLED)
    assert _launched(fresh, policy, few)[1] == start["block_threads"]
    fresh.set_layout(policy, LAYOUT_THREAD)
    assert [_launched(fresh, policy, n) for n in sizes] == want
    # the values that are already set change nothing
    fresh.set_layout(policy, LAYOUT_THREAD)
    fresh.set_launch(policy, start["block_threads"], 0)
    assert [_launched(fresh, policy, n) for n in sizes] == want


@pytest.mark.parametrize("policy", [0, 1, 2])
@pytest.mark.parametrize("limit", [0, 1])
@pytest.mark.parametrize("more", [-1, 0, 1])
@pytest.mark.parametrize("ragged", [False, True])
def test_outcomes_on_either_side_of_the_limits(fresh, policy, limit, more, ragged):
    total = _limits(fresh, policy)[limit] + more
    if ragged:
        rng = np.random.default_rng(total)
        cuts = np.sort(rng.integers(0, total + 1, 199))
        reps = np.diff(np.concatenate([[0], cuts, [total]])).astype(np.uint32)
        pos = L.random_positions(total, len(reps), 40, 120)
    else:
        reps = np.ones(total, np.uint32)
        pos = np.resize(L.random_positions(total, 997, 40, 120), (total, 4))
    got = fresh.playouts(pos, reps if ragged else None, seed=17, stream_base=3, policy=policy)
    exp, _ = L.replay_batch(pos, reps, seed=17, stream_base=3, policy=policy)
    np.testing.assert_array_equal(got, exp)


def test_wide_blocks_on_a_small_batch(fresh):
    """512-thread blocks where the size rule would take smaller ones."""
    pos = L.random_positions(21, 64, 0, 30)
    reps = np.random.default_rng(1).integers(0, 300, 64).astype(np.uint32)
    fresh.set_launch(0, 512, 1)
    got = fresh.playouts(pos, reps, seed=21, stream_base=5)
    exp, _ = L.replay_batch(pos, reps, seed=21, stream_base=5)
    np.testing.assert_array_equal(got, exp)
