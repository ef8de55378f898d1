"""Selections that stop at the depth limit, in a build of the library whose
limit is 3 levels (with the kernels' bounds checks): the call reports the limit
and nothing else, every leaf slot of the step is the search's own -- the slots
left over play out the root -- and the visits and scores of every node are
those of the leaf slots below it, also after a search was removed and its slot
and node range given to another one."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
LIMIT = 8  # the status bit of the depth limit (search.cu)


def _build_limited() -> str:
    from gpu_ai_gb300 import build as B
    out = os.path.join(HERE, "_build")
    os.makedirs(out, exist_ok=True)
    obj, so = os.path.join(out, "search_depth.o"), os.path.join(out, "libgpuai_depth.so")
    subprocess.run([B.nvcc()] + B.NVCC_FLAGS + ["-DGPUAI_CHECKS", "-DGPUAI_MAX_SELECT_DEPTH=3", "-c",
                                               os.path.join(B.CSRC, "search.cu"), "-o", obj], check=True)
    rest = [u for u in B.CUDA_UNITS if u != "search.cu"] + B._host_units()
    subprocess.run([B.nvcc(), "-shared", "-Xcompiler", "-fPIC"] + B.ARCH + ["-o", so, obj] +
                   [os.path.join(B.OBJ, u + ".o") for u in rest] + ["-lpthread"], check=True)
    return so


def _poll(gpu):
    """done and the status word (Searches.poll raises on any status)."""
    u64p = ctypes.POINTER(ctypes.c_uint64)
    done, budget = np.zeros(gpu.max_searches, np.uint64), np.zeros(gpu.max_searches, np.uint64)
    st = ctypes.c_uint32()
    gpu.lib.gpuai_searches_poll(gpu.h, done.ctypes.data_as(u64p), budget.ctypes.data_as(u64p), gpu.max_searches,
                                ctypes.byref(st))
    return done, st.value


def _run(learned, q, ppl, seed):
    import oracle_lib as L
    from gpu_ai_gb300 import Net, Searches
    from test_gpu_search_oracle import _peaky_params
    roots = list(L.random_positions(seed, 4, 0, 30))
    gpu = Searches(4, 40000, q, playouts_per_leaf=ppl, policy=0, seed=seed)
    unit = ppl
    if learned:
        net = Net(0, max_batch=256, seed=1)
        net.set_params(_peaky_params(5))
        gpu.set_net(net, value_weight=0.5, c_puct=1.5)
        unit = 64  # visit units per leaf slot
    live = {}  # slot -> visits and half points of its nodes, as the leaf slots add up

    def add(i, cap):
        slot = gpu.add(roots[i], 10**6, cap, (i + 1) << 36)
        live[slot] = np.zeros((cap, 2), np.int64)

    limits = 0
    for i, cap in enumerate((9000, 30, 12000)):
        add(i, cap)
    for step in range(10):
        if step == 4:  # its leaf entries of the last step stay behind
            gpu.remove(0)
            del live[0]
        if step == 7:
            add(3, 500)
        gpu.step(1, q, step % 2 == 0)
        done, st = _poll(gpu)
        assert st in (0, LIMIT), f"step {step}: status {st}"
        limits += st == LIMIT
        lv = gpu.leaves()
        np.testing.assert_array_equal(lv["search"], np.repeat(sorted(live), q))
        for slot, sums in live.items():
            t = gpu.nodes(slot)
            mine = lv["search"] == slot
            assert (lv["node"][mine] >= 0).all() and (lv["node"][mine] < len(t["info"])).all()
            np.testing.assert_array_equal(lv["boards"][mine], t["boards"][lv["node"][mine]])
            for n, o in zip(lv["node"][mine], lv["outcomes"][mine].astype(int)):
                while n >= 0:
                    first = int(t["boards"][n][3]) & 1  # PLAYER_1 moved into the node
                    sums[n] += unit, ((o == 0) + 2 * (o == (1 if first else -1))).sum()
                    n = t["parent"][n]
            k = len(t["info"])
            np.testing.assert_array_equal(t["info"][:, 2], sums[:k, 0], err_msg=f"step {step}: visits")
            if not learned:
                np.testing.assert_array_equal(t["info"][:, 3], sums[:k, 1], err_msg=f"step {step}: half points")
            assert done[slot] * unit == sums[0, 0] * ppl
    assert limits >= 3
    gpu.close()


@pytest.mark.gpu
def test_selections_that_stop_at_the_depth_limit(lib_built):
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], env=dict(os.environ, GPUAI_LIB=_build_limited()),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]


if __name__ == "__main__":
    sys.path[:0] = [HERE, os.path.dirname(HERE)]
    for learned, q, ppl in ((False, 512, 2), (False, 200, 1), (True, 33, 2), (True, 128, 1)):
        _run(learned, q, ppl, 40 + q)
