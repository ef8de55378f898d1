"""The playout kernels' rotated-bitboard plies (rot.cuh) against the plies of
rules.cuh they stand for, on the CPU: the same move, the same number of draws
and the same board after it, on random boards of every density (either side,
many kings: every multi-jump path) and along whole games, and the same plies
deferred."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gpu_ai_gb300", "csrc")


@pytest.fixture(scope="module")
def rot():
    src, so = os.path.join(HERE, "rot_host.cpp"), os.path.join(HERE, "_build", "librot_host.so")
    deps = [src] + [os.path.join(CSRC, f) for f in ("rot.cuh", "rules.cuh")]
    if not os.path.exists(so) or max(map(os.path.getmtime, deps)) > os.path.getmtime(so):
        os.makedirs(os.path.dirname(so), exist_ok=True)
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wno-unknown-pragmas", "-o", so, src],
                       check=True)
    lib = ctypes.CDLL(so)
    for f in (lib.rot_boards, lib.rot_games):
        f.argtypes = [ctypes.c_uint64, ctypes.c_uint64, ctypes.c_int, ctypes.POINTER(ctypes.c_uint64)]
        f.restype = ctypes.c_long
    u32, u64 = ctypes.c_uint32, ctypes.c_uint64
    lib.rot_positions.argtypes = [u64, u32, u32, u32, ctypes.c_int, ctypes.c_void_p]
    lib.rot_positions.restype = None
    return lib


@pytest.mark.parametrize("policy", [0, 1, 2])
def test_plies_match_on_random_boards(rot, policy):
    kind = (ctypes.c_uint64 * 4)()
    assert rot.rot_boards(1_500_000, 11 + policy, policy, kind) == 0
    assert min(kind) > 2_000  # every kind of ply was met


@pytest.mark.parametrize("policy", [0, 1, 2])
def test_plies_match_along_games(rot, policy):
    kind = (ctypes.c_uint64 * 4)()
    assert rot.rot_games(20_000, 5 + policy, policy, kind) == 0
    assert min(kind) > 500


@pytest.mark.gpu
@pytest.mark.parametrize("policy", [0, 1, 2])
@pytest.mark.parametrize("n,lo,hi", [(1, 0, 0), (1, 7, 7), (255, 0, 60), (257, 0, 1), (4000, 0, 90), (200_003, 0, 40),
                                     (600, 300, 5000)])
def test_positions_equal_the_plies_one_at_a_time(rot, engine, policy, n, lo, hi):
    """Seeded positions on the GPU: one game, part of a block, one more than a
    block, blocks that claim in bulk, games that are all played to their end."""
    import torch
    out = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    engine.selfplay_positions(99 + n, n, lo, hi, policy, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = np.zeros((n, 4), np.uint32)
    rot.rot_positions(99 + n, n, lo, hi, policy, want.ctypes.data)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
