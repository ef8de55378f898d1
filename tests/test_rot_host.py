"""The playout kernels' rotated-bitboard plies (rot.cuh) against the plies of
rules.cuh they stand for, on the CPU: the same move, the same number of draws
and the same board after it, on random boards of every density (either side,
many kings: every multi-jump path) and along whole games, and the same plies
deferred."""
import ctypes
import os
import subprocess

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
