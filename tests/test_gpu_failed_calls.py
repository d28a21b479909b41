"""Calls whose CUDA runtime call fails: an out-of-memory or an instantiation
error code comes from a preloaded library (tests/cpp/fake_cudart.cpp) in place
of the call, in a process of its own."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PRELUDE = """
import ctypes as C
import numpy as np
import torch
from oracle import oracle
from tdmd_claude_b200 import *
from tdmd_claude_b200 import workloads as W
fake = C.CDLL(None)
fake.fake_runs.restype = C.c_long
def fail(call, nth, code):
    fake.fake_fail(call, C.c_long(nth), code)
def runs(call=b"cudaMalloc"):
    return fake.fake_runs(call)
OOM = 2
"""


@pytest.fixture(scope="module")
def child(cuda, tmp_path_factory):
    """child(script): runs it with the preloaded library; its output."""
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run([gxx, "-shared", "-fPIC", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I",
                    os.path.join(CUDA_HOME, "include"),
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), "-o", so, "-ldl"],
                   check=True, capture_output=True, text=True)

    def run(script):
        r = subprocess.run([sys.executable, "-c", PRELUDE + script], cwd=ROOT, timeout=240,
                           env={**os.environ, "LD_PRELOAD": so, "PYTHONPATH": ROOT},
                           capture_output=True, text=True)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout
    return run


def test_list_build_without_room_for_padded_rows(child):
    """A list handle whose padded rows (second build) or whose list beside them
    cannot be allocated builds the list all the same; rows that a dense clump
    would size are not asked for."""
    child("""
rng = np.random.default_rng(8)
a = rng.uniform(0, 30.0, (1500, 3))
clump = np.concatenate([a[:1200], 15 + rng.uniform(-1, 1, (300, 3))])
nl = DeviceNeighborList()
def build(p):
    p = np.ascontiguousarray(p % 30.0)
    n0 = runs()
    nl.build(torch.as_tensor(p, device="cuda"), len(p), Box.make((0,) * 3, (30.0,) * 3), 4.0, 0.3)
    n1 = runs()
    want = oracle.neighbor_list(p, (0,) * 3, (30.0,) * 3, 4.0, 0.3, half=False)
    for g, w in zip(nl.host_csr(), want):
        assert np.array_equal(g, w)
    return n1 - n0
for p in (a, a):
    torch.as_tensor(p, device="cuda").cpu()  # (torch's own allocations are made)
build(a)
fail(b"cudaMalloc", 1, OOM)
assert build(a) == 1                 # the rows: refused
assert build(a) == 1                 # the rows: there
assert build(a) == 0
fail(b"cudaMalloc", 1, OOM)
assert build(15 + 0.96 * (a - 15)) == 2   # the list: refused beside the rows, then there
assert build(a) == 1                 # the rows again
build(clump)
assert build(clump) == 0             # 300 neighbors an atom of the clump: two sweeps
""")
