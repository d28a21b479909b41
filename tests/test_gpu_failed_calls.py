"""Calls whose CUDA runtime call fails: an out-of-memory or an instantiation
error code comes from a preloaded library (tests/cpp/fake_cudart.cpp) in place
of the call, in a process of its own.  The same library counts allocations."""
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
fake.fake_runs.restype = fake.fake_bytes.restype = C.c_long
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


def test_fit_without_room_for_the_adjoint_window(child):
    """The one-element adjoint's 10 MB of block partials: handles of several
    elements never hold them, a handle that could not allocate them works and
    asks again at the first gradient, and a captured first gradient has its
    own in the graph."""
    child("""
from tdmd_claude_b200.fitting import ForceMatch, eam_coeff_tensors, eam_table_meta
rng = np.random.default_rng(3)
lat = W.fcc_lattice(4, 4, 4, 3.615)
pos = np.stack([(lat + rng.normal(0, 0.1, lat.shape)) % (4 * 3.615) for _ in range(20)])
tgt = rng.normal(0, 0.3, pos.shape)
def make(types):
    b, n = fake.fake_bytes(), runs()
    fm = ForceMatch(pos, types, Box.make((0,) * 3, (4 * 3.615,) * 3), 5.0, "fp64")
    fm.set_targets(tgt)
    return fm, fake.fake_bytes() - b, runs() - n
one = np.ones(pos.shape[:2], np.int32)
_, bytes3, n3 = make(rng.integers(1, 4, pos.shape[:2]).astype(np.int32))
fm, bytes1, n1 = make(one)
assert n3 == n1 - 1 and bytes3 < bytes1 - 9e6
t = W.cu_eam_tables()
eam = EamAlloy.from_tables(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F, t.rho, t.rphi)
meta, c = eam_table_meta(eam), eam_coeff_tensors(eam)
loss, *g = [torch.empty_like(x) for x in (c[0][0, :1], *c)]
def gradient(fm, allocations):
    n = runs()
    fm.eam(meta, *c, loss, *g)
    assert runs() == n + allocations
    return [x.cpu().numpy().copy() for x in (loss, *g)]
def same(a, b):  # the adds' order is free: up to 1e4 terms an entry, some 100 times its size
    for x, y in zip(a, b):
        assert np.abs(x - y).max() <= 1e-10 * np.abs(y).max()
want = gradient(fm, 1)               # the spline rows
same(gradient(fm, 0), want)
fail(b"cudaMalloc", n1 - 1, OOM)
fm, _, n = make(one)
assert n == n1
same(gradient(fm, 2), want)          # the rows and the window
fail(b"cudaMalloc", n1 - 1, OOM)
fm = make(one)[0]
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    fm.eam(meta, *c, loss, *g)
for x in (loss, *g):
    x.fill_(7.0)
graph.replay()
torch.cuda.synchronize()
same([x.cpu().numpy() for x in (loss, *g)], want)
""")


def test_failed_window_leaves_its_start(child):
    """A graph that cannot be instantiated in the middle of a window: the error
    is reported, the state is the window's start, the next window runs from
    there, and a new upload has nothing of the old one."""
    child("""
s = W.fcc_system(4, 3.615, 600.0, 3)
t = W.cu_eam_tables()
eam = EamAlloy.from_tables(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F, t.rho, t.rphi)
L = np.array(s.hi) - np.array(s.lo)
moved = (s.positions + np.random.default_rng(1).normal(0, 0.1, s.positions.shape) - s.lo) % L + s.lo
def make(pot, precision, batch):
    cfg = make_config(r_skin=0.5, rebuild_every=6, precision=precision, lanes_per_atom=8)
    p = MorseParams.make(*W.MORSE_CU) if pot == "morse" else eam
    return (ReplicaBatch([Box.make(s.lo, s.hi)], [s.n], p, cfg) if batch else
            FastPipelineScheduler(Box.make(s.lo, s.hi), s.n, p, cfg))
def up(m, x, batch):
    if batch:
        m.upload(x, s.velocities, s.types, s.masses)
    else:
        m.upload(x, s.velocities, None, s.types, s.ids, s.masses)
def state(m, batch):
    d = m.download()
    return [np.array(v) for v in (d if batch else (d.positions, d.velocities, d.forces))]
for pot in ("morse", "eam"):
    for precision in ("fp64", "mixed"):
        for batch in (False, True):
            for end in (30, 31):      # an odd and an even number of fused drifts
                m, good = make(pot, precision, batch), make(pot, precision, batch)
                up(m, s.positions, batch), up(good, s.positions, batch)
                m.run_until(5), good.run_until(5)
                start = state(good, batch)
                fail(b"cudaGraphInstantiate", 2, OOM)
                try:
                    m.run_until(end)
                    raise SystemExit("no error")
                except TdmdError as e:
                    assert "OUT_OF_MEMORY" in str(e), e
                for a, b in zip(state(m, batch)[:2], start):
                    assert np.array_equal(a, b), (pot, precision, batch)
                m.run_until(end), good.run_until(end)   # (the lists' steps differ)
                tol = 1e-9 if precision == "fp64" else 1e-4
                d = state(m, batch)[0] - state(good, batch)[0]
                assert np.abs(d - np.round(d / L) * L).max() <= tol
                fail(b"cudaGraphInstantiate", 2, OOM)
                try:
                    m.run_until(end + 26)
                    raise SystemExit("no error")
                except TdmdError:
                    pass
                new = make(pot, precision, batch)
                for x in (m, new):
                    up(x, moved, batch)
                    x.run_until(1)
                for a, b in zip(state(m, batch), state(new, batch)):
                    assert np.array_equal(a, b), (pot, precision, batch)
""")


def test_batch_without_room_for_second_positions(child):
    """A Morse batch whose second position buffers cannot be allocated drifts
    in launches of its own: the same bits."""
    child("""
s = W.fcc_system(4, 3.615, 600.0, 3)
# a first window allocates its snapshot (2 arrays, 3 in mixed), then these (1, 2)
for precision, refused in (("fp64", 3), ("mixed", 4), ("mixed", 5)):
    out = []
    for nth in (0, refused):
        cfg = make_config(r_skin=0.5, rebuild_every=6, precision=precision, lanes_per_atom=8)
        m = ReplicaBatch([Box.make(s.lo, s.hi)], [s.n], MorseParams.make(*W.MORSE_CU), cfg)
        m.upload(s.positions, s.velocities, s.types, s.masses)
        m.run_until(0)
        n = runs()
        fail(b"cudaMalloc", nth, OOM)
        m.run_until(8)
        assert not nth or runs() - n == nth
        for t in (8, 17, 40):
            m.run_until(t)
            out.append([np.array(v) for v in m.download()])
    for a, b in zip(out[:3], out[3:]):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
""")


def test_overflow_without_room_for_longer_rows(child):
    """Rows that overflow in a window and cannot grow: the error is reported,
    the state is the window's start, and the next window makes its rows anew
    and reaches the state of an undisturbed run."""
    child("""
rng = np.random.default_rng(3)
L, n = 30.0, 300
x = rng.uniform(0, L, (n, 3))
v, types, masses = 15.0 - x, np.ones(n, np.int32), np.array([1.0, 63.546])
box = Box.make((0,) * 3, (L,) * 3)
def make(batch):
    cfg = make_config(r_skin=1.0, rebuild_every=5, dt=0.002, lanes_per_atom=8)
    p = MorseParams.make(0.01, 1.0, 3.0, 5.0)
    m = ReplicaBatch([box], [n], p, cfg) if batch else FastPipelineScheduler(box, n, p, cfg)
    m.upload(x, v, types, masses) if batch else m.upload(x, v, None, types, None, masses)
    m.run_until(5)
    return m
def state(m, batch):
    d = m.download()
    return [np.array(a) for a in (d[:2] if batch else (d.positions, d.velocities))]
for batch in (False, True):
    m, good = make(batch), make(batch)
    assert good.stats().nlist_retries == 0
    start = state(good, batch)
    fail(b"cudaMalloc", 1, OOM)
    try:
        m.run_until(200)
        raise SystemExit("no error")
    except TdmdError as e:
        assert "OUT_OF_MEMORY" in str(e), e
    for a, b in zip(state(m, batch), start):
        assert np.array_equal(a, b)
    m.run_until(200), good.run_until(200)
    assert good.stats().nlist_retries >= 1
    d = state(m, batch)[0] - state(good, batch)[0]  # (the lists' steps differ)
    assert np.abs(d - np.round(d / L) * L).max() <= 1e-8
""")
