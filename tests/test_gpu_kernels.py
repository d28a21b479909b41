"""Edges of the kernels' ranges: branches of the pair arithmetic, of the list
build and of the force-matching adjoint, at the sizes where they change."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(torch, a, dtype=None):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda", dtype=dtype)


def _spline(c, x, h):
    """(value, derivative) of packed a|b|c|d coefficients at x."""
    ns = len(c) // 4
    k = min(max(int(x / h), 0), ns - 1)
    dx = x - k * h
    a, b, cc, d = (c[m * ns + k] for m in range(4))
    return a + dx * (b + dx * (cc + dx * d)), b + dx * (2 * cc + 3 * d * dx)


# below the FP32 seed's range, tiny, on spline knots (dr = 5/1999), ordinary, at
# the cutoff's two sides
@pytest.mark.parametrize("r", [1e-18, 1e-3, 400 * 5 / 1999, 1000 * 5 / 1999, 2.556, 4.9999999, 5.0])
@pytest.mark.parametrize("wrapped", [False, True])
def test_fp64_pair_radius(cuda, r, wrapped):
    """Two atoms r apart, directly or through the periodic face: density, F'
    and force against numpy's square root and divisions.  A rounding of r
    moves phi' by |phi''/phi'| ulp(r) < 20 ulp: 1e-14 relative, ten times
    that allowed."""
    from tdmd_claude_b200 import Box, DeviceEam, EamAlloy
    from tdmd_claude_b200 import workloads as W
    t = W.cu_eam_tables()
    eam = EamAlloy.from_tables(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F, t.rho, t.rphi)
    lo, hi = -10.0, 22.0
    pos = np.array([[lo, 1.0, 2.0], [hi - r, 1.0, 2.0]] if wrapped else
                   [[0.0, 1.0, 2.0], [r, 1.0, 2.0]])
    dx = pos[0, 0] - pos[1, 0] + ((hi - lo) if wrapped else 0.0)
    r = abs(dx)
    if r == 0.0:
        pytest.skip("the face swallows this separation")
    de = DeviceEam()
    de.upload_tables(eam)
    f64 = cuda.float64
    f = cuda.zeros((2, 3), dtype=f64, device="cuda")
    rho = cuda.zeros(2, dtype=f64, device="cuda")
    fp = cuda.zeros(2, dtype=f64, device="cuda")
    nbr = _dev(cuda, np.array([1, 0], np.int32))
    off = _dev(cuda, np.array([0, 1], np.int32))
    cnt = _dev(cuda, np.array([1, 1], np.int32))
    de.compute(_dev(cuda, pos), f, _dev(cuda, np.ones(2, np.int32)), nbr.data_ptr(),
               off.data_ptr(), cnt.data_ptr(), 2, Box.make((lo,) * 3, (hi,) * 3), d_rho=rho,
               d_fp=fp)
    want_rho = want_f = want_fp = 0.0
    if r * r < t.cutoff ** 2:
        want_rho, drho = _spline(eam.coeffs(1, 0), r, t.dr)
    want_fp = _spline(eam.coeffs(0, 0), want_rho, t.drho)[1]
    if r * r < t.cutoff ** 2:
        want_f = -(_spline(eam.coeffs(2, 0), r, t.dr)[1] + 2 * want_fp * drho) / r * dx
    assert np.allclose(rho.cpu(), want_rho, rtol=1e-13, atol=1e-16)
    assert np.allclose(fp.cpu(), want_fp, rtol=1e-13)
    got = f.cpu().numpy()
    assert np.allclose(got[:, 0], [want_f, -want_f], rtol=1e-13, atol=1e-15)
    assert not got[:, 1:].any()


# nr = 600: every interval inside the shared-memory window; 2000: the window's
# lower edge at 1.8 A, below all pairs; 5001: at 3.72 A, so that the nearest
# shell's pairs add to global memory and the others to the window
@pytest.mark.parametrize("nr", [600, 2000, 5001])
@pytest.mark.parametrize("ntypes", [1, 3])
@pytest.mark.parametrize("nsnap", [1, 3])
def test_eam_adjoint_window_edges(cuda, oracle, nr, ntypes, nsnap):
    """EAM loss and gradient vs the FP64 oracle over the window's cases and a
    grid of fewer blocks than SMs, atoms in random order: 1e-10 of the loss,
    1e-9 of each spline's largest entry (sums of up to 1e4 terms of both
    signs), as the other FP64 gradient tests."""
    from tdmd_claude_b200 import Box, EamAlloy
    from tdmd_claude_b200 import workloads as W
    from tdmd_claude_b200.fitting import ForceMatch, eam_coeff_tensors, eam_table_meta
    rng = np.random.default_rng(40 + nr + ntypes)
    kw = {} if ntypes == 1 else dict(beta_f=(4.8, 5.0, 5.2), A_phi=(0.55, 0.60, 0.65),
                                     E_F=(1.1, 1.2, 1.3))
    t = W.analytic_eam(nr=nr, **kw)
    eam = EamAlloy.from_tables(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F, t.rho, t.rphi)
    lat = W.fcc_lattice(3, 3, 3, 3.615)
    pos = np.stack([rng.permutation(lat + rng.normal(0, 0.1, lat.shape)) for _ in range(nsnap)])
    L = 3 * 3.615
    pos %= L
    types = rng.integers(1, ntypes + 1, size=pos.shape[:2]).astype(np.int32)
    tgt = rng.normal(0.0, 0.3, size=pos.shape)
    fm = ForceMatch(pos, types, Box.make((0,) * 3, (L,) * 3), t.cutoff, "fp64")
    fm.set_targets(tgt)
    F, rho, phi = eam_coeff_tensors(eam)
    loss = cuda.zeros(1, dtype=cuda.float64, device="cuda")
    g = [cuda.empty_like(x) for x in (F, rho, phi)]
    fm.eam(eam_table_meta(eam), F, rho, phi, loss, *g)
    oe = oracle.OracleEam(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F, t.rho, t.rphi)
    lo, *want = oe.fm_loss_grad(pos, types, (0,) * 3, (L,) * 3, tgt)
    assert abs(loss.item() - lo) <= 1e-10 * lo
    for got, ref in zip(g, want):
        for sp in range(ref.shape[0]):
            assert np.abs(got[sp].cpu().numpy() - ref[sp]).max() <= 1e-9 * np.abs(ref[sp]).max()


# rows shorter than a sweep, one past whole sweeps, and longer; every lane count
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("lanes", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("batch", [2, 4])
def test_lane_slots_cover_every_row(cuda, oracle, precision, lanes, batch):
    """A gas whose rows hold 0 to ~70 entries: every slot of every row is
    taken once whatever the lanes and sweep (forces vs the oracle to 1e-10 of
    their RMS in FP64, 1e-5 in mixed, the library's bounds)."""
    from tdmd_claude_b200 import Box, FastPipelineScheduler, MorseParams, make_config
    rng = np.random.default_rng(6)
    pos = np.concatenate([rng.uniform(0, 30.0, (150, 3)), rng.uniform(10.0, 18.0, (65, 3))])
    n, morse = len(pos), (0.05, 1.0, 3.0, 5.0)
    s = FastPipelineScheduler(Box.make((0,) * 3, (30.0,) * 3), n, MorseParams.make(*morse),
                              make_config(r_skin=0.4, precision=precision, lanes_per_atom=lanes,
                                          nbr_batch=batch))
    masses = np.array([1.0, 63.546])
    s.upload(pos, np.zeros((n, 3)), None, np.ones(n, np.int32), None, masses)
    s.run_until(0)
    cnt = s.neighbor_list()[0]
    assert cnt.min() == 0 and cnt.max() > 32
    want = oracle.md_run(pos, np.zeros((n, 3)), np.ones(n, np.int32), masses, (0,) * 3,
                         (30.0,) * 3, 0.001, 0.4, 10, [0], morse=morse)["forces"]
    d = s.download().forces - want
    rms = np.sqrt((want ** 2).mean())
    assert np.sqrt((d ** 2).mean()) <= (1e-10 if precision == "fp64" else 1e-5) * rms


def test_neighbor_list_handle_reused(cuda, oracle):
    """One handle over changing inputs: the first build (two sweeps), the same
    atoms again, a squeezed system whose rows overflow the kept capacity, a
    dilute one, another atom count: rows bit-exact to the oracle each time."""
    from tdmd_claude_b200 import Box, DeviceNeighborList
    rng = np.random.default_rng(8)
    a = rng.uniform(0, 30.0, (1500, 3))
    squeezed = 9.0 + a * 0.4
    cases = [a, a, a + 0.01, squeezed, squeezed, a, a[:777], a[:1], a]
    nl = DeviceNeighborList()
    for k, p in enumerate(cases):
        p = np.ascontiguousarray(p % 30.0)
        nl.build(_dev(cuda, p), len(p), Box.make((0,) * 3, (30.0,) * 3), 4.0, 0.3)
        c, o, nb = nl.host_csr()
        ec, eo, enb = oracle.neighbor_list(p, (0,) * 3, (30.0,) * 3, 4.0, 0.3, half=False)
        assert np.array_equal(c, ec) and np.array_equal(o, eo) and np.array_equal(nb, enb), k
        assert nl.max_neighbors() == int(ec.max()) and nl.total_pairs() == enb.size


# two cells per SM are 296 on a B200: 270 and 540 cells with 3-cell axes, 294
# and 300 without
@pytest.mark.parametrize("nc", [(3, 3, 30), (3, 3, 60), (7, 7, 6), (5, 6, 10)])
def test_row_build_block_sizes(cuda, oracle, nc):
    """The list on both sides of the few-cells rule, with and without 3-cell
    axes, a dense corner included: bit-exact to the oracle."""
    from tdmd_claude_b200 import Box, DeviceNeighborList
    rng = np.random.default_rng(9)
    r, hi = 4.4, np.array(nc) * 4.5
    p = np.concatenate([rng.uniform(0, 1, (10 * int(np.prod(nc)), 3)) * hi,
                        rng.uniform(0, 1, (300, 3)) * 6.0])
    nl = DeviceNeighborList()
    nl.build(_dev(cuda, p), len(p), Box.make((0,) * 3, hi), r - 0.3, 0.3)
    got = nl.host_csr()
    want = oracle.neighbor_list(p, (0,) * 3, tuple(hi), r - 0.3, 0.3, half=False)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


# small systems, in one block or not, and cells of up to ~150 members
@pytest.mark.parametrize("n,nc", [(1, (3, 3, 3)), (31, (3, 4, 5)), (4096, (8, 8, 8)),
                                  (4097, (8, 8, 8)), (4000, (9, 8, 8)), (4096, (3, 3, 3))])
def test_cell_list_one_block(cuda, oracle, n, nc):
    """Cell lists bit-exact, with cells above 32 and above 128 members (27
    cells of ~150 atoms)."""
    _check_cell_list(cuda, oracle, n, nc)


# the one-block rule's two limits (3072 atoms, 192 cells) and both sides of each
@pytest.mark.parametrize("n,nc", [(3072, (4, 6, 8)), (3073, (4, 6, 8)), (3072, (5, 5, 8)),
                                  (2, (4, 6, 8)), (3072, (3, 3, 3)), (1025, (3, 3, 21))])
def test_cell_list_one_block_limits(cuda, oracle, n, nc):
    _check_cell_list(cuda, oracle, n, nc)


def _check_cell_list(cuda, oracle, n, nc):
    from tdmd_claude_b200 import Box, DeviceCellList
    rng = np.random.default_rng(n)
    hi = np.array(nc) * 5.0 + 0.1
    p = rng.uniform(-0.01, 1.01, (n, 3)) * hi  # some atoms outside: clamped
    cl = DeviceCellList()
    cl.build(_dev(cuda, p), n, Box.make((0,) * 3, hi), 5.0)
    got = cl.arrays()
    want = oracle.cell_list(p, (0,) * 3, tuple(hi), 5.0)
    assert tuple(got[0]) == nc
    enc, ecc, eco, eca, eac = want
    for g, w in zip(got, (enc, eca, eco, ecc, eac)):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("energy_every", [0, 3])
@pytest.mark.parametrize("batch", [False, True])
def test_morse_fused_kick_equals_unfused(cuda, precision, energy_every, batch):
    """Morse graph windows drift inside the force pass, into a second position
    buffer; windows launched one by one do not.  Windows of one step, of odd
    and even lengths, across rebuilds and past one graph segment, with and
    without energy-log steps: the same bits, and energies of the state that
    each window leaves."""
    from tdmd_claude_b200 import (Box, FastPipelineScheduler, MorseParams, ReplicaBatch,
                                  make_config)
    from tdmd_claude_b200 import workloads as W
    s = W.fcc_system(4, 3.615, 600.0, 3)
    out = []
    for graphs in (True, False):
        cfg = make_config(r_skin=0.3, rebuild_every=70, precision=precision, lanes_per_atom=8,
                          use_graphs=graphs, energy_every=energy_every, energy_log_capacity=256)
        p = MorseParams.make(*W.MORSE_CU)
        if batch:
            m = ReplicaBatch([Box.make(s.lo, s.hi)] * 2, [s.n, s.n], p, cfg)
            m.upload(np.concatenate([s.positions, s.positions]),
                     np.concatenate([s.velocities, 0.5 * s.velocities]),
                     np.concatenate([s.types] * 2), s.masses)
        else:
            m = FastPipelineScheduler(Box.make(s.lo, s.hi), s.n, p, cfg)
            m.upload(s.positions, s.velocities, None, s.types, s.ids, s.masses)
        for t in (1, 3, 6, 16, 27, 160, 161):
            m.run_until(t)
            st = m.download()
            out.append([*(st if batch else (st.positions, st.velocities, st.forces)),
                        *m.energies()])
        m.close()
    half = len(out) // 2
    for a, b in zip(out[:half], out[half:]):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


# on spline knots (dr = 5/1999), inside an interval, in the last one before the
# cutoff
@pytest.mark.parametrize("r", [400 * 5 / 1999, 1000 * 5 / 1999, 2.556, 4.4, 4.9985])
def test_mixed_pair_interval(cuda, r):
    """Two atoms r apart in mixed precision: FP32 rounds the distance (6e-8 of
    it), the offset and about ten products and sums: 1e-6 of the density (and
    3e-7 A of its slope), 3e-6 of the force's two terms before they cancel."""
    from tdmd_claude_b200 import Box, DeviceEam, EamAlloy
    from tdmd_claude_b200 import workloads as W
    t = W.cu_eam_tables()
    eam = EamAlloy.from_tables(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F, t.rho, t.rphi)
    de = DeviceEam()
    de.upload_tables(eam)
    pos = np.array([[0.0, 1.0, 2.0], [r, 1.0, 2.0]])
    f = cuda.zeros((2, 3), dtype=cuda.float32, device="cuda")
    rho = cuda.zeros(2, dtype=cuda.float64, device="cuda")
    nbr, off, cnt = (_dev(cuda, np.array(x, np.int32)) for x in ([1, 0], [0, 1], [1, 1]))
    de.compute(_dev(cuda, pos), f, _dev(cuda, np.ones(2, np.int32)), nbr.data_ptr(),
               off.data_ptr(), cnt.data_ptr(), 2, Box.make((-10.0,) * 3, (22.0,) * 3), d_rho=rho,
               precision="mixed")
    want, drho = _spline(eam.coeffs(1, 0), r, t.dr)
    assert np.abs(rho.cpu().numpy() - want).max() <= 1e-6 * want + 3e-7 * abs(drho)
    fp = _spline(eam.coeffs(0, 0), want, t.drho)[1]
    dphi = _spline(eam.coeffs(2, 0), r, t.dr)[1]
    wf = (dphi + 2 * fp * drho)  # on atom 0, towards atom 1 when positive
    bound = 3e-6 * (abs(dphi) + abs(2 * fp * drho)) + 1e-7
    assert np.abs(f.cpu().numpy()[:, 0] - [wf, -wf]).max() <= bound


# lanes per atom change between these sizes (8 at 40 000 atoms, 16 at 30 000 on
# 148 SMs), so that the smaller system needs more block partials
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_device_eam_graphs_keep_their_scratch(cuda, precision):
    """DeviceEam evaluations with energies, captured after a larger system was
    evaluated, and replayed after a smaller one: the same bits as uncaptured."""
    from tdmd_claude_b200 import Box, DeviceEam, DeviceNeighborList, EamAlloy
    from tdmd_claude_b200 import workloads as W
    t = W.cu_eam_tables()
    de = DeviceEam()
    de.upload_tables(EamAlloy.from_tables(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F,
                                          t.rho, t.rphi))
    a = 3.615

    class Case:
        def __init__(self, nz):
            rng = np.random.default_rng(nz)
            x = W.fcc_lattice(20, 25, nz, a)
            hi = np.array([20, 25, nz]) * a
            self.n, self.box = len(x), Box.make((0,) * 3, tuple(hi))
            self.x = _dev(cuda, (x + rng.normal(0, 0.05, x.shape)) % hi)
            self.types = cuda.ones(self.n, dtype=cuda.int32, device="cuda")
            self.nl = DeviceNeighborList()
            self.nl.build(self.x, self.n, self.box, t.cutoff, 0.3)
            self.e, self.w = (cuda.zeros(k, dtype=cuda.float64, device="cuda")
                              for k in (1, 6))
            self.f = cuda.zeros((self.n, 3), device="cuda",
                                dtype=cuda.float64 if precision == "fp64" else cuda.float32)
            cuda.cuda.synchronize()

        def run(self, prec=precision, stream=None, f=None):
            de.compute(self.x, self.f if f is None else f, self.types, self.nl.d_neighbors(),
                       self.nl.d_offsets(), self.nl.d_counts(), self.n, self.box, d_energy=self.e,
                       d_virial=self.w, precision=prec, stream=stream)

        def capture(self):
            g = cuda.cuda.CUDAGraph()
            with cuda.cuda.graph(g):
                self.run(stream=cuda.cuda.current_stream())
            return g

        def out(self):
            cuda.cuda.synchronize()
            r = [x.cpu().numpy().copy() for x in (self.f, self.e, self.w)]
            for x in (self.f, self.e, self.w):
                x.zero_()
            cuda.cuda.synchronize()
            return r

    big, small = Case(20), Case(15)
    big.run()
    want_big = big.out()
    g_small = small.capture()  # nothing of this size ran before
    small.out()
    small.run()
    want_small = small.out()
    g_big = big.capture()
    big.out()
    small.run()
    other = cuda.zeros((small.n, 3), device="cuda",
                       dtype=cuda.float32 if precision == "fp64" else cuda.float64)
    small.run(prec="mixed" if precision == "fp64" else "fp64", f=other)
    small.out()
    for case, g, want in ((big, g_big, want_big), (small, g_small, want_small)):
        g.replay()
        for got, w in zip(case.out(), want):
            assert np.array_equal(got, w)


# the lattice constant and its double on an odd and an even knot, exactly
# (dr = 1/256) or as the quotient rounds (dr = 0.005)
@pytest.mark.parametrize("a,dr", [(513 / 256, 1 / 256), (2.005, 0.005), (3.615, 0.005)])
@pytest.mark.parametrize("ntypes", [1, 3])
def test_eam_fit_pairs_on_knots(cuda, oracle, a, dr, ntypes):
    """Ideal simple-cubic snapshots (with vacancies, so that the densities
    differ) whose shells sit on spline knots, with coefficients that jump
    there: loss and gradient belong to the interval int(r / dr), as in the
    oracle (the bounds of the other FP64 fits)."""
    from tdmd_claude_b200 import Box, EamAlloy
    from tdmd_claude_b200 import workloads as W
    from tdmd_claude_b200.fitting import ForceMatch, eam_coeff_tensors, eam_table_meta
    rng = np.random.default_rng(ntypes)
    kw = {} if ntypes == 1 else dict(beta_f=(4.8, 5.0, 5.2), A_phi=(0.55, 0.60, 0.65),
                                     E_F=(1.1, 1.2, 1.3))
    t = W.analytic_eam(nr=int(round(5.0 / dr)) + 1, **kw)
    assert abs(t.dr - dr) < 1e-15
    eam = EamAlloy.from_tables(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F, t.rho, t.rphi)
    oe = oracle.OracleEam(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F, t.rho, t.rphi)
    m = int(10.0 / a) + 1
    x = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3) * a
    pos = np.stack([rng.permutation(x)[:-9] for _ in range(2)])
    types = rng.integers(1, ntypes + 1, size=pos.shape[:2]).astype(np.int32)
    tgt = rng.normal(0.0, 0.3, size=pos.shape)
    fm = ForceMatch(pos, types, Box.make((0,) * 3, (m * a,) * 3), t.cutoff, "fp64")
    fm.set_targets(tgt)
    F, rho, phi = eam_coeff_tensors(eam)
    for kind, c in ((1, rho), (2, phi)):
        c *= _dev(cuda, 1.0 + 0.1 * rng.normal(size=c.shape))
        for k in range(len(c)):
            oe.set_coeffs(kind, k, c[k].cpu().numpy())
    loss = cuda.zeros(1, dtype=cuda.float64, device="cuda")
    g = [cuda.empty_like(v) for v in (F, rho, phi)]
    fm.eam(eam_table_meta(eam), F, rho, phi, loss, *g)
    lo, *want = oe.fm_loss_grad(pos, types, (0,) * 3, (m * a,) * 3, tgt)
    assert abs(loss.item() - lo) <= 1e-10 * lo
    for got, ref in zip(g, want):
        for sp in range(ref.shape[0]):
            assert np.abs(got[sp].cpu().numpy() - ref[sp]).max() <= 1e-9 * np.abs(ref[sp]).max()


def test_fit_divides_by_the_radius_once(cuda):
    """Snapshots of two atoms, one pair to an interval, all coefficients zero:
    the gradient of phi's b is a single quotient (G_i - G_j) . d / r, and
    every one has the bits of the division."""
    from tdmd_claude_b200 import Box
    from tdmd_claude_b200.fitting import ForceMatch
    rng = np.random.default_rng(12)
    nsnap, nr, dr = 300, 2001, 0.0025
    k = 5 * np.arange(nsnap) + 500
    pos = np.full((nsnap, 2, 3), 6.0)
    pos[:, 1, 0] += (k + rng.uniform(0.1, 0.9, nsnap)) * dr
    tgt = rng.normal(size=pos.shape)
    fm = ForceMatch(pos, np.ones((nsnap, 2), np.int32), Box.make((0,) * 3, (20.0,) * 3), 5.0,
                    "fp64")
    fm.set_targets(tgt)
    z = [cuda.zeros((1, 4 * (nr - 1)), dtype=cuda.float64, device="cuda") for _ in range(3)]
    g = [cuda.empty_like(v) for v in z]
    loss = cuda.zeros(1, dtype=cuda.float64, device="cuda")
    fm.eam(dict(ntypes=1, nrho=nr, drho=0.01, nr=nr, dr=dr), *z, loss, *g)
    c = 1.0 / (3.0 * 2 * nsnap)
    G = (2.0 * c) * (0.0 - tgt[:, :, 0])
    d = pos[:, 0, 0] - pos[:, 1, 0]
    want = np.zeros(nr - 1)
    want[k] = -(((G[:, 0] - G[:, 1]) * d) / np.abs(d))
    assert np.array_equal(g[2].cpu().numpy()[0, nr - 1:2 * (nr - 1)], want)


def _pair_eam(torch, eam, r, precision):
    """(density, x force of atom 0) of two atoms r apart."""
    from tdmd_claude_b200 import Box, DeviceEam
    de = DeviceEam()
    de.upload_tables(eam)
    f = torch.zeros((2, 3), device="cuda",
                    dtype=torch.float64 if precision == "fp64" else torch.float32)
    rho = torch.zeros(2, dtype=torch.float64, device="cuda")
    nbr, off, cnt = (_dev(torch, np.array(x, np.int32)) for x in ([1, 0], [0, 1], [1, 1]))
    out = []
    for x in r:
        de.compute(_dev(torch, np.array([[0.0, 1.0, 2.0], [x, 1.0, 2.0]])), f,
                   _dev(torch, np.ones(2, np.int32)), nbr.data_ptr(), off.data_ptr(),
                   cnt.data_ptr(), 2, Box.make((-10.0,) * 3, (22.0,) * 3), d_rho=rho,
                   precision=precision)
        assert float(f[0, 0]) == -float(f[1, 0])
        out.append((rho.cpu().numpy().copy(), float(f[0, 0])))
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_eam_table_of_ten_million_knots(cuda, precision):
    """Distances on both sides of 2^22 knots, where an FP32 sum with 1.5 * 2^23
    stops being spaced by one, and of 2^23, past FP32 intervals: density and force of smooth
    functions (FP32 distance, product and sum roundings: 1e-6 and 3e-6)."""
    from tdmd_claude_b200 import EamAlloy
    nr, dr = 10_000_001, 5e-7
    x = np.arange(nr) * dr
    F = -0.5 * np.arange(100) * 0.1  # F' = -1/2
    eam = EamAlloy.from_tables(1, 100, 0.1, nr, dr, 5.0, F[None], np.exp(-x)[None],
                               (x * np.exp(-2 * x))[None])
    rs = [1.5, (2 ** 22 - 3) * dr, (2 ** 22 + 3.5) * dr, 2.9, (2 ** 23 - 3) * dr,
          (2 ** 23 + 3.5) * dr, 4.5, 4.9]
    for r, (rho, fx) in zip(rs, _pair_eam(cuda, eam, rs, precision)):
        assert np.abs(rho / np.exp(-r) - 1).max() <= 1e-6
        want = -2 * np.exp(-2 * r) + np.exp(-r)  # phi' + 2 F' rho', on atom 0 along +x
        assert abs(fx - want) <= 3e-6 * np.exp(-r)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ntypes", [1, 2])
def test_wide_table_windows(cuda, precision, ntypes):
    """Windows, energies and replicas with a table of 2^22 + 2 knots equal
    those with one of 2000 knots of the same functions, to the coarse table's
    interpolation and twice the mixed bound: 3e-5 of the largest force (1e-5
    from the batch, which sums in another order)."""
    from tdmd_claude_b200 import Box, EamAlloy, FastPipelineScheduler, ReplicaBatch, make_config
    from tdmd_claude_b200 import workloads as W
    rng = np.random.default_rng(2)
    x = W.fcc_lattice(4, 4, 4, 3.615)
    x = (x + rng.normal(0, 0.05, x.shape)) % (4 * 3.615)
    n, box = len(x), Box.make((0,) * 3, (4 * 3.615,) * 3)
    types = rng.integers(1, ntypes + 1, n).astype(np.int32)
    masses = np.array([1.0] + [63.546] * ntypes)
    kw = {} if ntypes == 1 else dict(beta_f=(4.8, 5.2), A_phi=(0.55, 0.65), E_F=(1.1, 1.3))
    out = []
    for nr in (2000, 2 ** 22 + 2):
        t = W.analytic_eam(nr=nr, **kw)
        eam = EamAlloy.from_tables(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F, t.rho,
                                   t.rphi)
        cfg = make_config(r_skin=0.3, precision=precision, energy_every=4, lanes_per_atom=8)
        s = FastPipelineScheduler(box, n, eam, cfg)
        s.upload(x, np.zeros((n, 3)), None, types, None, masses)
        b = ReplicaBatch([box] * 2, [n, n], eam, cfg)
        b.upload(np.concatenate([x, x]), np.zeros((2 * n, 3)), np.concatenate([types] * 2), masses)
        for m in (s, b):
            m.run_until(11)
        pe, ke, w = s.energies()
        bpe, bke = b.energies()
        f = s.download().forces
        assert np.abs(b.download()[2][:n] - f).max() <= 1e-5 * np.abs(f).max()
        assert np.allclose(bpe, pe, rtol=1e-6) and np.allclose(bke, ke, rtol=1e-4)
        out.append((f, pe, w))
    (f0, e0, w0), (f1, e1, w1) = out
    assert np.abs(f1 - f0).max() <= 3e-5 * np.abs(f0).max()
    assert np.allclose(e1, e0, rtol=1e-6) and np.abs(w1 - w0).max() <= 1e-4 * np.abs(w0).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_eam_cutoff_far_beyond_the_table(cuda, precision):
    """A table of ten knots that ends 2^32 spacings before the pair: the last
    cubic goes on (exact straight lines here)."""
    from tdmd_claude_b200 import EamAlloy
    nr, dr = 10, 2.0 ** -33
    k = np.arange(nr, dtype=float)
    eam = EamAlloy.from_samples(1, nr, 1.0, nr, dr, 5.0, k[None], k[None], 3 * k[None])
    for r, (rho, fx) in zip((2.5, 0.75), _pair_eam(cuda, eam, (2.5, 0.75), precision)):
        assert np.allclose(rho, r / dr, rtol=1e-6)
        assert np.allclose(fx, (3 + 2) / dr, rtol=1e-6)


# a Morse force whose two exponentials overflow together, and two atoms so close
# that r^2 underflows
@pytest.mark.parametrize("alpha,d", [(400.0, (1.1, -1.2, 1.3)), (1.4, (1e-170, -1e-171, 1e-170))])
def test_infinite_forces_keep_their_sign(cuda, alpha, d):
    """FP64 pair forces beyond the range are infinities of the sign that the
    division gives, not NaN."""
    from tdmd_claude_b200 import Box, MorseParams, compute_morse_gpu
    pos = np.array([[0.0, 0.0, 0.0], d])
    f = cuda.zeros((2, 3), dtype=cuda.float64, device="cuda")
    nbr, off, cnt = (_dev(cuda, np.array(x, np.int32)) for x in ([1, 0], [0, 1], [1, 1]))
    compute_morse_gpu(_dev(cuda, pos), f, nbr.data_ptr(), off.data_ptr(), cnt.data_ptr(), 2,
                      Box.make((-10.0,) * 3, (10.0,) * 3), MorseParams.make(0.3, alpha, 3.0, 5.0))
    want = np.sign(pos[0] - pos[1]) * np.inf  # repulsive
    assert np.array_equal(f.cpu().numpy(), [want, -want])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_fused_batch_window_overflow(cuda, precision):
    """Two Morse gases that drift to their centres overflow the padded rows of
    a fused graph window (odd and even lengths): the window is done again from
    its start, with the bits of unfused windows whose rows overflow as well,
    and of a single system."""
    from tdmd_claude_b200 import (Box, FastPipelineScheduler, MorseParams, ReplicaBatch,
                                  make_config)
    rng = np.random.default_rng(3)
    L, n = 30.0, 300
    x = rng.uniform(0, L, size=(n, 3))
    v, types, masses = 15.0 - x, np.ones(n, np.int32), np.array([1.0, 63.546])
    boxes, p = [Box.make((0,) * 3, (L,) * 3)] * 2, MorseParams.make(0.01, 1.0, 3.0, 5.0)
    for windows in ((200,), (99, 200)):
        out = []
        for graphs in (True, False):
            cfg = make_config(r_skin=1.0, rebuild_every=5, dt=0.002, precision=precision,
                              lanes_per_atom=8, use_graphs=graphs)
            b = ReplicaBatch(boxes, [n, n], p, cfg)
            b.upload(np.concatenate([x, x]), np.concatenate([v, 0.9 * v]),
                     np.concatenate([types] * 2), masses)
            s = FastPipelineScheduler(boxes[0], n, p, cfg)
            s.upload(x, v, None, types, None, masses)
            for t in windows:
                b.run_until(t)
                s.run_until(t)
            assert b.stats().nlist_retries >= 1 and s.stats().nlist_retries >= 1
            st = s.download()
            out.append((b.download(), (st.positions, st.velocities, st.forces)))
        (gb, gs), (ub, us) = out
        for i in range(3):
            assert np.array_equal(gb[i], ub[i]) and np.array_equal(gs[i], us[i])
        for i in range(2):
            assert np.array_equal(gb[i][:n], gs[i])
