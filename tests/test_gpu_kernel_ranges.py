"""Kernels whose launch shape or algorithm depends on the size, at the sizes
where the rule switches, against the oracle.

* Lennard-Jones term: a warp per particle up to 37 chunks of 256 particles,
  8 lanes above; against a numpy sum over the same list (FP64: forces to
  1e-12 relative RMS, sums of ~100 terms; FP32: 2e-5, the rounding of a
  minimum-image displacement (L 2^-24 / r ~ 1.3e-6) amplified 14-fold by
  r^-14).
* neighbour rows (HOOMD layout and pair list): cells of half the list radius
  (few cells, or full ones) with 4 and >= 5 cells per axis and both at once and
  with more than 8 and more than 32 particles in a cell; cells of the list
  radius, sparse and 27,000 and 125,000 of them (scanned by 7 and 31 CTAs);
  capacities that are no multiple of 4, and more excluded partners than the
  kernel keeps in shared memory: the rows are the oracle's sets.
* tile shares: few tiles, their particles shared out over several CTAs, with
  full, nearly empty and empty tiles at once, supports 5..8 (the rotated walk
  of the interpolation) and 4 and 10; long-range forces against the oracle
  within the parity tests' FP32 tolerance (5e-6), and per-particle and total
  energies within what the potential's tolerance (5e-6 of the largest mesh
  value) and 1e-6 for the FP32 stencil sum leave of them: 0.5 |q| 6e-6
  max|phi| times the sum of the particle's weights.
* FP64 pair term: a warp per particle up to 148 chunks of 32 particles, 8 lanes
  above, with and without the virial, on the last size of the one and the first
  of the other; against the oracle within the FP64 tests' tolerances (forces
  1e-8, energy 1e-10, virial 2e-8, the oracle's own finite difference).
* overlapped starts (below 192 chunks of 256 particles) and accumulators left
  clear: two position sets in turn through one context with nothing waited for,
  and after a charge spread and a long-range-only call, give what a fresh
  context gives for each (FP32 1e-6 of the RMS force and of the energies'
  magnitudes, the order of the FP64 mesh sums seen through one FP32 rounding
  per stage; FP64 1e-12).
* one-kernel sort (small systems): tiles above the shared-memory capacity, FP32
  on both sides of its 64 chunks, FP64 (up to 96 chunks; its other side is in
  test_gpu_tile_sort64) below; long-range forces against the oracle (FP32 5e-6,
  FP64 1e-8).
* FFT passes with 256, 512 and 1,024 threads per plane or slab, one and three
  systems: forces, energy and virial against the oracle within the parity
  tests' FP32 tolerances (5e-6, 2e-6, 1e-5).
* tile sort: tiles of a few particles, above the 512-thread switch, and above
  the shared-memory capacity (2,048); permutation bit-exact.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from esp_hoomd_b200 import native, systems, tables  # noqa: E402
from esp_hoomd_b200._lib import ESP_LONG_RANGE, ESP_SHORT_RANGE  # noqa: E402
from oracle import esp_ref as R  # noqa: E402


def _lj_numpy(pos, box, head, cnt, lst, eps, sig, rc):
    i = np.repeat(np.arange(len(cnt)), cnt)
    j = np.concatenate([lst[h:h + c] for h, c in zip(head, cnt)]).astype(np.int64)
    L = np.asarray(box)
    d = pos[i] - pos[j]
    d -= L * np.rint(d / L)
    r2 = (d * d).sum(1)
    ok = r2 < rc * rc
    i, d, r2 = i[ok], d[ok], r2[ok]
    s6 = (sig * sig / r2) ** 3
    f = (24 * eps * (2 * s6 * s6 - s6) / r2)[:, None] * d
    F = np.stack([np.bincount(i, f[:, k], len(pos)) for k in range(3)], 1)
    e = np.bincount(i, 2 * eps * (s6 * s6 - s6), len(pos))
    return F, e


@pytest.mark.parametrize("shape", [(7, 7, 7), (10, 10, 10), (22, 22, 20)])
@pytest.mark.parametrize("f64", [False, True])
def test_lj_lane_counts(shape, f64):
    s = systems.rocksalt(0, seed=sum(shape), shape=shape)
    s.pos = s.pos.astype(np.float32).astype(np.float64)
    head, cnt, lst = R.neighbor_list(s.pos, s.box, 3.4)
    b = native.Batch(native.make_params(precision=int(f64)), [s.N], [s.box])
    dt = torch.float64 if f64 else torch.float32
    pos = torch.zeros((s.N, 4), dtype=dt, device="cuda")
    pos[:, :3] = torch.as_tensor(s.pos, device="cuda")
    nl = tuple(torch.as_tensor(a.astype(np.int32), device="cuda") for a in (head, cnt, lst))
    force = torch.ones((s.N, 4), dtype=dt, device="cuda")  # the term is added
    energy = torch.zeros(1, dtype=torch.float64, device="cuda")
    b.lj(pos, nl, 1.0, 0.9, 2.5, force, energy)
    F, e = _lj_numpy(s.pos, s.box, head, cnt, lst, 1.0, 0.9, 2.5)
    f = force.double().cpu().numpy() - 1.0
    tol = 1e-12 if f64 else 2e-5
    assert R.rel_rms(f[:, :3], F) <= tol
    assert np.abs(f[:, 3] - e).max() <= 10 * tol * np.abs(e).max()
    assert abs(energy.item() - e.sum()) <= 10 * tol * np.abs(e).sum()


@pytest.mark.parametrize("n,mesh", [(400, 24), (3000, 12), (6000, 12), (20000, 24)])
def test_tile_sort_bit_exact(n, mesh):
    rng = np.random.default_rng(n)
    L = 10.0
    pos = rng.uniform(0, L, (n, 3)).astype(np.float32).astype(np.float64)
    ctx = native.Context(native.make_params(order=6, mesh=(mesh,) * 3), (L, L, L), n)
    p4 = torch.zeros((n, 4), device="cuda")
    p4[:, :3] = torch.as_tensor(pos, device="cuda")
    q = torch.as_tensor(rng.choice([-1.0, 1.0], n), dtype=torch.float32, device="cuda")
    ctx.spread(p4, q)
    key, perm = ctx.sort_state(n)
    inf = ctx.info()
    k_ref, p_ref = R.bin_sort(pos, (L, L, L), (mesh,) * 3, inf["order"], inf["tile"])
    assert np.array_equal(key.cpu().numpy().astype(np.uint32), k_ref)
    assert np.array_equal(perm.cpu().numpy().astype(np.uint32), p_ref)


def _rows(head, cnt, lst):
    return [sorted(lst[h:h + c].tolist()) for h, c in zip(head, cnt)]


def _check_lists(pos, box, rlist, cap, excl=None):
    pos = pos.astype(np.float32).astype(np.float64)
    n = len(pos)
    b = native.Batch(native.make_params(rcut=rlist, mesh=(16, 16, 16)), [n], [box])
    p4 = torch.zeros((n, 4), device="cuda")
    p4[:, :3] = torch.as_tensor(pos, device="cuda")
    if excl is not None:
        b.set_exclusions(torch.as_tensor(excl[0].astype(np.int32), device="cuda"),
                         torch.as_tensor(excl[1].astype(np.int32), device="cuda"), excl[2])
    head = torch.zeros(n, dtype=torch.int32, device="cuda")
    nn = torch.zeros_like(head)
    nl = torch.zeros(n * cap, dtype=torch.int32, device="cuda")
    b.build_nlist(p4, rlist, cap, head, nn, nl)
    b.nlist_check()
    ref = R.neighbor_list(pos, box, rlist)
    if excl is not None:
        ref = R.remove_pairs(ref, *excl)
    got = tuple(t.cpu().numpy() for t in (head, nn, nl))
    assert np.array_equal(got[1], ref[1].astype(np.int32))
    assert _rows(*got) == _rows(ref[0], ref[1], ref[2])
    # the pair list holds the same pairs: equal forces up to the summation order
    q = torch.as_tensor(np.where(np.arange(n) % 2 == 0, 1.0, -1.0), dtype=torch.float32, device="cuda")
    f = [torch.zeros((n, 4), device="cuda") for _ in range(2)]
    b.compute(p4, q, f[0], nlist=(head, nn, nl), flags=ESP_SHORT_RANGE)
    b.build_pairlist(p4, rlist, cap)
    b.pairlist_check()
    b.compute(p4, q, f[1], flags=ESP_SHORT_RANGE)
    a, c = (x.double().cpu().numpy()[:, :3] for x in f)
    assert R.rel_rms(c, a) <= 1e-6


@pytest.mark.parametrize("box,n,rlist,cap", [
    ((7.0, 7.3, 8.4), 400, 3.4, 253),     # 4 cells on every axis
    ((7.5, 12.0, 31.0), 2500, 3.0, 256),  # 5 cells on one axis, more on the others
    ((6.2, 20.0, 20.0), 2000, 3.0, 256),  # 4 cells on one axis only
    ((9.0, 9.0, 9.0), 6000, 2.0, 512),    # 8 particles per cell and more
    ((40.0, 40.0, 40.0), 300, 1.5, 16),   # a cell holds a particle rarely: cells enlarged
    ((60.0, 60.0, 60.0), 20000, 2.0, 64),  # 27,000 cells of the list radius
])
def test_neighbour_rows(box, n, rlist, cap):
    rng = np.random.default_rng(n)
    _check_lists(rng.uniform(0, 1, (n, 3)) * np.asarray(box), box, rlist, cap)


def test_neighbour_rows_of_many_cells():
    rng = np.random.default_rng(125)
    _check_lists(rng.uniform(0, 100.0, (20000, 3)), (100.0, 100.0, 100.0), 2.0, 16)


def test_neighbour_rows_of_a_dense_cell():
    rng = np.random.default_rng(9)
    pos = np.concatenate([rng.uniform(0, 20.0, (1000, 3)), rng.uniform(5.0, 6.5, (300, 3))])
    _check_lists(pos, (20.0, 20.0, 20.0), 3.0, 600)


@pytest.mark.parametrize("per_mol", [2, 9, 12])  # 1, 8 and 11 excluded partners
@pytest.mark.parametrize("n_mol,L", [(60, 9.0), (900, 28.0)])  # both row kernels
def test_neighbour_rows_exclusions(per_mol, n_mol, L):
    rng = np.random.default_rng(per_mol)
    pos = np.mod(np.repeat(rng.uniform(0, L, (n_mol, 3)), per_mol, 0) + rng.normal(0, 0.3, (n_mol * per_mol, 3)), L)
    _check_lists(pos, (L, L, L), 2.0, 256, R.molecule_exclusions(n_mol, per_mol))


@pytest.mark.parametrize("order", [4, 5, 6, 7, 8, 10])
@pytest.mark.parametrize("n", [37, 700])
def test_tile_shares(order, n):
    rng = np.random.default_rng(order * 1000 + n)
    L = 10.0
    pos = rng.uniform(0, L, (n, 3))
    pos[: 3 * n // 4] = rng.uniform(0, 3.0, (3 * n // 4, 3))  # most of them in one tile
    pos = pos.astype(np.float32).astype(np.float64)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    ctx = native.Context(native.make_params(order=order, mesh=(24, 24, 24)), (L, L, L), n)
    inf = ctx.info()
    p4 = torch.zeros((n, 4), device="cuda")
    p4[:, :3] = torch.as_tensor(pos, device="cuda")
    force = torch.zeros((n, 4), device="cuda")
    ctx.compute(p4, torch.as_tensor(q, dtype=torch.float32, device="cuda"), force, flags=ESP_LONG_RANGE)
    prm = tables.ESPParams(mesh=(24, 24, 24), box=(L, L, L), rcut=inf["rcut"],
                           split=tables.split_cached(inf["c_split"]),
                           window=tables.window_cached(inf["order"], inf["c_window"], inf["window_degree"]))
    empty = (np.zeros(n, np.uint32), np.zeros(n, np.uint32), np.zeros(0, np.uint32))
    _, F, _ = R.esp(pos, q, prm, nlist=empty)
    assert R.rel_rms(force.double().cpu().numpy()[:, :3], F) <= 5e-6


@pytest.mark.parametrize("order", [4, 5, 6, 7, 8, 10])
@pytest.mark.parametrize("n", [37, 700])
def test_tile_shares_energies(order, n):
    rng = np.random.default_rng(order * 1000 + n)
    L = 10.0
    pos = rng.uniform(0, L, (n, 3))
    pos[: 3 * n // 4] = rng.uniform(0, 3.0, (3 * n // 4, 3))  # most of them in one tile
    pos = pos.astype(np.float32).astype(np.float64)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    ctx = native.Context(native.make_params(order=order, mesh=(24, 24, 24)), (L, L, L), n)
    inf = ctx.info()
    p4 = torch.zeros((n, 4), device="cuda")
    p4[:, :3] = torch.as_tensor(pos, device="cuda")
    force = torch.zeros((n, 4), device="cuda")
    energy = torch.zeros(1, dtype=torch.float64, device="cuda")
    ctx.compute(p4, torch.as_tensor(q, dtype=torch.float32, device="cuda"), force, energy, flags=ESP_LONG_RANGE)
    prm = tables.ESPParams(mesh=(24, 24, 24), box=(L, L, L), rcut=inf["rcut"],
                           split=tables.split_cached(inf["c_split"]),
                           window=tables.window_cached(inf["order"], inf["c_window"], inf["window_degree"]))
    empty = (np.zeros(n, np.uint32), np.zeros(n, np.uint32), np.zeros(0, np.uint32))
    E, _, _, parts = R.esp(pos, q, prm, nlist=empty, return_parts=True)
    e = 0.5 * q * parts["pot"] + R.self_energy(q, prm) / (q * q).sum() * q * q
    _, t = R.stencil_origin(R.grid_coords(pos, prm.box, prm.mesh), order)
    weights = np.prod([prm.window.weights(t[:, d]).sum(1) for d in range(3)], 0)
    tol = 0.5 * np.abs(q) * 6e-6 * np.abs(parts["phi"]).max() * weights
    assert (np.abs(force.double().cpu().numpy()[:, 3] - e) <= tol).all()
    assert abs(energy.item() - E) <= tol.sum()


@pytest.mark.parametrize("shape", [(16, 16, 18), (18, 17, 16)])  # 4,608 and 4,896 ions
@pytest.mark.parametrize("virial", [False, True])
def test_fp64_pair_lane_counts(shape, virial):
    s = systems.rocksalt(0, seed=sum(shape), shape=shape)
    s.pos = s.pos.astype(np.float32).astype(np.float64)
    nlist = R.neighbor_list(s.pos, s.box, 3.0)
    ctx = native.Context(native.make_params(mesh=(32, 32, 32), precision=1), s.box, s.N)
    inf = ctx.info()
    pos = torch.zeros((s.N, 4), dtype=torch.float64, device="cuda")
    pos[:, :3] = torch.as_tensor(s.pos, device="cuda")
    nl = tuple(torch.as_tensor(a.astype(np.int32), device="cuda") for a in nlist)
    force = torch.zeros_like(pos)
    energy = torch.zeros(1, dtype=torch.float64, device="cuda")
    w = torch.zeros(6, dtype=torch.float64, device="cuda") if virial else None
    ctx.compute_f64(pos, torch.as_tensor(s.q, dtype=torch.float64, device="cuda"), force, energy, w, nlist=nl)
    prm = tables.ESPParams(mesh=(32, 32, 32), box=tuple(s.box), rcut=inf["rcut"],
                           split=tables.make_split(inf["c_split"], tol=1e-12),
                           window=tables.window_cached(inf["order"], inf["c_window"], inf["window_degree"]))
    E, F, W = R.esp(s.pos, s.q, prm, nlist=nlist)
    assert R.rel_rms(force.cpu().numpy()[:, :3], F) <= 1e-8
    assert abs(energy.item() - E) <= 1e-10 * abs(E)
    if virial:
        assert np.abs(w.cpu().numpy() - W).max() <= 2e-8 * np.abs(W).max()


@pytest.mark.parametrize("shape", [(8, 8, 8), (18, 20, 22), (36, 36, 38)])  # 2, 31 and 193 chunks
@pytest.mark.parametrize("f64", [False, True])
def test_back_to_back_evaluations(shape, f64):
    dt = torch.float64 if f64 else torch.float32
    par = native.make_params(mesh=(30, 32, 36), precision=int(f64))
    sets = []
    for seed in (1, 2):
        s = systems.rocksalt(0, seed=seed, shape=shape)
        p4 = torch.zeros((s.N, 4), dtype=dt, device="cuda")
        p4[:, :3] = torch.as_tensor(s.pos, device="cuda")
        nl = tuple(torch.as_tensor(a.astype(np.int32), device="cuda") for a in R.neighbor_list(s.pos, s.box, 3.0))
        sets.append((p4, torch.as_tensor(s.q, dtype=dt, device="cuda"), nl))

    def run(ctx, p4, q, nl, **kw):
        f, e = torch.zeros_like(p4), torch.zeros(1, dtype=torch.float64, device="cuda")
        (ctx.compute_f64 if f64 else ctx.compute)(p4, q, f, e, nlist=nl, **kw)
        return f, e

    want = []
    for a in sets:
        want.append(run(native.Context(par, s.box, s.N), *a))
        torch.cuda.synchronize()
    ctx = native.Context(par, s.box, s.N)
    got = []
    for k in range(6):
        if k == 3:
            run(ctx, *sets[0][:2], None, flags=ESP_LONG_RANGE)
            if not f64:
                ctx.spread(*sets[1][:2])
        got.append([run(ctx, *a) for a in sets])
    torch.cuda.synchronize()
    tol = 1e-12 if f64 else 1e-6
    for pair in got:
        for (f, e), (F, E) in zip(pair, want):
            assert R.rel_rms(f.double().cpu().numpy()[:, :3], F.double().cpu().numpy()[:, :3]) <= tol
            assert abs(e.item() - E.item()) <= tol * F[:, 3].double().abs().sum().item()


@pytest.mark.parametrize("n,mesh", [(400, 24), (4200, 24), (6000, 12), (16384, 24), (16640, 24)])
@pytest.mark.parametrize("f64", [False, True])
def test_one_kernel_sort(n, mesh, f64):
    # long-range forces through the sort of a whole evaluation: one kernel up to
    # 64 chunks in FP32 (the last size is above) and 96 in FP64; the third size
    # has tiles above 2,048 particles
    rng = np.random.default_rng(n)
    L = 10.0
    pos = rng.uniform(0, L, (n, 3)).astype(np.float32).astype(np.float64)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    dt = torch.float64 if f64 else torch.float32
    ctx = native.Context(native.make_params(order=6, mesh=(mesh,) * 3, precision=int(f64)), (L, L, L), n)
    inf = ctx.info()
    p4 = torch.zeros((n, 4), dtype=dt, device="cuda")
    p4[:, :3] = torch.as_tensor(pos, device="cuda")
    force = torch.zeros_like(p4)
    run = ctx.compute_f64 if f64 else ctx.compute
    for _ in range(2):  # the second finds the tile counts clear
        run(p4, torch.as_tensor(q, dtype=dt, device="cuda"), force, flags=ESP_LONG_RANGE)
    split = tables.make_split(inf["c_split"], tol=1e-12) if f64 else tables.split_cached(inf["c_split"])
    prm = tables.ESPParams(mesh=(mesh,) * 3, box=(L, L, L), rcut=inf["rcut"], split=split,
                           window=tables.window_cached(inf["order"], inf["c_window"], inf["window_degree"]))
    empty = (np.zeros(n, np.uint32), np.zeros(n, np.uint32), np.zeros(0, np.uint32))
    _, F, _ = R.esp(pos, q, prm, nlist=empty)
    assert R.rel_rms(force.double().cpu().numpy()[:, :3], F) <= (1e-8 if f64 else 5e-6)


@pytest.mark.parametrize("mesh,copies", [((16, 18, 20), 1), ((20, 24, 30), 1), ((64, 60, 72), 1), ((64, 60, 72), 3),
                                         ((128, 120, 27), 1)])
def test_fft_block_sizes(mesh, copies):
    s = systems.rocksalt(8, seed=sum(mesh))
    s.pos = s.pos.astype(np.float32).astype(np.float64)
    nlist = R.neighbor_list(s.pos, s.box, 3.0)
    b = native.Batch(native.make_params(mesh=mesh), [s.N] * copies, [s.box] * copies)
    inf = native.Context(native.make_params(mesh=mesh), s.box, s.N).info()
    pos = torch.zeros((s.N * copies, 4), device="cuda")
    pos[:, :3] = torch.as_tensor(np.tile(s.pos, (copies, 1)), device="cuda")
    q = torch.as_tensor(np.tile(s.q, copies), dtype=torch.float32, device="cuda")
    head = np.concatenate([nlist[0] + k * len(nlist[2]) for k in range(copies)])
    nl = tuple(torch.as_tensor(a.astype(np.int32), device="cuda")
               for a in (head, np.tile(nlist[1], copies), np.tile(nlist[2], copies)))
    force = torch.zeros_like(pos)
    energy = torch.zeros(copies, dtype=torch.float64, device="cuda")
    w = torch.zeros((copies, 6), dtype=torch.float64, device="cuda")
    b.compute(pos, q, force, energy, w, nlist=nl)
    prm = tables.ESPParams(mesh=mesh, box=tuple(s.box), rcut=inf["rcut"], split=tables.split_cached(inf["c_split"]),
                           window=tables.window_cached(inf["order"], inf["c_window"], inf["window_degree"]))
    E, F, W = R.esp(s.pos, s.q, prm, nlist=nlist)
    f = force.double().cpu().numpy().reshape(copies, s.N, 4)
    for k in range(copies):
        assert R.rel_rms(f[k, :, :3], F) <= 5e-6
        assert abs(energy[k].item() - E) <= 2e-6 * abs(E)
        assert np.abs(w[k].cpu().numpy() - W).max() <= 1e-5 * np.abs(W).max()
