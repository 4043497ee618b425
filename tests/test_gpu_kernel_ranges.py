"""Kernels whose launch shape or algorithm depends on the size, at the sizes
where the rule switches, against the oracle.

* Lennard-Jones term: a warp per particle up to 37 chunks of 256 particles,
  8 lanes above; against a numpy sum over the same list (FP64: forces to
  1e-12 relative RMS, sums of ~100 terms; FP32: 2e-5, the rounding of a
  minimum-image displacement (L 2^-24 / r ~ 1.3e-6) amplified 14-fold by
  r^-14).
* tile sort: tiles of a few particles, above the 512-thread switch, and above
  the shared-memory capacity (2,048); permutation bit-exact.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from esp_hoomd_b200 import native, systems  # noqa: E402
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
