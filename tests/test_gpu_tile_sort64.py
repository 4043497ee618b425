"""FP64 tile sorts at the sizes where their rules switch: keys and permutation bit-exact (a stable sort
by tile), long-range forces against the oracle within the FP64 tests' tolerance (1e-8).

* 96 chunks of 256 particles and fewer: scan, scatter and tile sort as one kernel; above, three kernels;
* up to 2,048 particles per tile in shared memory (ordinary and full tiles, 2,048 exactly), above that
  laid out by index ranges in global memory (2,049, a few thousand, most of the system in one tile);
* indices scattered over the tiles, in the order of the tiles, and a tile of one far index.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from esp_hoomd_b200 import native, tables  # noqa: E402
from esp_hoomd_b200._lib import ESP_LONG_RANGE  # noqa: E402
from oracle import esp_ref as R  # noqa: E402

L = 10.0


def _positions(n, mesh, layout):
    rng = np.random.default_rng(n + mesh)
    pos = rng.uniform(0, L, (n, 3))
    if layout == "ordered":
        key, _ = R.bin_sort(pos, (L,) * 3, (mesh,) * 3, 6, 11)
        pos = pos[np.argsort(key, kind="stable")]
    elif layout == "far":  # one tile of neighbouring indices and the last one
        pos[:] = rng.uniform(0.62 * L, L, (n, 3))
        pos[:3000] = rng.uniform(0.15 * L, 0.25 * L, (3000, 3))
        pos[-1] = 0.2 * L
    elif layout.startswith("one-"):  # that many particles in one tile, no other particle near it
        k = int(layout[4:])
        pos[:] = rng.uniform(0.62 * L, L, (n, 3))
        pos[rng.permutation(n)[:k]] = rng.uniform(0.15 * L, 0.25 * L, (k, 3))
    return pos


@pytest.mark.parametrize("n,mesh,layout", [
    # three kernels: more than 96 chunks
    (24577, 36, "any"), (25000, 24, "any"), (25000, 24, "ordered"), (30000, 12, "any"), (30000, 12, "ordered"),
    (25000, 36, "one-2048"), (25000, 36, "one-2049"), (25000, 36, "far"),
    # one kernel
    (24576, 36, "any"), (24576, 24, "any"), (24576, 24, "ordered"), (6000, 12, "any"),
    (5000, 36, "one-2048"), (5000, 36, "one-2049"), (5000, 36, "far"),
])
def test_fp64_tile_sort(n, mesh, layout, monkeypatch):
    # the oracle's mesh stages read float32 positions: here it takes them as they are
    monkeypatch.setattr(R, "grid_coords", lambda x, box, m: np.asarray(x) * (np.asarray(m) / np.asarray(box)))
    pos = _positions(n, mesh, layout)
    q = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    ctx = native.Context(native.make_params(order=6, mesh=(mesh,) * 3, precision=1), (L,) * 3, n)
    inf = ctx.info()
    assert inf["tile"] == 11
    p4 = torch.zeros((n, 4), dtype=torch.float64, device="cuda")
    p4[:, :3] = torch.as_tensor(pos, device="cuda")
    force = torch.zeros_like(p4)
    for _ in range(2):  # the second finds the tile counts clear
        ctx.compute_f64(p4, torch.as_tensor(q, device="cuda"), force, flags=ESP_LONG_RANGE)
    key, perm = (t.cpu().numpy().astype(np.uint32) for t in ctx.sort_state(n))
    ref, _ = R.bin_sort(pos, (L,) * 3, (mesh,) * 3, 6, 11)
    assert np.array_equal(key, ref)
    if layout.startswith("one-"):
        assert np.bincount(ref).max() >= int(layout[4:]) and int(layout[4:]) in np.bincount(ref)
    assert np.array_equal(perm, np.argsort(ref, kind="stable").astype(np.uint32))
    prm = tables.ESPParams(mesh=(mesh,) * 3, box=(L,) * 3, rcut=inf["rcut"],
                           split=tables.make_split(inf["c_split"], tol=1e-12),
                           window=tables.window_cached(inf["order"], inf["c_window"], inf["window_degree"]))
    empty = (np.zeros(n, np.uint32), np.zeros(n, np.uint32), np.zeros(0, np.uint32))
    _, F, _ = R.esp(pos, q, prm, nlist=empty)
    assert R.rel_rms(force.cpu().numpy()[:, :3], F) <= 1e-8
