"""The gridding kernels against a host sum of the same cells: sorted heights by
columns (one to eight levels), more by bisection, unsorted by the scan, over
populations from one column to one slot per column, with sizes around the
quads and passes of the kernel."""
from __future__ import annotations

import numpy as np
import pytest

from flexpart_gpu import api
from flexpart_gpu.records import PARTICLE_DTYPE

pytestmark = pytest.mark.gpu

HEIGHTS = {1: [900.0], 2: [100.0, 900.0], 5: [100.0, 500.0, 500.0, 2000.0, 5000.0],
           8: [50.0, 100.0, 200.0, 400.0, 800.0, 1600.0, 3200.0, 6400.0], 9: [100.0 * k for k in range(1, 10)],
           40: [60.0 * k for k in range(1, 41)]}


def _records(n, order, nx, ny, seed):
    rng = np.random.default_rng(seed)
    rec = np.zeros(n, PARTICLE_DTYPE)
    cells = {"column": np.full(n, 7), "sorted": np.sort(rng.integers(0, nx * ny, n)) // 3,
             "mixed": np.sort(rng.integers(0, nx * ny, n)), "random": rng.integers(0, nx * ny, n)}[order]
    if order == "mixed":                                  # neighbouring columns interleaved
        cells = cells ^ rng.integers(0, 4, n)
    rec["cell_x"], rec["cell_y"] = cells // ny, cells % ny
    rec["pos_z"] = rng.uniform(0, 7000, n)
    rec["flags"] = np.where(rng.random(n) < 0.15, 2, 3)
    rec["mass"][:, 0] = rng.uniform(0, 1e-2, n)
    if n > 300:
        rec["pos_z"][5:11] = [np.nan, np.inf, -np.inf, 100.0, 500.0, -3.0]
        rec["mass"][20:26, 0] = [np.nan, np.inf, -1.0, 1e30, 0.0, 5000.0]
        rec["cell_x"][30:33], rec["cell_y"][33:36] = [-4, nx, 10**6], [-1, ny, 10**6]
    return rec


@pytest.mark.parametrize("n", [1, 3, 4, 5, 127, 1023, 1024, 1025, 40_003, 700_001])
@pytest.mark.parametrize("order", ["column", "sorted", "mixed", "random"])
def test_grid_equals_the_host_sum(n, order):
    ctx = api.Context(0)
    nx, ny = 37, 23
    rec = _records(n, order, nx, ny, n)
    p = api.Particles(ctx, n)
    p.upload(rec)
    live = (rec["flags"] & 1) != 0
    ix, iy = np.clip(rec["cell_x"], 0, nx - 1).astype(np.int64), np.clip(rec["cell_y"], 0, ny - 1).astype(np.int64)
    m = np.fmax(rec["mass"][:, 0], np.float32(0)).astype(np.float32)
    scaled = m * np.float32(1e6) + np.float32(0.5)
    full = scaled >= np.float32(4294967295.0)
    q = np.where(m <= 0, 0.0, np.where(full, 0.0, scaled).astype(np.float64)).astype(np.uint64)
    q[full] = 0xFFFFFFFF
    for heights in (*HEIGHTS.values(), [500.0, 100.0, 2000.0]):
        nz = len(heights)
        h = np.asarray(heights, np.float32)
        below = rec["pos_z"][:, None] <= h[None, :]
        iz = np.where(below.any(1), below.argmax(1), nz - 1)
        cell = ((ix * ny + iy) * nz + iz)[live]
        counts = np.bincount(cell, minlength=nx * ny * nz).astype(np.uint32)
        mass = np.zeros(nx * ny * nz, np.uint64)
        np.add.at(mass, cell, q[live])
        grid = api.Grid(ctx, nx, ny, nz)
        grid.accumulate(p, 0, 1e6, h)
        got_counts, got_mass, _ = grid.download()
        assert np.array_equal(got_counts, counts), (nz, order)
        assert np.array_equal(got_mass, (mass & np.uint64(0xFFFFFFFF)).astype(np.uint32)), (nz, order)
