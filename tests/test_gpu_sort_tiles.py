"""The reorder's radix sort at the edges of its tiles and passes: the
permutation against a stable host sort of the oracle's keys, with one to
three digits, presorted, reversed, equal and random keys."""
from __future__ import annotations

import numpy as np
import pytest

from flexpart_gpu import api
from helpers import population
from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 511, 4095, 4096, 4097, 8192, 3 * 4096 + 17, 1_060_000])
@pytest.mark.parametrize("shape", [(3, 5, 4), (40, 30, 12), (200, 150, 30)])     # 6, 14 and 20 key bits
@pytest.mark.parametrize("order", ["random", "equal", "reversed"])
def test_reorder_is_the_stable_order(n, shape, order):
    if n > 100_000 and (order != "random" or shape[0] != 200):
        pytest.skip("one large population is enough")
    ctx = api.Context(0)
    nx, ny, nz = shape
    rec = population(nx, ny, n, seed=n, z_max=2500.0, inactive_every=11 if n > 11 else 0)
    if order == "equal":
        for name in ("cell_x", "cell_y", "pos_x", "pos_y", "pos_z"):
            rec[name] = rec[name][0]
    elif order == "reversed":
        rec = rec[np.lexsort((rec["pos_z"], rec["cell_y"], rec["cell_x"]))][::-1].copy()
    rec["time"] = np.arange(n, dtype=np.int32)
    heights = (2000.0 * (np.arange(1, nz + 1) / nz) ** 2).astype(np.float32)
    m = api.Met(ctx, nx, ny, nz)
    m.set_level_heights(heights)
    p = api.Particles(ctx, n)
    p.upload(rec)
    perm = api.DeviceArray(ctx, n, np.uint32)
    sorter = api.Sorter(ctx, n)
    for _ in range(2):                                       # the second sorts what the first left
        ref, ref_perm = orc.sort_by_cell(rec, n, heights, shape)
        sorter.sort(p, m, perm)
        assert np.array_equal(perm.numpy(), ref_perm)
        assert np.array_equal(p.download(), ref)
        rec = ref
