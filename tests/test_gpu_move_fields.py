"""Compaction at the edges of its tiles and of its two offset forms: every
field of every slot against the stable order formed on the host."""
from __future__ import annotations

import numpy as np
import pytest

from flexpart_gpu import api
from flexpart_gpu.records import FIELDS

pytestmark = pytest.mark.gpu


def _expected(flags, values, n):
    alive = np.flatnonzero(flags & 1)
    out = values.copy()
    out[:alive.size] = values[alive]
    cleared = flags.copy()
    cleared[:alive.size] = flags[alive]
    cleared[alive.size:] &= ~np.uint32(1)
    return alive, out, cleared


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 2047, 2048, 2049, 6 * 2048 + 3])
@pytest.mark.parametrize("dead", [0.0, 0.4, 1.0])
def test_compaction_moves_every_field_in_slot_order(n, dead):
    ctx = api.Context(0)
    rng = np.random.default_rng(n + int(10 * dead))
    p = api.Particles(ctx, n)
    host = {}
    for name, dt in FIELDS:
        host[name] = rng.integers(1, 1 << 20, n).astype(dt)
    host["flags"] = np.where(rng.random(n) < dead, 6, 7).astype(np.uint32)
    for name, _ in FIELDS:
        p.write_field(name, host[name])
    c = api.Compaction(ctx, n)
    for indices in (None, api.DeviceArray(ctx, n, np.uint32)):   # with and without the caller's index array
        count = c.compact(p, indices)
        alive, _, flags = _expected(host["flags"], host["pos_x"], n)
        assert count == alive.size == p.dispatch_count
        moved = {name: _expected(host["flags"], host[name], n)[1] for name, _ in FIELDS} | {"flags": flags}
        for name, _ in FIELDS:
            assert np.array_equal(p.read_field(name), moved[name]), name
        host = moved
        if indices is not None:
            assert np.array_equal(indices.numpy()[:count], np.arange(count))


@pytest.mark.parametrize("tiles", [8192, 8193])
def test_compaction_order_on_both_sides_of_the_scan_rule(tiles):
    n = tiles * 2048 - 5
    ctx = api.Context(0)
    rng = np.random.default_rng(tiles)
    p = api.Particles(ctx, n)
    flags = (rng.random(n) < 0.7).astype(np.uint32)
    ids = np.arange(n, dtype=np.int32)
    p.write_field("flags", flags)
    p.write_field("release_point", ids)
    count = api.Compaction(ctx, n).compact(p)
    alive, want, cleared = _expected(flags, ids, n)
    assert count == alive.size
    assert np.array_equal(p.read_field("release_point"), want)
    assert np.array_equal(p.read_field("flags"), cleared)
