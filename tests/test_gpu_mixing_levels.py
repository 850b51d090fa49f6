"""The level search of convective mixing: columns that take the bucket table
and columns that are bisected, against the oracle's scan, bit for bit."""
import numpy as np
import pytest

from flexpart_gpu import api
from flexpart_gpu import convection as cv
from flexpart_gpu.records import PARTICLE_DTYPE
from oracle import orc

pytestmark = pytest.mark.gpu

COLUMNS = {
    "one": [0.0, 4000.0],
    "two": [10.0, 11.0, 9000.0],
    "uniform60": np.linspace(0.0, 20_000.0, 61),
    "offset": 1.0e6 + np.linspace(0.0, 64.0, 34),
    "stretched60": np.cumsum(np.r_[0.0, 20.0 * 1.12 ** np.arange(60)]),
    "edge": np.r_[0.0, np.linspace(1.0, 20.0, 8), 9000.0],          # eight levels in one bucket
    "crowded": np.r_[0.0, 1e-3 * 1.2 ** np.arange(60), 9000.0],     # bisected: many levels in the first bucket
    "many": np.linspace(-500.0, 500.0, 4001),                       # bisected: four levels a bucket
}


@pytest.mark.parametrize("name", COLUMNS)
def test_every_level_search_finds_the_scan_level(name):
    ctx = api.Context(0)
    iface = np.asarray(COLUMNS[name], np.float32)
    L = len(iface) - 1
    assert np.all(np.diff(iface) > 0)
    rng = np.random.default_rng(5)
    z = np.concatenate([iface, np.nextafter(iface, np.float32(np.inf)), np.nextafter(iface, np.float32(-np.inf)),
                        rng.uniform(iface[0] - 10, iface[-1] + 10, 20_001).astype(np.float32),
                        np.float32([np.nan, np.inf, -np.inf, 0.0, -0.0])])
    rec = np.zeros(len(z), PARTICLE_DTYPE)
    rec["pos_z"] = z
    rec["flags"] = 1
    rec["flags"][::7] = 0
    matrix = np.eye(L, dtype=np.float32).reshape(-1)
    p = api.Particles(ctx, len(z))
    p.upload(rec)
    cm = cv.ConvectiveMixing(ctx, L)
    cm.set_matrix(matrix, iface)
    cm.apply(p)
    assert p.download().tobytes() == orc.convective_mixing(rec, matrix, iface).tobytes()
