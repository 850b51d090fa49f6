"""Philox counters at the last value whose blocks do not carry out of the first
word, and past it, where the passes with a Philox head of their own fall back
to the full counter arithmetic: a batch scenario's and the fused CBL sampler's.
"""
import numpy as np
import pytest

from flexpart_gpu import api, cbl, synthetic
from flexpart_gpu import batch as bt
from helpers import population

pytestmark = pytest.mark.gpu

N = 1003
TOP = 2**32


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def test_batch_scenarios_at_the_carry(ctx):
    """Scenarios that reach the carry in different steps (a step uses 2 N
    blocks; the first is the last step without, the second carries at once),
    with upper words that propagate it; the production pass against the
    general body, bit for bit."""
    met = synthetic.MetSpec(nx=40, ny=30, nz=16, dx_deg=1.0, dy_deg=1.0, xlon0=-20.0, ylat0=30.0, n_frames=3,
                            frame_seconds=3600, seed=5, wet=True)
    starts = [(TOP - 2 * N, 5, 6, 7), (TOP - 2 * N + 1, TOP - 1, 3, 4), (TOP - 6 * N + 1, TOP - 1, TOP - 1, 9),
              (TOP - 8 * N, TOP - 1, TOP - 1, TOP - 1), (TOP - 1, 0, 0, 0), (0, 1, 2, 3)]
    ens = synthetic.config2(n_scenarios=len(starts), lo=200, hi=2000, hours=2, met=met, seed=11)
    for src in ens.sources:
        src.particle_count = N
        src.start = src.end = ens.start                     # all released at once

    def run(shape):
        scenarios = bt.ensemble_scenarios(ens)
        for scenario, start in zip(scenarios, starts):
            for k, word in enumerate(start):
                scenario.counter[k] = word
        b = bt.Batch(ctx, bt.ensemble_config(ens), scenarios, (met.nx, met.ny, met.nz),
                     synthetic.level_heights(met.nz, met.top_m))
        bt.upload_ensemble_met(b, ens)
        b.tuning = shape
        before = ctx.form_launches["step"]
        b.run(5)
        return b.particles.download(), ctx.form_launches["step"] - before

    shapes = bt.tuning_candidates()
    production, took = run(next(t for t in shapes if t["particles_per_thread"] == 0))
    general, none = run(next(t for t in shapes if t["particles_per_thread"] == 1))
    assert (took, none) == (5, 0)
    assert int((production["flags"] & 1).sum()) == N * len(starts)
    assert production.tobytes() == general.tobytes()


@pytest.mark.parametrize("upper", [(5, 6, 7), (TOP - 1, 3, 4), (TOP - 1, TOP - 1, TOP - 1)])
@pytest.mark.parametrize("past", [0, 1, 500, N - 1])
def test_fused_cbl_sampler_at_the_carry(ctx, past, upper):
    """Slots of a launch whose last `past` blocks lie past the carry, against
    the same slots sampled in two launches that do not carry."""
    nx, ny = 20, 20
    rng = np.random.default_rng(8)
    pbl = api.Pbl(ctx, nx, ny)
    cells = nx * ny
    pbl.upload(rng.uniform(0.05, 0.8, cells), rng.uniform(0.0, 2.5, cells), rng.uniform(60, 2500, cells),
               rng.normal(0, 0.02, cells))
    rec = population(nx, ny, N)

    def sample(records, counter):
        p = api.Particles(ctx, len(records))
        p.upload(records)
        return cbl.sample_cbl_vertical_velocity_philox(ctx, p, pbl, (0xCAFEBABE, 0x12345678), counter)

    first = N - past
    want = [sample(rec[:first], (TOP - first, *upper))]
    if past:
        words, carry = [], 1
        for word in upper:
            words.append((word + carry) % TOP)
            carry = int(carry and words[-1] == 0)
        want.append(sample(rec[first:], (0, *words)))
    assert sample(rec, (TOP - first, *upper)).tobytes() == np.concatenate(want).tobytes()
