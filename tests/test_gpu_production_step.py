"""The step's production form (its own kernels, compile-time settings, no
sanitising where it cannot fire) against the general body, bit for bit: the
general body runs when a launch shape is selected by hand."""
from __future__ import annotations

import numpy as np
import pytest

from flexpart_gpu import api, cbl
from flexpart_gpu.records import FIELDS
from helpers import population, production_params, small_met

pytestmark = pytest.mark.gpu

GENERAL = {"block_threads": 256, "min_blocks_per_sm": 4, "particles_per_thread": 1}
PRODUCTION = {"block_threads": 256, "min_blocks_per_sm": 5, "particles_per_thread": 1}
ODD = np.array([0.0, -1.0, np.nan, np.inf, 1e-30, 5e2, 2e3, 1e12], np.float32)


@pytest.fixture(scope="module")
def world():
    ctx = api.Context(0)
    spec, frames, met = small_met()
    m = api.Met(ctx, spec.nx, spec.ny, spec.nz)
    m.upload_frame(0, met["u0"], met["v0"], met["w0"])
    m.upload_frame(1, met["u1"], met["v1"], met["w1"])
    m.set_level_heights(met["heights"])
    cells = spec.nx * spec.ny
    rng = np.random.default_rng(3)
    # every regime, and some cells outside any real boundary layer
    ust = rng.uniform(0.05, 0.8, cells).astype(np.float32)
    wst = np.where(rng.random(cells) < 0.5, rng.uniform(0, 2.5, cells), 0).astype(np.float32)
    h = rng.uniform(60, 2500, cells).astype(np.float32)
    oli = rng.normal(0, 0.02, cells).astype(np.float32)
    for field in (ust, wst, h, oli):
        at = rng.choice(cells, 24, replace=False)
        field[at] = np.resize(ODD, 24)
    pbl = api.Pbl(ctx, spec.nx, spec.ny)
    pbl.upload(ust, wst, h, oli)
    wet = api.CellField(ctx, spec.nx, spec.ny)
    lam = np.where(rng.random(cells) < 0.4, rng.uniform(0, 5e-4, cells), 0).astype(np.float32)
    frac = rng.uniform(-0.1, 1.1, cells).astype(np.float32)
    lam[:6], frac[6:12] = np.resize(ODD, 6), np.resize(ODD, 6)
    wet.upload(lam, frac)
    return ctx, spec, m, pbl, wet


def _records(spec, n):
    rec = population(spec.nx, spec.ny, n, seed=n)
    rng = np.random.default_rng(n)
    if n > 64:
        for k, name in enumerate(("turb_u", "turb_v", "turb_w", "pos_z")):
            at = rng.choice(np.arange(16, n), 12, replace=False)
            rec[name][at] = np.resize(np.array([np.nan, np.inf, -np.inf, 1e35, -3e29, 2e4], np.float32), 12)
        rec["cell_x"][20:24] = [-3, 1000, spec.nx - 1, 0]
        rec["pos_x"][22:24] = [0.7, -0.5]
    rec["mass"][:, 1:] = 0.0
    rec["cbt"] = np.where(rng.random(n) < 0.5, 1, -1)
    return rec


def _run(world, rec, shape, steps, **kw):
    ctx, spec, m, pbl, wet = world
    p = api.Particles(ctx, len(rec))
    p.upload(rec)
    api.set_step_tuning(ctx, shape)
    prm = production_params(**kw)
    for _ in range(steps):
        prm.counter[:] = api.step(ctx, p, m, pbl, prm, wet if prm.wet_mode == 3 else None)
        prm.dt_seconds = -prm.dt_seconds
    api.set_step_tuning(ctx, PRODUCTION)
    return {name: p.read_field(name).view(np.uint32) for name, _ in FIELDS}


def _same(a, b):
    for name in a:
        if not np.array_equal(a[name], b[name]):
            at = np.flatnonzero(a[name] != b[name])
            raise AssertionError(f"{name}: {at.size} slots differ, first {at[:5]}: "
                                 f"{a[name][at[:5]].view(np.float32)} {b[name][at[:5]].view(np.float32)}")


@pytest.mark.parametrize("n", [1, 31, 33, 1003, 148 * 24 * 32, 148 * 24 * 32 + 1])
@pytest.mark.parametrize("wet", [0, 3])
def test_production_form_gives_the_general_bits(world, n, wet):
    rec = _records(world[1], n)
    kw = dict(wet_mode=wet, rho_grad_over_rho=-1e-4)
    _same(_run(world, rec, PRODUCTION, 3, **kw), _run(world, rec, GENERAL, 3, **kw))


@pytest.mark.parametrize("counter", [(0xFFFFFFFF - 2005, 0xFFFFFFFF, 3, 4), (0xFFFFFFFF - 2006, 7, 0xFFFFFFFF, 1),
                                     (0xFFFFFFF0, 0xFFFFFFFF, 0xFFFFFFFF, 2)])
def test_counters_at_the_edge_of_a_carry(world, counter):
    rec = _records(world[1], 1003)
    kw = dict(counter=counter, key=(0xDECAFBAD, 0x12345678))
    _same(_run(world, rec, PRODUCTION, 2, **kw), _run(world, rec, GENERAL, 2, **kw))


@pytest.mark.parametrize("n", [1, 3, 4, 5, 63, 65, 1027])
@pytest.mark.parametrize("species,shift,prob", [(1, 0, True), (3, 0, False), (4, 1, True)])
def test_stage_kernels_give_the_general_bits(world, n, species, shift, prob):
    """One stage per call; `shift` moves the per-slot forcing off 16 bytes,
    where the general body runs."""
    ctx, spec, m, pbl, _ = world
    rec = _records(spec, n)
    rng = np.random.default_rng(n)
    rec["mass"][:, 1:species] = rng.uniform(0, 1, (n, species - 1))
    arrays = []
    for lo, hi in ((-1e-3, 4e-3), (-1e-4, 4e-4), (-0.2, 1.2)):
        a = rng.uniform(lo, hi, n + shift).astype(np.float32)
        a[shift::5] = np.resize(ODD, a[shift::5].size)
        arrays.append(api.DeviceArray.from_numpy(ctx, a))

    def run(shape):
        p = api.Particles(ctx, n)
        p.upload(rec)
        out = [api.DeviceArray.from_numpy(ctx, np.full(n + shift, -7.0, np.float32)) for _ in range(2)]
        at = [type("At", (), {"ptr": a.ptr + 4 * shift}) for a in arrays + out]
        api.set_step_tuning(ctx, shape)
        for k in range(2):
            api.langevin_fused(ctx, p, pbl, 900.0, 0.0, 4, 0.01, (7, 9), [k, 0, 0, 0])
            api.advect_dual_wind(ctx, p, m, 0.3, 900.0 * (1 - 2 * k), 2.5e-5, 1.8e-5)
            api.langevin_fused(ctx, p, pbl, 900.0, -1e-4, 4, 0.01, (42, 0), [5 + k, 0, 0, 0])
            api.dry_deposition(ctx, p, at[0], 900.0, 15.0, at[3] if prob else None)
            api.wet_deposition(ctx, p, at[1], at[2], 900.0, at[4] if prob else None)
        api.set_step_tuning(ctx, PRODUCTION)
        return {name: p.read_field(name).view(np.uint32) for name, _ in FIELDS} | {
            "dry": out[0].numpy().view(np.uint32), "wet": out[1].numpy().view(np.uint32)}

    _same(run(PRODUCTION), run(GENERAL))


@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 2049])
@pytest.mark.parametrize("n_sub", [1, 2, 3, 4])
def test_record_kernel_gives_the_general_bits(world, n, n_sub):
    """Records on a 32-byte boundary against the same records 16 bytes off it,
    where the general kernel runs; some hold what no boundary layer does."""
    ctx, spec, _, pbl, _ = world
    rec = _records(spec, n)
    rng = np.random.default_rng(n)

    def particles():
        p = api.Particles(ctx, n)
        p.upload(rec)
        return p

    hanna = cbl.compute_hanna_params_gpu(ctx, particles(), pbl)
    assert not hanna[(rec["flags"] & 1) == 0].view(np.uint32).any()
    words = hanna.view(np.float32).reshape(n, 16)
    at = rng.random((n, 13)) < 0.03
    words[:, :13][at] = np.resize(ODD, int(at.sum()))

    def run(offset):
        p = particles()
        d = api.DeviceArray.from_numpy(ctx, np.concatenate([np.zeros(offset, np.float32), words.reshape(-1)]))
        at = api.DeviceArray.__new__(api.DeviceArray)
        at.ctx, at.n, at.dtype, at.ptr = ctx, n, cbl.HANNA_PARAMS_DTYPE, d.ptr + 4 * offset
        for k in range(2):
            cbl.update_particles_turbulence_langevin_gpu(ctx, p, at, 900.0, -1e-4, n_sub, 0.01, (42, 0), [9 + k, 0, 0, 0])
        at.ptr = None
        return {name: p.read_field(name).view(np.uint32) for name, _ in FIELDS}

    _same(run(0), run(4))


# Philox blocks under key (42, 0) whose word (1 or 3: the angle of a pair) lies
# exactly between two quadrants, where the rounding of the quadrant is a tie
TIES = [(1, 34705893), (1, 7291534), (1, 49559575), (1, 15432739), (3, 16559396), (3, 34779132), (3, 15007975),
        (3, 1106156)]


@pytest.mark.parametrize("word,block", TIES)
def test_box_muller_at_quadrant_ties(world, word, block):
    rec = _records(world[1], 33)
    rec["flags"] = 1
    for first in (block - 16, block - 17):          # slot 8's first block, and its second
        kw = dict(counter=(first, 0, 0, 0), key=(42, 0))
        _same(_run(world, rec, PRODUCTION, 1, **kw), _run(world, rec, GENERAL, 1, **kw))


def test_largest_shape(world):
    rec = np.resize(_records(world[1], 50_021), 4_000_001)
    _same(_run(world, rec, PRODUCTION, 1, wet_mode=3), _run(world, rec, GENERAL, 1, wet_mode=3))


@pytest.mark.parametrize("kw", [dict(n_substeps=2), dict(min_height_m=1.5), dict(dry_mode=0), dict(rho_grad_over_rho=5e3),
                                dict(turb_dt_seconds=2e6)])
def test_settings_outside_the_form_run_the_general_body(world, kw):
    rec = _records(world[1], 1003)
    _same(_run(world, rec, PRODUCTION, 2, **kw), _run(world, rec, GENERAL, 2, **kw))
