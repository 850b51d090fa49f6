"""Which kernel a particle pass runs: the ones compiled for common settings
(whole step, one-stage seam calls, Hanna records) where their rule takes a
call, the general one everywhere else."""
from __future__ import annotations

import numpy as np
import pytest

from flexpart_gpu import api, cbl, synthetic
from flexpart_gpu import batch as bt
from helpers import population, production_params, small_met

pytestmark = pytest.mark.gpu

N = 1003
GENERAL = {"block_threads": 256, "min_blocks_per_sm": 4, "particles_per_thread": 1}


@pytest.fixture(scope="module")
def world():
    ctx = api.Context(0)
    spec, frames, met = small_met()
    m = api.Met(ctx, spec.nx, spec.ny, spec.nz)
    m.upload_frame(0, met["u0"], met["v0"], met["w0"])
    m.upload_frame(1, met["u1"], met["v1"], met["w1"])
    m.set_level_heights(met["heights"])
    cells = spec.nx * spec.ny
    pbl = api.Pbl(ctx, spec.nx, spec.ny)
    pbl.upload(np.full(cells, 0.3, np.float32), np.full(cells, 1.0, np.float32), np.full(cells, 900.0, np.float32),
               np.full(cells, -0.01, np.float32))
    wet = api.CellField(ctx, spec.nx, spec.ny)
    wet.upload(np.full(cells, 1e-4, np.float32), np.full(cells, 0.5, np.float32))
    return ctx, spec, m, pbl, wet


def _particles(world, n=N, species=1):
    ctx, spec = world[:2]
    rec = population(spec.nx, spec.ny, n)
    rec["mass"][:, 1:] = 0.0
    rec["mass"][:, 1:species] = 1.0
    p = api.Particles(ctx, n)
    p.upload(rec)
    return p


def _took(ctx, call):
    """The forms the call's passes ran, name -> launches."""
    before = ctx.form_launches
    call()
    return {k: v - before[k] for k, v in ctx.form_launches.items() if v != before[k]}


@pytest.mark.parametrize("kw", [dict(), dict(wet_mode=3), dict(rho_grad_over_rho=-1e-4), dict(dt_seconds=-900.0),
                                dict(counter=(2**32 - 2 * N, 0, 0, 0))])
def test_step_in_the_production_form(world, kw):
    ctx, _, m, pbl, wet = world
    prm = production_params(**kw)
    p = _particles(world)
    assert _took(ctx, lambda: api.step(ctx, p, m, pbl, prm, wet if prm.wet_mode == 3 else None)) == {"step": 1}


@pytest.mark.parametrize("kw", [dict(n_substeps=2), dict(min_height_m=1.5), dict(dry_mode=0), dict(rho_grad_over_rho=5e3),
                                dict(turb_dt_seconds=2e6), dict(wet_mode=1, wet_lambda_s_inv=1e-4, wet_fraction=1.0),
                                dict(counter=(2**32 - 2 * N + 1, 0, 0, 0))])
def test_step_outside_the_production_form(world, kw):
    ctx, _, m, pbl, _ = world
    prm = production_params(**kw)
    p = _particles(world)
    assert _took(ctx, lambda: api.step(ctx, p, m, pbl, prm)) == {}


def test_species_and_a_shape_selected_by_hand_run_the_general_body(world):
    ctx, _, m, pbl, _ = world
    p2 = _particles(world, species=2)
    assert _took(ctx, lambda: api.step(ctx, p2, m, pbl, production_params())) == {}
    p = _particles(world)
    api.set_step_tuning(ctx, GENERAL)
    assert _took(ctx, lambda: api.step(ctx, p, m, pbl, production_params())) == {}
    api.set_step_tuning(ctx, api.step_tuning_candidates()[0])
    assert _took(ctx, lambda: api.step(ctx, p, m, pbl, production_params())) == {"step": 1}


@pytest.mark.parametrize("n", [97, 1003, 40_001, 300_007])
def test_tuning_settings_without_a_form_leaves_the_forms_on(world, n):
    """Whatever shape wins for two species, calls with a form still run it;
    a tuning of those keeps a shape it measured, and selecting shape 0 by hand
    brings the forms back."""
    ctx, _, m, pbl, _ = world
    p2, p = _particles(world, n, species=2), _particles(world, n)
    best, cands = api.step_autotune(ctx, p2, m, pbl, production_params(), reps=3)
    assert best["step_ms"] == min(c["step_ms"] for c in cands)
    got = api.get_step_tuning(ctx)
    assert all(got[k] == best[k] for k in ("block_threads", "min_blocks_per_sm", "particles_per_thread"))
    assert _took(ctx, lambda: api.step(ctx, p2, m, pbl, production_params())) == {}
    assert _took(ctx, lambda: api.step(ctx, p, m, pbl, production_params())) == {"step": 1}
    assert _took(ctx, lambda: api.advect_dual_wind(ctx, p, m, 0.3, 900.0, 2.5e-5, 1.8e-5)) == {"advection": 1}
    first = api.step_tuning_candidates()[0]
    best, _ = api.step_autotune(ctx, p, m, pbl, production_params(), reps=3)
    in_form = all(best[k] == first[k] for k in ("block_threads", "min_blocks_per_sm", "particles_per_thread"))
    assert _took(ctx, lambda: api.step(ctx, p, m, pbl, production_params())) == ({"step": 1} if in_form else {})
    api.set_step_tuning(ctx, first)
    assert _took(ctx, lambda: api.step(ctx, p, m, pbl, production_params())) == {"step": 1}


@pytest.mark.parametrize("species,shift", [(1, 0), (4, 0), (1, 1)])
def test_seam_calls(world, species, shift):
    ctx, _, m, pbl, _ = world
    p = _particles(world, species=species)
    arrays = [api.DeviceArray.from_numpy(ctx, np.full(N + shift, 1e-4, np.float32)) for _ in range(3)]
    at = [type("At", (), {"ptr": a.ptr + 4 * shift}) for a in arrays]
    deposition = {} if shift else {"deposition": 1}
    assert _took(ctx, lambda: api.advect_dual_wind(ctx, p, m, 0.3, 900.0, 2.5e-5, 1.8e-5)) == {"advection": 1}
    assert _took(ctx, lambda: api.langevin_fused(ctx, p, pbl, 900.0, 0.0, 4, 0.01, (42, 0), [0] * 4)) == {"turbulence": 1}
    assert _took(ctx, lambda: api.langevin_fused(ctx, p, pbl, 900.0, 0.0, 3, 0.01, (42, 0), [0] * 4)) == {}
    assert _took(ctx, lambda: api.dry_deposition(ctx, p, at[0], 900.0, 15.0)) == deposition
    assert _took(ctx, lambda: api.wet_deposition(ctx, p, at[0], at[1], 900.0, at[2])) == deposition


@pytest.mark.parametrize("offset,n_sub,counter,took", [
    (0, 4, 0, True), (0, 1, 0, True), (0, 4, 2**32 - 2 * N, True), (0, 2, 2**32 - N, True),
    (0, 4, 2**32 - 2 * N + 1, False), (0, 5, 0, False), (4, 4, 0, False)])
def test_record_calls(world, offset, n_sub, counter, took):
    """`offset`: floats between a 32-byte boundary and the records."""
    ctx, _, _, pbl, _ = world
    p = _particles(world)
    hanna = cbl.compute_hanna_params_gpu(ctx, p, pbl).view(np.float32).reshape(-1)
    d = api.DeviceArray.from_numpy(ctx, np.concatenate([np.zeros(offset, np.float32), hanna]))
    at = api.DeviceArray.__new__(api.DeviceArray)
    at.ctx, at.n, at.dtype, at.ptr = ctx, N, cbl.HANNA_PARAMS_DTYPE, d.ptr + 4 * offset
    got = _took(ctx, lambda: cbl.update_particles_turbulence_langevin_gpu(ctx, p, at, 900.0, -1e-4, n_sub, 0.01, (42, 0),
                                                                         [counter, 0, 0, 0]))
    at.ptr = None
    assert got == ({"record": 1} if took else {})


@pytest.mark.parametrize("graph", [True, False])
def test_batched_pass(graph):
    ctx = api.Context(0)
    met = synthetic.MetSpec(nx=40, ny=30, nz=16, dx_deg=1.0, dy_deg=1.0, xlon0=-20.0, ylat0=30.0, n_frames=3,
                            frame_seconds=3600, seed=5, wet=True)
    ens = synthetic.config2(n_scenarios=3, lo=200, hi=2000, hours=2, met=met, seed=11)

    def batch(dry):
        ens.dry_velocity = dry
        b = bt.Batch(ctx, bt.ensemble_config(ens), bt.ensemble_scenarios(ens), (met.nx, met.ny, met.nz),
                     synthetic.level_heights(met.nz, met.top_m))
        bt.upload_ensemble_met(b, ens)
        return b

    b = batch(0.002)
    assert _took(ctx, lambda: b.run(3, graph=graph)) == {"step": 3}
    b.tuning = {"block_threads": 256, "min_blocks_per_sm": 4, "particles_per_thread": 1}
    assert _took(ctx, lambda: b.run(2, graph=graph)) == {}
    assert _took(ctx, lambda: batch(0.0).run(3, graph=graph)) == {}


def test_tuner_times_one_kernel_once():
    """In the production form the flat shapes of 128 threads run one kernel and
    report one time; in the general body they are two."""
    ctx = api.Context(0)
    met = synthetic.MetSpec(nx=40, ny=30, nz=16, dx_deg=1.0, dy_deg=1.0, xlon0=-20.0, ylat0=30.0, n_frames=3,
                            frame_seconds=3600, seed=5, wet=True)
    ens = synthetic.config2(n_scenarios=3, lo=200, hi=2000, hours=2, met=met, seed=11)
    times = {}
    for dry in (0.002, 0.0):
        ens.dry_velocity = dry
        b = bt.Batch(ctx, bt.ensemble_config(ens), bt.ensemble_scenarios(ens), (met.nx, met.ny, met.nz),
                     synthetic.level_heights(met.nz, met.top_m))
        bt.upload_ensemble_met(b, ens)
        launches = ctx.kernel_launches
        best, cands = b.autotune(reps=1)
        assert best["step_ms"] == min(c["step_ms"] for c in cands) > 0.0
        flat = [c["step_ms"] for c in cands if c["particles_per_thread"] == 0 and c["block_threads"] == 128]
        times[dry] = (len(cands), ctx.kernel_launches - launches, flat)
    (n, launches, flat), (n_general, launches_general, _) = times[0.002], times[0.0]
    assert len(flat) == 2 and flat[0] == flat[1]
    assert n == n_general and launches_general == 2 * n and launches == 2 * (n - 1)


def test_sequential_path_launches_what_a_step_of_the_scenario_alone_would():
    ctx = api.Context(0)
    met = synthetic.MetSpec(nx=40, ny=30, nz=16, dx_deg=1.0, dy_deg=1.0, xlon0=-20.0, ylat0=30.0, n_frames=3,
                            frame_seconds=3600, seed=5, wet=True)
    ens = synthetic.config2(n_scenarios=3, lo=200, hi=2000, hours=2, met=met, seed=11)
    for src in ens.sources:
        src.start = src.end = ens.start                      # all released at once
    scenarios = bt.ensemble_scenarios(ens)
    scenarios[2].counter[0] = 2**32 - 1                     # carries in the first step
    b = bt.Batch(ctx, bt.ensemble_config(ens), scenarios, (met.nx, met.ny, met.nz),
                 synthetic.level_heights(met.nz, met.top_m))
    bt.upload_ensemble_met(b, ens)
    assert _took(ctx, lambda: b.run_sequential(1)) == {"step": 2}
    assert _took(ctx, lambda: b.run_sequential(2)) == {"step": 6}
