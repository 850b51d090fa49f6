"""Kernels launched into the tail of the one before them: a long chain of
dependent calls queued without waiting gives the bits of the same calls with
a wait after each."""
from __future__ import annotations

import numpy as np
import pytest

from flexpart_gpu import api, cbl, convection
from flexpart_gpu.records import CBL_OUTPUT_DTYPE, FIELDS, HANNA_PARAMS_DTYPE
from helpers import population, production_params, small_met

pytestmark = pytest.mark.gpu


def _chain(n, wait):
    ctx = api.Context(0)
    spec, frames, met = small_met()
    m = api.Met(ctx, spec.nx, spec.ny, spec.nz)
    m.upload_frame(0, met["u0"], met["v0"], met["w0"])
    m.upload_frame(1, met["u1"], met["v1"], met["w1"])
    m.set_level_heights(met["heights"])
    surf = api.Surface(ctx, spec.nx, spec.ny)
    surf.upload(0, frames[0]["surface"])
    surf.upload(1, frames[1]["surface"])
    pbl = api.Pbl(ctx, spec.nx, spec.ny)
    p = api.Particles(ctx, n)
    p.upload(population(spec.nx, spec.ny, n, seed=n))
    hanna = api.DeviceArray(ctx, n, HANNA_PARAMS_DTYPE)
    inputs = api.DeviceArray.from_numpy(ctx, cbl.sampling_inputs(*np.random.default_rng(1).random((3, n))))
    out = api.DeviceArray(ctx, n, CBL_OUTPUT_DTYPE)
    mix = convection.ConvectiveMixing(ctx, 8)
    mix.set_matrix((0.5 * np.eye(8) + 0.5 / 8).astype(np.float32).reshape(-1), np.linspace(0, 6000, 9))
    sorter = api.Sorter(ctx, n)
    prm = production_params()
    done = ctx.synchronize if wait else (lambda: None)
    counter = [0, 0, 0, 0]
    for k in range(24):
        api.pbl_diagnostics(ctx, surf, k / 24.0, pbl)
        done()
        prm.counter[:] = api.step(ctx, p, m, pbl, prm)
        done()
        cbl.dispatch_hanna_params_gpu(ctx, p, pbl, hanna)
        done()
        counter = cbl.update_particles_turbulence_langevin_gpu(ctx, p, hanna, 900.0, 0.0, 4, 0.01, (1, 2), counter)
        done()
        cbl.sample_cbl_vertical_velocity_gpu(ctx, p, hanna, inputs, out)
        done()
        api.advect_dual_wind(ctx, p, m, 0.5, -900.0, 2.5e-5, 1.8e-5)
        done()
        if k % 8 == 3:
            mix.apply(p)
            done()
        if k % 8 == 5:
            sorter.sort(p, m)
            done()
    ctx.synchronize()
    fields = {name: p.read_field(name).view(np.uint32) for name, _ in FIELDS}
    return fields | {"hanna": hanna.numpy().view(np.uint32), "cbl": out.numpy().view(np.uint32)}


@pytest.mark.parametrize("n", [97, 20_011, 300_007])
def test_a_chain_without_waits_gives_the_same_bits(n):
    a, b = _chain(n, True), _chain(n, False)
    for name in a:
        assert np.array_equal(a[name], b[name]), name
