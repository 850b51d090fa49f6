"""The two forms of the inversion's reverse: a bracket's steps in one launch up
to 4,096 work items of 256 slots, one launch a step above."""
import numpy as np
import pytest

from flexpart_gpu import synthetic

pytestmark = pytest.mark.gpu

api = pytest.importorskip("flexpart_gpu.api")
adj = pytest.importorskip("flexpart_gpu.adjoint")

ITEMS = 4096


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def problem():
    """Four sources of 1,024 items each and a fifth of 200 slots (one item),
    released over the first hour of 4 h (17 steps, two met brackets), every
    cell of the lowest layer observed at every step; and dL/dsim."""
    inv = synthetic.config3(n_particles=5 * 64, n_sources=5, n_receptors=10, hours=4)
    spec = inv.ensemble.met
    inv.receptors = [(0, i, j) for i in range(spec.nx) for j in range(spec.ny)]
    inv.sample_every = 1
    for s, src in enumerate(inv.ensemble.sources):
        src.start = inv.ensemble.start
        src.end = src.start + 3600
        src.particle_count = ITEMS // 4 * 256 if s < 4 else 200
    return inv, np.random.default_rng(2).standard_normal(len(inv.receptors))


def _gradient(ctx, problem, sources, K, W):
    """The gradient of the inversion of `sources` alone, and the kernels its
    backward launched."""
    inv, d_sim = problem
    ens = inv.ensemble
    part = synthetic.Ensemble(ens.name, ens.met, [ens.sources[s] for s in sources], [ens.keys[s] for s in sources],
                              start=ens.start, end=ens.end, dt=ens.dt, out_shape=ens.out_shape,
                              outheights=ens.outheights, dry_velocity=ens.dry_velocity)
    model = adj.SourceInversion(ctx, synthetic.Inversion(
        inv.name, part, inv.receptors, [0] * len(sources), sample_every=1, receptor_top_m=inv.receptor_top_m,
        receptor_ramp_m=inv.receptor_ramp_m, checkpoint_every=K, tape_tail_windows=W))
    model.forward(model.mass0, model.position0)
    before = ctx.kernel_launches
    return model.backward(d_sim), ctx.kernel_launches - before


@pytest.mark.parametrize("K,W", [(0, 0), (4, 0), (5, 2)])
def test_both_forms_of_the_reverse_give_the_same_gradient(ctx, problem, K, W):
    """For a given dL/dsim the loss is linear in the particles: a source's
    gradient does not depend on the others, and the bias gradient is the sum
    of the parts'.  So the four large sources give at 4,096 items what they
    give beside the fifth at 4,097.  The f32 partial sums of a source are the
    same warps' in both (rtol: the order of their f64 sums).  The bias goes
    through a CTA's f32 sums per node and step, at most 8 warps of 7 items with
    up to 32 lanes' groups each: 2^-24 times the square root of 1,792 random
    terms, 2.5e-6 in norm."""
    small, bracket_launches = _gradient(ctx, problem, range(4), K, W)
    one, _ = _gradient(ctx, problem, [4], K, W)
    both, step_launches = _gradient(ctx, problem, range(5), K, W)
    assert step_launches > bracket_launches                 # the two forms did run
    for name in ("mass", "position"):
        np.testing.assert_allclose(both[name][:4], small[name], rtol=1e-9, atol=1e-300)
        np.testing.assert_allclose(both[name][4:], one[name], rtol=1e-9, atol=1e-300)
    whole = both["wind_bias"].astype(np.float64)
    parts = small["wind_bias"].astype(np.float64) + one["wind_bias"]
    assert np.linalg.norm(parts) > 0.0
    assert np.linalg.norm(whole - parts) <= 1e-5 * np.linalg.norm(parts)
