"""The work that a user of the framework has it do, as cases to be timed.

A case is one kind of call (``kind``) at one size, through the public entry
points of ``flexpart_gpu``.  The meteorology, the particle counts and the
release geometry are those of the repository's own configurations
(``flexpart_gpu/synthetic.py``) and tests, from one launch that fills a
fraction of the GPU to the ten-million-particle global run.

Winds and clocks are arranged so that a state can be run any number of times
without leaving the situation it stands for: single steps alternate their
advection direction (forward and backward runs are both supported), and the
looped drivers see a wind that swings from +U to -U and back between frames.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "flexpart-gpu_b200"))

from flexpart_gpu import api, batch, cbl, convection, synthetic, timeloop  # noqa: E402
from flexpart_gpu import adjoint  # noqa: E402
from flexpart_gpu._lib import check, lib  # noqa: E402
from flexpart_gpu.records import CBL_OUTPUT_DTYPE, FIELDS, HANNA_PARAMS_DTYPE, MetBracket, StepParams  # noqa: E402

# (nx, ny, nz, cell size in degrees) of the configurations' meteorology:
# regional, ensemble and global.
METS = {"regional": (90, 60, 20, 0.5), "ensemble": (180, 90, 40, 2.0), "global": (360, 180, 60, 1.0)}
KEY = (42, 0)
DT = 900.0
STEP_FLOPS = 750          # floating-point operations of one particle-step (two dual-time samples, Hanna, four sub-steps)


def listed():
    return [
        # one release of a few hundred to a few thousand particles, the size of the framework's own unit
        # tests: a quick look, or a time loop just after its start.  Latency of one launch.
        {"name": "step_1k", "kind": "step", "n": 1003, "met": "regional", "wet": False},
        # the regional forward run of 100 k particles: one step
        {"name": "step_100k", "kind": "step", "n": 100_000, "met": "regional", "wet": False},
        # the global run of ten million particles with per-cell scavenging: one step of the headline benchmark
        {"name": "step_10M", "kind": "step", "n": 10_000_000, "met": "global", "wet": True},
        # the four seam calls one at a time with per-slot forcing and probability outputs, three species and a
        # third of the slots dead: how the reference's time loop drives the kernels
        {"name": "seam_1M", "kind": "seam", "n": 999_983, "met": "regional", "species": 3, "dead": 0.3},
        # the validation and backward path: Hanna records per slot, then the Langevin update from them
        {"name": "records_3M", "kind": "records", "n": 3_000_001, "met": "ensemble", "substeps": 4},
        # a convective step: column mixing, then the skewed vertical velocity of every particle
        {"name": "convective_4M", "kind": "convective", "n": 4_000_000, "met": "global", "levels": 60},
        # the output time of the global run: concentrations on 360 x 180 x 5
        {"name": "grid_10M", "kind": "grid", "n": 10_000_000, "met": "global", "out_levels": 5},
        # a store whose dead particles are dropped: 30 % of 5 M slots, the mask as a sink term leaves it
        {"name": "compact_5M", "kind": "compact", "n": 5_000_011, "met": "regional", "dead": 0.3},
        # the reorder by met cell after a step has mixed the columns
        {"name": "reorder_6M", "kind": "reorder", "n": 6_000_000, "met": "global"},
        # the forward time loop over one three-hour met bracket (12 steps) with met streaming, one reorder,
        # scavenging from precipitation, and the concentration grid read back at its end
        {"name": "loop_300k", "kind": "loop", "n": 300_000, "met": "ensemble", "sort": 12},
        # a small part of the batched ensemble: 24 scenarios of 10 k to 300 k particles, 8 steps
        {"name": "ensemble_24", "kind": "ensemble", "scenarios": 24, "lo": 10_000, "hi": 300_000, "met": "ensemble",
         "steps": 8},
        # the source inversion on the regional met, 160 k particles over 6 h: forward, misfit, backward
        {"name": "inversion_160k", "kind": "inversion", "n": 160_000, "sources": 16, "receptors": 200, "hours": 6,
         "checkpoint": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "seam", "records", "convective", "grid", "compact", "reorder", "loop",
                       "ensemble", "inversion"])
    met = rng.choice(sorted(METS))
    if kind == "step":
        return {"kind": kind, "n": _log(rng, 97, 9_000_000), "met": met, "wet": rng.random() < 0.5}
    if kind == "seam":
        return {"kind": kind, "n": _log(rng, 1_000, 3_000_000), "met": met, "species": rng.randint(1, 4),
                "dead": round(rng.uniform(0.0, 0.6), 3)}
    if kind == "records":
        return {"kind": kind, "n": _log(rng, 1_000, 6_000_000), "met": met, "substeps": rng.choice([1, 2, 4])}
    if kind == "convective":
        return {"kind": kind, "n": _log(rng, 1_000, 8_000_000), "met": met, "levels": rng.randint(4, 80)}
    if kind == "grid":
        return {"kind": kind, "n": _log(rng, 1_000, 10_000_000), "met": met, "out_levels": rng.randint(1, 12)}
    if kind == "compact":
        return {"kind": kind, "n": _log(rng, 1_000, 8_000_000), "met": "regional", "dead": round(rng.uniform(0.0, 0.9), 3)}
    if kind == "reorder":
        return {"kind": kind, "n": _log(rng, 10_000, 8_000_000), "met": met}
    if kind == "loop":
        return {"kind": kind, "n": _log(rng, 1_000, 1_000_000), "met": rng.choice(["regional", "ensemble"]),
                "sort": rng.choice([0, 6, 12])}
    if kind == "ensemble":
        lo = _log(rng, 1_000, 30_000)
        return {"kind": kind, "scenarios": rng.randint(2, 64), "lo": lo, "hi": lo * rng.randint(2, 20),
                "met": rng.choice(["regional", "ensemble"]), "steps": rng.choice([4, 8])}
    return {"kind": kind, "n": _log(rng, 8_000, 400_000), "sources": rng.randint(1, 16),
            "receptors": rng.randint(20, 200), "hours": rng.choice([3, 6]), "checkpoint": rng.choice([0, 8])}


# ---- device memory as tensors ------------------------------------------------

_CTX = None


def _ctx():
    """The program's one context."""
    global _CTX
    if _CTX is None:
        torch.zeros(1, device="cuda")
        _CTX = api.Context(torch.cuda.current_device())
    return _CTX


class _Device:
    """A view of device memory that keeps the handles owning it alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (int(ptr), False), "version": 2}


def _tensor(owner, ptr, shape, dtype=np.float32):
    kind = {"f": "<f4", "i": "<i4", "u": "<i4"}[np.dtype(dtype).kind]
    return torch.as_tensor(_Device(owner, ptr, tuple(shape), kind), device="cuda")


def _fields(p, n, names=None, owner=None):
    return {name: _tensor(owner or p, p.field_ptr(name), (n,), dt) for name, dt in FIELDS if names is None or name in names}


STEP_FIELDS = ("pos_x", "pos_y", "pos_z", "cell_x", "cell_y", "mass0", "vel_u", "vel_v", "vel_w", "turb_u", "turb_v",
               "turb_w", "cbt")


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _rand(g, n, lo=0.0, hi=1.0):
    return torch.rand(n, generator=g, device="cuda") * (hi - lo) + lo


def _normal(g, shape, mean, std):
    return torch.randn(shape, generator=g, device="cuda") * std + mean


# ---- meteorology -----------------------------------------------------------------


def _spec(met, wet=False, frames=2):
    nx, ny, nz, d = METS[met]
    return synthetic.MetSpec(nx=nx, ny=ny, nz=nz, dx_deg=d, dy_deg=d, xlon0=-0.5 * (nx - 1) * d,
                             ylat0=-0.5 * (ny - 1) * d, n_frames=frames, wet=wet)


def _smooth(g, shape, mean, std):
    """N(mean, std) with a Gaussian filter of three cells (periodic), renormalised."""
    a = torch.randn(shape, generator=g, device="cuda")
    f = torch.fft.rfft2(a, dim=(0, 1))
    kx = torch.fft.fftfreq(shape[0], device="cuda")[:, None, None]
    ky = torch.fft.rfftfreq(shape[1], device="cuda")[None, :, None]
    a = torch.fft.irfft2(f * torch.exp(-2.0 * (math.pi * 3.0) ** 2 * (kx * kx + ky * ky)), s=shape[:2], dim=(0, 1))
    return ((a - a.mean()) / a.std() * std + mean).contiguous()


def _frames(spec, seed, swing=False):
    """The frames' wind (device tensors, z fastest) and surface records.  With
    `swing` every second frame has the reversed wind of its predecessor."""
    g = _gen(seed, 1)
    shape = (spec.nx, spec.ny, spec.nz)
    n = spec.nx * spec.ny
    h, us, oli = _rand(g, n, 300.0, 1500.0), _rand(g, n, 0.1, 0.6), _normal(g, n, 0.0, 0.01)
    out = []
    for k in range(spec.n_frames):
        if swing and k % 2:
            u, v, w = (-out[-1][c] for c in "uvw")
        else:
            u, v, w = _smooth(g, shape, 5.0, 3.0), _smooth(g, shape, 5.0, 3.0), _normal(g, shape, 0.0, 0.05)
        cells = synthetic.surface_cells(
            spec, u.cpu().numpy(), v.cpu().numpy(), (h * _rand(g, n, 0.9, 1.1)).cpu().numpy(),
            (us * _rand(g, n, 0.9, 1.1)).cpu().numpy(), (oli * _rand(g, n, 0.9, 1.1)).cpu().numpy())
        out.append({"u": u.contiguous(), "v": v.contiguous(), "w": w.contiguous(), "surface": cells})
    return out


def _precipitation(spec, seed):
    g = _gen(seed, 2)
    n = spec.nx * spec.ny
    p = torch.exp(_normal(g, n, -1.0, 1.0))
    return torch.where(_rand(g, n) < 0.30, p, torch.zeros_like(p))


def _met(ctx, spec, frames):
    m = api.Met(ctx, spec.nx, spec.ny, spec.nz)
    torch.cuda.synchronize()
    for k in (0, 1):
        ptrs = [ctypes.c_void_p(frames[k][c].data_ptr()) for c in "uvw"]
        check(lib.fpg_met_upload_frame_device(m.h, k, *ptrs, None), "fpg_met_upload_frame_device")
    ctx.synchronize()
    m.set_level_heights(synthetic.level_heights(spec.nz, spec.top_m))
    return m


ALPHA = 0.4


def _pbl(ctx, spec, frames):
    s = api.Surface(ctx, spec.nx, spec.ny)
    s.upload(0, frames[0]["surface"])
    s.upload(1, frames[1]["surface"])
    p = api.Pbl(ctx, spec.nx, spec.ny)
    api.pbl_diagnostics(ctx, s, ALPHA, p)
    ctx.synchronize()
    return p, s


# ---- the population -------------------------------------------------------------


def _population(p, n, spec, seed):
    """Plumes of eight point sources two days after the start of a continuous
    release: grid distance from the source grows with age, heights fill the
    boundary layer with a tail above it.  Slots in release order."""
    g = _gen(seed, 3)
    src_x, src_y = _rand(g, 8, 0.2, 0.7) * (spec.nx - 1), _rand(g, 8, 0.2, 0.7) * (spec.ny - 1)
    age = torch.linspace(1.0, 0.0, n, device="cuda")                       # fraction of 48 h
    s = torch.randint(0, 8, (n,), generator=g, device="cuda")
    drift = 5.0 * 48 * 3600 / (111_000.0 * spec.dx_deg)                     # cells in 48 h
    drift = min(drift, 0.25 * spec.ny)
    wid = 0.05 + 0.12 * drift * age
    x = src_x[s] + drift * age + wid * _normal(g, n, 0.0, 1.0)
    y = src_y[s] + drift * age + wid * _normal(g, n, 0.0, 1.0)
    x, y = x.clamp(0, spec.nx - 1.001), y.clamp(0, spec.ny - 1.001)
    z = torch.where(_rand(g, n) < 0.85, _rand(g, n, 1.0, 1400.0), 1400.0 + 400.0 * -torch.log(_rand(g, n, 1e-6, 1.0)))
    f = _fields(p, n)
    f["cell_x"].copy_(x.floor().int())
    f["cell_y"].copy_(y.floor().int())
    f["pos_x"].copy_(x - x.floor())
    f["pos_y"].copy_(y - y.floor())
    f["pos_z"].copy_(z)
    f["flags"].fill_(1)
    f["mass0"].fill_(384.0 / n)
    f["turb_u"].copy_(_normal(g, n, 0.0, 0.5))
    f["turb_v"].copy_(_normal(g, n, 0.0, 0.5))
    f["turb_w"].copy_(_normal(g, n, 0.0, 0.3))
    f["release_point"].copy_(s.int())
    f["cbt"].fill_(1)
    torch.cuda.synchronize()


def _dead(p, n, share, seed):
    m = (_rand(_gen(seed, 4), n) >= share).int()
    if n > 1:
        m[0] = 1
    return m


def _params(spec, wet, **kw):
    xs, ys, zs = synthetic.velocity_scale(spec)
    return StepParams.production(alpha=ALPHA, dt_seconds=DT, turb_dt_seconds=DT, x_grid_per_meter=xs,
                                 y_grid_per_meter=ys, z_grid_per_meter=zs, key=KEY, dry_mode=1,
                                 dry_velocity_m_s=0.002, wet_mode=3 if wet else 0, **kw)


def _base(case, seed, wet=False, sort=True):
    """Met, PBL and a population in the order the last reorder left it."""
    ctx = _ctx()
    spec = _spec(case["met"], wet)
    frames = _frames(spec, seed)
    s = {"case": case, "ctx": ctx, "spec": spec, "frames": frames, "n": case["n"], "met": _met(ctx, spec, frames)}
    s["pbl"], s["surface"] = _pbl(ctx, spec, frames)
    s["p"] = api.Particles(ctx, case["n"])
    _population(s["p"], case["n"], spec, seed)
    if sort:
        sorter = api.Sorter(ctx, case["n"])
        sorter.sort(s["p"], s["met"])
        ctx.synchronize()
        s["sorter"] = sorter
    if wet:
        s["wet"] = api.CellField(ctx, spec.nx, spec.ny)
        s["prec"] = _precipitation(spec, seed)
        s["wet"].from_precipitation(s["prec"].cpu().numpy())
    s["out"] = _fields(s["p"], case["n"], STEP_FIELDS)
    return s


# ---- prepare and run, kind by kind -------------------------------------------------


def _prepare_step(case, seed):
    s = _base(case, seed, case["wet"])
    s["prm"] = _params(s["spec"], case["wet"])
    del s["sorter"]
    return s


def _run_step(s):
    """One fused step; the advection direction alternates."""
    prm = s["prm"]
    nxt = api.step(s["ctx"], s["p"], s["met"], s["pbl"], prm, s.get("wet"))
    prm.counter[:] = nxt
    prm.dt_seconds = -prm.dt_seconds
    return s["out"]


def _prepare_seam(case, seed):
    s = _base(case, seed)
    n, g = case["n"], _gen(seed, 5)
    flags = _fields(s["p"], n, ("flags",))["flags"]
    flags.copy_(_dead(s["p"], n, case["dead"], seed))
    names = ["mass%d" % k for k in range(case["species"])]
    for k in range(1, case["species"]):
        s["p"].write_field("mass%d" % k, _rand(g, n, 1e-6, 1e-3).cpu().numpy())
    for name, lo, hi in (("vdep", 0.0, 0.004), ("lam", 0.0, 2e-4), ("frac", 0.0, 1.0)):
        s[name] = api.DeviceArray.from_numpy(s["ctx"], _rand(g, n, lo, hi).cpu().numpy())
    s["pd"], s["pw"] = api.DeviceArray(s["ctx"], n), api.DeviceArray(s["ctx"], n)
    s["dt"], s["counter"] = DT, [0, 0, 0, 0]
    s["out"] = _fields(s["p"], n, STEP_FIELDS + tuple(names))
    s["out"]["dry_probability"], s["out"]["wet_probability"] = _tensor(s["pd"], s["pd"].ptr, (n,)), _tensor(s["pw"], s["pw"].ptr, (n,))
    s["scale"] = synthetic.velocity_scale(s["spec"])
    torch.cuda.synchronize()
    return s


def _run_seam(s):
    ctx, p = s["ctx"], s["p"]
    api.advect_dual_wind(ctx, p, s["met"], ALPHA, s["dt"], *s["scale"])
    s["counter"] = api.langevin_fused(ctx, p, s["pbl"], DT, 0.0, 4, 0.01, KEY, s["counter"])
    api.dry_deposition(ctx, p, s["vdep"], DT, 15.0, s["pd"])
    api.wet_deposition(ctx, p, s["lam"], s["frac"], DT, s["pw"])
    s["dt"] = -s["dt"]
    return s["out"]


def _prepare_records(case, seed):
    s = _base(case, seed)
    n = case["n"]
    s["hanna"] = api.DeviceArray(s["ctx"], n, HANNA_PARAMS_DTYPE)
    s["counter"] = [0, 0, 0, 0]
    s["out"] = _fields(s["p"], n, ("pos_z", "turb_u", "turb_v", "turb_w", "cbt"))
    s["out"]["hanna"] = _tensor(s["hanna"], s["hanna"].ptr, (n, 16))
    return s


def _run_records(s):
    cbl.dispatch_hanna_params_gpu(s["ctx"], s["p"], s["pbl"], s["hanna"])
    s["counter"] = cbl.update_particles_turbulence_langevin_gpu(
        s["ctx"], s["p"], s["hanna"], DT, 0.0, s["case"]["substeps"], 0.01, KEY, s["counter"])
    return s["out"]


def _interfaces(case):
    return np.linspace(0.0, 12_000.0, case["levels"] + 1, dtype=np.float32)


def _matrix(case, seed):
    """A column-stochastic redistribution matrix (column-major): most mass
    stays, the rest spreads over the column."""
    L = case["levels"]
    m = torch.rand((L, L), generator=_gen(seed, 6), device="cuda", dtype=torch.float64)
    m = 0.3 * m / m.sum(1, keepdim=True) + 0.7 * torch.eye(L, device="cuda", dtype=torch.float64)
    return m.float().cpu().numpy()


def _prepare_convective(case, seed):
    s = _base(case, seed)
    n = case["n"]
    s["mix"] = convection.ConvectiveMixing(s["ctx"], case["levels"])
    s["mix"].set_matrix(_matrix(case, seed).reshape(-1), _interfaces(case))
    s["cbl"] = api.DeviceArray(s["ctx"], n, CBL_OUTPUT_DTYPE)
    s["out"] = _fields(s["p"], n, ("pos_z", "cbt"))
    s["out"]["cbl"] = _tensor(s["cbl"], s["cbl"].ptr, (n, 12))
    s["counter"] = [7, 0, 0, 0]
    return s


def _run_convective(s):
    cbl.sample_cbl_vertical_velocity_philox(s["ctx"], s["p"], s["pbl"], KEY, s["counter"], s["cbl"])
    s["mix"].apply(s["p"])
    return s["out"]


def _heights(k):
    return [100.0, 500.0, 1000.0, 2000.0, 5000.0][:k] + [5000.0 + 700.0 * i for i in range(1, k - 4)]


def _prepare_grid(case, seed):
    s = _base(case, seed)
    # the heights mix within the columns from the first step after a reorder on
    prm = _params(s["spec"], False)
    for _ in range(2):
        prm.counter[:] = api.step(s["ctx"], s["p"], s["met"], s["pbl"], prm)
        prm.dt_seconds = -prm.dt_seconds
    s["ctx"].synchronize()
    nx, ny = s["spec"].nx, s["spec"].ny
    s["grid"] = api.Grid(s["ctx"], nx, ny, case["out_levels"])
    lib.fpg_grid_counts_device.restype = lib.fpg_grid_mass_device.restype = ctypes.c_void_p
    shape = (nx * ny * case["out_levels"],)
    s["out"] = {"counts": _tensor(s["grid"], lib.fpg_grid_counts_device(s["grid"].h), shape, np.uint32),
                "mass": _tensor(s["grid"], lib.fpg_grid_mass_device(s["grid"].h), shape, np.uint32)}
    s["oh"] = _heights(case["out_levels"])
    return s


def _run_grid(s):
    s["grid"].accumulate(s["p"], 0, 1.0e6, s["oh"])
    return s["out"]


def _prepare_compact(case, seed):
    s = _base(case, seed)
    n = case["n"]
    s["mask"] = _dead(s["p"], n, case["dead"], seed)
    s["compaction"] = api.Compaction(s["ctx"], n)
    s["views"] = {}
    torch.cuda.synchronize()
    return s


def _moved(s):
    """The particle fields wherever the last move left them (the handle swaps
    between two blocks)."""
    at = s["p"].field_ptr("pos_x")
    if at not in s["views"]:
        s["views"][at] = _fields(s["p"], s["n"], owner=(s["p"], s.get("sorter"), s.get("compaction"), s.get("d")))
    return s["views"][at]


def _run_compact(s):
    """The mask of a sink term goes into the flags, then the dead are dropped."""
    s["p"].dispatch_count = s["n"]
    check(lib.fpg_memcpy(s["ctx"].h, s["p"].field_ptr("flags"), s["mask"].data_ptr(), 4 * s["n"], 2, None), "fpg_memcpy")
    alive = s["compaction"].compact(s["p"])
    return {"alive": alive, **_moved(s)}


def _prepare_reorder(case, seed):
    s = _base(case, seed)
    s["prm"] = _params(s["spec"], False)
    s["views"] = {}
    return s


def _run_reorder(s):
    _run_step(s)
    s["sorter"].sort(s["p"], s["met"])
    return _moved(s)


START = synthetic.EPOCH_2024


def _prepare_loop(case, seed):
    ctx = _ctx()
    spec = _spec(case["met"], True)
    frames = _frames(spec, seed, swing=True)
    g = np.random.default_rng(seed)
    n, src = case["n"], 4
    sources = [synthetic.Source(lon=float(spec.xlon0 + g.uniform(0.3, 0.6) * (spec.nx - 1) * spec.dx_deg),
                                lat=float(spec.ylat0 + g.uniform(0.3, 0.6) * (spec.ny - 1) * spec.dy_deg),
                                z_min=50.0, z_max=50.0, mass_kg=1.0,
                                particle_count=n // src + (1 if k < n % src else 0), start=START, end=START + 9000)
               for k in range(src)]
    scn = synthetic.Scenario("loop", spec, sources, start=START, end=START + 400 * 365 * 86400, dt=900,
                             out_shape=(spec.nx, spec.ny, 3), outheights=[100.0, 500.0, 1000.0], capacity=n)
    cfg = timeloop.scenario_config(scn, sort_interval_steps=case["sort"])
    d = timeloop.ForwardDriver(ctx, cfg, timeloop.scenario_releases(scn), timeloop.scenario_domain(scn), n,
                               (spec.nx, spec.ny, spec.nz), synthetic.level_heights(spec.nz, spec.top_m))
    d.enable_met_ring(3)
    wet = api.CellField(ctx, spec.nx, spec.ny)
    wet.from_precipitation(_precipitation(spec, seed).cpu().numpy())
    surf = [torch.from_numpy(f["surface"].view(np.float32).copy()).cuda() for f in frames]
    s = {"case": case, "ctx": ctx, "spec": spec, "frames": frames, "surf": surf, "n": n, "d": d, "wet": wet, "views": {},
         "forcing": timeloop.cell_forcing(wet, 0.002), "grid": api.Grid(ctx, *scn.out_shape), "p": d.particles,
         "oh": scn.outheights, "bracket": 0}
    torch.cuda.synchronize()
    _run_loop(s)                       # the release window lies in the first bracket
    ctx.synchronize()
    return s


def _prefetch(s, k):
    f, sf = s["frames"][k % 2], s["surf"][k % 2]
    s["d"].prefetch_frame(START + 10800 * k, f["u"].data_ptr(), f["v"].data_ptr(), f["w"].data_ptr(), sf.data_ptr())


def _run_loop(s):
    k = s["bracket"]
    _prefetch(s, k)
    _prefetch(s, k + 1)
    bracket = MetBracket(time_t0_seconds=START + 10800 * k, time_t1_seconds=START + 10800 * (k + 1))
    for _ in range(12):
        rep = s["d"].run_timestep(bracket, s["forcing"])
    s["bracket"] = k + 1
    counts, mass, kg = s["d"].accumulate_concentration_grid(s["grid"], 0, 1.0e6, s["oh"])
    return {"counts": counts.view(np.int32), "mass": mass.view(np.int32), "kg": kg,
            "active": int(rep.active_particle_count), **_moved(s)}


def _prepare_ensemble(case, seed):
    ctx = _ctx()
    spec = _spec(case["met"], True)
    frames = _frames(spec, seed, swing=True)
    ens = synthetic.config2(case["scenarios"], case["lo"], case["hi"], hours=24, met=spec, seed=int(seed) % (1 << 31))
    ens.end = ens.start + 400 * 365 * 86400
    m = case["scenarios"]
    for k, src in enumerate(ens.sources):   # counts log-uniform, all released in the first steps
        src.start, src.end = ens.start, ens.start + 3600
        src.particle_count = int(case["lo"] * (case["hi"] / case["lo"]) ** ((k * 7 % m + 0.5) / m))
    b = batch.Batch(ctx, batch.ensemble_config(ens, output_every_steps=case["steps"]), batch.ensemble_scenarios(ens),
                    (spec.nx, spec.ny, spec.nz), synthetic.level_heights(spec.nz, spec.top_m), ens.outheights)
    prec = _precipitation(spec, seed).cpu().numpy()
    for k, f in enumerate(frames):
        b.upload_frame(k, {"u": f["u"].cpu().numpy(), "v": f["v"].cpu().numpy(), "w": f["w"].cpu().numpy(),
                           "surface": f["surface"]}, prec)
    p = b.particles
    s = {"case": case, "ctx": ctx, "b": b, "n": p.capacity, "p": p,
         "out": _fields(p, p.capacity, STEP_FIELDS + ("flags",), b), "particles": ens.total_particles}
    b.run(case["steps"])
    ctx.synchronize()
    return s


def _run_ensemble(s):
    s["b"].run(s["case"]["steps"])
    return s["out"]


def _prepare_inversion(case, seed):
    ctx = _ctx()
    spec = _spec("regional")
    frames = _frames(spec, seed)
    inv = synthetic.config3(case["n"], case["sources"], case["receptors"], case["hours"], met=spec,
                            seed=int(seed) % (1 << 31))
    inv.sample_every, inv.checkpoint_every = 4, case["checkpoint"]
    # receptors where the plumes pass: cells downwind of the sources
    g = np.random.default_rng(seed)
    cells = set()
    while len(cells) < case["receptors"]:
        src = inv.ensemble.sources[int(g.integers(0, len(inv.ensemble.sources)))]
        i = int((src.lon - spec.xlon0) / spec.dx_deg + g.integers(-1, 9))
        j = int((src.lat - spec.ylat0) / spec.dy_deg + g.integers(-1, 9))
        cells.add((min(max(i, 0), spec.nx - 1), min(max(j, 0), spec.ny - 1)))
    inv.receptors = [(0, i, j) for i, j in sorted(cells)]
    host = [{"u": f["u"].cpu().numpy(), "v": f["v"].cpu().numpy(), "w": f["w"].cpu().numpy(), "surface": f["surface"]}
            for f in frames]
    model = adjoint.SourceInversion(ctx, inv, host)
    obs = g.uniform(0.0, 1e-3, len(inv.receptors))
    return {"case": case, "ctx": ctx, "model": model, "obs": obs,
            "mass": model.mass0 * g.lognormal(0.0, 0.5, model.n_sources)}


def _run_inversion(s):
    """One gradient of the receptor misfit, as an optimiser asks for it."""
    sim = s["model"].forward(s["mass"], s["model"].position0)
    loss, d_sim = adjoint.misfit(sim, s["obs"])
    return {"sim": sim, "loss": loss, **s["model"].backward(d_sim)}


_KINDS = {"step": (_prepare_step, _run_step), "seam": (_prepare_seam, _run_seam),
          "records": (_prepare_records, _run_records), "convective": (_prepare_convective, _run_convective),
          "grid": (_prepare_grid, _run_grid), "compact": (_prepare_compact, _run_compact),
          "reorder": (_prepare_reorder, _run_reorder), "loop": (_prepare_loop, _run_loop),
          "ensemble": (_prepare_ensemble, _run_ensemble), "inversion": (_prepare_inversion, _run_inversion)}


def prepare(case, seed):
    s = _KINDS[case["kind"]][0](case, seed)
    s["run"] = _KINDS[case["kind"]][1]
    return s


def run(state):
    return state["run"](state)


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    met = METS[case.get("met", "regional")]
    cells = met[0] * met[1]
    step = 96.0                        # 44 B read and 52 B written per particle-step, one species
    if kind == "step":
        return {"bytes": step * n, "flops": STEP_FLOPS * n}
    if kind == "seam":
        live = n * (1.0 - case["dead"])
        return {"bytes": 4 * n + live * (88 + 8 * case["species"] + 12) + 8 * n, "flops": STEP_FLOPS * live}
    if kind == "records":
        return {"bytes": n * (24 + 64 + 20 + 52 + 20.0), "flops": 450.0 * n}
    if kind == "convective":
        return {"bytes": n * (24 + 48 + 16.0), "flops": 250.0 * n}
    if kind == "grid":
        return {"bytes": 20.0 * n + 8.0 * cells * case["out_levels"], "flops": 4.0 * n}
    if kind == "compact":
        return {"bytes": 2 * 92.0 * n + 8.0 * n, "flops": 0.0}
    if kind == "reorder":
        return {"bytes": (step + 20 + 2 * 92.0) * n, "flops": STEP_FLOPS * n}
    if kind == "loop":
        return {"bytes": 12 * (step * n + 140.0 * cells) + (20.0 * n + 24.0 * cells) +
                (2 * 92.0 * n if case["sort"] else 0.0) * (12 // max(case["sort"], 1)) + 56.0 * cells * met[2],
                "flops": 12.0 * STEP_FLOPS * n}
    if kind == "ensemble":
        lo, hi = case["lo"], case["hi"]
        mean = (hi - lo) / math.log(hi / lo)
        total = case["scenarios"] * mean
        return {"bytes": case["steps"] * (step * total + 140.0 * cells) + 20.0 * total +
                8.0 * 3 * cells * case["scenarios"], "flops": case["steps"] * STEP_FLOPS * total}
    steps = 4.0 * case["hours"] + 1
    # each step once forward and once taped or reversed; a quarter of the particle-steps lie before the releases
    return {"bytes": 0.75 * n * steps * (step + 160.0) + 24.0 * cells * met[2], "flops": 3.0 * STEP_FLOPS * 0.75 * n * steps}


# ---- the same in 64 bits, in plain torch --------------------------------------------

_D = torch.float64


def _philox(counter, offset, key):
    """Philox4x32-10 blocks at counter + offset, as four int64 tensors."""
    m32 = 0xFFFFFFFF
    c0 = counter[0] + offset
    carry = c0 >> 32
    c = [c0 & m32]
    for k in (1, 2, 3):
        v = counter[k] + carry
        carry = v >> 32
        c.append(v & m32)
    k0, k1 = key

    def mul(a, b):                     # 32 x 32 -> (high, low) within int64
        ah, al, bh, bl = a >> 16, a & 0xFFFF, b >> 16, b & 0xFFFF
        low = al * bl
        mid = ah * bl + (low >> 16)
        mid2 = al * bh + (mid & 0xFFFF)
        return ah * bh + (mid >> 16) + (mid2 >> 16), ((mid2 & 0xFFFF) << 16) | (low & 0xFFFF)

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return c


def _gauss(a, b):
    u0 = ((a >> 8).to(_D) / 16777216.0).clamp(1.17549435e-38, 0.99999994039535522)
    u1 = (b >> 8).to(_D) / 16777216.0
    r, t = torch.sqrt(-2.0 * torch.log(u0)), 2.0 * math.pi * u1
    return r * torch.cos(t), r * torch.sin(t)


def _lerp(a, b, t):
    return a * (1.0 - t) + b * t


def _axis(x, n):
    c = x.clamp(0, n - 1)
    lo = c.floor()
    i = lo.long()
    return i, (i + 1).clamp(max=n - 1), c - lo


def _level(z, h):
    k = torch.searchsorted(h, z, right=False).clamp(min=1)          # first k >= 1 with z <= h[k]
    top = h.numel() - 1
    kk = k.clamp(max=top)
    lv = (kk - 1).to(_D) + (z - h[kk - 1]) / (h[kk] - h[kk - 1])
    lv = torch.where(k > top, torch.full_like(z, float(top)), lv)
    return torch.where(z <= h[0], z / h[0], lv)


def _wind(frames, spec, h, x, y, z):
    x0, x1, tx = _axis(x, spec.nx)
    y0, y1, ty = _axis(y, spec.ny)
    z0, z1, tz = _axis(_level(z, h), spec.nz)
    out = []
    for c in "uvw":
        both = []
        for f in frames[:2]:
            a = f[c].reshape(-1)

            def at(i, j, k):
                return a[(i * spec.ny + j) * spec.nz + k].to(_D)

            both.append(_lerp(_lerp(_lerp(at(x0, y0, z0), at(x1, y0, z0), tx), _lerp(at(x0, y1, z0), at(x1, y1, z0), tx), ty),
                              _lerp(_lerp(at(x0, y0, z1), at(x1, y0, z1), tx), _lerp(at(x0, y1, z1), at(x1, y1, z1), tx), ty),
                              tz))
        out.append(_lerp(both[0], both[1], float(np.float32(ALPHA))))
    return out


def _exact_pbl(frames, spec):
    """u*, w*, h and L per cell: the met provides u*, h and 1/L, w* follows
    from the heat flux."""
    a, b = ({k: torch.from_numpy(f["surface"][k].astype(np.float64)).cuda() for k in f["surface"].dtype.names}
            for f in frames[:2])
    i = {k: _lerp(a[k], b[k], float(np.float32(ALPHA))) for k in a}
    rho = i["surface_pressure_pa"] / (287.05 * i["temperature_2m_k"])
    ust = i["friction_velocity_ms"].clamp(min=1e-4)
    shf = i["sensible_heat_flux_w_m2"]
    ol = -(rho * 1004.6 * i["temperature_2m_k"] * ust ** 3) / (0.4 * 9.81 * shf)
    ol = torch.where((shf.abs() < 1.0) | (ol.abs() > 1e5), torch.full_like(ol, math.inf), ol)
    oli = torch.where(i["inv_obukhov_length_per_m"].abs() >= 1e-5, i["inv_obukhov_length_per_m"], 1.0 / ol)
    h = i["mixing_height_m"].clamp(100.0, 4500.0)
    flux = shf / (rho * 1004.6) * 9.81 / i["temperature_2m_k"]
    wst = torch.where(shf > 0, (flux.clamp(min=0) * h) ** (1.0 / 3.0), torch.zeros_like(h))
    return ust, wst, h, torch.where(oli.abs() < 1e-5, torch.full_like(oli, math.inf), 1.0 / oli)


def _hanna(ust, wst, h, ol, z_in):
    """Hanna's profiles at z: a dict, the vertical parts as the sub-steps use them too."""
    z = torch.minimum(z_in.clamp(min=0), h)
    zeta = (z / h).clamp(0, 1)
    neutral = torch.isinf(ol) | (h / ol.abs() < 1)
    unstable = ~neutral & (ol < 0)
    corr = z / ust
    su_n, sw_n = 1e-2 + 2 * ust * torch.exp(-3e-4 * corr), 1.3 * ust * torch.exp(-2e-4 * corr)
    ds_n, sw_n = -2e-4 * sw_n, sw_n + 1e-2
    tl_n = 0.5 * z / sw_n / (1 + 1.5e-3 * corr)
    third = 1.0 / 3.0
    su_u = 1e-2 + ust * (12 - 0.5 * h / ol).clamp(min=0) ** third
    tlu_u = (0.15 * h / su_u).clamp(min=10)
    z23 = zeta ** (2 * third)
    sw_u = torch.sqrt(1.2 * wst ** 2 * (1 - 0.9 * zeta) * z23 + (1.8 - 1.4 * zeta) * ust ** 2) + 1e-2
    ds_u = 0.5 / sw_u / h * (-1.4 * ust ** 2 + wst ** 2 * (0.8 * zeta.clamp(min=1e-3) ** -third - 1.8 * z23))
    tlw_u = torch.where(z < ol.abs(), 0.1 * z / (sw_u * (0.55 - 0.38 * (z / ol).abs())),
                        torch.where(zeta < 0.1, 0.59 * z / sw_u, 0.15 * h / sw_u * (1 - torch.exp(-5 * zeta))))
    su_s, sv_s = 1e-2 + 2 * ust * (1 - zeta), 1e-2 + 1.3 * ust * (1 - zeta)
    tlu_s, tlw_s = 0.15 * h / su_s * torch.sqrt(zeta), 0.1 * h / sv_s * zeta ** 0.8

    def pick(n, u, s):
        return torch.where(neutral, n, torch.where(unstable, u, s))

    return {"ust": ust, "wst": wst, "ol": ol, "h": h, "zeta": zeta, "sigu": pick(su_n, su_u, su_s),
            "sigv": pick(sw_n, su_u, sv_s), "sigw": pick(sw_n, sw_u, sv_s), "dsigwdz": pick(ds_n, ds_u, -1.3 * ust / h),
            "tlu": pick(tl_n, tlu_u, tlu_s).clamp(min=10), "tlv": pick(tl_n, tlu_u, 0.467 * tlu_s).clamp(min=10),
            "tlw": pick(tl_n, tlw_u, tlw_s).clamp(min=30)}


def _ou(prev, sig, tl, dt, eta, drift=None):
    r = dt / tl
    c = torch.exp(-r)
    small = (1 - r) * prev + eta * sig * torch.sqrt(2 * r)
    large = c * prev + eta * sig * torch.sqrt((1 - c * c).clamp(min=0))
    if drift is not None:
        small, large = small + dt * drift, large + tl * (1 - c) * drift
    return torch.where(r < 0.5, small, large)


def _turbulence(f, pbl_of, n_sub, n):
    """Langevin update with vertical sub-steps, in place in the dict `f`."""
    blocks = 1 if n_sub <= 2 else 2
    slot = torch.arange(n, device="cuda", dtype=torch.int64) * blocks
    b0 = _philox([0, 0, 0, 0], slot, KEY)
    e = [_gauss(b0[0], b0[1]), _gauss(b0[2], b0[3])]
    if blocks > 1:
        b1 = _philox([0, 0, 0, 0], slot + 1, KEY)
        e.append(_gauss(b1[0], b1[1]))
    cell = pbl_of
    hn = _hanna(*cell, f["pos_z"])
    f["turb_u"] = _ou(f["turb_u"], hn["sigu"], hn["tlu"], DT, e[0][0])
    f["turb_v"] = _ou(f["turb_v"], hn["sigv"], hn["tlv"], DT, e[0][1])
    etas = [e[1][0], e[1][1]] + ([e[2][0], e[2][1]] if blocks > 1 else [])
    dt, h, z, w, zmin, cbt = DT / n_sub, cell[2], f["pos_z"], f["turb_w"], float(np.float32(0.01)), f["cbt"]
    cur = hn
    for k in range(n_sub):
        w = _ou(w, cur["sigw"], cur["tlw"], dt, etas[k], cur["sigw"] * cur["dsigwdz"])
        z = z + w * dt
        for _ in range(10):
            lo, hi = z < zmin, z > h
            hi = hi & ~lo
            z = torch.where(lo, 2 * zmin - z, torch.where(hi, 2 * h - z, z))
            w = torch.where(lo | hi, -w, w)
            cbt = torch.where(lo | hi, -cbt, cbt)
        z = torch.maximum(torch.minimum(z, h), torch.full_like(z, zmin))
        if k < n_sub - 1:
            cur = _hanna(*cell, z)
    f["pos_z"], f["turb_w"], f["cbt"] = z, w, cbt
    return hn


def _start(s, names):
    f = {k: v.clone() for k, v in _fields(s["p"], s["n"], names).items()}
    return {k: v.to(_D) if v.is_floating_point() else v for k, v in f.items()}


def _cell_of(spec, x, y):
    return x.clamp(0, spec.nx - 1).floor().long() * spec.ny + y.clamp(0, spec.ny - 1).floor().long()


def _advect(s, f, h, dt):
    spec, (xs, ys, zs) = s["spec"], synthetic.velocity_scale(s["spec"])
    x, y, z = f["cell_x"].to(_D) + f["pos_x"], f["cell_y"].to(_D) + f["pos_y"], f["pos_z"]
    top = float(h[-1])
    u0, v0, w0 = _wind(s["frames"], spec, h, x, y, z)
    u0, v0 = u0 + f["turb_u"], v0 + f["turb_v"]
    u1, v1, w1 = _wind(s["frames"], spec, h, (x + u0 * xs * dt).clamp(0, spec.nx - 1),
                       (y + v0 * ys * dt).clamp(0, spec.ny - 1), (z + w0 * zs * dt).clamp(0, top))
    u, v, w = 0.5 * (u0 + u1 + f["turb_u"]), 0.5 * (v0 + v1 + f["turb_v"]), 0.5 * (w0 + w1)
    x, y = (x + u * xs * dt).clamp(0, spec.nx - 1), (y + v * ys * dt).clamp(0, spec.ny - 1)
    f["pos_z"] = (z + w * zs * dt).clamp(0, top)
    f["vel_u"], f["vel_v"], f["vel_w"] = u, v, w
    f["cell_x"], f["cell_y"] = x.floor().int(), y.floor().int()
    f["pos_x"], f["pos_y"] = x - x.floor(), y - y.floor()
    return x, y


def _exact_step(s, f):
    case, spec = s["case"], s["spec"]
    h = torch.from_numpy(synthetic.level_heights(spec.nz, spec.top_m).astype(np.float64)).cuda()
    x, y = _advect(s, f, h, DT)
    c = _cell_of(spec, x, y)
    pbl = [q[c] for q in _exact_pbl(s["frames"], spec)]
    _turbulence(f, pbl, 4, s["n"])
    vd = s["vdep"] if "vdep" in s else float(np.float32(0.002))
    low = f["pos_z"] < 30.0
    dry = torch.where(low, torch.exp(-(vd * DT / 30.0) * torch.ones_like(f["pos_z"])), torch.ones_like(f["pos_z"]))
    wet = torch.ones_like(dry)
    if "lam" in s:
        wet = 1 - (1 - torch.exp(-s["lam"] * DT)) * s["frac"]
    elif case.get("wet"):
        p = s["prec"].to(_D)
        cls = torch.tensor([0.5, 0.65, 0.8, 0.9, 0.95], device="cuda", dtype=_D)
        area = cls[(p > 1).long() + (p > 3).long() + (p > 8).long() + (p > 20).long()].clamp(0.05, 1.0)
        on = p >= 0.01
        lam = torch.where(on, float(np.float32(1e-4)) * (p / area) ** float(np.float32(0.8)), torch.zeros_like(p))
        wet = 1 - (1 - torch.exp(-lam[c] * DT)) * torch.where(on, area, torch.zeros_like(p))[c]
    return dry, wet


def _exact_fused(case, seed):
    s = _prepare_step(case, seed)
    f = _start(s, STEP_FIELDS)
    dry, wet = _exact_step(s, f)
    f["mass0"] = f["mass0"] * dry * wet
    return {k: f[k] for k in s["out"]}


def _exact_seam(case, seed):
    s = _prepare_seam(case, seed)
    names = [k for k in s["out"] if "probability" not in k]
    before = _start(s, names)
    live = _fields(s["p"], s["n"], ("flags",))["flags"] != 0
    f = dict(before)
    t = dict(s)
    for k in ("vdep", "lam", "frac"):
        t[k] = _tensor(s[k], s[k].ptr, (s["n"],)).to(_D)
    dry, wet = _exact_step(t, f)
    for k in range(case["species"]):
        f["mass%d" % k] = f["mass%d" % k] * dry * wet
    out = {k: torch.where(live, f[k], before[k]) for k in names}
    zero = torch.zeros_like(dry)
    out["dry_probability"], out["wet_probability"] = torch.where(live, 1 - dry, zero), torch.where(live, 1 - wet, zero)
    return out


def _exact_records(case, seed):
    s = _prepare_records(case, seed)
    f = _start(s, STEP_FIELDS)
    c = _cell_of(s["spec"], f["cell_x"].to(_D) + f["pos_x"], f["cell_y"].to(_D) + f["pos_y"])
    hn = _turbulence(f, [q[c] for q in _exact_pbl(s["frames"], s["spec"])], case["substeps"], s["n"])
    # an infinite Obukhov length (neutral cells) stays what it is in the records
    cols = [hn[k] for k in ("ust", "wst", "ol", "h", "zeta", "sigu", "sigv", "sigw", "dsigwdz")]
    cols += [2 * hn["sigw"] * hn["dsigwdz"], hn["tlu"], hn["tlv"], hn["tlw"]]
    zero = torch.zeros_like(cols[0])
    return {"pos_z": f["pos_z"], "turb_u": f["turb_u"], "turb_v": f["turb_v"], "turb_w": f["turb_w"], "cbt": f["cbt"],
            "hanna": torch.stack(cols + [zero, zero, zero], 1)}


def _exact_convective(case, seed):
    s = _prepare_convective(case, seed)
    n, spec = s["n"], s["spec"]
    f = _start(s, STEP_FIELDS)
    c = _cell_of(spec, f["cell_x"].to(_D) + f["pos_x"], f["cell_y"].to(_D) + f["pos_y"])
    ust, wst, h, ol = (q[c] for q in _exact_pbl(s["frames"], spec))
    hn = _hanna(ust, wst, h, ol, f["pos_z"])
    z = torch.minimum(f["pos_z"].clamp(min=0), h)
    zoh, sw = z / h, hn["sigw"]
    ratio = -h / ol
    trans = torch.where(ratio < 15, torch.sin((ratio + 10) / 10 * math.pi) * 0.5 + 0.5, torch.ones_like(h)).clamp(0, 1)
    trans = torch.where(torch.isinf(ol), torch.ones_like(h), trans)
    w2 = sw * sw
    w3 = (1.2 * zoh * (1 - zoh).clamp(min=0) ** 1.5 + 1e-6) * wst ** 3 * trans
    skew = w3 / w2 ** 1.5
    fl = 2.0 / 3.0 * skew.clamp(min=0) ** (1.0 / 3.0)
    fl2 = fl * fl
    flat = (skew.abs() <= 1e-6) | (fl.abs() <= 1e-6)
    r = ((1 + fl2) ** 3 * skew ** 2 / ((3 + fl2) ** 2 * fl2).clamp(min=1e-6)).clamp(min=0)
    aw = (0.5 * (1 - torch.sqrt(r) / torch.sqrt(4 + r))).clamp(1e-4, 1 - 1e-4)
    bw = 1 - aw
    sa, sb = sw * torch.sqrt(bw / (aw * (1 + fl2))), sw * torch.sqrt(aw / (bw * (1 + fl2)))
    half, zero = torch.full_like(h, 0.5), torch.zeros_like(h)
    aw, bw, am, bm = (torch.where(flat, q, v) for q, v in ((half, aw), (half, bw), (zero, fl * sa), (zero, -fl * sb)))
    sa, sb = torch.where(flat, sw, sa), torch.where(flat, sw, sb)
    b = _philox(s["counter"], torch.arange(n, device="cuda", dtype=torch.int64), KEY)
    eta = _gauss(b[1], b[2])[0]
    w = torch.where((b[0] >> 8).to(_D) / 16777216.0 < aw, am + sa * eta, bm + sb * eta)
    cols = torch.stack([w, aw, am, sa, bw, bm, sb, w2, w3, skew, trans, zoh], 1)
    iface = torch.from_numpy(_interfaces(case).astype(np.float64)).cuda()
    m = torch.from_numpy(_matrix(case, seed).astype(np.float64)).cuda().clamp(min=0)
    centre = 0.5 * (iface[1:] + iface[:-1])
    to = ((m * centre).sum(1) / m.sum(1)).clamp(float(iface[0]), float(iface[-1]))
    zc = f["pos_z"].clamp(float(iface[0]), float(iface[-1]))
    lev = (torch.searchsorted(iface, zc, right=True) - 1).clamp(0, case["levels"] - 1)
    return {"pos_z": to[lev], "cbt": lev.int(), "cbl": cols}


def exact(case, seed):
    """The outputs of run() in 64 bits; None where the outputs are whole
    numbers or moved values, and for the runs of many steps (their releases,
    reorders and atomics are the framework's own)."""
    of = {"step": _exact_fused, "seam": _exact_seam, "records": _exact_records, "convective": _exact_convective}
    if case["kind"] not in of:
        return None
    return of[case["kind"]](case, seed)
