"""The work a user of the engine has it do, as timed cases.

Every mover case is one MHD frame of the reference driver's loop
(src/programs/stochastic-mhd.f90:312-567) from a checkpoint: counters and
particles go in, particle_mover moves them over one MHD interval,
split_particle, f(p) and quick_check follow, and the particles come back to
pinned host memory.  The split-precision path bins particles by cell, so its
sets come back in an order of their own; they are put in the order of their
lineage tags.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "stochastic-parker_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from gpat import _abi, configs, fields  # noqa: E402
from gpat.engine import (Batch, Engine, Mlp, ParticleSet, make_mhd_config, make_params,  # noqa: E402
                         mover_learned_stats, set_mover_learned, window_params)

P0 = 0.1


def listed():
    return [
        # The planar-shock configuration at its grid, in the default (FP64)
        # precision, with the handful of particles of a first try: one call
        # whose time is latency.
        dict(name="planar_fp64_1e3", kind="frame", flow="planar", precision=0, grid=512, nptl=1000,
             pushes=1000, time_interp=0, split=1),
        # The planar-shock configuration (512 x 64, 1e5 particles), split precision.
        dict(name="planar_mixed_1e5", kind="frame", flow="planar", precision=1, grid=512,
             nptl=100_000, pushes=1000, time_interp=0, split=1),
        # The benchmark: 2048^2 turbulent shock, 1000 pushes a particle.
        dict(name="shock2d_mixed_2e6", kind="frame", flow="shock", precision=1, grid=2048,
             nptl=2_000_000, pushes=1000, time_interp=0, split=1),
        # 3D compressible turbulence: adaptive steps, particles that start
        # anywhere in the interval, an odd particle count.
        dict(name="turb3d_mixed_1e6", kind="frame", flow="turb3d", precision=1, grid=128,
             nptl=1_000_003, pushes=500, time_interp=0, split=0),
        # The shock in the default precision, 512^2.
        dict(name="shock2d_fp64_5e4", kind="frame", flow="shock", precision=0, grid=512,
             nptl=50_001, pushes=1000, time_interp=0, split=1),
        # 3D turbulence in the default precision, two field frames
        # interpolated in time.
        dict(name="turb3d_fp64_2e4", kind="frame", flow="turb3d", precision=0, grid=64,
             nptl=20_000, pushes=250, time_interp=1, split=0),
        # Focused transport (pitch angle and speed as state) on a 2D shock.
        dict(name="focused2d_2e4", kind="focused", grid=256, nptl=20_000, pushes=250),
        # Solar-wind style run: 3D spherical coordinates on a stretched grid.
        dict(name="sphere3d_2e4", kind="sphere", grid=48, nptl=20_000, pushes=250),
        # A parameter study: six runs of uneven size moved as one batch.
        dict(name="batch6_mixed", kind="batch", grid=512, nptl=200_000, nruns=6, pushes=500),
        # Learned splitting inside the split-precision 3D mover.
        dict(name="learned3d_2e5", kind="learned", grid=64, nptl=200_000, pushes=250),
        # A new MHD frame: fields in, gradients, the compression count and
        # injection that read them, frame 2 taking frame 1's place.
        dict(name="frame3d_128", kind="newframe", grid=128, nptl=100_000),
        # The diagnostics of an output step over a resident set.
        dict(name="diag_4e6", kind="diag", grid=1024, nptl=4_000_000, nmu=8),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("planar", "shock", "shock", "turb3d", "turb3d", "focused", "sphere", "batch",
                       "learned", "newframe", "diag"))
    if kind in ("planar", "shock", "turb3d"):
        mixed = rng.randrange(2)
        c = dict(kind="frame", flow=kind, precision=mixed, time_interp=rng.randrange(2),
                 split=0 if kind == "turb3d" else 1)
        if kind == "planar":
            c.update(grid=rng.choice((256, 500, 512)), pushes=1000,
                     nptl=_logint(rng, 500, 200_000 if mixed else 20_000))
        elif kind == "shock":
            c.update(grid=rng.choice((300, 512, 777, 1024)), pushes=rng.choice((250, 500, 1000)),
                     nptl=_logint(rng, 1000, 1_000_000 if mixed else 50_000))
        else:
            c.update(grid=rng.choice((33, 48, 64, 96)), pushes=rng.choice((125, 250)),
                     nptl=_logint(rng, 1000, 500_000 if mixed else 20_000))
        return c
    if kind == "focused":
        return dict(kind="focused", grid=rng.choice((64, 200, 256)), nptl=_logint(rng, 500, 20_000),
                    pushes=rng.choice((100, 250)))
    if kind == "sphere":
        return dict(kind="sphere", grid=rng.choice((24, 37, 48)), nptl=_logint(rng, 500, 20_000),
                    pushes=rng.choice((100, 250)))
    if kind == "batch":
        return dict(kind="batch", grid=rng.choice((128, 256, 500)), nruns=rng.randint(2, 6),
                    nptl=_logint(rng, 2000, 200_000), pushes=rng.choice((250, 500)))
    if kind == "learned":
        return dict(kind="learned", grid=rng.choice((32, 48, 64)), nptl=_logint(rng, 2000, 200_000),
                    pushes=rng.choice((125, 250)))
    if kind == "newframe":
        return dict(kind="newframe", grid=rng.choice((40, 63, 96, 120)),
                    nptl=_logint(rng, 1000, 100_000))
    return dict(kind="diag", grid=rng.choice((256, 1000, 1024)), nptl=_logint(rng, 1000, 4_000_000),
                nmu=rng.choice((1, 8, 32)))


# -- inputs ------------------------------------------------------------------------
def _pinned(n):
    """A ParticleSet in pinned host memory."""
    dt = {"f8": torch.float64, "i1": torch.int8, "i4": torch.int32, "u4": torch.int32}
    arrays = {}
    for name, t in _abi.PARTICLE_FIELDS:
        k = np.dtype(t)
        a = torch.zeros(max(1, n), dtype=dt[k.kind + str(k.itemsize)], pin_memory=True).numpy()
        arrays[name] = a[:n].view(k)
    return ParticleSet(arrays)


def _checkpoint(eng, margin=1.0):
    """The injected particles in pinned memory, buffers for the result, the counters."""
    start = eng.get_particles()
    first = _pinned(len(start))
    for name, a in first.arrays.items():
        a[:] = start[name]
    return dict(eng=eng, first=first, out=_pinned(int(len(start) * margin) + 64),
                counters=eng.counters())


def _restore(s):
    s["eng"].set_counters(s["counters"])
    s["eng"].put_particles(s["first"])


def _turb3d(grid, seed):
    """turbulence_3d's frame: v rms 0.3 with 30 % compressive power, B = z +
    solenoidal dB of 0.3, both with Kolmogorov spectra, drawn on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = grid
    k1 = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64)
    k3 = torch.fft.rfftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64)
    k = torch.stack(torch.meshgrid(k1, k1, k3, indexing="ij"))
    kk = k.square().sum(0).sqrt()
    ok = (kk >= 1) & (kk <= n // 2)
    amp = torch.where(ok, kk.clamp(min=1.0) ** ((-5.0 / 3.0 - 2.0) / 2.0), torch.zeros_like(kk))
    kh = k / kk.clamp(min=1.0)

    def parts():
        h = torch.randn((2, 3) + kk.shape, generator=g, device="cuda", dtype=torch.float64)
        h = torch.complex(h[0], h[1]) * amp
        comp = (h * kh).sum(0) * kh
        real = lambda v: torch.fft.irfftn(v, s=(n, n, n), dim=(1, 2, 3))  # noqa: E731
        return real(h - comp), real(comp)

    sol, comp = parts()
    v = sol * math.sqrt(0.7 / float(sol.square().sum(0).mean())) + \
        comp * math.sqrt(0.3 / float(comp.square().sum(0).mean()))
    v *= 0.3 / math.sqrt(float(v.square().sum(0).mean()))
    b, _ = parts()
    b *= 0.3 / math.sqrt(float(b.square().sum(0).mean()))
    b[2] += 1.0
    a = torch.cat([v, torch.ones_like(v[:1]), b, b.square().sum(0).sqrt()[None]])
    a = torch.nn.functional.pad(a[None].float(), (2, 2, 2, 2, 2, 2), mode="circular")[0]
    return a.permute(3, 2, 1, 0).contiguous().cpu().numpy()


def _shock(grid, seed, r=3.5, w=0.001):
    db = fields.kolmogorov_az_2d(grid, grid, 1.0, 1.0, db_rms=0.5, kmin=2.0 * np.pi,
                                 kmax=min(512.0 * np.pi, np.pi * grid / 2), seed=seed)
    return fields.planar_shock_2d(grid, grid, 0.0, 1.0, 0.0, 1.0, u1=1.0, r=r, w=w, x0=0.5, db=db)


def _engine(params, cfg, frames, tstamps, grid_positions=None):
    eng = Engine(make_params(**params), cfg, 0)
    eng.set_tstamps(tstamps)
    if grid_positions is not None:
        eng.set_grid_positions(*grid_positions)
    for k, f in enumerate(frames):
        eng.set_fields(f, k)
        eng.calc_fields_gradients(k)
    return eng


BOX = (0.0, 0.0, 0.0, 1.0, 1.0, 1.0)


def _prepare_frame(c, seed):
    n, grid, ti = c["nptl"], c["grid"], c["time_interp"]
    if c["flow"] == "planar":
        w = configs.planar_shock(nx=grid, ny=64, precision=c["precision"], seed=seed)
        params, cfg, frame = w.params, w.mhd_config, w.frame
        second = fields.planar_shock_2d(grid, 64, 0.0, 1.0, 0.0, 0.125, r=3.5, w=0.004, x0=0.5)
        dt_out = 0.1
    elif c["flow"] == "shock":
        dt_out = 0.01
        params = dict(p0=P0, pmin=P0, pmax=1e4 * P0, kpara0=0.01, kret=0.05,
                      dt_min_rel=1.0 / c["pushes"], dt_max_rel=1e-2, ndim=2, pbcx=1,
                      precision=c["precision"], seed=seed)
        cfg = make_mhd_config(grid, grid, 1, 0.0, 1.0, 0.0, 1.0, dt_out=dt_out)
        frame = _shock(grid, seed)
        second = _shock(grid, seed + 1) if ti else None
    else:
        dt_out = 0.05
        params = dict(p0=P0, pmin=P0, pmax=10 * P0, kpara0=0.01, kret=0.02,
                      dt_min_rel=0.1 / c["pushes"], dt_max_rel=1.0 / c["pushes"], ndim=3,
                      precision=c["precision"], seed=seed)
        cfg = make_mhd_config(grid, grid, grid, 0.0, 1.0, 0.0, 1.0, dt_out=dt_out, ndim=3)
        frame = _turb3d(grid, seed)
        second = _turb3d(grid, seed + 1) if ti else None
    params = dict(params, nptl_max=2 * n + 64, time_interp=ti)
    eng = _engine(params, cfg, [frame, second] if ti else [frame], np.arange(3) * dt_out)
    if c["flow"] == "turb3d":
        eng.inject_particles_spatial_uniform(n, 1e-7, 2, 1.0, 1, BOX, 1.0)
    else:
        # momenta up to pmax as a shock that has run for a while has them
        eng.inject_particles_at_x(n, 0.5, 1e-7, 2, 1.0, 1, 7.0)
    s = _checkpoint(eng, 2.0)
    s["frame"] = frame
    return s


def _prepare_focused(c, seed):
    n, grid = c["nptl"], c["grid"]
    cfg = make_mhd_config(grid, grid, 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02)
    params = dict(ndim=2, p0=P0, pmin=P0, pmax=1e3 * P0, kpara0=3e-3, kret=0.1,
                  dt_min_rel=1.0 / c["pushes"], dt_max_rel=5e-2, pbcx=1, duu0=10.0, seed=seed,
                  nptl_max=n + 64)
    eng = _engine(params, cfg, [_shock(grid, seed, r=3.0, w=0.02)], np.arange(3) * 0.02)
    eng.inject_particles_spatial_uniform(n, 1e-6, 1, 2.0, 1, BOX)
    return _checkpoint(eng)


def _prepare_sphere(c, seed):
    n, grid = c["nptl"], c["grid"]
    lo, hi = (0.5, 0.6, 0.0), (1.5, math.pi - 0.6, 1.2)
    cfg = make_mhd_config(grid, grid, grid, lo[0], hi[0], lo[1], hi[1], zmin=lo[2], zmax=hi[2],
                          dt_out=0.02, ndim=3)
    rng = np.random.default_rng(seed)
    pos = []
    for a in range(3):
        x = np.concatenate([[0.0], np.cumsum(rng.uniform(0.6, 1.4, grid + 3))])
        pos.append(lo[a] + (x - x[2]) * (hi[a] - lo[a]) / (x[grid + 2] - x[2]))
    params = dict(ndim=3, p0=P0, pmin=0.5 * P0, pmax=1e3 * P0, kpara0=2e-3, kret=0.1,
                  dt_min_rel=1.0 / c["pushes"], dt_max_rel=5e-2, pbcx=1, pbcy=1, spherical_coord=1,
                  nonuniform_grid=1, seed=seed, nptl_max=n + 64)
    eng = _engine(params, cfg, [_turb3d(grid, seed)], np.arange(3) * 0.02, pos)
    box = [lo[a] + 0.1 * (hi[a] - lo[a]) for a in range(3)] + \
          [hi[a] - 0.1 * (hi[a] - lo[a]) for a in range(3)]
    eng.inject_particles_spatial_uniform(n, 1e-6, 1, 1.0, 1, box)
    return _checkpoint(eng)


def _prepare_batch(c, seed):
    runs = []
    rng = np.random.default_rng(seed)
    frame = _shock(c["grid"], seed)
    for r in range(c["nruns"]):
        n = max(64, int(c["nptl"] * 10.0 ** -(1.5 * r / max(1, c["nruns"] - 1))))
        params = dict(p0=P0, pmin=P0, pmax=1e4 * P0, kpara0=10.0 ** rng.uniform(-3, -1),
                      kret=rng.uniform(0.01, 0.2), dt_min_rel=1.0 / c["pushes"], dt_max_rel=1e-2,
                      ndim=2, pbcx=1, precision=1, seed=seed + r, nptl_max=2 * n)
        cfg = make_mhd_config(c["grid"], c["grid"], 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.01)
        eng = _engine(params, cfg, [frame], np.arange(3) * 0.01)
        eng.inject_particles_at_x(n, 0.5, 1e-7, 2, 1.0, 1, 7.0)
        runs.append(_checkpoint(eng, 2.0))
    return dict(runs=runs, batch=Batch([s["eng"] for s in runs]))


def _prepare_learned(c, seed):
    n, grid = c["nptl"], c["grid"]
    params = dict(p0=P0, pmin=P0, pmax=1e3 * P0, kpara0=0.01, kret=0.02,
                  dt_min_rel=0.1 / c["pushes"], dt_max_rel=1.0 / c["pushes"], ndim=3, precision=1,
                  seed=seed, nptl_max=2 * n + 64)
    cfg = make_mhd_config(grid, grid, grid, 0.0, 1.0, 0.0, 1.0, dt_out=0.05, ndim=3)
    eng = _engine(params, cfg, [_turb3d(grid, seed)], np.arange(3) * 0.05)
    eng.inject_particles_spatial_uniform(n, 1e-7, 2, 1.0, 1, BOX, 7.0)
    # a run some intervals in: importances that vary by a third, so that the
    # window splits or kills a few particles
    rng = np.random.default_rng(seed)
    shapes = [(64, 8), (64,), (64, 64), (64,), (64, 64), (64,), (64,), (1,)]
    par = np.concatenate([(rng.normal(size=s) / math.sqrt(s[-1] if len(s) > 1 else 64)).ravel()
                          for s in shapes]).astype(np.float32)
    mean = np.array([0.5, 0.5, 0.5, 0.2, 0.0, 1.0, 5.0, 0.5], np.float32)
    inv = np.array([3.0, 3.0, 3.0, 5.0, 0.2, 3.0, 0.2, 3.0], np.float32)
    mlp = Mlp(seed=1)
    mlp.set_params(par, np.concatenate([mean, inv]))
    z = mlp.forward(mean + rng.normal(size=(4096, 8)).astype(np.float32) / inv)
    par[-65:] *= np.float32(0.3) / z.std()   # the output layer
    mlp.set_params(par)
    s = _checkpoint(eng, 2.0)
    _, lse, lsw = mlp.score(eng, 0.1)
    z_ref, z_floor = window_params(lse, lsw, n)
    set_mover_learned(eng, mlp, 0.2, 1.0, z_ref, 4.0, 3, z_floor)
    s["mlp"] = mlp   # outlives the setting
    return s


def _prepare_newframe(c, seed):
    grid = c["grid"]
    params = dict(p0=P0, pmin=P0, pmax=10 * P0, kpara0=0.01, kret=0.02, dt_min_rel=2e-4,
                  dt_max_rel=2e-3, ndim=3, precision=1, seed=seed, nptl_max=c["nptl"] + 64,
                  time_interp=1)
    cfg = make_mhd_config(grid, grid, grid, 0.0, 1.0, 0.0, 1.0, dt_out=0.05, ndim=3)
    eng = Engine(make_params(**params), cfg, 0)
    eng.set_tstamps(np.arange(4) * 0.05)
    frames = [_turb3d(grid, seed), _turb3d(grid, seed + 1)]
    return dict(eng=eng, frames=frames, counters=eng.counters(), first=ParticleSet.empty(0),
                out=_pinned(c["nptl"] + 64), nptl=c["nptl"])


def _diag_particles(n, grid, seed):
    """A set some time into a shock run: spread about the shock, a power-law
    momentum distribution, weights halved by splitting."""
    rng = np.random.default_rng(seed)
    p = ParticleSet.empty(n).arrays
    p["x"][:] = np.clip(rng.normal(0.5, 0.1, n), 0.0, 1.0)
    p["y"][:] = rng.random(n)
    p["p"][:] = P0 * rng.random(n) ** (-1.0 / 3.0) * 0.9
    p["mu"][:] = rng.uniform(-0.99, 0.99, n)
    p["v"][:] = 1.0
    k = rng.integers(0, 6, n)
    p["weight"][:] = 0.5 ** k
    p["split_times"][:] = k
    p["dt"][:] = 1e-5 * (1.0 + rng.random(n))
    p["count_flag"][:] = 1
    p["tag_injected"][:] = np.arange(n) + 1
    p["tag_splitted"][:] = 1
    return p


LOCAL = dict(pmin=P0, pmax=1e3 * P0, npbins=32, nmu=1, rx=16, ry=16, rz=1)


def _prepare_diag(c, seed):
    n, grid = c["nptl"], c["grid"]
    params = dict(p0=P0, pmin=P0, pmax=1e4 * P0, kpara0=0.01, kret=0.05, dt_min_rel=1e-3, ndim=2,
                  pbcx=1, precision=1, seed=seed, nptl_max=n)
    cfg = make_mhd_config(grid, grid, 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.01)
    eng = Engine(make_params(**params), cfg, 0)
    eng.put_particles(ParticleSet(_diag_particles(n, grid, seed)))
    return dict(eng=eng, nmu=c["nmu"])


def prepare(case, seed):
    s = {"frame": _prepare_frame, "focused": _prepare_focused, "sphere": _prepare_sphere,
         "batch": _prepare_batch, "learned": _prepare_learned, "newframe": _prepare_newframe,
         "diag": _prepare_diag}[case["kind"]](case, seed % 1_000_003)
    s["case"] = dict(case)
    return s


# -- one pass ----------------------------------------------------------------------
# Sets come back in buffers of the checkpoint's capacity, zero past their end,
# so that they have one shape whatever splits or leaves.
def _by_tags(s):
    """The set on the GPU in the order of its lineage tags."""
    ps = s["eng"].get_particles(s["out"])
    a = {k: torch.from_numpy(v.view(np.int32) if v.dtype == np.uint32 else v).cuda()
         for k, v in ps.arrays.items()}
    key = (a["tag_injected"].long() << 32) | (a["tag_splitted"].long() & 0xFFFFFFFF)
    order = torch.argsort(key)
    cap = len(s["out"])
    return {k: torch.cat([v[order], v.new_zeros(cap - len(v))]) for k, v in a.items()}


def _in_order(s):
    """The set in its own order (the FP64 path keeps it)."""
    s["eng"].get_particles(s["out"])
    return {k: v.view(np.int32) if v.dtype == np.uint32 else v
            for k, v in s["out"].arrays.items()}


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "diag":
        eng = s["eng"]
        f, n = eng.calc_particle_distributions()
        fm, nm = eng.particle_distributions_mu(s["nmu"])
        fl, nl = eng.local_distribution(**LOCAL)
        return dict(f=f, n=n.view(np.int64), fm=fm, nm=nm.view(np.int64), fl=fl,
                    nl=nl.view(np.int64), check=eng.quick_check(), pmax=eng.get_pmax_global())
    if kind == "newframe":
        eng = s["eng"]
        _restore(s)
        for k in (0, 1):
            eng.set_fields(s["frames"][k], k)
            eng.calc_fields_gradients(k)
        ncells = eng.count_cells_large(_abi.LARGE_DIVV, 1.0, BOX)
        eng.inject_particles_at_large(_abi.LARGE_DIVV, s["nptl"], 1e-7, 2, 1.0, 1, True, 1.0, 1,
                                      BOX, 1.0)
        particles = _in_order(s)
        eng.copy_fields()
        return dict(particles=particles, ncells=ncells, shock=eng.locate_shock_xpos())
    if kind == "batch":
        for r in s["runs"]:
            _restore(r)
        s["batch"].particle_mover()
        res = []
        for r in s["runs"]:
            eng = r["eng"]
            eng.split_particle(2.72, 2.0)
            f, n = eng.calc_particle_distributions()
            a = _by_tags(r)
            res.append(dict(f=f, n=n.view(np.int64), rng_ctr=a["rng_ctr"],
                            **{k: a[k] for k in ("x", "y", "p", "t", "weight")}))
        return res
    eng = s["eng"]
    _restore(s)
    eng.particle_mover(focused_transport=kind == "focused")
    if c.get("split"):
        eng.split_particle(2.72, 2.0)
    if kind == "focused":
        f, n = eng.particle_distributions_mu(8)
    else:
        f, n = eng.calc_particle_distributions()
    res = dict(f=f, n=n.view(np.int64), check=eng.quick_check(),
               steps=int(eng.counters().last_mover_steps))
    if kind == "learned":
        res["learned"] = mover_learned_stats(eng)
    res["particles"] = _by_tags(s) if eng.params.precision == _abi.PREC_MIXED else _in_order(s)
    return res


# -- what a pass cannot do without ---------------------------------------------------
STATE = 98   # bytes of a particle's record


def work(case):
    kind, n, grid = case["kind"], case["nptl"], case["grid"]
    # floating-point operations of one push: 4 or 8 corners of the fields and
    # gradients it reads, kappa and its gradients, drift, step, noise
    per = {2: 300, 3: 700}
    if kind == "frame":
        d = 3 if case["flow"] == "turb3d" else 2
        nodes = grid ** 3 if d == 3 else grid * (64 if case["flow"] == "planar" else grid)
        # 3D: steps between dt_max and dt_max / 10, starts spread over the interval
        pushes = case["pushes"] * (0.5 * 2.5 if d == 3 else 1.0)
        if case["flow"] == "planar":
            pushes = 300
        return {"bytes": 2.0 * STATE * n + 32.0 * nodes * (1 + case["time_interp"]),
                "flops": float(n) * pushes * per[d]}
    if kind in ("focused", "sphere"):
        d = 3 if kind == "sphere" else 2
        return {"bytes": 2.0 * STATE * n + 32.0 * grid ** d,
                "flops": float(n) * 0.5 * case["pushes"] * (per[d] + 200)}
    if kind == "batch":
        total = sum(max(64, int(n * 10.0 ** -(1.5 * r / max(1, case["nruns"] - 1))))
                    for r in range(case["nruns"]))
        return {"bytes": 2.0 * STATE * total + 32.0 * grid ** 2,
                "flops": float(total) * case["pushes"] * per[2]}
    if kind == "learned":
        return {"bytes": 2.0 * STATE * n + 32.0 * grid ** 3,
                "flops": float(n) * (0.5 * 2.5 * case["pushes"] * per[3] + 2 * 8961)}
    if kind == "newframe":
        return {"bytes": 2 * 32.0 * (grid + 4) ** 3 * 4 + STATE * n,
                "flops": 2 * 24.0 * 3 * grid ** 3}
    nl = 2 * 8 * 32 * (-(-grid // 16)) ** 2
    return {"bytes": n * (8.0 * 6) + nl + 16.0 * 128 * (1 + case["nmu"]), "flops": 40.0 * n}


# -- the same in 64 bits, without the engine -----------------------------------------
def exact(case, seed):
    if case["kind"] == "diag":
        return _exact_diag(case, seed % 1_000_003)
    if case["kind"] == "frame" and case["flow"] != "turb3d" and not case["precision"] and \
            not case["time_interp"]:
        # in split precision rounding decides whether the last push of an
        # interval lands or is redone with other increments: no such value
        return _exact_frame(case, seed % 1_000_003)
    return None


def _exact_diag(case, seed):
    n, grid, nmu = case["nptl"], case["grid"], case["nmu"]
    p = _diag_particles(n, grid, seed)
    lo, hi = math.log10(P0), math.log10(1e4 * P0)
    npp = 128
    ok = (p["p"] > P0) & (p["p"] <= 1e4 * P0)
    ip = np.floor((np.log10(p["p"]) - lo) / ((hi - lo) / npp)).astype(np.int64)
    ok &= (ip >= 0) & (ip < npp)
    w = p["weight"]
    f = np.bincount(ip[ok], w[ok], npp)
    dmu = float(np.float32(2.0) / np.float32(nmu))
    im = np.floor((p["mu"] + 1.0) / dmu).astype(np.int64)
    okm = ok & (im >= 0) & (im < nmu)
    fm = np.bincount(ip[okm] * nmu + im[okm], w[okm], npp * nmu).reshape(npp, nmu)
    nr = -(-grid // LOCAL["rx"])
    lp = (math.log10(LOCAL["pmax"]) - math.log10(LOCAL["pmin"])) / LOCAL["npbins"]
    il = np.floor((np.log10(p["p"]) - math.log10(LOCAL["pmin"])) / lp).astype(np.int64) + 1
    ix = np.floor(p["x"] / (1.0 / nr)).astype(np.int64)
    iy = np.floor(p["y"] / (1.0 / nr)).astype(np.int64)
    okl = (il > 0) & (il < LOCAL["npbins"]) & (ix >= 0) & (ix < nr) & (iy >= 0) & (iy < nr)
    nb = LOCAL["npbins"]
    fl = np.bincount((iy[okl] * nr + ix[okl]) * nb + il[okl] - 1, w[okl], nr * nr * nb)
    dt = p["dt"]
    check = dict(nptl_current=float(n), nptl_split=0.0, ntot=float(w.sum()), leak=0.0,
                 leak_negp=0.0, pdt_min=float(dt.min()), pdt_max=float(dt.max()),
                 pdt_avg=math.fsum(dt) / n)
    return dict(f=f, n=None, fm=fm, nm=None, fl=fl.reshape(1, nr, nr, nb, 1), nl=None, check=check,
                pmax=float(p["p"].max()))


def _philox(ctr, word, ti, ts, key0, key1):
    """Philox-4x32-10 on int64 tensors holding 32-bit words."""
    m32 = 0xFFFFFFFF
    c = [ctr & m32, torch.full_like(ctr, word), ti & m32, ts & m32]
    k = [key0, key1]
    for r in range(10):
        if r:
            k = [(k[0] + 0x9E3779B9) & m32, (k[1] + 0xBB67AE85) & m32]
        a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((b >> 32) & m32) ^ c[1] ^ k[0], b & m32, ((a >> 32) & m32) ^ c[3] ^ k[1], a & m32]
    return c


def _exact_frame(case, seed):
    """push_particle_2d (particle_module.f90:3358-3606) and the mover cycle
    around it (:1481-1833) for the 2D shock cases, over all particles at once."""
    s = _prepare_frame(case, seed)
    eng, first, frame = s["eng"], s["first"], s["frame"]
    prm, cfg = eng.params, eng.cfg
    dev = "cuda"
    a = {k: torch.from_numpy(v.astype(np.float64 if v.dtype.kind == "f" else np.int64)).to(dev)
         for k, v in first.arrays.items()}
    f8 = torch.from_numpy(frame[0]).to(dev).double()        # (nyg, nxg, 8)
    nyg, nxg = f8.shape[:2]
    dx, dy = cfg.dx, cfg.dy
    gx = torch.gradient(f8, dim=1, edge_order=2)[0] / dx
    gy = torch.gradient(f8, dim=0, edge_order=2)[0] / dy
    # vx vy bx by bz dvx/dx dvy/dy dbx/dx dbx/dy dby/dx dby/dy dbz/dx dbz/dy db/dx db/dy
    rec = torch.stack([f8[..., 0], f8[..., 1], f8[..., 4], f8[..., 5], f8[..., 6], gx[..., 0],
                       gy[..., 1], gx[..., 4], gy[..., 4], gx[..., 5], gy[..., 5], gx[..., 6],
                       gy[..., 6], gx[..., 7], gy[..., 7]], -1).reshape(-1, 15)
    dtf = 0.1 if case["flow"] == "planar" else 0.01
    dtmin, dtmax = prm.dt_min_rel * dtf, prm.dt_max_rel * dtf
    key0, key1 = prm.seed & 0xFFFFFFFF, prm.seed >> 32
    x, y, p, t, dt = a["x"], a["y"], a["p"], a["t"], a["dt"]
    ctr, ti, ts, nsp = a["rng_ctr"], a["tag_injected"], a["tag_splitted"], a["nsteps_pushed"]
    flag = a["count_flag"].clone()
    xlo, xhi = cfg.xmin, cfg.xmin + cfg.nx * dx
    ylo, yhi = cfg.ymin, cfg.ymin + cfg.ny * dy
    leak = 0.0

    def bounds(x, y, flag, h):
        nonlocal leak
        out = (flag == 1) & ((x < xlo - h * dx) | (x > xhi + h * dx))
        leak += float(a["weight"][out].sum())
        flag = torch.where(out, torch.where(x < xlo, -1, -2), flag)
        per = (yhi + h * dy) - (ylo - h * dy)
        y = torch.where((flag == 1) & (y < ylo - h * dy), y + per, y)
        y = torch.where((flag == 1) & (y > yhi + h * dy), y - per, y)
        return y, flag

    def push(x, y, p, dt, fixed, ctr):
        px, py = (x - xlo) / dx, (y - ylo) / dy
        ix, iy = px.floor().clamp(-2, nxg - 4), py.floor().clamp(-2, nyg - 4)
        rx, ry = px - ix, py - iy
        base = (iy.long() + 2) * nxg + ix.long() + 2
        v = 0.0
        for j in (0, 1):
            for i in (0, 1):
                wt = (rx if i else 1.0 - rx) * (ry if j else 1.0 - ry)
                v = v + rec[base + i + nxg * j] * wt[:, None]
        vx, vy, bx, by, bz, dvx, dvy, bxx, bxy, byx, byy, bzx, bzy, mx, my = v.unbind(1)
        b = (bx * bx + by * by + bz * bz).sqrt()
        ib = 1.0 / b
        kpara = prm.kpara0 * (p / prm.p0) ** prm.pindex
        kperp = kpara * prm.kret
        kpp = kpara - kperp
        sa, sr, sp = (2 * kpara).sqrt(), (2 * kperp).sqrt(), (2 * kpp).sqrt()
        i2, i3 = ib * ib, ib * ib * ib
        kxx = 2 * kpp * bx * (bxx * b - bx * mx) * i3
        kyy = 2 * kpp * by * (byy * b - by * my) * i3
        kxyx = kpp * ((bxx * by + bx * byx) * i2 - 2 * bx * by * mx * i3)
        kxyy = kpp * ((bxy * by + bx * byy) * i2 - 2 * bx * by * my * i3)
        q1, q2 = prm.drift1 * prm.p0 / p, prm.drift2 * prm.p0 ** 2 / (p * p)
        vd = float(np.float32(1.0) / np.float32(3 * prm.charge)) / (q1 * q1 + q2 * q2).sqrt()
        ax = vx + vd * (bzy * i2 - 2 * bz * my * i3) + kxx + kxyy
        ay = vy + vd * (2 * bz * mx * i3 - bzx * i2) + kxyx + kyy
        ap = -p * (dvx + dvy) / 3.0
        m = torch.minimum((0.5 * dx / sa) ** 2, (0.5 * dy / sa) ** 2)
        m = torch.minimum(m, torch.minimum((sr / ax) ** 2, (sr / ay) ** 2))
        m = torch.minimum(m, float(np.float32(0.1)) * p / ap.abs())
        m = torch.where((ax != 0) & (ay != 0) & (ap != 0), m, torch.full_like(m, dtmin))
        dt = torch.where(fixed, dt, m.clamp(dtmin, dtmax))
        w = _philox(ctr, 0, ti, ts, key0, key1) + _philox(ctr, 1, ti, ts, key0, key1)
        r = [(2.0 * ((w[2 * k] >> 5) * 67108864 + (w[2 * k + 1] >> 6)).double() / 2.0 ** 53 - 1.0)
             * math.sqrt(3.0) for k in range(3)]
        sd = dt.sqrt()
        return (ax * dt + r[0] * sr * sd + r[2] * sp * sd * bx * ib,
                ay * dt + r[1] * sr * sd + r[2] * sp * sd * by * ib, ap * dt, dt)

    def apply(go, x, y, p, t, ctr, d):
        pn = p + d[2]
        low = pn < 0.25 * prm.p0
        dp = torch.where(low, 0.25 * prm.p0 - p, d[2])
        return (torch.where(go, x + d[0], x), torch.where(go, y + d[1], y),
                torch.where(go, torch.where(low, torch.full_like(p, 0.25 * prm.p0), pn), p),
                torch.where(go, t + d[3], t), torch.where(go, ctr + 1, ctr), dp)

    last = [torch.zeros_like(x) for _ in range(3)]
    for it in range(10 ** 6):
        go = (flag == 1) & (t < dtf)
        if it % 16 == 0 and not bool(go.any()):
            break
        yb, fb = bounds(x, y, torch.where(go, flag, torch.zeros_like(flag)), 0.5)
        y, flag = torch.where(go, yb, y), torch.where(go, fb, flag)
        go = go & (flag == 1)
        d = push(x, y, p, dt, torch.zeros_like(go), ctr)
        x, y, p, t, ctr, dp = apply(go, x, y, p, t, ctr, d)
        dt = torch.where(go, d[3], dt)
        last = [torch.where(go, u, l) for u, l in zip((d[0], d[1], dp), last)]
    over = (flag == 1) & (t > dtf)
    x, y, p, t = (torch.where(over, u - l, u) for u, l in zip((x, y, p, t), last + [dt]))
    rest = dtf - t
    redo = over & (rest > 0)
    d = push(x, y, p, rest, torch.ones_like(redo), ctr)
    x, y, p, t, ctr, _ = apply(redo, x, y, p, t, ctr, d)
    yb, fb = bounds(x, y, flag, 0.5)
    y, flag = yb, fb
    y, flag = bounds(x, y, flag, 0.0)
    keep = flag == 1
    g = {k: v[keep] for k, v in dict(a, x=x, y=y, p=p, t=t, dt=dt).items()}
    parents = g["p"].numel()
    if case.get("split"):
        sel = (g["p"] > 2.0 * prm.p0 * 2.72 ** g["split_times"].double()) & (g["p"] <= prm.pmax)
        g["weight"][sel] = 0.5 ** (g["split_times"][sel] + 1).double()
        kids = {k: v[sel].clone() for k, v in g.items()}
        kids["tag_splitted"] = kids["tag_splitted"] + 2 ** kids["split_times"]
        g = {k: torch.cat([v, kids[k]]) for k, v in g.items()}
    total = g["weight"]
    lo, hi = math.log10(prm.pmin), math.log10(prm.pmax)
    ok = (g["p"] > prm.pmin) & (g["p"] <= prm.pmax)
    ip = ((g["p"].log10() - lo) / ((hi - lo) / prm.npp_global)).floor().long()
    ok &= (ip >= 0) & (ip < prm.npp_global)
    f = torch.zeros(prm.npp_global, dtype=torch.float64, device=dev)
    f.index_add_(0, ip[ok], total[ok])
    check = dict(nptl_current=float(len(total)), nptl_split=float(len(total) - parents),
                 ntot=float(total.sum()), leak=leak, leak_negp=0.0, pdt_min=float(g["dt"].min()),
                 pdt_max=float(g["dt"].max()), pdt_avg=float(g["dt"].mean()))
    cap = len(s["out"])
    part = {k: torch.cat([v, v.new_zeros(cap - len(v))]).cpu()
            if k in ("x", "y", "z", "p", "v", "mu", "weight", "t", "dt") else None
            for k, v in g.items()}
    return dict(f=f.cpu(), n=None, check=check, steps=None, particles=part)
