"""Both builds of the FP64 mover (mover_fp64.cu with one lane a particle, and with
teams of eight for calls of up to 16 particles an SM) and the work order (more than
128 an SM), for every kind of run: against the oracle just above the teams' limit
and at it, and particle for particle the same bits in calls of all three sizes,
which the kinds that call pow(), sin() or log() are compared by as well.

Tolerances against the oracle are those of the tests of each kind: equal bits
without library functions on the path, else 1e-9 relative (spherical focused
transport 1e-5) on 99.5 % of the particles."""
import math

import numpy as np
import pytest

import oracle
from gpat import fields
from gpat.engine import Engine, ParticleSet, make_mhd_config, make_params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

STATE = ("x", "y", "z", "p", "v", "mu", "weight", "t", "dt", "count_flag", "nsteps_pushed",
         "tag_injected", "tag_splitted", "rng_ctr")
FT = dict(focused_transport=True)
NLGC = dict(nlgc=True, kperp_kpara=0.05)


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() \
        else 152


# name: (ndim, engine options, mover options, exact against the oracle); options in
# capitals are the grid's and the arrays', the others make_params'
KINDS = {
    "1d": (1, {}, {}, True),
    "1d_nonuniform_nlgc_wave": (1, dict(NONUNIFORM=1, dpp_wave=1), NLGC, True),
    "1d_spherical": (1, dict(SPHERICAL=1), {}, False),
    "1d_focused": (1, dict(duu0=0.0), FT, True),
    "1d_focused_scattering": (1, dict(duu0=3.0), FT, False),
    "2d": (2, {}, {}, True),
    "2d_drift_z": (2, dict(check_drift_2d=1, BZ=0.4), {}, True),
    "2d_bz": (2, dict(BZ=0.4), {}, True),
    "2d_no_diffusion": (2, dict(kpara0=0.0), {}, True),
    "2d_two_frames": (2, dict(time_interp=1), {}, True),
    "2d_kappa_p_b": (2, dict(momentum_dependency=1, mag_dependency=1), {}, False),
    "2d_gaussian": (2, dict(noise=1), {}, False),
    "2d_nlgc": (2, {}, NLGC, True),
    "2d_region": (2, dict(acc_region_flag=1, acc_region=(0.0, 0.5, 0.0, 0.7, 0.0, 1.0)), {}, True),
    "2d_wave": (2, dict(dpp_wave=1), {}, True),
    "2d_shear": (2, dict(dpp_shear=1, weak_scattering=1, tau0=0.5), {}, False),
    "2d_variance": (2, dict(deltab_flag=1, FLUCT="variance"), {}, True),
    "2d_fluctuations_nlgc": (2, dict(deltab_flag=1, correlation_flag=1, FLUCT="all"), NLGC, False),
    "2d_nonuniform": (2, dict(NONUNIFORM=1), {}, True),
    "2d_spherical": (2, dict(SPHERICAL=1), {}, False),
    "2d_spherical_nonuniform": (2, dict(SPHERICAL=1, NONUNIFORM=1), {}, False),
    "2d_include_3rd": (2, dict(include_3rd_dim=1, BZ=0.4), {}, True),
    "2d_include_3rd_spherical": (2, dict(include_3rd_dim=1, BZ=0.4, SPHERICAL=1), {}, False),
    "2d_focused": (2, dict(duu0=0.0), FT, True),
    "2d_focused_scattering": (2, dict(duu0=10.0), FT, False),
    "2d_focused_spherical": (2, dict(duu0=3.0, SPHERICAL=1, momentum_dependency=1), FT, 1e-5),
    "2d_focused_variance": (2, dict(duu0=0.0, deltab_flag=1, FLUCT="variance"), FT, True),
    "2d_focused_include_3rd": (2, dict(include_3rd_dim=1, BZ=0.4, duu0=0.0), FT, True),
    "3d": (3, {}, {}, True),
    "3d_two_frames_nlgc": (3, dict(time_interp=1), NLGC, True),
    "3d_wave_shear": (3, dict(dpp_wave=1, dpp_shear=1, momentum_dependency=1), {}, False),
    "3d_nonuniform": (3, dict(NONUNIFORM=1), {}, True),
    "3d_spherical": (3, dict(SPHERICAL=1), {}, False),
    "3d_surfaces": (3, dict(time_interp=1, acc_region_flag=1, SURFACES=1), {}, True),
    "3d_focused": (3, dict(duu0=0.0), FT, True),
    "3d_focused_scattering": (3, dict(duu0=10.0), FT, False),
}


def _stretched(n, lo, hi, seed):
    h = np.random.default_rng(seed).uniform(0.6, 1.4, n + 3)
    x = np.concatenate([[0.0], np.cumsum(h)])
    return lo + (x - x[2]) * (hi - lo) / (x[n + 2] - x[2])


def _smooth(n, seed, lo, hi):
    rng = np.random.default_rng(seed)
    x = fields.node_coords(n, 0.0, 1.0 / n)
    X, Y = np.meshgrid(x, x)
    f = sum(np.sin(2 * np.pi * (a * X + b * Y) + c) for a, b, c in
            zip(rng.integers(1, 4, 4), rng.integers(1, 4, 4), rng.uniform(0, 6.28, 4)))
    f = (f - f.min()) / (f.max() - f.min())
    return (lo + (hi - lo) * f)[None].astype(np.float32)


def _height(n, seed, base, amp):
    u = np.linspace(0.0, 1.0, n + 4)
    A, B = np.meshgrid(u, u)
    return base + amp * np.sin(2 * np.pi * (A + B) + seed)


def _frame(ndim, n, lo, hi, seed, bz):
    if ndim == 3:
        return fields.turbulence_3d(n, seed=seed)
    if ndim == 2:
        db = fields.kolmogorov_az_2d(n, n, 1.0, 1.0, 0.5, 2 * np.pi, np.pi * n / 2, seed)
        f = fields.planar_shock_2d(n, n, 0.0, 1.0, 0.0, 1.0, u1=1.0, r=3.0, w=0.05, x0=0.5, db=db)
        if bz:
            f = f.astype(np.float64)
            x = np.linspace(0, 1, n + 4)
            X, Y = np.meshgrid(x, x)
            f[0, :, :, 2] = 0.1 * np.sin(2 * np.pi * X)
            f[0, :, :, 6] = bz + 0.2 * np.cos(2 * np.pi * Y)
            f[0, :, :, 7] = np.sqrt((f[0, :, :, 4:7] ** 2).sum(-1))
        return f.astype(np.float32)
    x = np.linspace(lo, hi, n + 4)[None, None, :]
    z = np.zeros((1, 1, n + 4))
    vx = 1.0 - 0.6 * (1 + np.tanh((x - 0.5 * (lo + hi)) / 0.05)) / 2
    by = 0.5 + 0.2 * np.sin(2 * np.pi * (x - lo) / (hi - lo))
    return fields.assemble_frame(vx + z, 0.1 * by + z, z, 1.0 + z, 1.0 + z, by + z,
                                 0.3 + z).astype(np.float32)


class _Run:
    """One kind of run, in the engine and the oracle."""

    def __init__(self, kind, nptl):
        ndim, opts, self.mover_kw, self.exact = KINDS[kind]
        o = dict(opts)
        sph, non = o.pop("SPHERICAL", 0), o.pop("NONUNIFORM", 0)
        bz, fluct, surfaces = o.pop("BZ", 0.0), o.pop("FLUCT", None), o.pop("SURFACES", 0)
        n = {1: 64, 2: 32, 3: 16}[ndim]
        lo, hi = ((0.5, 0.6, 0.0), (1.5, math.pi - 0.6, 1.2)) if sph else ((0.0,) * 3, (1.0,) * 3)
        if ndim == 1:
            lo, hi = (lo[0], 0.0, 0.0), (hi[0], 1.0, 1.0)
        elif ndim == 2:
            lo, hi = lo[:2] + (0.0,), hi[:2] + (1.0,)
        self.cfg = cfg = make_mhd_config(n, n if ndim > 1 else 1, n if ndim == 3 else 1, lo[0], hi[0],
                                         lo[1], hi[1], zmin=lo[2], zmax=hi[2], dt_out=0.02, ndim=ndim)
        base = dict(ndim=ndim, p0=0.1, pmin=0.05, pmax=100.0, kpara0=2e-3, kret=0.1, dt_min_rel=1e-2,
                    dt_max_rel=1e-1, pbcx=1, pbcy=0 if ndim == 2 else 1, pbcz=0, momentum_dependency=0,
                    nptl_max=nptl, seed=31, spherical_coord=sph, nonuniform_grid=non)
        base.update(o)
        self.prm = prm = make_params(**base)
        self.eng = eng = Engine(prm, cfg, 0)
        eng.set_tstamps(np.arange(4) * 0.02)
        d = (cfg.dx, cfg.dy, cfg.dz)
        self.pos = [_stretched(n, lo[a], hi[a], 3 + a) if non else
                    oracle.uniform_grid_positions(n + 4, d[a], lo[a]) for a in range(ndim)]
        if non:
            eng.set_grid_positions(*self.pos)
        two = base.get("time_interp", 0)
        frames = [_frame(ndim, n, lo[0], hi[0], 3 + k, bz) for k in range(1 + two)]
        for k, f in enumerate(frames):
            eng.set_fields(f, k)
            eng.calc_fields_gradients(k)
        self._grid()
        self.full = [oracle.full_fields(f, ndim, cfg, nonuniform=bool(non)) for f in frames]
        for k, f in enumerate(self.full):
            assert np.array_equal(eng.get_fields(k), f)
        self.aux = None
        if fluct:
            arrays = (_smooth(n, 1, 0.5, 2.0),) + ((None,) * 3 if fluct == "variance" else
                                                   tuple(_smooth(n, s, 0.4, 1.4) for s in (2, 3, 4)))
            eng.set_fluctuations(0, *arrays)
            self.aux = oracle.aux_fields(*arrays, ndim, cfg)
        self.surfaces = None
        if surfaces:
            s = [_height(n, k, 0.4 + 0.05 * k, 0.15) for k in range(4)]
            eng.init_acc_surface("+z", "-x", True)
            eng.set_acc_surface(0, s[0], s[2])
            eng.set_acc_surface(1, s[1], s[3])
            self.surfaces = dict(norm2="-x", s21=s[2], s22=s[3], intersection=True,
                                 shape=(n + 4,) * 3), s[0], s[1]
        box = tuple(lo[a] + 0.1 * (hi[a] - lo[a]) for a in range(3)) + \
            tuple(hi[a] - 0.1 * (hi[a] - lo[a]) for a in range(3))
        eng.inject_particles_spatial_uniform(nptl, 1e-6, 1, 2.0, 1, box)
        self.start = eng.get_particles()

    def _grid(self):
        oracle.set_grid_positions(*(self.pos + [None] * (3 - len(self.pos))))

    def moved(self, n):
        """The first n particles over an interval, by tag."""
        self.eng.put_particles(self.start.take(np.arange(n)))
        before = self.eng.counters().steps
        self.eng.particle_mover(mhd_tframe=1, num_fine_steps=2, **self.mover_kw)
        return self.eng.get_particles().order_by_tags(), self.eng.counters().steps - before

    def oracle(self, n):
        parts = oracle.Particles(n, self.start.take(np.arange(n)).arrays)
        cnt = oracle.OrcCounters()
        kw = dict(self.mover_kw)
        if len(self.full) > 1:
            kw["f2"] = self.full[1]
        if self.aux is not None:
            kw["aux1"] = self.aux
        self._grid()
        if self.surfaces:
            skw, s1, s2 = self.surfaces
            oracle.set_acc_surface("+z", s1, s2, **skw)
        try:
            oracle.mover(oracle.params_from(self.prm), oracle.config_from(self.cfg), self.full[0],
                         parts, 0.0, 0.02, num_fine_steps=2, counters=cnt, **kw)
        finally:
            oracle.set_grid_positions(None)
            if self.surfaces:
                oracle.set_acc_surface(None)
        return ParticleSet(parts.view()).order_by_tags(), cnt.steps


@pytest.mark.parametrize("kind", KINDS)
def test_all_sizes_of_call(kind):
    team, order = 16 * _sms(), 128 * _sms() + 1
    run = _Run(kind, order)
    try:
        results = {n: run.moved(n) for n in (team, team + 1, order)}
        # the same particles, whatever the size of the call
        whole = results[order][0]
        for n in (team, team + 1):
            got = results[n][0]
            at = np.isin(whole["tag_injected"], run.start["tag_injected"][:n])
            assert len(got) == at.sum() > 0.3 * n
            for k in STATE:
                assert np.array_equal(got[k], whole[k][at]), (n, k)
        for n in (team, team + 1):
            got, steps = results[n]
            ref, ref_steps = run.oracle(n)
            if run.exact is True:
                assert len(got) == len(ref) and steps == ref_steps
                for k in STATE:
                    if k in ("v", "mu") and not run.mover_kw.get("focused_transport"):
                        continue
                    assert np.array_equal(got[k], ref[k]), (n, k)
            else:
                rtol = run.exact or 1e-9
                both = np.intersect1d(got["tag_injected"], ref["tag_injected"])
                assert len(both) >= 0.995 * max(len(got), len(ref))
                g = got.take(np.isin(got["tag_injected"], both))
                r = ref.take(np.isin(ref["tag_injected"], both))
                ok = np.ones(len(g), bool)
                for k in ("x", "y", "z", "p", "t"):
                    ok &= np.isclose(g[k], r[k], rtol=rtol, atol=rtol * 1e-3)
                assert ok.mean() >= 0.995, (n, ok.mean())
                assert abs(steps - ref_steps) <= 1e-2 * ref_steps
    finally:
        run.eng.close()
        oracle.set_grid_positions(None)


@pytest.mark.parametrize("extra", [0, 1])
def test_tracked_particles(extra):
    """Particle records at the teams' limit and above it, against the oracle."""
    from test_gpu_tracking import _equal, _records_equal, _table
    n = 16 * _sms() + extra
    cfg = make_mhd_config(32, 32, 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02)
    prm = make_params(ndim=2, p0=0.1, pmin=0.1, pmax=100.0, kpara0=1e-2, kret=0.1, dt_min_rel=5e-3,
                      dt_max_rel=5e-2, pbcx=1, pbcy=0, momentum_dependency=0, nptl_max=2 * n, seed=11)
    frame = _frame(2, 32, 0.0, 1.0, 5, 0.0)
    eng = Engine(prm, cfg, 0)
    eng.set_tstamps(np.arange(4) * 0.02)
    eng.set_fields(frame, 0)
    eng.calc_fields_gradients(0)
    eng.init_particle_tracking(_table(), 3)
    trk = oracle.Tracking(_table(), prm.dt_min_rel, 3)
    try:
        box = (0.0, 0.0, 0.0, 1.0, 1.0, 1.0)
        eng.inject_particles_spatial_uniform(n, 1e-6, 1, 2.0, 1, box)
        oprm, parts, cnt = oracle.params_from(prm), oracle.Particles(2 * n), oracle.OrcCounters()
        oracle.inject_spatial_uniform(oprm, parts, n, 1e-6, 1, 2.0, 0.0, 0.02, box, cnt)
        eng.particle_mover(mhd_tframe=1, nsteps_interval=3, num_fine_steps=2)
        oracle.mover(oprm, oracle.config_from(cfg), oracle.full_fields(frame, 2, cfg), parts, 0.0, 0.02,
                     counters=cnt, nsteps_interval=3, num_fine_steps=2)
        _equal(eng.get_particles(), parts)
        rec = eng.get_tracked_particles()
        _records_equal(rec, trk.sync())
        assert (rec["tag_splitted"] < 0).sum() > 8
    finally:
        trk.detach()
        eng.close()
