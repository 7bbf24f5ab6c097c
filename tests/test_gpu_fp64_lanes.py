"""The FP64 mover's work list and its integer forms, bit for bit against the
oracle: fewer particles than warps, the most that are moved in teams of lanes
and one more, one more than the lanes of the small grid (taken in work order),
enough for the large grid; cells of different sizes; fields with subnormal
values and zeros."""
import numpy as np
import pytest

import oracle
from gpat import fields
from gpat.engine import Engine, ParticleSet, make_mhd_config, make_params

pytestmark = pytest.mark.gpu

STATE = ("x", "y", "z", "p", "mu", "weight", "t", "dt", "count_flag", "nsteps_pushed",
         "tag_injected", "tag_splitted", "rng_ctr")
BOX = (0.0, 0.0, 0.0, 1.0, 1.0, 1.0)


def _pair(ndim, n, frame, second=None, shape=(32, 32, 1), **kw):
    """n particles with start times spread over the interval, in both."""
    base = dict(ndim=ndim, p0=0.1, pmin=0.1, pmax=1.0, kpara0=3e-3, kret=0.1, dt_min_rel=2e-2,
                dt_max_rel=2e-1, pbcx=1, pbcy=0, pbcz=0, momentum_dependency=0, nptl_max=n, seed=17,
                time_interp=int(second is not None))
    base.update(kw)
    nx, ny, nz = shape
    cfg = make_mhd_config(nx, ny, nz, 0.0, 1.0, 0.0, 1.0, dt_out=0.02, ndim=ndim)
    prm = make_params(**base)
    eng = Engine(prm, cfg, 0)
    eng.set_tstamps(np.arange(4) * 0.02)
    full = []
    for k, f in enumerate([frame] if second is None else [frame, second]):
        eng.set_fields(f, k)
        eng.calc_fields_gradients(k)
        full.append(eng.get_fields(k))
    eng.inject_particles_spatial_uniform(n, 1e-6, 2, 1.0, 1, BOX, 1.0)
    parts = oracle.Particles(n, eng.get_particles().arrays)
    eng.particle_mover(mhd_tframe=1)
    cnt = oracle.OrcCounters()
    extra = {} if second is None else dict(f2=full[1])
    oracle.mover(oracle.params_from(prm), oracle.config_from(cfg), full[0], parts, 0.0, 0.02,
                 counters=cnt, **extra)
    # the oracle removes escaped particles by swapping, the engine keeps the order
    got, ref = eng.get_particles().order_by_tags(), ParticleSet(parts.view()).order_by_tags()
    assert len(got) == len(ref)
    for k in STATE:
        assert np.array_equal(got[k], ref[k]), k
    assert eng.counters().steps == cnt.steps
    eng.close()
    return got


def _frame2d(nx, ny, seed=3):
    db = fields.kolmogorov_az_2d(nx, ny, 1.0, 1.0, 0.5, 2 * np.pi, np.pi * min(nx, ny) / 2, seed)
    return fields.planar_shock_2d(nx, ny, 0.0, 1.0, 0.0, 1.0, r=3.0, w=0.05, x0=0.5, db=db)


@pytest.mark.parametrize("n", [1, 3, 700, 2432, 2433, 19457, 97281])
def test_particle_counts_around_the_grids(n):
    _pair(2, n, _frame2d(32, 32))


@pytest.mark.parametrize("ndim,shape", [(2, (32, 20, 1)), (3, (20, 12, 16))])
def test_cells_of_different_sizes_and_two_frames(ndim, shape):
    if ndim == 2:
        frames = [_frame2d(shape[0], shape[1], s) for s in (3, 4)]
    else:
        cube = [fields.turbulence_3d(32, seed=s) for s in (3, 4)]
        frames = [np.ascontiguousarray(c[:shape[2] + 4, :shape[1] + 4, :shape[0] + 4])
                  for c in cube]
    _pair(ndim, 4000, frames[0], frames[1], shape=shape)


@pytest.mark.parametrize("what", ["zeros", "subnormal"])
def test_fields_with_special_values(what):
    f = _frame2d(32, 32).copy()
    if what == "zeros":
        f[0, ::3, ::2, 0:3] = 0.0      # velocities 0 beside values of both signs
    else:
        f[0, ::5, ::4, 1] = 1e-41      # vy
        f[0, ::7, ::3, 6] = -3e-43     # Bz
    _pair(2, 2000, f)
