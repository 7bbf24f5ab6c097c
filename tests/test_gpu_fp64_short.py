"""The FP64 mover where particles make one to a few pushes an interval, so that lanes
wait for the others of their warp before they take the next particle: more particles
than lanes, in work order, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
from gpat import fields
from gpat.engine import Engine, ParticleSet, make_mhd_config, make_params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

STATE = ("x", "y", "z", "p", "v", "mu", "weight", "t", "dt", "count_flag", "nsteps_pushed",
         "tag_injected", "tag_splitted", "rng_ctr")


@pytest.mark.parametrize("dt_min", [0.9, 0.4, 0.15, 0.02])
@pytest.mark.parametrize("ndim,mover_kw", [(2, {}), (3, {}), (2, dict(focused_transport=True))])
def test_few_pushes(ndim, mover_kw, dt_min):
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() \
        else 152
    n, m = 128 * sms * 6 + 5, 16         # two warps a scheduler
    cfg = make_mhd_config(m, m, m if ndim == 3 else 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02, ndim=ndim)
    prm = make_params(ndim=ndim, p0=0.1, pmin=0.1, pmax=1.0, kpara0=1e-3, kret=0.1, dt_min_rel=dt_min,
                      dt_max_rel=0.95, pbcx=1, pbcy=0, pbcz=0, momentum_dependency=0, duu0=0.0,
                      nptl_max=n, seed=17)
    eng = Engine(prm, cfg, 0)
    eng.set_tstamps(np.arange(3) * 0.02)
    if ndim == 3:
        frame = fields.turbulence_3d(m, seed=3)
    else:
        db = fields.kolmogorov_az_2d(m, m, 1.0, 1.0, 0.5, 2 * np.pi, np.pi * m / 2, 3)
        frame = fields.planar_shock_2d(m, m, 0.0, 1.0, 0.0, 1.0, r=3.0, w=0.1, x0=0.5, db=db)
    eng.set_fields(frame, 0)
    eng.calc_fields_gradients(0)
    eng.inject_particles_spatial_uniform(n, 1e-6, 1, 2.0, 1, (0.1, 0.1, 0.1, 0.9, 0.9, 0.9), 1.0)
    parts = oracle.Particles(n, eng.get_particles().arrays)
    cnt = oracle.OrcCounters()
    eng.particle_mover(mhd_tframe=1, **mover_kw)
    oracle.mover(oracle.params_from(prm), oracle.config_from(cfg), oracle.full_fields(frame, ndim, cfg),
                 parts, 0.0, 0.02, counters=cnt, **mover_kw)
    got, ref = eng.get_particles().order_by_tags(), ParticleSet(parts.view()).order_by_tags()
    assert len(got) == len(ref) and eng.counters().steps == cnt.steps
    assert cnt.steps < 200 * n
    for k in STATE:
        if k in ("v", "mu") and not mover_kw:
            continue
        assert np.array_equal(got[k], ref[k]), k
    eng.close()
