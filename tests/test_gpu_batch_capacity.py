"""Batched runs with room for many more particles than they have, or with enough
of them for the binning's second pass: each gives what it gives alone."""
import numpy as np
import pytest

from gpat import fields
from gpat.engine import Batch, Engine, make_mhd_config, make_params

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "p", "v", "mu", "weight", "t", "dt", "split_times", "count_flag", "origin",
        "nsteps_pushed", "tag_injected", "tag_splitted", "rng_ctr")


@pytest.mark.parametrize("nptl,cap", [(500, 600_000), (500, 599_999), (599_999, 700_000),
                                      (600_000, 700_000), (650_000, 650_000)])
def test_capacity_and_count_around_the_second_pass(nptl, cap):
    engs, alone = [], []
    for k in range(2):
        cfg = make_mhd_config(24, 24, 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02)
        prm = make_params(ndim=2, p0=0.1, pmin=0.1, pmax=1.0, kpara0=3e-3, kret=0.1,
                          dt_min_rel=5e-2, dt_max_rel=2e-1, pbcx=1, pbcy=0, nptl_max=cap,
                          seed=5 + k, precision=1, bin_interval=8)
        eng = Engine(prm, cfg, 0)
        eng.set_tstamps(np.arange(3) * 0.02)
        eng.set_fields(fields.planar_shock_2d(24, 24, 0.0, 1.0, 0.0, 1.0, r=3.0, w=0.05, x0=0.5), 0)
        eng.calc_fields_gradients(0)
        eng.inject_particles_spatial_uniform(nptl, 1e-6, 2, 1.0, 1, (0.0, 0.0, 0.0, 1.0, 1.0, 1.0),
                                             1.0)
        start, counters = eng.get_particles(), eng.counters()
        start["origin"][:] = np.arange(nptl)
        start["split_times"][:] = np.arange(nptl) % 7
        eng.put_particles(start)
        eng.particle_mover(mhd_tframe=1)
        alone.append(eng.get_particles().order_by_tags())
        eng.set_counters(counters)
        eng.put_particles(start)
        engs.append(eng)
    batch = Batch(engs)
    batch.particle_mover(mhd_tframe=1)
    for eng, ref in zip(engs, alone):
        got = eng.get_particles().order_by_tags()
        assert 0 < len(ref) < nptl          # some left through the open faces
        for k in KEYS:
            assert np.array_equal(got[k], ref[k]), k
    batch.close()
    for eng in engs:
        eng.close()
