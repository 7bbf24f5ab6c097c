"""The brick mover where most pushes end near a face of the box: steps of half a
cell on a small periodic grid, so that lanes go into the boundary test at
different times and meet again before the push.  Against the global-gather form,
with test_gpu_tile's tolerances (FP32 rounding carried over the interval where a
particle pauses)."""
import numpy as np
import pytest

from gpat import fields
from gpat.engine import Engine, make_mhd_config, make_params

pytestmark = pytest.mark.gpu


def _moved(ndim, n, nptl, bricks):
    cfg = make_mhd_config(n, n, n if ndim == 3 else 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02, ndim=ndim)
    frame = fields.turbulence_3d(n, seed=2) if ndim == 3 else fields.planar_shock_2d(
        n, n, 0.0, 1.0, 0.0, 1.0, r=3.0, w=0.05, x0=0.5,
        db=fields.kolmogorov_az_2d(n, n, 1.0, 1.0, 0.5, 2 * np.pi, np.pi * n / 2, 2))
    # (0.5 / n)^2 / (2 kappa) = dt_max: half a cell a push
    dt_max = 0.02 / 60
    prm = make_params(ndim=ndim, p0=0.1, pmin=0.01, pmax=100.0, kpara0=0.125 / n ** 2 / dt_max,
                      kret=0.2, dt_min_rel=1 / 240, dt_max_rel=1 / 60, pbcx=0, pbcy=0, pbcz=0,
                      momentum_dependency=0, precision=1, nptl_max=nptl, seed=9, bin_interval=32)
    eng = Engine(prm, cfg, 0)
    eng.set_tstamps(np.arange(3) * 0.02)
    eng.set_fields(frame, 0)
    eng.calc_fields_gradients(0)
    if bricks:
        eng.set_mover_tiles(*bricks)
    eng.inject_particles_spatial_uniform(nptl, 1e-6, 1, 1.0, 1, (0, 0, 0, 1, 1, 1))
    eng.particle_mover(mhd_tframe=1)
    out = eng.get_particles().order_by_tags(), eng.counters().steps
    eng.close()
    return out


@pytest.mark.parametrize("ndim,n,bricks", [(2, 16, (8, 8)), (3, 12, (6, 6, 6, 2, 2, 2))])
def test_pushes_across_the_faces(ndim, n, bricks):
    a, steps_a = _moved(ndim, n, 6000, None)
    b, steps_b = _moved(ndim, n, 6000, bricks)
    assert np.array_equal(a["tag_injected"], b["tag_injected"])
    assert abs(steps_a - steps_b) <= 0.005 * steps_a
    # the step is half a cell: a particle meets the other side of the box often
    assert steps_a > 20 * len(a)
    ok = np.isclose(a["p"], b["p"], rtol=1e-4)
    for k in ("x", "y", "z")[:ndim]:
        d = np.abs(a[k] - b[k])
        ok &= np.minimum(d, 1.0 + 1.0 / n - d) * n < 1e-3
    assert ok.mean() >= 0.99, ok.mean()
