"""Binning by cell at both sides of the size from which the particles are moved in
a second pass: every particle that stays is there once, with all its values, in
the order of the cells; particles that left the box are gone."""
import numpy as np
import pytest

from gpat import fields
from gpat.engine import Engine, make_mhd_config, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("n", [599999, 600000, 600257])
def test_binning_keeps_every_particle(n, ndim):
    m = 12
    cfg = make_mhd_config(m, m, m if ndim == 3 else 1, 0.0, 1.0, 0.0, 1.0, dt_out=1e-3, ndim=ndim)
    prm = make_params(ndim=ndim, p0=0.1, pmin=0.1, pmax=1.0, kpara0=1e-9, kret=0.1, dt_min_rel=0.4,
                      dt_max_rel=0.5, pbcx=1, pbcy=1, pbcz=1, nptl_max=600300, seed=3, precision=1)
    eng = Engine(prm, cfg, 0)
    eng.set_tstamps(np.arange(3) * 1e-3)
    frame = fields.turbulence_3d(m, seed=3) if ndim == 3 else \
        fields.planar_shock_2d(m, m, 0.0, 1.0, 0.0, 1.0, r=3.0, w=0.05, x0=0.5)
    eng.set_fields(frame, 0)
    eng.calc_fields_gradients(0)
    eng.inject_particles_spatial_uniform(n, 1e-6, 2, 1.0, 1, (0.0, 0.0, 0.0, 1.0, 1.0, 1.0), 1.0)
    ps = eng.get_particles()
    rng = np.random.default_rng(n)
    gone = rng.permutation(n)[:1000]
    ps["x"][gone] = 1.5                      # past the open face
    ps["t"][:] = 1e-3                        # nothing left to do: only binned
    ps["origin"][:] = rng.integers(0, 1 << 30, n)
    ps["split_times"][:] = rng.integers(0, 30, n)
    ps["rng_ctr"][:] = rng.integers(0, 1 << 30, n)
    ps["mu"][:] = rng.uniform(-1, 1, n)
    want = {int(t) for t in np.delete(ps["tag_injected"], gone)}
    eng.put_particles(ps)
    eng.particle_mover(mhd_tframe=1)
    got = eng.get_particles()
    assert len(got) == n - 1000 and set(got["tag_injected"].tolist()) == want
    first = np.argsort(ps["tag_injected"], kind="stable")
    at = first[np.searchsorted(ps["tag_injected"][first], got["tag_injected"])]
    for k in ("x", "y", "z", "p", "v", "mu", "weight", "t", "origin", "split_times", "rng_ctr",
              "tag_splitted"):
        assert np.array_equal(got[k], ps[k][at]), k
    cell = np.floor(got["x"] * m).astype(int) + 64 * np.floor(got["y"] * m).astype(int)
    if ndim == 3:
        cell += 4096 * np.floor(got["z"] * m).astype(int)
    assert (np.diff(cell) >= 0).mean() > 0.9999
    eng.close()
