"""The split-precision mover gathers records by groups of lanes: what a particle
computes must not depend on the particles beside it.  Sets of every size
around a warp and a block give each particle the bits it has when it is moved
alone, in 2D and 3D, with one and two frames, with chunks that end mid-way and
with particles that have left the box or start late beside it."""
import numpy as np
import pytest

from gpat import fields
from gpat.engine import Engine, make_mhd_config, make_params

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "p", "t", "dt", "count_flag", "nsteps_pushed", "rng_ctr")


def _engine(ndim, two, nmax=200):
    n = 20 if ndim == 3 else 36
    cfg = make_mhd_config(n, n, n if ndim == 3 else 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02, ndim=ndim)
    prm = make_params(ndim=ndim, p0=0.1, pmin=0.1, pmax=1.0, kpara0=3e-3, kret=0.1, dt_min_rel=1e-2,
                      dt_max_rel=1e-1, pbcx=1, pbcy=0, pbcz=0, nptl_max=nmax, seed=5, precision=1,
                      time_interp=int(two), bin_interval=16)
    eng = Engine(prm, cfg, 0)
    eng.set_tstamps(np.arange(3) * 0.02)
    for k in range(2 if two else 1):
        if ndim == 3:
            frame = fields.turbulence_3d(n, seed=3 + k)
        else:
            db = fields.kolmogorov_az_2d(n, n, 1.0, 1.0, 0.5, 2 * np.pi, np.pi * n / 2, 7 + k)
            frame = fields.planar_shock_2d(n, n, 0.0, 1.0, 0.0, 1.0, r=3.0, w=0.05, x0=0.5, db=db,
                                           b0=(1.0, 0.0, 0.2))
        eng.set_fields(frame, k)
        eng.calc_fields_gradients(k)
    return eng


@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("ndim", [2, 3])
def test_a_particle_does_not_depend_on_its_neighbours(ndim, two):
    eng = _engine(ndim, two)
    eng.inject_particles_spatial_uniform(131, 1e-6, 2, 1.0, 1, (0.0, 0.0, 0.0, 1.0, 1.0, 1.0), 1.0)
    start = eng.get_particles()
    start["x"][5] = -0.2            # leaves at once through the open face
    start["x"][6] = 1.0 - 1e-9      # at the edge of the box
    start["t"][7] = 0.02            # has nothing left to do

    def moved(idx):
        eng.put_particles(start.take(idx))
        eng.particle_mover(mhd_tframe=1)
        out = eng.get_particles()
        return {int(t): {k: out[k][j] for k in KEYS} for j, t in enumerate(out["tag_injected"])}

    alone = {}
    for j in range(131):
        alone.update(moved(np.array([j])))
    for size in (2, 3, 4, 31, 32, 33, 127, 128, 129, 131):
        got = moved(np.arange(131)[-size:])
        tags = {int(t) for t in start["tag_injected"][-size:]} & set(alone)
        assert set(got) == tags
        for t, p in got.items():
            for k in KEYS:
                assert p[k] == alone[t][k] or (p[k] != p[k] and alone[t][k] != alone[t][k]), (t, k)
    eng.close()


@pytest.mark.parametrize("ndim,two", [(2, False), (3, False), (3, True)])
def test_a_particle_does_not_depend_on_the_lanes_of_a_launch(ndim, two):
    """Launches that give a particle 1 to 32 lanes, at both sides of each line
    on 152 SMs: the bits are those of the particle in the whole set."""
    eng = _engine(ndim, two, 80000)
    eng.inject_particles_spatial_uniform(80000, 1e-6, 2, 1.0, 1, (0.0, 0.0, 0.0, 1.0, 1.0, 1.0), 1.0)
    start = eng.get_particles()

    def moved(idx):
        eng.put_particles(start.take(idx))
        eng.particle_mover(mhd_tframe=1)
        out = eng.get_particles()
        order = np.argsort(out["tag_injected"], kind="stable")
        return {k: out[k][order] for k in KEYS + ("tag_injected",)}

    whole = moved(np.arange(80000))
    for n in (38913, 38912, 19457, 19456, 9729, 9728, 4865, 2432, 1217, 1216, 608, 33, 1):
        idx = np.sort(np.random.default_rng(n).permutation(80000)[:n])
        got = moved(idx)
        at = np.isin(whole["tag_injected"], start["tag_injected"][idx])
        for k in KEYS + ("tag_injected",):
            assert np.array_equal(got[k], whole[k][at]), (n, k)
    eng.close()
