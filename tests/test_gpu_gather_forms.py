"""Both gathers of the split-precision mover give a particle the same bits: runs
whose longest step puts the launch on either side of the rule (gather_form.h),
moved whole, so that the launch has many particles a cell, and in parts small
enough for the other form or for several lanes a particle; 2D and 3D, one and two
frames, alone, in a batch and with the network."""
import numpy as np
import pytest

from gpat import fields
from gpat.engine import Batch, Engine, Mlp, make_mhd_config, make_params, set_mover_learned

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "p", "t", "dt", "count_flag", "nsteps_pushed", "rng_ctr", "tag_injected",
        "tag_splitted")
BOX = (0.0, 0.0, 0.0, 1.0, 1.0, 1.0)


def _engine(ndim, two, step, n, nmax, seed=5, pushes=64):
    cfg = make_mhd_config(n, n, n if ndim == 3 else 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02, ndim=ndim)
    dt_max = 0.02 / pushes
    prm = make_params(ndim=ndim, p0=0.1, pmin=0.1, pmax=1.0, kpara0=(step / n) ** 2 / (2 * dt_max),
                      kret=0.1, dt_min_rel=0.1 / pushes, dt_max_rel=1 / pushes, pbcx=1, pbcy=0, pbcz=0,
                      momentum_dependency=0, nptl_max=nmax, seed=seed, precision=1,
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


def _moved(eng, start, idx, **kw):
    eng.put_particles(start.take(idx))
    eng.particle_mover(mhd_tframe=1, **kw)
    out = eng.get_particles()
    order = np.argsort(out["tag_injected"], kind="stable")
    return {k: out[k][order] for k in KEYS}


# the whole set and its parts fall on different sides of the rule: 2D one frame by
# the number of particles, two frames below one particle a cell, 3D by the lanes a
# particle has
@pytest.mark.parametrize("nlgc", [False, True])
@pytest.mark.parametrize("ndim,two,step,n,total,parts", [
    (2, False, 0.5, 36, 40000, (9000, 3000, 300, 33, 1)),   # groups -> lanes
    (2, True, 0.1, 128, 40000, (12000, 3000, 1)),           # lanes -> groups -> lanes
    (2, True, 3.0, 100, 20000, (9000, 3000, 2000, 1)),      # groups -> lanes at 2000
    (3, False, 0.05, 20, 60000, (20000, 3000, 1)),          # lanes -> groups
    (3, True, 0.01, 20, 60000, (20000, 3000, 1)),
])
def test_the_same_bits_on_both_sides(ndim, two, step, n, total, parts, nlgc):
    eng = _engine(ndim, two, step, n, total)
    eng.inject_particles_spatial_uniform(total, 1e-6, 2, 1.0, 1, BOX, 1.0)
    start = eng.get_particles()
    start["x"][5] = -0.2            # leaves at once through the open face
    start["t"][7] = 0.02            # has nothing left to do
    kw = dict(nlgc=True, kperp_kpara=0.05) if nlgc else {}
    whole = _moved(eng, start, np.arange(total), **kw)
    assert len(whole["x"]) > 0.5 * total
    for m in parts:
        idx = np.sort(np.random.default_rng(m).permutation(total)[:m])
        got = _moved(eng, start, idx, **kw)
        at = np.isin(whole["tag_injected"], start["tag_injected"][idx])
        for k in KEYS:
            assert np.array_equal(got[k], whole[k][at]), (m, k)
    eng.close()


@pytest.mark.parametrize("ndim,two", [(2, False), (2, True), (3, True)])
def test_launches_of_few_pushes(ndim, two):
    """By single lanes as a whole, the last particles of a 3D set by groups."""
    eng = _engine(ndim, two, 0.5, 20 if ndim == 3 else 128, 60000, pushes=1.2)
    eng.inject_particles_spatial_uniform(60000, 1e-6, 2, 1.0, 1, BOX, 1.0)
    start = eng.get_particles()
    whole = _moved(eng, start, np.arange(60000))
    for m in (45000, 20000, 300):
        got = _moved(eng, start, np.arange(m))
        at = np.isin(whole["tag_injected"], start["tag_injected"][:m])
        for k in KEYS:
            assert np.array_equal(got[k], whole[k][at]), (m, k)
    eng.close()


def test_a_batch_and_its_runs_in_different_forms():
    """Two runs whose own launches gather in different forms, and the batch, which
    takes the form of most of its particles, both ways round."""
    for sizes in ((40000, 500), (500, 40000)):
        engs, alone = [], []
        for step, m in zip((0.5, 0.1), sizes):
            eng = _engine(2, False, step, 36, 40000, seed=11)
            eng.inject_particles_spatial_uniform(m, 1e-6, 2, 1.0, 1, BOX, 1.0)
            start = eng.get_particles()
            alone.append(_moved(eng, start, np.arange(m)))
            eng.put_particles(start)
            engs.append(eng)
        with_batch = Batch(engs)
        with_batch.particle_mover(mhd_tframe=1)
        for eng, ref in zip(engs, alone):
            out = eng.get_particles()
            order = np.argsort(out["tag_injected"], kind="stable")
            for k in KEYS:
                assert np.array_equal(out[k][order], ref[k]), k
        with_batch.close()
        for eng in engs:
            eng.close()


@pytest.mark.parametrize("ndim,step,n,total,part", [(2, 0.5, 36, 40000, 9000),
                                                    (3, 0.05, 20, 60000, 20000)])
def test_learned_launches_in_both_forms(ndim, step, n, total, part):
    """A window no particle leaves: the launch moves them as the plain one does."""
    eng = _engine(ndim, False, step, n, total)
    eng.inject_particles_spatial_uniform(total, 1e-6, 2, 1.0, 1, BOX, 1.0)
    start = eng.get_particles()
    idx = np.arange(part)
    plain = [_moved(eng, start, i) for i in (np.arange(total), idx)]
    mlp = Mlp(seed=1)
    set_mover_learned(eng, mlp, 0.2, 1.0, 0.0, 1e12, 1, -50.0)
    learned = [_moved(eng, start, i) for i in (np.arange(total), idx)]
    for a, b in zip(plain, learned):
        for k in KEYS:
            assert np.array_equal(a[k], b[k]), k
    eng.close()
