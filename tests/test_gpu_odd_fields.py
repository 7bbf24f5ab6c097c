"""Field values that the FP64 mover's integer products do not take (subnormal,
infinite, NaN) and every way by which the mover learns of them, in both of its
builds (teams of eight lanes for up to 16 particles an SM, one lane above), bit
for bit against the oracle: frames with and without their gradients, the second
frame alone, a frame that takes the first one's place, counters put back in
between, fluctuation arrays, and ordinary frames after such ones."""
import numpy as np
import pytest

import oracle
from gpat import fields
from gpat.engine import Engine, GPATError, ParticleSet, make_mhd_config, make_params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N = 24
BOX = (0.0, 0.0, 0.0, 1.0, 1.0, 1.0)
STATE = ("x", "y", "z", "p", "v", "mu", "weight", "t", "dt", "count_flag", "nsteps_pushed",
         "tag_injected", "tag_splitted", "rng_ctr")


def _counts():
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() \
        else 152
    return [16 * sms, 16 * sms + 1]


def _frame(ndim, seed=3, odd=None):
    if ndim == 3:
        f = fields.turbulence_3d(N, seed=seed).copy()
    else:
        db = fields.kolmogorov_az_2d(N, N, 1.0, 1.0, 0.5, 2 * np.pi, np.pi * N / 2, seed)
        f = fields.planar_shock_2d(N, N, 0.0, 1.0, 0.0, 1.0, r=3.0, w=0.05, x0=0.5, db=db).copy()
    cells = f.reshape(-1, 8)
    if odd == "subnormal":
        cells[::5, 1] = 1e-41      # vy
        cells[::7, 6] = -3e-43     # Bz
    elif odd == "one":
        cells[len(cells) // 2, 0] = 2e-40
    return f


def _engine(ndim, nptl, two=False, **kw):
    cfg = make_mhd_config(N, N, N if ndim == 3 else 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02, ndim=ndim)
    base = dict(ndim=ndim, p0=0.1, pmin=0.1, pmax=1.0, kpara0=3e-3, kret=0.1, dt_min_rel=3e-2,
                dt_max_rel=2e-1, pbcx=1, pbcy=0, pbcz=0, momentum_dependency=0, nptl_max=nptl, seed=17,
                time_interp=int(two))
    base.update(kw)
    prm = make_params(**base)
    eng = Engine(prm, cfg, 0)
    eng.set_tstamps(np.arange(4) * 0.02)
    return eng, prm, cfg


def _compare(eng, prm, cfg, nptl, full1, full2=None, aux=None, aux2=None, inject=True):
    """One interval on both sides from the same particles."""
    if inject:
        eng.inject_particles_spatial_uniform(nptl, 1e-6, 2, 1.0, 1, BOX, 1.0)
    parts = oracle.Particles(nptl, eng.get_particles().arrays)
    eng.particle_mover(mhd_tframe=1)
    kw = {k: v for k, v in dict(f2=full2, aux1=aux, aux2=aux2).items() if v is not None}
    oracle.mover(oracle.params_from(prm), oracle.config_from(cfg), full1, parts, 0.0, 0.02, **kw)
    got, ref = eng.get_particles().order_by_tags(), ParticleSet(parts.view()).order_by_tags()
    assert len(got) == len(ref) > 0.5 * nptl
    for k in STATE:
        assert np.array_equal(got[k], ref[k]), k


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("odd", ["subnormal", "one"])
def test_both_builds(ndim, odd, which):
    n = _counts()[which]
    f = _frame(ndim, odd=odd)
    eng, prm, cfg = _engine(ndim, n)
    eng.set_fields(f, 0)
    eng.calc_fields_gradients(0)
    _compare(eng, prm, cfg, n, oracle.full_fields(f, ndim, cfg))
    eng.close()


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("odd", [(None, "one"), ("one", None), ("subnormal", "subnormal")])
def test_either_frame(odd, which):
    n = _counts()[which]
    fr = [_frame(2, 3 + k, odd[k]) for k in (0, 1)]
    eng, prm, cfg = _engine(2, n, two=True)
    for k in (0, 1):
        eng.set_fields(fr[k], k)
        eng.calc_fields_gradients(k)
    full = [oracle.full_fields(f, 2, cfg) for f in fr]
    _compare(eng, prm, cfg, n, full[0], full[1])
    eng.close()


@pytest.mark.parametrize("which", [0, 1])
def test_a_frame_that_takes_the_other_ones_place(which):
    """copy_fields with values of either kind on top of the other, and counters put
    back in between."""
    n = _counts()[which]
    plain, odd = _frame(2, 3), _frame(2, 4, "subnormal")
    for first, second in ((plain, odd), (odd, plain)):
        eng, prm, cfg = _engine(2, n, two=True)
        for k, f in enumerate((first, second)):
            eng.set_fields(f, k)
            eng.calc_fields_gradients(k)
        eng.copy_fields()
        eng.set_fields(first, 1)
        eng.calc_fields_gradients(1)
        eng.set_counters(eng.counters())
        full = [oracle.full_fields(f, 2, cfg) for f in (second, first)]
        _compare(eng, prm, cfg, n, full[0], full[1])
        eng.close()


@pytest.mark.parametrize("which", [0, 1])
def test_frames_with_their_gradients_and_plain_ones_after_them(which):
    n = _counts()[which]
    eng, prm, cfg = _engine(3, n)
    for odd in ("one", None, "subnormal"):
        full = oracle.full_fields(_frame(3, 5, odd), 3, cfg)
        eng.set_fields(full, 0)              # 32 variables
        eng.put_particles(ParticleSet.empty(0))
        _compare(eng, prm, cfg, n, full)
    eng.close()


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("value", [1e-40, None])
def test_fluctuation_arrays(value, which):
    """dB^2 with subnormal gradients (nearly constant) or ordinary ones, one array
    after the other in the same slot."""
    n = _counts()[which]
    eng, prm, cfg = _engine(2, n, deltab_flag=1)
    f = _frame(2)
    eng.set_fields(f, 0)
    eng.calc_fields_gradients(0)
    full = oracle.full_fields(f, 2, cfg)
    x = fields.node_coords(N, 0.0, 1.0 / N)
    smooth = (1.0 + 0.3 * np.sin(2 * np.pi * x)[None, None, :] + 0 * x[None, :, None]).astype(np.float32)
    for db2 in (smooth, smooth * 0 + 1):
        if value is not None:
            db2 = db2.copy()
            db2d = np.full_like(db2, 1.0)
            db2d[0, ::3, ::4] = value
        else:
            db2d = None
        eng.set_fluctuations(0, db2, db2d, None, None)
        aux = oracle.aux_fields(db2, db2d, None, None, 2, cfg)
        assert np.array_equal(eng.get_fluctuations(0), aux)
        eng.put_particles(ParticleSet.empty(0))
        _compare(eng, prm, cfg, n, full, aux=aux)
    eng.close()


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_infinities_and_nan(bad, which):
    """Far from every particle they change nothing; met by one they are reported,
    not turned into numbers."""
    n = _counts()[which]
    f = _frame(2)
    f[0, 2:6, 2:6, 4] = bad               # Bx in a corner of the box
    eng, prm, cfg = _engine(2, n, dt_min_rel=0.25, dt_max_rel=0.5, kpara0=1e-6)
    eng.set_fields(f, 0)
    eng.calc_fields_gradients(0)
    eng.inject_particles_spatial_uniform(n, 1e-6, 2, 1.0, 1, (0.5, 0.5, 0.0, 0.9, 0.9, 1.0), 1.0)
    _compare(eng, prm, cfg, n, oracle.full_fields(f, 2, cfg), inject=False)
    eng.put_particles(ParticleSet.empty(0))
    eng.inject_particles_spatial_uniform(n, 1e-6, 2, 1.0, 1, (0.05, 0.05, 0.0, 0.1, 0.1, 1.0), 1.0)
    with pytest.raises(GPATError):
        eng.particle_mover(mhd_tframe=1)
    eng.close()
