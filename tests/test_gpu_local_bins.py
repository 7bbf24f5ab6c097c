"""Local distributions where their sums can go wrong: all, most or none of a warp's
particles in one bin, with weights that carry through every limb, and tables on
either side of the sizes at which the bins change their form (2^23), the results
come back in parts (2^22) and the buffer is not kept (64 MiB).  Counts and weights
are exact."""
import numpy as np
import pytest

from gpat.engine import Engine, ParticleSet, make_mhd_config, make_params

pytestmark = pytest.mark.gpu

PMIN, PMAX = 0.1, 100.0


def _engine(n, nx, ny=None):
    cfg = make_mhd_config(nx, ny or nx, 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02)
    return Engine(make_params(ndim=2, p0=0.1, pmin=PMIN, pmax=PMAX, npp_global=16, nptl_max=n,
                              seed=1), cfg, 0)


def _set(n, seed):
    rng = np.random.default_rng(seed)
    ps = ParticleSet.empty(n)
    # multiples of 2^-64: exact in the engine's fixed point
    raw = rng.integers(1, 1 << 53, n).astype(np.uint64)
    exp = rng.integers(-64, -20, n)
    w = np.ldexp(raw.astype(np.float64), exp)
    w[::3] = np.ldexp(float((1 << 53) - 1), -40)     # limbs of ones
    w[::5] = 2.0 ** -64
    for k, v in dict(p=PMIN * 10.0 ** rng.uniform(0.01, 2.99, n), mu=rng.uniform(-0.99, 0.99, n),
                     weight=w, x=rng.random(n), y=rng.random(n), v=np.ones(n), dt=np.full(n, 1e-3),
                     count_flag=np.ones(n)).items():
        ps[k][:] = v
    ps["tag_injected"][:] = np.arange(n) + 1
    ps["tag_splitted"][:] = 1
    return ps


def _check(eng, ps, npb, nx, ny, rx, ry):
    f, c = eng.local_distribution(PMIN, PMAX, npb, 1, rx, ry, 1)
    nrx, nry = -(-nx // rx), -(-ny // ry)
    lo, hi = np.log10(PMIN), np.log10(PMAX)
    ip = np.floor((np.log10(ps["p"]) - lo) / ((hi - lo) / npb)).astype(int) + 1
    ix = np.floor(ps["x"] / (1.0 / nrx)).astype(int)
    iy = np.floor(ps["y"] / (1.0 / nry)).astype(int)
    ok = (ip > 0) & (ip < npb)
    index = ((iy * nrx + ix) * npb + ip - 1)[ok]
    sums = {}
    for i, w in zip(index.tolist(), ps["weight"][ok].tolist()):
        num, den = w.as_integer_ratio()
        s = sums.get(i, (0, 0))
        sums[i] = (s[0] + 1, s[1] + (num << 64) // den)
    f, c = f.ravel(), c.ravel()
    assert f.size == npb * nrx * nry
    at = np.fromiter(sums, np.int64)
    assert np.array_equal(c[at], np.array([v[0] for v in sums.values()], np.uint64))
    mask = (1 << 64) - 1
    want = np.array([float(v[1] >> 64) + float(v[1] & mask) / 2.0 ** 64 for v in sums.values()])
    assert np.array_equal(f[at], want)
    assert int(c.sum()) == len(index) and np.count_nonzero(f) == len(at)


@pytest.mark.parametrize("share", [0.0, 0.05, 0.5, 0.9, 1.0])
@pytest.mark.parametrize("n", [1, 31, 33, 1000, 100_003])
def test_particles_that_share_a_bin(n, share):
    ps = _set(n, n)
    hot = np.random.default_rng(7).random(n) < share
    ps["p"][hot], ps["x"][hot], ps["y"][hot] = 0.3, 0.4, 0.6
    eng = _engine(n, 16)
    eng.put_particles(ps)
    _check(eng, ps, 12, 16, 16, 4, 4)
    _check(eng, ps, 12, 16, 16, 16, 16)
    eng.close()


# 2^21 words of 40 bytes pass 64 MiB; 2^22 and 2^23 bins exactly, one row more
@pytest.mark.parametrize("npb,nx,ny", [(16, 256, 300), (16, 512, 512), (16, 512, 513), (16, 1024, 512),
                                       (16, 1024, 513), (31, 640, 640)])
def test_large_tables(npb, nx, ny):
    n = 40_000
    ps = _set(n, nx + ny)
    ps["x"][:5000], ps["y"][:5000], ps["p"][:5000] = 0.9999, 0.9999, 99.0   # the last bins
    eng = _engine(n, nx, ny)
    eng.put_particles(ps)
    _check(eng, ps, npb, nx, ny, 1, 1)
    eng.close()
