"""The distributions' bins and exact weights against numpy with the plain
expressions: momenta in, at and around the range and either side of the bin
edges, pitch angles at +-1, weights from 2^-70 to 2^20 that are no powers of
two, more particles than one table word holds between flushes, and tables in
shared memory, past it, and of one bin."""
from fractions import Fraction

import numpy as np
import pytest

from gpat.engine import Engine, ParticleSet, make_mhd_config, make_params

pytestmark = pytest.mark.gpu

PMIN, PMAX = 0.1, 100.0


def _set(n, npp, seed):
    rng = np.random.default_rng(seed)
    ps = ParticleSet.empty(n)
    p = PMIN * 10.0 ** rng.uniform(-0.1, 3.1, n)
    edges = 10.0 ** (np.log10(PMIN) + np.arange(npp + 1) * (np.log10(PMAX) - np.log10(PMIN)) / npp)
    special = np.concatenate([edges * (1 - 1e-9), edges * (1 + 1e-9), [0.0, 1e-310, 1e300]])[:n]
    p[:len(special)] = special
    mu = rng.uniform(-1.05, 1.05, n)
    mu[:4] = [1.0, -1.0, np.nextafter(1.0, 2), np.nextafter(-1.0, -2)][:min(4, n)]
    w = rng.random(n) * 2.0 ** rng.integers(-20, 3, n)
    w[::7] = 0.5 ** rng.integers(0, 30, len(w[::7]))
    w[::1001] = 2.0 ** rng.integers(-70, 21, len(w[::1001])) * 1.2345
    for k, v in dict(p=p, mu=mu, weight=w, x=rng.random(n), y=rng.random(n), v=np.ones(n),
                     dt=rng.random(n) * 1e-3 + 1e-9, count_flag=np.ones(n)).items():
        ps[k][:] = v
    ps["tag_injected"][:] = np.arange(n) + 1
    ps["tag_splitted"][:] = 1
    return ps


def _engine(n, npp):
    cfg = make_mhd_config(32, 32, 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02)
    return Engine(make_params(ndim=2, p0=0.1, pmin=PMIN, pmax=PMAX, npp_global=npp, nptl_max=n,
                              seed=1), cfg, 0)


def _weights(index, w, nbins):
    """Exact sums of weights cut below 2^-64, rounded as high and low words."""
    out = [0] * nbins
    for i, x in zip(index.tolist(), w.tolist()):
        out[i] += int(Fraction(x) * 2 ** 64)
    hi, lo = [v >> 64 for v in out], [v & (2 ** 64 - 1) for v in out]
    return np.array(hi, np.float64) + np.array(lo, np.uint64).astype(np.float64) / 2.0 ** 64


def _log_bins(p, lo, hi, n):
    with np.errstate(divide="ignore"):
        q = (np.log10(p) - np.log10(lo)) / ((np.log10(hi) - np.log10(lo)) / n)
    return np.floor(np.clip(q, -1e6, 1e6)).astype(int)


@pytest.mark.parametrize("n,npp,nmu", [(1, 128, 0), (257, 1, 0), (20000, 128, 0), (20000, 2048, 0),
                                       (300000, 7, 0), (20000, 128, 3), (20000, 128, 32),
                                       (20000, 2048, 3), (20000, 2048, 32), (300000, 1, 1)])
def test_global_bins(n, npp, nmu):
    ps = _set(n, npp, n + npp)
    eng = _engine(n, npp)
    eng.put_particles(ps)
    p, mu, w = ps["p"], ps["mu"], ps["weight"]
    ip = _log_bins(p, PMIN, PMAX, npp)
    ok = (p > PMIN) & (p <= PMAX) & (mu >= -1.0) & (mu <= 1.0) & (ip >= 0) & (ip < npp)
    if nmu == 0:
        f, c = eng.calc_particle_distributions()
        index, nb = ip, npp
    else:
        f, c = eng.particle_distributions_mu(nmu)
        im = np.floor((mu + 1.0) / float(np.float32(2.0) / np.float32(nmu))).astype(int)
        ok &= (im >= 0) & (im < nmu)
        index, nb = ip * nmu + im, npp * nmu
    assert np.array_equal(c.ravel(), np.bincount(index[ok], minlength=nb).astype(np.uint64))
    assert np.array_equal(f.ravel(), _weights(index[ok], w[ok], nb))
    eng.close()


@pytest.mark.parametrize("n,rx,npb", [(1, 1, 4), (50000, 4, 16), (50000, 32, 2)])
def test_local_bins_and_quick_check(n, rx, npb):
    ps = _set(n, 64, 11)
    eng = _engine(n, 64)
    eng.put_particles(ps)
    w = ps["weight"]
    ip = _log_bins(ps["p"], 0.2, 50.0, npb) + 1
    nr = -(-32 // rx)
    ix = np.floor(ps["x"] / (1.0 / nr)).astype(int)
    iy = np.floor(ps["y"] / (1.0 / nr)).astype(int)
    im = np.floor((ps["mu"] + 1.0) / 2.0).astype(int)
    ok = (ip > 0) & (ip < npb) & (im == 0)
    f, c = eng.local_distribution(0.2, 50.0, npb, 1, rx, rx, 1)
    index, nb = (iy * nr + ix) * npb + ip - 1, nr * nr * npb
    assert np.array_equal(c.ravel(), np.bincount(index[ok], minlength=nb).astype(np.uint64))
    assert np.array_equal(f.ravel(), _weights(index[ok], w[ok], nb))
    got = eng.quick_check()
    zero = np.zeros(n, int)
    assert got["ntot"] == _weights(zero, w, 1)[0]
    assert got["pdt_min"] == ps["dt"].min() and got["pdt_max"] == ps["dt"].max()
    assert got["pdt_avg"] == _weights(zero, ps["dt"], 1)[0] / n
    eng.close()
