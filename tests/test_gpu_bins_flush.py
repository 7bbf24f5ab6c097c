"""f(p) of more particles than one word of a block's table takes: 65 536 weights with
a limb of 0xffff in the same bin fill 32 bits, so each block adds its table to the
global one every 256 turns.  More than that many turns of all blocks, every particle
in one or two bins, weights whose limbs are all ones: counts and weights exact."""
import numpy as np
import pytest

from gpat.engine import Engine, ParticleSet, make_mhd_config, make_params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ONES = float((1 << 53) - 1) * 2.0 ** -37     # 16 bits above the point and 37 below


@pytest.mark.parametrize("npp", [1, 2])
def test_tables_flushed_on_the_way(npp):
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() \
        else 152
    n = 4 * sms * 256 * 262 + 77             # 263 turns
    ps = ParticleSet.empty(n)
    weights = np.array([ONES, ONES * 2.0 ** -27, 1.0, ONES, ONES])
    momenta = np.array([0.5, 20.0])
    ps["p"][:] = np.resize(momenta, n)
    ps["weight"][:] = np.resize(weights, n)
    eng = Engine(make_params(ndim=2, p0=0.1, pmin=0.1, pmax=100.0, npp_global=npp, nptl_max=n, seed=1),
                 make_mhd_config(16, 16, 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02), 0)
    eng.put_particles(ps)
    per = np.bincount(np.arange(10 * (n // 10), n) % 10, minlength=10) + n // 10
    count, total = [0] * npp, [0] * npp
    for k in range(10):
        b = 0 if npp == 1 else k % 2         # 0.1 .. 3.16 .. 100
        num, den = float(weights[k % 5]).as_integer_ratio()
        count[b] += int(per[k])
        total[b] += int(per[k]) * ((num << 64) // den)
    mask = (1 << 64) - 1
    want = np.array([float(t >> 64) + float(t & mask) / 2.0 ** 64 for t in total])
    for f, c in (eng.calc_particle_distributions(), eng.particle_distributions_mu(1)):
        assert c.ravel().tolist() == count
        assert np.array_equal(f.ravel(), want)
    eng.close()
