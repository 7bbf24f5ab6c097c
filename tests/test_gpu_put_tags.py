"""The tag range of a received particle set, on both sides of the size from which
it is found on the GPU: the injection counter moves past every tag."""
import numpy as np
import pytest

from gpat.engine import Engine, ParticleSet, make_mhd_config, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 16384, 16385, 400001])
def test_tag_max_is_past_every_tag(n):
    cfg = make_mhd_config(8, 8, 1, 0.0, 1.0, 0.0, 1.0, dt_out=0.02, ndim=2)
    eng = Engine(make_params(ndim=2, nptl_max=n, seed=1), cfg, 0)
    ps = ParticleSet({k: np.zeros_like(v) for k, v in ParticleSet.empty(n).arrays.items()})
    seen = 0
    for at, tag in ((n - 1, -7), (0, 5), (n // 2, 3), (n - 1, 2**31 - 2), (0, 9), (0, 2**31 - 1)):
        ps["tag_injected"][:] = -1
        ps["tag_injected"][at] = tag
        ps["tag_splitted"][:] = -2**31
        eng.put_particles(ps)
        seen = max(seen, tag + 1)
        assert eng.counters().tag_max == seen
    eng.put_particles(ParticleSet.empty(0))
    assert eng.counters().tag_max == seen
    eng.close()
