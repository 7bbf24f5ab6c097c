"""What an engine takes on the device: per field slot and cell the 32 variables
(128 bytes) and a packed record of 64 (2D) or 96 (3D) bytes, so that the largest
frames the card holds stay what they are."""
import numpy as np
import pytest

from gpat import fields
from gpat.engine import Engine, make_mhd_config, make_params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _taken(ndim, n, slots):
    cfg = make_mhd_config(n, n, n if ndim == 3 else 1, 0.0, 1.0, 0.0, 1.0, ndim=ndim)
    prm = make_params(ndim=ndim, nptl_max=16, time_interp=slots - 1)
    free = torch.cuda.mem_get_info(0)[0]
    eng = Engine(prm, cfg, 0)
    taken = free - torch.cuda.mem_get_info(0)[0]
    eng.close()
    return taken


@pytest.mark.parametrize("slots", [1, 2])
@pytest.mark.parametrize("ndim,n,record", [(2, 1500, 64), (3, 128, 96)])
def test_bytes_per_cell_and_slot(ndim, n, record, slots):
    _taken(ndim, 16, slots)                   # the context and the modules
    cells = (n + 4) ** ndim
    taken = _taken(ndim, n, slots)
    # allocations are rounded up to 2 MiB each
    assert taken <= slots * cells * (128 + record) + (16 << 20), taken / (slots * cells)


def test_bytes_per_particle_of_the_split_precision_mover():
    """Two sets of 98 bytes, a key of 4 and a pause flag of 1, through a call that
    bins more particles than are moved in one pass."""
    cap, n = 20_000_000, 700_000
    _taken(2, 16, 1)
    cfg = make_mhd_config(32, 32, 1, 0.0, 1.0, 0.0, 1.0, dt_out=1e-3)
    prm = make_params(ndim=2, p0=0.1, pmin=0.1, pmax=1.0, kpara0=1e-9, dt_min_rel=0.4, dt_max_rel=0.5,
                      nptl_max=cap, seed=3, precision=1)
    free = torch.cuda.mem_get_info(0)[0]
    eng = Engine(prm, cfg, 0)
    eng.set_tstamps(np.arange(3) * 1e-3)
    eng.set_fields(fields.planar_shock_2d(32, 32, 0.0, 1.0, 0.0, 1.0, r=3.0, w=0.05, x0=0.5), 0)
    eng.calc_fields_gradients(0)
    eng.inject_particles_spatial_uniform(n, 1e-6, 2, 1.0, 1, (0.0, 0.0, 0.0, 1.0, 1.0, 1.0), 1.0)
    eng.particle_mover(mhd_tframe=1)
    taken = free - torch.cuda.mem_get_info(0)[0]
    eng.close()
    assert taken <= cap * (2 * 98 + 4 + 1) + (24 << 20), taken / cap


def test_bytes_per_particle_of_the_fp64_mover():
    """Two sets of 98 bytes, through a call that orders its particles."""
    cap, n = 30_000_000, 100_000
    _taken(2, 16, 1)
    cfg = make_mhd_config(32, 32, 1, 0.0, 1.0, 0.0, 1.0, dt_out=1e-3)
    prm = make_params(ndim=2, p0=0.1, pmin=0.1, pmax=1.0, kpara0=1e-3, dt_min_rel=0.1, dt_max_rel=0.5,
                      nptl_max=cap, seed=3, precision=0)
    free = torch.cuda.mem_get_info(0)[0]
    eng = Engine(prm, cfg, 0)
    eng.set_tstamps(np.arange(3) * 1e-3)
    eng.set_fields(fields.planar_shock_2d(32, 32, 0.0, 1.0, 0.0, 1.0, r=3.0, w=0.05, x0=0.5), 0)
    eng.calc_fields_gradients(0)
    eng.inject_particles_spatial_uniform(n, 1e-6, 2, 1.0, 1, (0.0, 0.0, 0.0, 1.0, 1.0, 1.0), 1.0)
    eng.particle_mover(mhd_tframe=1)
    taken = free - torch.cuda.mem_get_info(0)[0]
    eng.close()
    assert taken <= cap * 2 * 98 + (24 << 20), taken / cap
