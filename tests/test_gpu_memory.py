"""What an engine takes on the device: per field slot and cell the 32 variables
(128 bytes) and a packed record of 64 (2D) or 96 (3D) bytes, so that the largest
frames the card holds stay what they are."""
import pytest

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
