"""FP32 transport on either side of the line between whole paths and the wavefront (4
packets per cell of more than 1.4e7 cells in large subgrids).  Packet k is the same on both
sides, so one packet more adds that packet's crossings and its path lengths and nothing
else: J of the other cells is the same sum in another order (merged in FP64 up to ~1e4
times, 1e4 x 2^-53 ~ 1e-12, tested at 1e-11)."""
import numpy as np
import pytest

from parallelcmacionize_b200 import GridSpec, TransportEngine
from parallelcmacionize_b200.engine import PARSEC

pytestmark = pytest.mark.gpu

BOX = (-5 * PARSEC,) * 3 + (10 * PARSEC,) * 3


def test_one_packet_more_across_the_line():
    ncell = (256, 256, 224)
    cells = int(np.prod(ncell))
    grid = GridSpec(box=BOX, ncell=ncell, num_subgrid=(16, 16, 14),
                    sources=[(0.3 * PARSEC, -0.2 * PARSEC, 0.1 * PARSEC, 4.26e49)],
                    num_photon=4 * cells - 1)
    with TransportEngine(grid, precision="fp32") as eng:
        eng.set_fields(0, np.full(cells, 1e8), np.full(cells, 1e-4))
        few = eng.shoot_packets(seed=3, iteration=1)[0]
        _, j_few = eng.get_fields(0, neutral_fraction=False)
        eng.set_packet_budget(0, 4 * cells)
        eng.set_intensity(0, np.zeros(cells))
        more = eng.shoot_packets(seed=3, iteration=1)[0]
        _, j_more = eng.get_fields(0, neutral_fraction=False)
    for st, n in ((few, 4 * cells - 1), (more, 4 * cells)):
        assert st["packets_absorbed"] + st["packets_escaped"] == n and st["error_flags"] == 0
    extra = more["cell_crossings"] - few["cell_crossings"]
    assert 0 < extra <= sum(ncell)
    assert 0 < more["subgrid_transits"] - few["subgrid_transits"] <= 16 + 16 + 14
    off = np.abs(j_more - j_few) > 1e-11 * j_few
    assert np.count_nonzero(off) <= extra
