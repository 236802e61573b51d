"""Whole-path transport (k_path) against the wavefront on the same packets.

``shoot_packets`` emits and walks its packets in one kernel; ``transport_packets``
takes the photons that ``emit_photons`` gives for the same seed and iteration
through the wavefront.  Both walk with the same operations, so every count is equal,
and J is the same sum in another order: the fixed-point tallies are exact in the path
kernel and merged in FP64 up to ~1e3 times in the wavefront (1e3 x 2^-53 ~ 1e-13,
tested at 1e-12); the FP64 walk adds up to 2e4 terms per cell on either side (2 x 2e4
x 2^-53 ~ 4.4e-12, tested at 5e-12).
"""
import numpy as np
import pytest

from parallelcmacionize_b200 import GridSpec, TransportEngine
from parallelcmacionize_b200.engine import PARSEC

pytestmark = pytest.mark.gpu

BOX = (-5 * PARSEC,) * 3 + (10 * PARSEC,) * 3
Q = 4.26e49
COUNTS = ("packets_absorbed", "packets_escaped", "cell_crossings", "subgrid_transits",
          "packets_reemitted")

# cells, subgrids, sources (in box sides from the lower corner), packets, reemission
CASES = {
    "one packet": ((16, 16, 16), (1, 1, 1), [(0.4, 0.5, 0.6)], 1, 0.0),
    "one-cell subgrids": ((8, 4, 4), (8, 4, 4), [(0.5, 0.5, 0.5)], 33, 0.0),
    "padded subgrids": ((33, 18, 14), (3, 2, 2), [(0.3, 0.7, 0.2), (0.9, 0.1, 0.5)], 4001, 0.0),
    "subgrid corner": ((32, 32, 32), (4, 4, 4), [(0.5, 0.5, 0.5)], 20_000, 0.0),
    "upper box corner": ((24, 24, 24), (3, 3, 3), [(1.0, 1.0, 1.0)], 500, 0.0),
    "faces of the box": ((24, 24, 24), (3, 3, 3), [(0.0, 0.5, 1.0), (1.0, 0.2, 0.3)], 999, 0.0),
    "long subgrids": ((300, 2, 2), (1, 1, 1), [(0.1, 0.6, 0.4)], 700, 0.0),
    "largest subgrid": ((16, 16, 16), (1, 1, 1), [(0.51, 0.49, 0.5)], 3000, 0.0),
    "fewer packets than shares": ((20, 20, 20), (2, 2, 2), [(0.2, 0.3, 0.4)] * 7, 13, 0.0),
    "many sources": ((40, 30, 20), (4, 3, 2), [((7 * k % 17 + 0.5) / 17, (5 * k % 13) / 13,
                                              (3 * k % 11 + 0.2) / 11) for k in range(17)],
                     10_000, 0.0),
    "reemission": ((32, 32, 32), (4, 4, 4), [(0.5, 0.5, 0.5), (0.25, 0.6, 0.8)], 5000, 0.45),
}


def _grid(ncell, nsub, sources, packets, p):
    src = [tuple(BOX[a] + s[a] * BOX[3 + a] for a in range(3)) + (Q * (1 + 0.3 * k),)
           for k, s in enumerate(sources)]
    return GridSpec(box=BOX, ncell=ncell, num_subgrid=nsub, sources=src, num_photon=packets,
                    reemission_probability=p)


def _fields(grid, seed):
    rng = np.random.default_rng(seed)
    return (np.exp(rng.normal(np.log(1e8), 0.7, grid.num_cells)),
            10.0 ** rng.uniform(-6, -1, grid.num_cells))


def _first_subgrids(grid, photons):
    """Subgrid of each photon's source (clamped to the box, as the engine places it)."""
    s = [np.clip((photons["position"][:, a] - grid.box[a]) / grid.box[3 + a]
                 * grid.num_subgrid[a], 0, grid.num_subgrid[a] - 1).astype(np.uint32)
         for a in range(3)]
    return (s[0] * grid.num_subgrid[1] + s[1]) * grid.num_subgrid[2] + s[2]


@pytest.mark.parametrize("precision", ["mixed", "fp32", "fp64"])
@pytest.mark.parametrize("name", list(CASES))
def test_path_equals_wavefront(name, precision):
    g = _grid(*CASES[name])
    nH, xH = _fields(g, 5)
    with TransportEngine(g, precision=precision) as eng:
        eng.set_fields(0, nH, xH)
        for it in (0, 3):
            ph = eng.emit_photons(seed=91, iteration=it)
            assert ph.size == g.num_photon
            eng.set_intensity(0, np.zeros(g.num_cells))
            want = eng.transport_packets(0, ph, _first_subgrids(g, ph))
            _, jw = eng.get_fields(0, neutral_fraction=False)
            eng.set_intensity(0, np.zeros(g.num_cells))
            got = eng.shoot_packets(seed=91, iteration=it)[0]
            _, jg = eng.get_fields(0, neutral_fraction=False)
            assert {k: got[k] for k in COUNTS} == {k: want[k] for k in COUNTS}
            assert got["rounds"] == want["rounds"] and got["error_flags"] == 0
            np.testing.assert_allclose(jg, jw, rtol=5e-12 if precision == "fp64" else 1e-12,
                                       atol=0)


@pytest.mark.parametrize("precision", ["mixed", "fp32", "fp64"])
def test_batch_equals_single_instances(precision):
    """Warps change the instance on the way: each instance's counts are those of the
    wavefront on its own photons, and J adds to what is there."""
    grids = [_grid(*CASES[n]) for n in ("padded subgrids", "subgrid corner", "one packet",
                                        "many sources", "reemission")]
    with TransportEngine(grids, precision=precision) as eng:
        fields = [_fields(g, 20 + i) for i, g in enumerate(grids)]
        for i, (n, x) in enumerate(fields):
            eng.set_fields(i, n, x)
        ph = eng.emit_photons(seed=12, iteration=1)
        first = np.cumsum([0] + [g.num_photon for g in grids])
        want = []
        for i, g in enumerate(grids):
            mine = ph[first[i]: first[i + 1]]
            want.append(eng.transport_packets(i, mine, _first_subgrids(g, mine)))
        jw = [eng.get_fields(i, neutral_fraction=False)[1] for i in range(len(grids))]
        got = eng.shoot_packets(seed=12, iteration=1)
        for i, g in enumerate(grids):
            assert {k: got[i][k] for k in COUNTS} == {k: want[i][k] for k in COUNTS}
            _, j = eng.get_fields(i, neutral_fraction=False)
            np.testing.assert_allclose(j, 2.0 * jw[i],
                                       rtol=5e-12 if precision == "fp64" else 1e-12, atol=0)


@pytest.mark.parametrize("precision", ["mixed", "fp32", "fp64"])
def test_many_packets_of_one_source(precision):
    """Above 1.5e6 packets of a source its cells have more tally copies.  Up to 1.6e6
    packets cross a cell: 2 x 1.6e6 x 2^-53 ~ 3.6e-10 for the FP64 sums; the fixed-point
    ones merge at most 1.6e4 times (1.8e-12, tested at 1e-11)."""
    for packets in (1_499_999, 1_600_000):
        g = _grid((16, 16, 16), (2, 2, 2), [(0.4, 0.5, 0.6)], packets, 0.0)
        nH, xH = _fields(g, 5)
        with TransportEngine(g, precision=precision) as eng:
            eng.set_fields(0, nH, xH)
            ph = eng.emit_photons(seed=91, iteration=2)
            want = eng.transport_packets(0, ph, _first_subgrids(g, ph))
            _, jw = eng.get_fields(0, neutral_fraction=False)
            eng.set_intensity(0, np.zeros(g.num_cells))
            got = eng.shoot_packets(seed=91, iteration=2)[0]
            _, jg = eng.get_fields(0, neutral_fraction=False)
            assert {k: got[k] for k in COUNTS} == {k: want[k] for k in COUNTS}
            np.testing.assert_allclose(jg, jw, rtol=4e-10 if precision == "fp64" else 1e-11,
                                       atol=0)
