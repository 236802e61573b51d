"""The dust photon loop by whole paths (k_dust_path) against the oracle at the edges of
its range; every count exact, the image within the order of its sums (up to 2e4 terms
per pixel: 2e4 x 2^-53 ~ 2e-12, tested at 1e-11)."""
import numpy as np
import pytest

import oracle as O
from parallelcmacionize_b200 import GridSpec, TransportEngine

pytestmark = pytest.mark.gpu

# cells, subgrids, source, packets, albedo, pixels, mean density
CASES = {
    "one packet": ((8, 8, 8), (1, 1, 1), (0.0, 0.0, 0.0), 1, 0.9, (3, 5), 1.0),
    "one-cell subgrids": ((6, 4, 4), (6, 4, 4), (0.1, 0.2, -0.3), 500, 0.5, (7, 7), 1.0),
    "padded subgrids": ((33, 18, 14), (3, 2, 2), (0.3, 0.5, -0.7), 5001, 0.8, (16, 9), 1.0),
    "source at a subgrid corner": ((16, 16, 16), (2, 2, 2), (0.0, 0.0, 0.0), 20_000, 0.5,
                                   (11, 11), 1.0),
    "source at the upper corner": ((16, 16, 16), (2, 2, 2), (1.0, 1.0, 1.0), 777, 0.5, (4, 4),
                                   1.0),
    "thick": ((12, 12, 12), (2, 2, 2), (0.0, 0.1, 0.2), 300, 0.98, (8, 8), 30.0),
    "empty": ((16, 16, 16), (2, 2, 2), (0.0, 0.1, 0.2), 300, 0.5, (8, 8), 0.0),
    "no scattering": ((16, 16, 16), (4, 4, 4), (0.0, 0.0, 0.0), 2000, 0.0, (8, 8), 1.0),
    "subgrid too long for the table": ((900, 2, 2), (1, 1, 1), (0.2, 0.1, 0.3), 400, 0.5, (5, 5),
                                       1.0),
}


def _run(name):
    ncell, nsub, src, n, albedo, npix, density = CASES[name]
    grid = GridSpec(box=(-1.0, -1.0, -1.0, 2.0, 2.0, 2.0), ncell=ncell, num_subgrid=nsub)
    rng = np.random.default_rng(8)
    nH = density * np.exp(rng.normal(0.0, 0.8, grid.num_cells))
    xH = rng.uniform(0.2, 1.0, grid.num_cells)
    lat = O.LatticeGrid(grid.box, ncell, nsub)
    si = [min(int((src[a] + 1.0) / 2.0 * nsub[a]), nsub[a] - 1) for a in range(3)]
    want = lat.dust_run(nH, xH, n, 31, albedo, src, (si[0] * nsub[1] + si[1]) * nsub[2] + si[2],
                        npix)
    return grid, nH, xH, (n, albedo, src, npix), want


@pytest.mark.parametrize("precision", ["mixed", "fp32", "fp64"])
@pytest.mark.parametrize("name", list(CASES))
def test_counts_and_image(name, precision):
    grid, nH, xH, (n, albedo, src, npix), (image, stats) = _run(name)
    with TransportEngine(grid, precision=precision,
                         rng="ranlux" if precision == "fp64" else "philox") as eng:
        eng.set_fields(0, nH, xH)
        for _ in range(2):  # the second call starts from the first one's buffers
            img, st = eng.dust_image(0, n, albedo, source=src, npix=npix, seed=31)
            assert st == stats
            np.testing.assert_allclose(img, image, rtol=1e-11, atol=1e-300)
