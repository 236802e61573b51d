"""cmi_traverse_buffer at the sizes where its launches change: one block that also groups
(up to 256 photons), blocks and a grouping launch, copies through pinned memory (up to 1
MiB) and past it.  A buffer of any size gives, group by group, the photons of its parts
in order; J is the same sum in another order (up to 2e4 terms: 2e4 x 2^-53 x 2 < 5e-12;
FP32: compensated sums of FP32 lengths, 1e-7)."""
import numpy as np
import pytest

from parallelcmacionize_b200 import PHOTON_DTYPE, GridSpec, TransportEngine
from parallelcmacionize_b200.engine import PARSEC, TravelDirection

pytestmark = pytest.mark.gpu


def _photons(n, side, seed=3):
    rng = np.random.default_rng(seed)
    ph = np.zeros(n, PHOTON_DTYPE)
    d = rng.normal(size=(n, 3))
    ph["position"] = rng.uniform(size=(n, 3)) * side
    ph["direction"] = d / np.linalg.norm(d, axis=1)[:, None]
    ph["tau"], ph["sigma"], ph["weight"] = rng.exponential(size=n), 6.3e-22, 1.0
    return ph


@pytest.mark.parametrize("precision", ["mixed", "fp32", "fp64"])
@pytest.mark.parametrize("n", [0, 1, 31, 33, 255, 256, 257, 4097, 20_000])
def test_buffer_equals_its_parts(n, precision):
    side = np.array([10.0, 7.0, 5.0]) * PARSEC
    grid = GridSpec(box=(0.0, 0.0, 0.0) + tuple(side), ncell=(12, 11, 10), num_subgrid=(1, 1, 1))
    rng = np.random.default_rng(4)
    ph = _photons(n, side)
    enabled = np.ones(27, np.uint8)
    enabled[[TravelDirection["FACE_Y_P"], TravelDirection["EDGE_X_PN"]]] = 0
    with TransportEngine(grid, precision=precision) as eng:
        eng.set_fields(0, np.exp(rng.normal(np.log(1e8), 1.0, grid.num_cells)),
                       10.0 ** rng.uniform(-5, -2, grid.num_cells))
        got, counts, done = eng.traverse_buffer(0, 0, 0, ph, enabled)
        _, J = eng.get_fields(0, neutral_fraction=False)
        eng.set_intensity(0, np.zeros(grid.num_cells))
        groups, lost = [[] for _ in range(27)], 0
        for k in range(0, n, 200):
            o, c, dn = eng.traverse_buffer(0, 0, 0, ph[k: k + 200], enabled)
            lost += dn
            for d, part in enumerate(np.split(o, np.cumsum(c)[:-1])):
                groups[d].append(part)
        _, Jp = eng.get_fields(0, neutral_fraction=False)
    want = [np.concatenate(g) if g else np.zeros(0, PHOTON_DTYPE) for g in groups]
    assert [w.size for w in want] == counts.tolist() and done == lost
    assert counts.sum() + done == n
    assert np.concatenate(want).tobytes() == got.tobytes()
    np.testing.assert_allclose(J, Jp, rtol=1e-7 if precision == "fp32" else 5e-12, atol=0)
