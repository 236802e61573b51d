"""Ray sums of the warm-start features (k_features) where its samples are found another
way: sources clear of the box's faces (no clamps), on a face, in a corner and outside the
box (clamped), grids of odd sides; against the same FP32 sum on the host (the tolerance of
the features' own test: the FP64 logarithm and scaling after equal sums)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from parallelcmacionize_b200 import GridSpec  # noqa: E402
from parallelcmacionize_b200.warmstart import UNet, stromgren_ratio  # noqa: E402

pytestmark = pytest.mark.gpu

PLACES = {"inside": (0.31, 0.62, 0.47), "face": (0.0, 0.4, 0.7), "upper face": (0.5, 1.0, 0.2),
          "corner": (1.0, 1.0, 0.0), "by a face": (0.5, 0.5, 1e-4), "outside": (1.4, -0.3, 0.5)}


@pytest.mark.parametrize("ncell", [(9, 7, 11), (32, 16, 8)])
@pytest.mark.parametrize("place", list(PLACES))
def test_ray_sums(place, ncell):
    box = (-2.0e16, -1.0e16, 0.0, 4.0e16, 3.0e16, 5.0e16)
    at = tuple(box[a] + PLACES[place][a] * box[3 + a] for a in range(3))
    grid = GridSpec(box=box, ncell=ncell, num_subgrid=(1, 1, 1),
                    sources=[at + (3.0e48,), (1.0e15, 2.0e15, 3.0e16, 1.0e48)])
    rng = np.random.default_rng(6)
    cube = np.exp(rng.normal(np.log(1e8), 1.0, ncell))
    with UNet() as net:
        f = net.features(torch.from_numpy(cube.ravel().copy()).cuda(), grid,
                         norm=np.array([0, 1] * 3, np.float32)).cpu().numpy()
    np.testing.assert_allclose(f[:, 2], stromgren_ratio(grid, cube).ravel(), rtol=1e-5, atol=1e-5)
