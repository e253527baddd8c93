"""The generator's device paths at their edges: percolation through one cell's
components joined over the tiling (rows longer than a warp, cells of one
voxel, snakes that only percolate through several tiles, no pores at all)
against the oracle's labelling of the whole tiling, and the device quantile
(ties, the extreme porosities, rows beyond a block) against numpy's."""
import numpy as np
import pytest

from flow_anizotropy_b200 import gen3d as G
from oracle import gen3d_oracle as GO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 70), (2, 3, 33), (4, 5, 64), (7, 2, 95), (12, 12, 12)])
@pytest.mark.parametrize("frac", [0.0, 0.35, 0.6, 0.75, 1.0])
def test_percolation(gpu, shape, frac):
    gen = G.Generator(size=8)
    for seed in range(4):
        solid = np.random.default_rng(seed).random(shape) < frac
        assert gen.percolates(solid.astype(np.uint8)) == tuple(GO.percolates(solid))


def test_diagonal_channel(gpu):
    """A channel that leaves the cell one row higher each time: it crosses the
    tiling along x only by climbing through the tiles along y."""
    for ny, climb in ((6, 2), (6, 5), (9, 3)):
        solid = np.ones((3, ny, 8), np.uint8)
        solid[1, 0, :4] = 0
        solid[1, :climb + 1, 4] = 0
        solid[1, climb, 4:] = 0
        assert G.Generator(size=8).percolates(solid) == tuple(GO.percolates(solid.astype(bool)))


@pytest.mark.parametrize("size,modes", [(3, 6), (31, 20), (80, 50), (150, 9), (260, 3)])
@pytest.mark.parametrize("por", [0.0, 0.31, 1.0])
def test_quantile(gpu, size, modes, por):
    rng = np.random.default_rng(size)
    q = rng.integers(-4, 5, (modes, 3))
    ph = rng.uniform(0, np.pi, modes)
    solid, t = G.Generator(size=size).structure(q, ph, por)
    p = G.axis_points(size)
    field = np.zeros((size, size, size))
    for (a, b, c), s in zip(q, ph):
        field += np.cos(((2 * np.pi * c) * p[:, None, None] + (2 * np.pi * b) * p[None, :, None])
                        + (2 * np.pi * a) * p[None, None, :] + s)
    field *= np.sqrt(2.0 / modes)
    assert abs(t - np.quantile(field, por)) <= 1e-12 * max(1.0, abs(t))
    # voxels further from the threshold than the cosine's last bits lie on its side
    sure = np.abs(field - t) > 1e-12
    assert np.array_equal(solid[sure], (field > t)[sure].astype(np.uint8))
