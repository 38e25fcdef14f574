"""The early-exit tables' geometry on blocks of 2 x 2 cells (cone.cu): the blocks of
all cells a ray visits after a cell lie in the cell's block + e + K, for some offset
e of the window [-(r + a + b), r] per axis, r = 1 + ceil((1 + 2 L (L + 1) 2^-24) / 2),
K the cone between two vectors a, b of the Farey set of order 4."""
import numpy as np
import pytest

from oracle import oracle as O
from test_cone_bound import cone_of, dda_cells, farey

ORDER, SIDE = 4, 2


def test_the_smaller_set_is_unimodular_too():
    F = farey(ORDER)
    assert F[0] == (1, 0) and F[-1] == (0, 1)
    for a, b in zip(F[:-1], F[1:]):
        assert a[0] * b[1] - a[1] * b[0] == 1


@pytest.mark.parametrize("flip", [False, True])
def test_later_blocks_lie_in_the_widened_cone(flip):
    """flip: blocks cut from the far side, as the grid's blocks look in the
    unsigned coordinates of a ray that runs against them."""
    bins = O.sky_bins(np.zeros((8760, 2), np.float32) + np.float32([180.0, 30.0]))
    dirs, _, upper = O.directions(bins)
    rng = np.random.default_rng(4)
    F = farey(ORDER)
    steps = 160
    r = 1 + int(np.ceil((1.0 + 2.0 * (steps + 4) * (steps + 5) / 16777216.0) / SIDE))
    checked = 0
    for d in rng.choice(np.flatnonzero(upper), 48, replace=False):
        cells, dX, dY = dda_cells(dirs[d, 0], dirs[d, 1], int(rng.integers(0, 50)), int(rng.integers(0, 50)), steps)
        blocks = -(-cells // SIDE) if flip else cells // SIDE
        a, b = cone_of(F, dX, dY)
        ex = np.arange(-(r + a[0] + b[0]), r + 1)
        ey = np.arange(-(r + a[1] + b[1]), r + 1)
        E = np.stack(np.meshgrid(ex, ey, indexing="ij"), -1).reshape(-1, 2)
        for k in range(0, steps - 1, 7):
            q = (blocks[k:] - blocks[k])[:, None, :] - E[None, :, :]
            in_k = ((a[0] * q[..., 1] - a[1] * q[..., 0]) >= 0) & ((q[..., 0] * b[1] - q[..., 1] * b[0]) >= 0)
            assert in_k.any(axis=1).all(), (d, k)
            checked += q.shape[0]
    assert checked > 40000
