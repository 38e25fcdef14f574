"""Scans of counts in one block (up to 16384) and in three launches (more): scenes
whose visiting order has 15360, 16384 and 20480 cell positions, and whose voxels
are fewer and more than 16384.  Lists and shadow bits equal the oracle's."""
import numpy as np
import pytest

from conftest import device_arrays, oracle_trace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(160, 96), (128, 128), (129, 128)])
def test_lists(cuda_lib, w, h):
    from solargpu_b200 import api, inputs
    rng = np.random.default_rng(w + h)
    z = (rng.random((h, w)) * 0.9).astype(np.float32)   # few walls: about as many voxels as cells
    for _ in range(4):
        y, x = rng.integers(0, h - 6), rng.integers(0, w - 6)
        z[y:y + 5, x:x + 5] += np.float32(7.0)
    s = inputs.scene_from_heightmap(f"scan{w}x{h}", z, 1.0, 15.592, 46.543, 1)
    _, off, ids, sh = oracle_trace(s)
    with api.Context(0) as c:
        r = c.trace(s, device_arrays(s), neighbor_format=api.CSR)
    np.testing.assert_array_equal(r["csr_off"], off)
    np.testing.assert_array_equal(r["csr_ids"], ids)
    np.testing.assert_array_equal(r["shadow"], sh)
