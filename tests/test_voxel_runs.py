"""GPU voxelization by runs of 1024 cells: sizes around a run, cells with more walls
than a block has threads, runs without any, against the host restatement.  Counts,
parents and heights are equal; angles within the 2e-6 rad by which CUDA's atan2f and
the host library's may differ (0 and 2 pi are one direction)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ANGLE_TOL = 2e-6


@pytest.mark.parametrize("w,h", [(1, 1), (1, 1023), (1024, 1), (1025, 1), (31, 33), (32, 32), (2, 1023), (37, 211),
                                 (2049, 3)])
@pytest.mark.parametrize("size", [1.0, 0.37])
@pytest.mark.parametrize("kind", ["flat", "rough", "towers"])
def test_runs(cuda_lib, w, h, size, kind):
    import torch
    from solargpu_b200 import api, inputs
    rng = np.random.default_rng(w * 7 + h)
    z = np.zeros((h, w), np.float32)
    if kind != "flat":
        z += (rng.random((h, w)) * 6.0).astype(np.float32)
    if kind == "towers":
        for k in rng.integers(0, w * h, 5):
            z.ravel()[k] += np.float32(rng.uniform(300.0, 900.0))
        z.ravel()[[0, -1]] += np.float32(500.0)
    with np.errstate(all="ignore"):
        total, top, pp, wz, sl, asp = inputs.voxelize(z, size)
    with api.Context(0) as c:
        for _ in range(2):   # the second call over the first one's sums
            r = c.voxelize(torch.from_numpy(z.ravel().copy()).cuda(), w, h, size)
    assert (r["num_total"], r["num_top"]) == (total, top)
    np.testing.assert_array_equal(r["pixel_parent"].cpu().numpy(), pp)
    np.testing.assert_array_equal(r["wall_z"].cpu().numpy()[:total - top], wz[:total - top])
    for got, want in ((r["slopes"].cpu().numpy(), sl), (r["aspects"].cpu().numpy(), asp)):
        d = np.abs(got.astype(np.float64) - want)
        d = np.minimum(d, np.abs(2.0 * np.pi - d))
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
        assert (d[~np.isnan(want)] <= ANGLE_TOL).all()
