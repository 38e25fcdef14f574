"""The azimuth sweep (sweep.cu) and what it rests on: a ray's crossing times
and cells relative to its voxel depend only on its direction and on the
binades of its origin."""
import dataclasses

import numpy as np
import pytest

from conftest import device_arrays


def test_origin_fraction_is_constant_in_a_binade(oracle_lib):
    """For every direction, the rounded origin gx + 2 c minus gx is one value
    for all gx whose rounded origin has the same exponent (>= 2^2), up to the
    widest grid the sweep takes."""
    O = oracle_lib
    from solargpu_b200 import inputs
    dirs = np.asarray(O.directions(O.sky_bins(inputs.sun_positions(15.65, 46.56, 1)))[0], np.float32).reshape(-1, 3)
    c2 = np.unique(dirs[:, :2] * np.float32(2.0)).astype(np.float32)
    gx = np.concatenate([np.arange(4200), np.arange(8180, 8210), np.arange(16370, 16400), np.arange(32750, 32768)])
    for c in c2:
        ox = gx.astype(np.float32) + c
        assert ox.dtype == np.float32
        e = (ox.view(np.uint32) >> 23).astype(np.int64) - 127
        off = ox.astype(np.float64) - gx
        for b in range(2, 15):
            assert np.unique(off[(e == b) & (ox > 0)]).size <= 1, (c, b)
        # the cell 2^b + 2, from which the times of binade b are taken, lies in it for every direction
        rep = (2.0 ** np.arange(2, 15) + 2).astype(np.float32) + c
        assert np.array_equal((rep.view(np.uint32) >> 23).astype(np.int64) - 127, np.arange(2, 15))


def _scene(w, h, kind, seed):
    from solargpu_b200 import inputs
    rng = np.random.default_rng(seed)
    z = (rng.random((h, w)) * 4.0).astype(np.float32)
    for _ in range(1 + w * h // 150):
        y, x = rng.integers(0, h), rng.integers(0, w)
        z[y:y + rng.integers(1, 5), x:x + rng.integers(1, 5)] += np.float32(rng.random() * 25.0)
    s = inputs.scene_from_heightmap(f"win_{w}x{h}_{kind}", z, 1.0, 15.592, 46.543, 1)
    g, wz = s.grid.copy(), s.wall_z.copy()
    if kind == "odd":      # after voxelization, which wants finite heights
        at = rng.permutation(g.size)[:min(g.size, 6)]
        g[at] = np.array([np.nan, np.inf, -np.inf, 1e31, -1e31, 3e38], np.float32)[:at.size]
        if wz.size >= 4:
            wz[[0, 1, 2, 3]] = np.array([np.nan, np.inf, -np.inf, 2e30], np.float32)
    elif kind == "below":  # lower rays start below 0 and end on the range test
        g, wz = g - np.float32(6.0), wz - np.float32(6.0)
    mz = np.float32(12.0) if kind == "capped" else s.max_height
    return dataclasses.replace(s, grid=g, wall_z=wz, max_height=mz)


# one and two cells, the first binades, a tile less and more one cell, strips
# longer than most tabulated times on both axes, several tiles and binades
SIZES = [(1, 1), (3, 2), (5, 9), (31, 33), (32, 32), (64, 65), (300, 5), (6, 290), (133, 70)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "odd", "below", "capped"])
@pytest.mark.parametrize("w,h", SIZES)
def test_sweep_matches_oracle(cuda_lib, oracle_lib, w, h, kind):
    """Lists and shadow bits bit for bit against the oracle; the same from the
    general tracer (a context with a memory limit takes no tables), from Stage 1
    in chunks, whose warps hold pieces of several tiles, and for a few voxels
    in no order (solar_gpu_trace_shadow_subset)."""
    from solargpu_b200 import api
    s = _scene(w, h, kind, 100 * w + h)
    bins = oracle_lib.sky_bins(s.sun)
    off, ids, sh = oracle_lib.trace(s, bins)
    with api.Context(0) as a, api.Context(0) as b:
        b.set_memory_limit(8 << 30)
        d = device_arrays(s)
        for r in (a.trace(s, d, neighbor_format=0), b.trace(s, d, neighbor_format=0),
                  a.trace(s, d, neighbor_format=0, chunk_voxels=1000)):
            np.testing.assert_array_equal(r["csr_off"], off)
            np.testing.assert_array_equal(r["csr_ids"], ids)
            np.testing.assert_array_equal(r["shadow"], sh)
        import torch
        from solargpu_b200 import surrogate
        v = np.random.default_rng(1).integers(0, s.num_total, 77).astype(np.int32)
        got, words = surrogate.exact_bits(a, s, d, torch.from_numpy(v).cuda())
        np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), sh[v])
