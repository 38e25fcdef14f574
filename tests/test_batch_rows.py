"""A batch's tiles work in one context's raw hit rows, tile after tile: growing and
shrinking tiles give the bits of runs of their own, on a first and a second
batch, and the other contexts hold no rows; contexts with a memory limit keep theirs.
The tiles are below 20,000 voxels, where a limit does not change the reflection's route."""
import numpy as np
import pytest

from conftest import device_arrays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("limit", [0, 64 << 30])
def test_tiles_share_rows(cuda_lib, fmt, limit):
    import torch
    from solargpu_b200 import api, inputs
    scenes = []
    for k, (w, h) in enumerate([(40, 33), (96, 70), (20, 20), (88, 86)]):
        z = (np.random.default_rng(k).random((h, w)) * 5.0).astype(np.float32)
        z[h // 2:h // 2 + 4, w // 3:w // 3 + 4] += np.float32(9.0)
        scenes.append(inputs.scene_from_heightmap(f"tile{k}", z, 1.0, 15.592, 46.543, 1, seed=k))
    devs = [device_arrays(s) for s in scenes]
    want, held = [], []
    for s, d in zip(scenes, devs):
        out = torch.zeros(s.num_total, dtype=torch.float32, device="cuda:0")
        with api.Context(0) as c:
            c.run_device(s, d, out, neighbor_format=fmt)
            torch.cuda.synchronize()
            held.append(c.memory_held())
        want.append(out)
    ctxs = [api.Context(0) for _ in scenes]
    try:
        for c in ctxs:
            c.set_memory_limit(limit)
        for _ in range(2):
            outs = [torch.zeros_like(w) for w in want]
            api.run_batch(ctxs, scenes, devs, outs, per_tile=[dict(neighbor_format=fmt)] * len(scenes))
            torch.cuda.synchronize()
            for got, w in zip(outs, want):
                assert torch.equal(got, w)
        if not limit:   # a context of its own holds the rows too
            for s, c, own in list(zip(scenes, ctxs, held))[1:]:
                assert c.memory_held() <= own - 4 * 2592 * s.num_total
    finally:
        for c in ctxs:
            c.close()
