"""Light cells of the tensor-core reflection: the weights of cells that few
voxels of a group see, multiplied by k_light instead of the MMAs.

The same scene and lists run with light cells and, under a memory limit,
without them.  Both multiply the same fp16 irradiance; what differs is the
weights' precision (FP32 against 22 bits of the largest weight) and the order
of FP32 sums of up to about 2500 terms a voxel and hour: a random walk of 2500
roundings of 2^-24 is 3e-6, the bound below is five times that.
"""
import numpy as np
import pytest

from conftest import device_arrays, load_scene

pytestmark = pytest.mark.gpu
RTOL = 1.5e-5


def _both(s, dev, lists, fmt, acc):
    import torch
    from solargpu_b200 import api
    outs = []
    for limit in (0, 16 << 30):
        out = torch.zeros(s.num_total, dtype=torch.float32, device="cuda:0")
        with api.Context(0) as c:
            if limit:
                c.set_memory_limit(limit)
            for _ in range(2):   # a second pass over the buffers of the first
                if lists is None:
                    c.run_device(s, dev, out, neighbor_format=fmt, accumulation=acc)
                else:
                    c.run_lists(s, dev, lists, out, accumulation=acc)
                torch.cuda.synchronize()
                outs.append(out.cpu().numpy().astype(np.float64))
    return outs


def _same(outs):
    light, again, dense, dense_again = outs
    assert np.array_equal(light, again) and np.array_equal(dense, dense_again)
    assert not np.array_equal(light, dense), "the light cells did not take part"
    assert np.isfinite(light).all()
    assert (np.abs(light - dense) <= RTOL * np.abs(dense)).all()


@pytest.mark.parametrize("fmt,acc", [(0, 0), (1, 1), (0, 2)])
def test_light_cells_match_the_dense_products(cuda_lib, fmt, acc):
    s = load_scene("dsm160")
    _same(_both(s, device_arrays(s), None, fmt, acc))


def test_lists_with_empty_long_and_repeated_entries(cuda_lib):
    """A caller's own lists: none, one cell hundreds of times (more entries of a
    cell than a byte counts), and one cell in every list (a cell's light list
    longer than a warp's share, and dense in full groups)."""
    from solargpu_b200 import api
    s = load_scene("dsm160")
    dev = device_arrays(s)
    with api.Context(0) as c:
        lists = c.trace(s, dev, neighbor_format=api.CSR)
    off, ids = lists["csr_off"], lists["csr_ids"]
    rows = [ids[off[v]:off[v + 1]] for v in range(s.num_total)]
    rng = np.random.default_rng(5)
    far = int(np.argmax(s.grid)) + 1
    for v in range(0, s.num_total, 97):
        rows[v] = np.zeros(0, np.int32)
    for v in range(11, s.num_total, 501):
        if rows[v].size:
            rows[v] = np.repeat(rows[v][:1], 600)
    for v in rng.permutation(s.num_total)[:s.num_total // 6]:
        rows[v] = np.append(rows[v], np.int32(far))
    lists = dict(lists, csr_off=np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int64),
                 csr_ids=np.concatenate(rows).astype(np.int32))
    _same(_both(s, dev, lists, 0, 0))
