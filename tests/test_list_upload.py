"""Saved lists from pageable arrays go to the device through pinned slots on several
threads (arrays from 8 MB on): the same result as from page-locked arrays, which
do not, call after call on one context and on several threads at once."""
import threading

import numpy as np
import pytest

from conftest import device_arrays, load_scene

pytestmark = pytest.mark.gpu


def test_pageable_lists_arrive_whole(cuda_lib):
    import torch
    from solargpu_b200 import api
    s = load_scene("dsm160")
    dev = device_arrays(s)
    with api.Context(0) as c:
        lists = c.trace(s, dev, neighbor_format=api.CSR)
    ids = lists["csr_ids"]
    assert ids.nbytes > 8 << 20 and ids.nbytes % (1 << 20), "large, and not whole slots"
    # another order of every list's ids: other bytes, for a second upload over the first
    keep = np.repeat(np.arange(s.num_total), np.diff(lists["csr_off"]))
    other = dict(lists, csr_ids=ids[np.lexsort((-ids, keep))].copy())

    def run(c, l):
        out = torch.zeros(s.num_total, dtype=torch.float32, device="cuda:0")
        c.run_lists(s, dev, l, out)
        torch.cuda.synchronize()
        return out.cpu().numpy()

    def pinned(l):
        return dict(l, csr_ids=torch.from_numpy(l["csr_ids"]).pin_memory().numpy())
    with api.Context(0) as c:
        want = [run(c, pinned(l)) for l in (lists, other)]
    assert not np.array_equal(want[0], want[1]) or not np.array_equal(ids, other["csr_ids"])
    got = {}

    def user(k):
        with api.Context(0) as c:
            got[k] = [run(c, l) for _ in range(3) for l in (lists, other)]   # slots from the second run on
    ts = [threading.Thread(target=user, args=(k,)) for k in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert sorted(got) == [0, 1, 2]
    for outs in got.values():
        for i, out in enumerate(outs):
            np.testing.assert_array_equal(out, want[i % 2])
