"""The one-pass ba-RLE encoder (barle.cu, lists of up to 1024 ids): the run
optimiser without its fixpoint, modelled here element by element, and the
kernel's bytes at the edges of its list sizes, against the oracle's encoder."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O

CLASS_EDGES = np.array([15, 255, 65535, 16777215], np.int64)


def _model(ids) -> bytes:
    """Merged run of one id = the id takes the next class; runs = maximal equal classes."""
    x = np.sort(np.asarray(ids, np.int64))[::-1]
    if x.size == 0:
        return b""
    d = np.concatenate([x[:1], x[:-1] - x[1:]])
    w = [int(np.searchsorted(CLASS_EDGES, v)) for v in d]
    n, joined, out = len(w), False, list(w)
    for i in range(1, n):
        single = w[i - 1] == w[i] + 1 and (i + 1 == n or w[i + 1] != w[i])
        joined = single and not joined
        out[i] += joined
    pieces, i = [], 0
    while i < n:
        j = i
        while j < n and out[j] == out[i] and j - i < 255:
            j += 1
        pieces.append((out[i], i, j))
        i = j
    b = bytearray()
    for q in range(0, len(pieces), 8):
        blk = pieces[q:q + 8]
        bits = 0
        for j in range(8):
            bits = (bits << 3) | (blk[j][0] if j < len(blk) else 7)
        b += bits.to_bytes(3, "big") + bytes(e - s for _, s, e in blk)
        for c, s, e in blk:
            if c == 0:
                v = [int(t) for t in d[s:e]] + [0]
                b += bytes((v[k] << 4 | v[k + 1]) & 0xFF for k in range(0, e - s, 2))
            else:
                for t in d[s:e]:
                    b += int(t).to_bytes(c, "big")
    return bytes(b)


def _list(rng, k, mix):
    """k distinct ids; mix: probabilities of the five delta classes."""
    lo = np.array([1, 16, 256, 65536, 16777216])
    hi = np.array([15, 255, 65535, 400000, 17000000])
    c = rng.choice(5, size=k, p=mix)
    d = rng.integers(lo[c], hi[c], endpoint=True)
    while d.sum() > 2 ** 31 - 1:   # ids stay positive ints
        d[np.argmax(d)] = rng.integers(1, 256)
    x = np.cumsum(d)
    return rng.permutation(x).astype(np.int32)


MIXES = [(0.5, 0.5, 0, 0, 0), (0.9, 0.08, 0.02, 0, 0), (0.25, 0.25, 0.25, 0.2, 0.05), (0.02, 0.96, 0.02, 0, 0),
         (1, 0, 0, 0, 0), (0, 0, 1, 0, 0), (0.3, 0.3, 0.2, 0.19, 0.01)]


def _lists(seed, sizes):
    rng = np.random.default_rng(seed)
    return [_list(rng, k, MIXES[i % len(MIXES)]) for i, k in enumerate(sizes)]


def test_one_pass_runs_match_the_fixpoint():
    rng = np.random.default_rng(3)
    sizes = [int(k) for k in rng.integers(1, 60, 3000)] + [254, 255, 256, 509, 510, 511, 512, 765, 766, 1024] * 7
    for x in _lists(4, sizes):
        assert _model(x) == O.barle_encode(x)
    # chains of classes, each a run of one id, after a run of 1 to 3 of the widest
    step = {0: 3, 1: 100, 2: 1000, 3: 100000, 4: 16777300}
    for top in range(1, 5):
        for lead in (1, 2, 3):
            for tail in range(6):
                cl = [top] * lead + list(range(top - 1, -1, -1)) + [(t * 2) % (top + 1) for t in range(tail)]
                d = np.array([step[c] for c in cl], np.int64)
                x = 2 ** 31 - 1 - np.cumsum(d[1:])   # the first id is absolute (widest class)
                x = np.concatenate([[2 ** 31 - 1], x]).astype(np.int32)
                assert _model(x) == O.barle_encode(x)


@pytest.mark.gpu
@pytest.mark.parametrize("part", range(4))
def test_encoder_bytes(cuda_lib, part):
    """Sizes around the lanes' shares (8, 16, 32 ids), the three ways through the
    kernels (256, 512, 1024 ids), pieces of 255, and the two-pass encoder beyond."""
    import torch
    from solargpu_b200 import api
    edges = [0, 1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 128, 129, 253, 254, 255, 256, 257, 258, 300, 383, 384, 385,
             509, 510, 511, 512, 513, 514, 600, 765, 766, 767, 1000, 1020, 1022, 1023, 1024, 1025, 1026, 1500, 2592]
    lists = _lists(100 + part, [k for k in edges for _ in range(7)])   # every size with every mix
    off = np.concatenate([[0], np.cumsum([x.size for x in lists])]).astype(np.int64)
    ids = torch.from_numpy(np.concatenate(lists)).cuda()
    offd = torch.from_numpy(off).cuda()
    want_off, want = O.barle_encode_csr(off, np.concatenate(lists))
    got_off = torch.zeros(len(lists) + 1, dtype=torch.int64, device="cuda")
    total = C.c_longlong()
    fn = api.lib().solar_gpu_barle_encode_noalloc
    buf = torch.zeros(want.size + 64, dtype=torch.uint8, device="cuda")
    shift = part   # streams start on every byte of a word
    rc = fn(C.c_void_p(offd.data_ptr()), C.c_void_p(ids.data_ptr()), len(lists), C.c_void_p(got_off.data_ptr()),
            C.c_void_p(buf.data_ptr() + shift), C.c_longlong(want.size), C.byref(total), None)
    assert rc == 0, api.lib().solar_gpu_last_error().decode()
    assert total.value == want.size
    np.testing.assert_array_equal(got_off.cpu().numpy(), want_off)
    b = buf.cpu().numpy()
    np.testing.assert_array_equal(b[shift:shift + want.size], want)
    assert not b[:shift].any() and not b[shift + want.size:].any()
