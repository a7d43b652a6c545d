"""The allocation-free pair query at the edges of its warps, chunks and kept
partners, against a brute-force restatement of the pair rule on the host:
sizes around multiples of the warp width and of the owners a warp or block
takes, owners with more partners than are kept, static and shared bodies,
bounds that touch or are inverted, and capacities that cut a bucket.
Integer work: exact."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def oracle_pairs(b, flags):
    """Pairs (a < b): in x the shape that starts first (lower id on ties)
    reaches the other's start, y and z overlap, different bodies, one
    dynamic."""
    out = []
    body, dyn = flags & 0x7FFFFFFF, flags >> 31
    for a in range(len(b)):
        o = b[a + 1:]
        first = o[:, 0] >= b[a, 0]
        hit = np.where(first, o[:, 0] <= b[a, 3], b[a, 0] <= o[:, 3])
        hit &= (body[a + 1:] != body[a]) & ((dyn[a + 1:] | dyn[a]) != 0)
        for k in (1, 2):
            hit &= ~((b[a, k] > o[:, 3 + k]) | (o[:, k] > b[a, 3 + k]))
        out.append(np.stack([np.full(hit.sum(), a), np.flatnonzero(hit) + a + 1], 1))
    return np.concatenate(out).astype(np.uint32) if out else np.zeros((0, 2), np.uint32)


def query(pkg, b, flags, cap):
    import torch
    n = len(b)
    bt = torch.from_numpy(np.ascontiguousarray(b).reshape(-1).view(np.int32)).cuda()
    ft = torch.from_numpy(np.ascontiguousarray(flags).view(np.int32)).cuda()
    p = torch.full((2 * max(cap, 1),), -1, dtype=torch.int32, device="cuda")
    c = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    msg = C.create_string_buffer(256)
    rc = pkg.lib().fyzz_b200_sap_pairs_static_scratch(bt.data_ptr(), ft.data_ptr(), n, p.data_ptr(), cap,
                                                      c.data_ptr(), None, msg, len(msg))
    assert rc == 0, msg.value
    torch.cuda.synchronize()
    return int(c.cpu()[0]), p.cpu().numpy().view(np.uint32).reshape(-1, 2)


@pytest.mark.parametrize("n,spread", [(1, 10), (2, 1), (3, 2), (31, 6), (32, 6), (33, 6), (63, 9), (64, 9), (65, 9),
                                      (127, 12), (129, 12), (257, 4), (1000, 60), (4097, 300), (8191, 500),
                                      (8192, 40)])
def test_matches_brute_force(pkg, n, spread):
    rng = np.random.default_rng(n)
    lo = rng.integers(0, 16 * spread, (n, 3)).astype(np.uint32) + np.uint32(1 << 31)
    b = np.concatenate([lo, lo + rng.integers(0, 24, (n, 3)).astype(np.uint32)], 1)
    swap = rng.random(n) < 0.02                    # inverted in x: the sweep's one-sided rule decides
    b[swap, 0], b[swap, 3] = b[swap, 3].copy(), b[swap, 0].copy()
    body = np.arange(n, dtype=np.uint32)
    body[1:] -= (rng.random(n - 1) < 0.2).astype(np.uint32)
    flags = body | ((body % 4 != 0).astype(np.uint32) << np.uint32(31))
    want = oracle_pairs(b, flags)
    cap = len(want) + 8
    total, got = query(pkg, b, flags, cap)
    assert total == len(want)
    np.testing.assert_array_equal(got[:total], want)
    assert np.all(got[total:] == 0xFFFFFFFF)
    if len(want) > 3:                              # a capacity inside the list: whole buckets that fit
        cap = len(want) // 2
        total, got = query(pkg, b, flags, cap)
        ends = np.flatnonzero(np.append(want[1:, 0] != want[:-1, 0], True)) + 1
        k = int(ends[ends <= cap].max(initial=0))
        assert total == len(want)
        np.testing.assert_array_equal(got[:k], want[:k])
        assert np.all(got[k:] == 0xFFFFFFFF)
