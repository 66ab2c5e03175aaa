"""Packing events of many windows, whose offsets a whole CTA finds, beside small ones, and in
a time that depends on the slots, not on how few events they belong to."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _packed(p2z, ctx, bsize, counts, repeat=0):
    """The permutation and the hit counts of an uneven sample of one or two layers, and the best time of a pack."""
    import torch
    counts = np.array(counts, dtype=np.int64)
    nl = 2
    cfg = p2z.make_config(bsize=bsize, nevts=len(counts), event_ntrks=counts, nlayer=nl)
    ns = p2z.num_batches(cfg) * bsize
    g = torch.Generator(device="cuda").manual_seed(ns)
    words = lambda *shape: torch.randint(-2 ** 31, 2 ** 31 - 1, shape, generator=g, device="cuda", dtype=torch.int32)  # noqa: E731
    t, h, m = words(ns // bsize, 28, bsize), words(ns // bsize, nl, 9, bsize), words(ns)
    pt, ph, pm = torch.empty_like(t), torch.empty_like(h), torch.empty_like(m)
    perm = torch.full((2 * ns,), -1, dtype=torch.int64, device="cuda")
    best = float("inf")
    for _ in range(1 + repeat):
        t0 = time.perf_counter()
        ctx.pack_by_hits_device(cfg, t, h, pt, ph, perm, d_mask_in=m, d_mask_out=pm)
        best = min(best, time.perf_counter() - t0)
    w = perm[:ns]
    assert torch.equal(pm, m[w])
    assert torch.equal(pt.transpose(0, 1).reshape(28, ns), t.transpose(0, 1).reshape(28, ns)[:, w])
    bits = m.cpu().numpy() & 3
    return counts, perm.cpu().numpy(), (bits & 1) + (bits >> 1), best


W = 512  # slots of a window; events of more than 32 windows take a CTA


@pytest.mark.parametrize("bsize", [8, 64])
@pytest.mark.parametrize("counts", [[32 * W, 33 * W, 1, 0, 32 * W + 1, 31 * W], [3, 65 * W - 1, 7, 64 * W],
                                    [1, 32 * 32 * W + 5, 0, 9], [1030 * W]])
def test_order(p2z, ctx, bsize, counts):
    counts, perm, hits, _ = _packed(p2z, ctx, bsize, counts)
    ns, first, want = len(hits), 0, []
    for n in counts:
        room = -(-int(n) // bsize) * bsize
        key = np.where(np.arange(room) < n, 2 - hits[first:first + room], 3)
        want.append(first + np.argsort(key, kind="stable"))
        first += room
    want = np.concatenate(want)
    inv = np.empty(ns, dtype=np.int64)
    inv[want] = np.arange(ns)
    assert np.array_equal(perm[:ns], want) and np.array_equal(perm[ns:], inv)


def test_one_event_takes_as_long_as_many(p2z, ctx):
    one = _packed(p2z, ctx, 32, [2_000_000], repeat=5)[3]
    many = _packed(p2z, ctx, 32, [20_000] * 100, repeat=5)[3]
    assert one < 1.5 * many, (one, many)
