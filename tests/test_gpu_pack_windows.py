"""Packing and unpacking at the edges of their windows of 512 slots: windows with
many events, events over many windows, a last window that is partly filled, more
layers than a CTA's share, arrays off a 16-byte boundary, large and small unpacks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    "tiny_events": (8, [1, 3, 8, 9, 0, 17, 2] * 40, 3),
    "one_event": (32, [5001], 7),
    "window_ends": (64, [512, 511, 513, 0, 0, 1024, 64, 1], 20),
    "one_batch": (16, [5], 32),
    "large": (16, [20011, 7, 300] * 28, 2),  # above the size from which unpacking sorts windows
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("shift", [0, 1])
def test_round_trip(p2z, ctx, name, shift):
    import torch
    bsize, counts, nlayer = CASES[name]
    counts = np.array(counts, dtype=np.int64)
    cfg = p2z.make_config(bsize=bsize, nevts=len(counts), event_ntrks=counts, nlayer=nlayer)
    ns = p2z.num_batches(cfg) * bsize
    g = torch.Generator(device="cuda").manual_seed(ns)

    def words(*shape):  # `shift` words past a 16-byte boundary
        n = int(np.prod(shape))
        w = torch.empty(n + shift, dtype=torch.int32, device="cuda")[shift:].view(*shape)
        return w.copy_(torch.randint(-2 ** 31, 2 ** 31 - 1, shape, generator=g, device="cuda"))

    t, h, m = words(ns // bsize, 28, bsize), words(ns // bsize, nlayer, 9, bsize), words(ns)
    pt, ph, pm, back = words(*t.shape), words(*h.shape), words(ns), words(*t.shape)
    perm = torch.full((2 * ns,), -1, dtype=torch.int64, device="cuda")
    ctx.pack_by_hits_device(cfg, t, h, pt, ph, perm, d_mask_in=m, d_mask_out=pm)
    # the order: per event, most hits first, equal counts as they were, padding last
    mm = m.cpu().numpy().view(np.uint32) & np.uint32((1 << nlayer) - 1)
    hits = np.array([bin(int(x)).count("1") for x in mm])
    want, first = [], 0
    for n in counts:
        room = -(-int(n) // bsize) * bsize
        key = np.where(np.arange(room) < n, 32 - hits[first:first + room], 33)
        want.append(first + np.argsort(key, kind="stable"))
        first += room
    want = np.concatenate(want)
    assert np.array_equal(perm[:ns].cpu().numpy(), want)
    inv = np.empty(ns, dtype=np.int64)
    inv[want] = np.arange(ns)
    assert np.array_equal(perm[ns:].cpu().numpy(), inv)
    w = torch.from_numpy(want).cuda()
    assert torch.equal(pm, m[w])
    assert torch.equal(pt.transpose(0, 1).reshape(28, ns), t.transpose(0, 1).reshape(28, ns)[:, w])
    flat = lambda x: x.permute(1, 2, 0, 3).reshape(nlayer, 9, ns)  # noqa: E731
    assert torch.equal(flat(ph), flat(h)[:, :, w])
    ctx.unpack_tracks_device(cfg, perm, pt, back)
    torch.cuda.synchronize()
    assert torch.equal(back, t)
