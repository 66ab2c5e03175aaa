"""Unpacking by windows (from 6 windows of 512 slots an SM on) and by scattered reads: both
sides of that limit, every batch width, arrays on and off a 16-byte boundary."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bsize", [8, 16, 32, 64])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("windows", [-1, 0, 0.5])
def test_gathers_by_the_inverse(p2z, ctx, bsize, shift, windows):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ns = int((6 * sms + windows) * 512) // bsize * bsize
    cfg = p2z.make_config(bsize=bsize, nevts=1, event_ntrks=np.array([ns], dtype=np.int64), nlayer=1)
    g = torch.Generator(device="cuda").manual_seed(ns)
    words = lambda: torch.empty(28 * ns + shift, dtype=torch.int32, device="cuda")[shift:].view(ns // bsize, 28, bsize)  # noqa: E731
    t = words().copy_(torch.randint(-2 ** 31, 2 ** 31 - 1, (ns // bsize, 28, bsize), generator=g, device="cuda"))
    out = words().fill_(-1)
    inv = torch.randperm(ns, generator=g, device="cuda")
    perm = torch.empty(2 * ns, dtype=torch.int64, device="cuda")
    perm[inv] = torch.arange(ns, device="cuda")
    perm[ns:] = inv
    ctx.unpack_tracks_device(cfg, perm, t, out)
    torch.cuda.synchronize()
    flat = lambda a: a.transpose(0, 1).reshape(28, ns)  # noqa: E731
    assert torch.equal(flat(out), flat(t)[:, inv])
