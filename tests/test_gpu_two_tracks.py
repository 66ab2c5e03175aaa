"""The kernel with two tracks per thread (flat launches that fill the GPU) and the
sorted windows that runs with schedule AUTO take for large masked samples: the
same bits as the one-track kernel in stored order, which a launch per event of
the same arrays takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLOTS = 640 * 148  # two tracks per thread from this many slots on (148 SMs)


def _both(p2z, ctx, cfg, dt, dh, dm=None):
    import torch
    outs, stats = [], []
    for schedule in ("auto", "per_event"):
        cfg.schedule = p2z.SCHED_NAMES[schedule]
        out = torch.full_like(dt, float("nan"))
        stats.append(ctx.run_device(cfg, dt, dh, out, d_mask=dm))
        torch.cuda.synchronize()
        outs.append(out.cpu().numpy().view(np.uint32))
    assert np.array_equal(outs[0], outs[1])
    assert stats[0].updates == stats[1].updates and stats[0].singular == stats[1].singular
    return stats


def _device(p2z, ctx, cfg, soa=False, params=None, masked=False):
    import torch
    nb, B, nl = p2z.num_batches(cfg), cfg.bsize, cfg.nlayer
    dt = torch.empty((nb, 28, B), device="cuda")
    dh = torch.empty((nb, nl, 9, B), device="cuda")
    dm = torch.empty(nb * B, dtype=torch.int32, device="cuda") if masked else None
    ctx.generate_physics_device(cfg, dt, dh, dm, params=params)
    if soa:
        dt = dt.permute(1, 0, 2).reshape(28, nb * B).contiguous()
        dh = dh.permute(1, 2, 0, 3).reshape(nl, 9, nb * B).contiguous()
        cfg.layout = p2z.LAYOUT_SOA
    return dt, dh, dm


# every layout, layer counts around the ring's depth, last warps that are partly filled
@pytest.mark.parametrize("layout", ["b8", "b16", "b32", "b64", "soa"])
@pytest.mark.parametrize("nlayer", [1, 2, 3, 4, 5, 20, 32])
def test_uniform(p2z, ctx, layout, nlayer):
    B = 8 if layout == "soa" else int(layout[1:])
    ntrks = (SLOTS // 7 // B + 1) * B  # 7 events: just past the threshold, and no multiple of 64 for B < 64
    cfg = p2z.make_config(bsize=B, nevts=7, ntrks=ntrks, nlayer=nlayer)
    dt, dh, _ = _device(p2z, ctx, cfg, soa=layout == "soa")
    stats = _both(p2z, ctx, cfg, dt, dh)
    assert stats[0].launches == 1 and stats[1].launches == 7


@pytest.mark.parametrize("bsize", [8, 32])
def test_padding(p2z, ctx, bsize):
    """Uneven events without a mask: one, both and none of a pair are padding."""
    counts = np.array([1, 0, 9000, 7, 12345, 31, 2] + [14999] * 5 + [33, 6], dtype=np.int64)
    cfg = p2z.make_config(bsize=bsize, nevts=len(counts), event_ntrks=counts, nlayer=6)
    dt, dh, _ = _device(p2z, ctx, cfg)
    # padding slots hold anything: here NaN, which their neighbours must not see
    first = np.concatenate([[0], np.cumsum((counts + bsize - 1) // bsize)])
    for e, n in enumerate(counts):
        if n % bsize:
            b = int(first[e + 1]) - 1
            dt[b, :, n % bsize:] = float("nan")
            dh[b, :, :, n % bsize:] = float("nan")
    assert _both(p2z, ctx, cfg, dt, dh)[0].singular == 0


@pytest.mark.parametrize("what", ["low_pt", "off_angles", "nonfinite", "indefinite"])
def test_rare_paths(p2z, ctx, what):
    """Tracks outside the plain ranges beside others: helix angles past 0.5 rad,
    angles that the first updates turn by more than the series cover, infinities
    and NaN, a covariance whose residual determinant is negative."""
    import torch
    params = p2z.physics_params(pt_min=0.05, pt_max=0.6) if what == "low_pt" else None
    cfg = p2z.make_config(bsize=32, nevts=10, ntrks=9600, nlayer=20)
    dt, dh, _ = _device(p2z, ctx, cfg, params=params)
    g = torch.Generator(device="cuda").manual_seed(3)
    some = torch.rand(dt[:, 0].shape, generator=g, device="cuda") < 0.1
    if what == "off_angles":
        for e, s in ((4, 0.05), (5, 0.05)):
            dt[:, e] += some * s * torch.randn(some.shape, generator=g, device="cuda")
        for e in (6 + 14, 6 + 20):
            dt[:, e] = torch.where(some, 2.5e-3, dt[:, e])
    elif what == "nonfinite":
        for e, v in ((0, float("inf")), (3, 0.0), (5, float("nan")), (6 + 9, float("inf")), (6 + 14, float("nan"))):
            dt[e::7, e, e % 5] = v
        dh[::11, 3, 3] = float("inf")
    elif what == "indefinite":
        dt[::5, 6, 2] = -1.0
    stats = _both(p2z, ctx, cfg, dt, dh)
    assert stats[0].singular == (1 if what in ("nonfinite", "indefinite") else 0)


def test_unaligned_arrays_take_the_one_track_kernel(p2z, ctx):
    """Arrays that start 4 bytes past a 16-byte boundary."""
    import torch
    cfg = p2z.make_config(bsize=32, nevts=11, ntrks=9600, nlayer=5)
    dt, dh, _ = _device(p2z, ctx, cfg)

    def shifted(t):
        return torch.empty(t.numel() + 1, device="cuda")[1:].view(t.shape).copy_(t)

    want = torch.empty_like(dt)
    ctx.run_device(cfg, dt, dh, want)
    for t, h, o in ((shifted(dt), dh, want), (dt, shifted(dh), want), (dt, dh, shifted(want))):
        out = torch.empty_like(want) if o is want else o
        ctx.run_device(cfg, t, h, out)
        assert torch.equal(out.view(torch.int32), want.view(torch.int32))


# slots of the last window: 1 to 128 of it
@pytest.mark.parametrize("last", [8, 40, 128])
@pytest.mark.parametrize("update", ["v2", "3x3_f64"])
def test_sorted_by_default(p2z, ctx, last, update):
    counts = np.array([9600] * 12 + [last], dtype=np.int64)
    cfg = p2z.make_config(bsize=8, nevts=len(counts), event_ntrks=counts, nlayer=32, update=update)
    dt, dh, dm = _device(p2z, ctx, cfg, masked=True)
    ctx.mask_layers_device(dm, dm.numel(), 32, min_hits=1, max_hits=32, drop_prob=0.2, seed=5)
    dm[3::97] = 0    # tracks without hits pass through
    dm[5::89] = -1   # and some have every layer
    _both(p2z, ctx, cfg, dt, dh, dm)
