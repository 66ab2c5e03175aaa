"""Masked 3-D updates under every launch: flat, sorted and per-event launches take hits through a
ring in shared memory, the queue kernels may not; each track's bits are the same, also where the hits
come from page-locked host memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("update", ["3x3_f64", "3x3_comp"])
@pytest.mark.parametrize("layout", ["b8", "b32", "soa"])
@pytest.mark.parametrize("nlayer", [1, 3, 20])
def test_same_bits(p2z, ctx, update, layout, nlayer):
    import torch
    counts = np.array([300, 0, 65, 1, 2100, 129], dtype=np.int64)
    B = 32 if layout == "soa" else int(layout[1:])
    cfg = p2z.make_config(bsize=B, nevts=len(counts), event_ntrks=counts, nlayer=nlayer, update=update)
    t, h, m = p2z.generate_physics(cfg, with_mask=True)
    p2z.mask_layers(m, nlayer, min_hits=1, max_hits=nlayer, drop_prob=0.3, seed=9)
    m[5::31] = 0
    if layout == "soa":
        t, h = p2z.tracks_to_soa(t), p2z.hits_to_soa(h)
        cfg.layout = p2z.LAYOUT_SOA
    dt, dh, dm = (torch.from_numpy(x).cuda() for x in (t, h, m.view(np.int32)))
    want = torch.empty_like(dt)
    cfg.schedule = p2z.SCHED_NAMES["staged" if layout == "b32" else "per_event"]
    ctx.run_device(cfg, dt, dh, want, d_mask=dm)
    same = lambda a: torch.equal(a.view(torch.int32), want.view(torch.int32))  # noqa: E731
    for schedule, flags, block in (("flat", 0, 0), ("flat", 0, 256), ("flat", p2z.FLAG_SORT_WINDOWS, 0),
                                   ("persistent", 0, 0), ("persistent", 0, 256), ("per_event", 0, 64)):
        cfg.schedule, cfg.flags, cfg.block_threads = p2z.SCHED_NAMES[schedule], flags, block
        out = torch.full_like(dt, float("nan"))
        ctx.run_device(cfg, dt, dh, out, d_mask=dm)
        assert same(out), (schedule, flags, block)
    if layout != "soa":
        out = torch.full_like(dt, float("nan"))
        torch.cuda.synchronize()
        assert p2z.lib.p2z_run_device_noalloc(p2z.C.byref(cfg), dt.data_ptr(), dh.data_ptr(), dm.data_ptr(),
                                              out.data_ptr(), None) == p2z.OK
        torch.cuda.synchronize()
        assert same(out)


@pytest.mark.parametrize("update", ["3x3_f64", "3x3_comp"])
@pytest.mark.parametrize("layout", ["b32", "b64", "soa"])
def test_uneven_events_from_page_locked_memory(p2z, ctx, update, layout):
    import torch
    counts = np.array([1, 0, 700, 33, 4097, 64], dtype=np.int64)
    B = 32 if layout == "soa" else int(layout[1:])
    cfg = p2z.make_config(bsize=B, nevts=len(counts), event_ntrks=counts, nlayer=9, update=update)
    t, h = p2z.generate_physics(cfg)
    if layout == "soa":
        t, h = p2z.tracks_to_soa(t), p2z.hits_to_soa(h)
        cfg.layout = p2z.LAYOUT_SOA
    dt, dh = torch.from_numpy(t).cuda(), torch.from_numpy(h).cuda()
    want = torch.empty_like(dt)
    cfg.schedule = p2z.SCHED_NAMES["persistent"]
    ctx.run_device(cfg, dt, dh, want)
    cfg.schedule = p2z.SCHED_NAMES["auto"]
    pt, ph = (torch.empty(x.shape, pin_memory=True).copy_(x) for x in (dt, dh))
    po = torch.empty(dt.shape, pin_memory=True)
    ctx.run(cfg, pt, ph, po)
    assert torch.equal(po.view(torch.int32), want.cpu().view(torch.int32))
