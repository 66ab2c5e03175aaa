"""p2z_run on page-locked arrays: the pass that reads and writes them over the link
and the copies it stands in for (pageable arrays, wide runs, narrow batches) give the
bits of p2z_run_device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(a, shift=0):
    import torch
    w = torch.empty(a.size + shift, dtype=torch.float32, pin_memory=True)[shift:].view(*a.shape)
    w.numpy().view(np.uint32)[...] = a.view(np.uint32)
    return w


@pytest.mark.parametrize("layout", ["b8", "b32", "b64", "soa"])
@pytest.mark.parametrize("form", ["uniform", "ragged", "in_place", "unaligned", "passes", "3x3", "two_threads"])
def test_same_bits(p2z, ctx, layout, form):
    import torch
    B = 32 if layout == "soa" else int(layout[1:])
    kw = dict(bsize=B, nlayer=7)
    if form == "ragged":
        counts = np.array([1, 0, 700, 33, 4097, 64], dtype=np.int64)
        kw.update(nevts=len(counts), event_ntrks=counts)
    else:
        kw.update(nevts=3, ntrks=1600 * (B // 32 or 1) // B * B)
    if form == "passes":
        kw["niter"] = 3
    if form == "3x3":
        kw["update"] = "3x3_f64"
    if form == "two_threads":
        kw["threads_per_track"] = 2
    cfg = p2z.make_config(**kw)
    t, h = p2z.generate_physics(cfg)
    if layout == "soa":
        t, h = p2z.tracks_to_soa(t), p2z.hits_to_soa(h)
        cfg.layout = p2z.LAYOUT_SOA
    dt, dh = torch.from_numpy(t).cuda(), torch.from_numpy(h).cuda()
    want = torch.empty_like(dt)
    ctx.run_device(cfg, dt, dh, want)
    want = want.cpu().numpy().view(np.uint32)
    shift = 1 if form == "unaligned" else 0
    pt, ph, po = _pinned(t, shift), _pinned(h, shift), _pinned(np.zeros_like(t), shift)
    if form == "in_place":
        po = pt
    st = ctx.run(cfg, pt, ph, po)
    assert np.array_equal(po.numpy().view(np.uint32), want)
    assert st.h2d_bytes > st.d2h_bytes > 0 and st.updates > 0
    out = np.zeros_like(t)
    st2 = ctx.run(cfg, t, h, out)  # pageable: copies
    assert np.array_equal(out.view(np.uint32), want)
    assert (st.h2d_bytes, st.d2h_bytes, st.updates) == (st2.h2d_bytes, st2.d2h_bytes, st2.updates)


@pytest.mark.parametrize("nevts", [44, 46])  # 251 and 262 MB of input: to both sides of the limit
def test_both_sides_of_the_limit(p2z, ctx, nevts):
    import torch
    cfg = p2z.make_config(bsize=32, nevts=nevts, ntrks=9600, nlayer=20)
    nb = p2z.num_batches(cfg)
    dt = torch.empty((nb, 28, 32), device="cuda")
    dh = torch.empty((nb, 20, 9, 32), device="cuda")
    ctx.generate_physics_device(cfg, dt, dh)
    want = torch.empty_like(dt)
    ctx.run_device(cfg, dt, dh, want)
    pt, ph = (torch.empty(x.shape, pin_memory=True).copy_(x) for x in (dt, dh))
    po = torch.empty(dt.shape, pin_memory=True)
    ctx.run(cfg, pt, ph, po)
    assert torch.equal(po.view(torch.int32), want.cpu().view(torch.int32))
