"""The launch shape of a run: the rules for what the caller leaves open, and whose
measurements a run takes."""
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_rules(tmp_path):
    """Measurements of runs without a mask, with uneven events' padding alone and with a caller's
    mask are kept apart; a caller's mask sorts windows from the slot limit on."""
    exe = tmp_path / "shape"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", f"-I{ROOT / 'include'}",
                        f"-I{ROOT / 'p2z-tests_b200' / 'csrc'}", "-o", str(exe),
                        str(ROOT / "tests" / "cpp" / "shape.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout.splitlines()
    assert out == ["none: block 0 schedule 1 tpt 1 sort never",
                   "padding: block 0 schedule 1 tpt 1 sort never",
                   "caller: block 0 schedule 1 tpt 1 sort from 113664",
                   "caller, flat asked: block 0 schedule 1 tpt 1 sort never",
                   "caller, sorting asked: block 64 schedule 3 tpt 2 sort from 0",
                   "caller, auto and sorting asked: block 0 schedule 1 tpt 1 sort from 0",
                   "8: block 0 schedule 1 tpt 1 sort never",
                   "8, sorting asked: block 0 schedule 1 tpt 1 sort from 0",
                   "8, 3-D: block 0 schedule 1 tpt 1 sort from 113664",
                   "16: block 0 schedule 1 tpt 1 sort from 113664",
                   "SoA of 8: block 0 schedule 1 tpt 1 sort from 113664",
                   "padding, measured: block 64 schedule 1 tpt 2 sort never",
                   "caller after padding: block 0 schedule 1 tpt 1 sort from 113664",
                   "none after padding: block 0 schedule 1 tpt 1 sort never",
                   "caller, measured: block 256 schedule 1 tpt 1 sort from 0",
                   "padding after caller: block 0 schedule 1 tpt 1 sort never",
                   "none after caller: block 0 schedule 1 tpt 1 sort never",
                   "caller, again: block 32 schedule 3 tpt 2 sort never",
                   "caller, staged: block 32 schedule 4 tpt 1 sort never",
                   "caller, all set: block 128 schedule 1 tpt 1 sort from 0"]


@pytest.mark.gpu
def test_tuned_without_a_mask_then_run_with_one(p2z):
    """Uneven events tuned without a mask, where one launch per event wins or does not: a run of
    them with a mask is one launch, as in a context that measured nothing."""
    import torch
    counts = np.array([9600] * 12 + [40], dtype=np.int64)
    cfg = p2z.make_config(bsize=32, nevts=len(counts), event_ntrks=counts, nlayer=5)
    t, h, m = p2z.generate_physics(cfg, with_mask=True)
    p2z.mask_layers(m, 5, min_hits=1, max_hits=5, drop_prob=0.2, seed=7)
    dt, dh, dm = (torch.from_numpy(x).cuda() for x in (t, h, m.view(np.int32)))
    want, out = torch.empty_like(dt), torch.empty_like(dt)
    with p2z.Context(0) as c:
        c.run_device(cfg, dt, dh, want, d_mask=dm)
        c.autotune(cfg, dt, dh, reps=1)
        st = c.run_device(cfg, dt, dh, out, d_mask=dm)
        assert st.launches == 1
        assert torch.equal(out.view(torch.int32), want.view(torch.int32))


def _masked(p2z, ctx, B, nslots, nlayer=4):
    """A masked sample of nslots slots (a multiple of B) in events of up to 9600 tracks, some without hits."""
    import torch
    counts = np.array([9600] * (nslots // 9600) + ([nslots % 9600] if nslots % 9600 else []), dtype=np.int64)
    cfg = p2z.make_config(bsize=B, nevts=len(counts), event_ntrks=counts, nlayer=nlayer)
    nb = p2z.num_batches(cfg)
    assert nb * B == nslots
    dt = torch.empty((nb, 28, B), device="cuda")
    dh = torch.empty((nb, nlayer, 9, B), device="cuda")
    dm = torch.empty(nslots, dtype=torch.int32, device="cuda")
    ctx.generate_physics_device(cfg, dt, dh, dm)
    ctx.mask_layers_device(dm, nslots, nlayer, min_hits=1, max_hits=nlayer, drop_prob=0.2, seed=5)
    dm[3::97] = 0
    return cfg, dt, dh, dm


@pytest.mark.gpu
@pytest.mark.parametrize("B", [8, 32, 64])
@pytest.mark.parametrize("past", [-64, 0, 64])
def test_bits_around_the_limit(p2z, ctx, B, past):
    """Runs just below, at and above the slots from which windows are sorted: the bits of stored order."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cfg, dt, dh, dm = _masked(p2z, ctx, B, 768 * sms + past)
    want, out = torch.empty_like(dt), torch.full_like(dt, float("nan"))
    for o, schedule, flags in ((want, "per_event", 0), (out, "auto", 0), (torch.full_like(dt, float("nan")), "flat", 0x80)):
        cfg.schedule, cfg.flags = p2z.SCHED_NAMES[schedule], flags
        ctx.run_device(cfg, dt, dh, o, d_mask=dm)
        assert torch.equal(o.view(torch.int32), want.view(torch.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [False, True])
def test_chunks_on_both_sides_of_the_limit(p2z, ctx, pinned):
    """p2z_run on 420,000 masked slots: the first chunk sorts its windows, the later ones do not."""
    import torch
    cfg, dt, dh, dm = _masked(p2z, ctx, 32, 420_000)
    want = torch.empty_like(dt)
    cfg.schedule = p2z.SCHED_NAMES["per_event"]
    ctx.run_device(cfg, dt, dh, want, d_mask=dm)
    cfg.schedule = p2z.SCHED_NAMES["auto"]
    t, h, m = (torch.empty(x.shape, dtype=x.dtype, pin_memory=pinned).copy_(x) for x in (dt, dh, dm))
    out = torch.empty(dt.shape, pin_memory=pinned)
    ctx.run(cfg, t, h, out, hit_mask=m)
    assert torch.equal(out.view(torch.int32), want.cpu().view(torch.int32))


@pytest.mark.gpu
def test_autotune_measures_a_sorted_launch_once(p2z, ctx):
    """Sorted windows are one flat launch under either schedule: both rows of the sweep give one
    figure, and the fastest row names the flat one."""
    cfg, dt, dh, dm = _masked(p2z, ctx, 32, 6400)
    with p2z.Context(0) as c:
        best, rows = c.autotune(cfg, dt, dh, d_mask=dm, reps=1)
    key = lambda r: (r["bsize"], r["layout"], r["threads_per_track"], r["block_threads"])  # noqa: E731
    flat, queue = ({key(r): r["ms"] for r in rows if r["schedule"] == s and r["sorted_windows"]}
                   for s in ("flat", "persistent"))
    assert len(flat) == 4 * 2 * 2 * 4 and flat == queue
    assert not (best["schedule"] == "persistent" and best["sorted_windows"])
