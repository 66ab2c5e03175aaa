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
    assert out == ["none: block 0 schedule 1 tpt 1 sort 0",
                   "padding: block 0 schedule 1 tpt 1 sort 0",
                   "caller, large: block 0 schedule 1 tpt 1 sort 1",
                   "caller, small: block 0 schedule 1 tpt 1 sort 0",
                   "caller, flat asked: block 0 schedule 1 tpt 1 sort 0",
                   "caller, sorting asked: block 64 schedule 3 tpt 2 sort 1",
                   "padding, measured: block 64 schedule 1 tpt 2 sort 0",
                   "caller after padding: block 0 schedule 1 tpt 1 sort 1",
                   "none after padding: block 0 schedule 1 tpt 1 sort 0",
                   "caller, measured: block 256 schedule 1 tpt 1 sort 1",
                   "padding after caller: block 0 schedule 1 tpt 1 sort 0",
                   "none after caller: block 0 schedule 1 tpt 1 sort 0",
                   "caller, again: block 32 schedule 3 tpt 2 sort 0",
                   "caller, staged: block 32 schedule 4 tpt 1 sort 0",
                   "caller, all set: block 128 schedule 1 tpt 1 sort 1"]


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
