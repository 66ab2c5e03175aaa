"""p2z_run's kernel reads and writes page-locked arrays itself only where that
cannot fault and no input shares a byte with the output: the rule on made-up
page-locked ranges, and calls on each side of it through the library."""
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_rule(tmp_path):
    exe = tmp_path / "direct"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", f"-I{ROOT / 'p2z-tests_b200' / 'csrc'}", "-o",
                        str(exe), str(ROOT / "tests" / "cpp" / "direct.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout.splitlines()
    assert out == ["whole 0x910000", "inside 0x910404", "last_byte_past 0", "first_byte_before 0", "pageable 0",
                   "off_a_word 0", "off_a_word 0", "off_a_word 0", "empty 0", "wraps 0", "not_mapped 0",
                   "two_pieces 0x910004", "hole_between 0", "device_gap 0", "most_pieces 0x910000",
                   "too_many_pieces 0", "same 0x3", "apart 0", "by_one 0x3", "within 0x3"]


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["aosoa", "soa"])
@pytest.mark.parametrize("form", ["bytes_1", "bytes_2", "bytes_3", "in_place", "out_over_tracks", "out_over_hits"])
def test_same_bits(p2z, ctx, form, layout):
    """Arrays off a word's boundary and outputs that overlap an input (one chunk: the
    copies bring every input in before the output goes back)."""
    import torch
    cfg = p2z.make_config(bsize=32, nevts=1, ntrks=96 * 32, nlayer=5)
    t, h = p2z.generate_physics(cfg)
    if layout == "soa":
        t, h = p2z.tracks_to_soa(t), p2z.hits_to_soa(h)
        cfg.layout = p2z.LAYOUT_SOA
    dt, dh = torch.from_numpy(t).cuda(), torch.from_numpy(h).cuda()
    want = torch.empty_like(dt)
    ctx.run_device(cfg, dt, dh, want)
    shift = int(form[6:]) if form.startswith("bytes") else 0
    at_t = shift
    at_h = at_t + t.nbytes + 4
    at_o = at_h + h.nbytes + 4
    if form == "in_place":
        at_o = at_t
    elif form == "out_over_tracks":
        at_h, at_o = at_h + t.nbytes, at_t + t.nbytes // 2 // 4 * 4
    elif form == "out_over_hits":
        at_o = at_h + h.nbytes // 3 // 4 * 4
    room = p2z.PinnedArray((at_o + at_h + t.nbytes + h.nbytes,), np.uint8)
    buf = room.array
    buf[at_t:at_t + t.nbytes] = t.view(np.uint8).reshape(-1)
    buf[at_h:at_h + h.nbytes] = h.view(np.uint8).reshape(-1)
    base = buf.ctypes.data
    rc = p2z.lib.p2z_run(ctx.h, p2z.C.byref(cfg), base + at_t, base + at_h, None, base + at_o, None)
    assert rc == p2z.OK
    assert np.array_equal(buf[at_o:at_o + t.nbytes], want.cpu().numpy().view(np.uint8).reshape(-1))
