"""The variates themselves that p2z_prepare_device draws: with a smearing factor so large that a word
is its variate times a power of two, against the polar method in numpy with the logarithm
rounded once from double, bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_every_bit(p2z, ctx):
    import torch
    n = 9600
    need = n * 27 // 2  # accepted attempts, two variates each
    state = ctypes.create_string_buffer(256)
    p2z.lib.p2z_ref_rng_seed(state, 1)
    draws = int(2 * need / (np.pi / 4) * 1.02) // 2 * 2
    rand = p2z.lib.p2z_ref_rng_rand
    d = np.array([rand(state) for _ in range(draws)], dtype=np.int32).reshape(-1, 2)
    f32 = np.float32
    u = f32(-1) + (d.astype(f32) / f32(2147483648.0)) * f32(2)
    w = (u.astype(np.float64) ** 2).sum(1).astype(f32)
    ok = (w < 1) & (w != 0)
    assert ok.sum() >= need
    u, w = u[ok][:need], w[ok][:need]
    mult = np.sqrt((f32(-2) * np.log(w.astype(np.float64)).astype(f32)) / w)
    want = (u * mult[:, None]).reshape(n, 27) * f32(2.0 ** 60)
    trk = p2z.make_atrk([1.0] * 6, [1.0] * 21, 1)
    hit = p2z.make_ahits([([1.0] * 3, [1.0] * 6)])
    dt = torch.empty((n // 32, 28, 32), device="cuda")
    dh = torch.empty((n // 32, 1, 9, 32), device="cuda")
    ctx.prepare_device(trk, hit, 32, 1, n, 1, dt, dh, smear=2.0 ** 60, cov_scale=1.0)
    got = dt.cpu().numpy()[:, :27].transpose(0, 2, 1).reshape(n, 27)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
