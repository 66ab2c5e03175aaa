"""The reference-rounding form's sin and cos (one shared reduction, series in
double) against the oracle's restatement with correctly rounded sin and cos, bit
for bit, where the reduction can go wrong: multiples of pi/2, zeros of either
sign, both sides of the limit past which CUDA's own functions take over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phi", ["quarter_turns", "zeros", "below_limit", "past_limit", "huge"])
def test_angles(p2z, oracle, ctx, phi):
    cfg = p2z.make_config(bsize=32, nevts=1, ntrks=256, nlayer=3, flags=p2z.FLAG_REFERENCE_ROUNDING)
    trk, hit = p2z.generate_physics(cfg)
    r = np.random.default_rng(11)
    shape = trk[:, 4].shape
    trk[:, 4] = {
        "quarter_turns": lambda: np.float32(np.pi / 2) * r.integers(-40, 41, shape).astype(np.float32),
        "zeros": lambda: np.where(r.random(shape) < 0.5, np.float32(0.0), np.float32(-0.0)),
        "below_limit": lambda: r.uniform(9e4, 99999.0, shape).astype(np.float32),
        "past_limit": lambda: -r.uniform(100001.0, 2e5, shape).astype(np.float32),
        "huge": lambda: r.uniform(1e7, 1e9, shape).astype(np.float32),
    }[phi]()
    if phi == "zeros":  # and no step in z on the first layer: a zero helix angle of either sign
        trk[:, 2] = hit[:, 0, 2]
    out = np.empty_like(trk)
    ctx.run(cfg, trk, hit, out)
    want = oracle.run_f32(trk, hit, cr_trig=True)
    assert np.isfinite(want[:, :27]).all()
    assert np.array_equal(out.view(np.uint32), want.view(np.uint32))
