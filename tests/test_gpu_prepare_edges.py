"""p2z_prepare_device against p2z_prepare, word for word, where its CTAs' ranges of
the stream can go wrong: fewer variates than one CTA holds, ranges that end in
the tracks, in the hits or between them, many layers in one range, one layer in
many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bsize,nevts,ntrks,nlayer", [(8, 1, 8, 1), (8, 1, 8, 32), (16, 3, 16, 20), (64, 1, 512, 1),
                                                      (8, 57, 8, 3), (32, 2, 224, 20), (64, 9, 1024, 2)])
@pytest.mark.parametrize("smear", [1e-7, 0.03])
def test_ranges(p2z, ctx, bsize, nevts, ntrks, nlayer, smear):
    import torch
    r = np.random.default_rng(nlayer)
    trk = p2z.make_atrk(r.uniform(-3, 3, 6), r.uniform(0.5, 1.5, 21), -1)
    hit = p2z.make_ahits([(r.uniform(-50, 50, 3), r.uniform(0.5, 1.5, 6)) for _ in range(nlayer)])
    t, h = p2z.prepare(trk, hit, bsize, nevts, ntrks, nlayer, smear=smear, cov_scale=100.0)
    dt = torch.full(t.shape, float("nan"), device="cuda")
    dh = torch.full(h.shape, float("nan"), device="cuda")
    ctx.prepare_device(trk, hit, bsize, nevts, ntrks, nlayer, dt, dh, smear=smear, cov_scale=100.0)
    t2, h2 = dt.cpu().numpy(), dh.cpu().numpy()
    assert np.array_equal(t[:, 27].view(np.uint32), t2[:, 27].view(np.uint32))
    if smear < 1e-3:  # the words hide the last place of the variate's logarithm (see p2z_prepare_device)
        assert np.array_equal(t.view(np.uint32), t2.view(np.uint32))
        assert np.array_equal(h.view(np.uint32), h2.view(np.uint32))
    else:  # one ulp of log moves the variate by one part in 2^23: the word by at most smear*|r| of that, and its own rounding
        for a, b in ((t[:, :27], t2[:, :27]), (h, h2)):
            assert np.abs(a.astype(np.float64) - b).max() <= np.abs(a).max() * (0.03 * 7 * 2.0 ** -22 + 2.0 ** -23)
