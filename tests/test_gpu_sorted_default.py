"""The sorted windows that runs with schedule AUTO take for large masked samples: the
same bits as stored order, which a launch per event of the same arrays takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(p2z, ctx, cfg, dt, dh, dm):
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


def _device(p2z, ctx, cfg):
    import torch
    nb, B, nl = p2z.num_batches(cfg), cfg.bsize, cfg.nlayer
    dt = torch.empty((nb, 28, B), device="cuda")
    dh = torch.empty((nb, nl, 9, B), device="cuda")
    dm = torch.empty(nb * B, dtype=torch.int32, device="cuda")
    ctx.generate_physics_device(cfg, dt, dh, dm)
    return dt, dh, dm


# slots of the last window: 1 to 128 of it
@pytest.mark.parametrize("last", [8, 40, 128])
@pytest.mark.parametrize("update", ["v2", "3x3_f64"])
def test_sorted_by_default(p2z, ctx, last, update):
    counts = np.array([9600] * 12 + [last], dtype=np.int64)
    cfg = p2z.make_config(bsize=8, nevts=len(counts), event_ntrks=counts, nlayer=32, update=update)
    dt, dh, dm = _device(p2z, ctx, cfg)
    ctx.mask_layers_device(dm, dm.numel(), 32, min_hits=1, max_hits=32, drop_prob=0.2, seed=5)
    dm[3::97] = 0    # tracks without hits pass through
    dm[5::89] = -1   # and some have every layer
    _both(p2z, ctx, cfg, dt, dh, dm)
