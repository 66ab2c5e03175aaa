"""p2z_run_device recorded into the caller's CUDA graph: flat launches carry the programmatic-launch
attribute there too, behind one another, behind launches spread over the context's ten streams and
in front of them; replays give the bits of the direct calls, also on other inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["uniform", "masked", "mixed"])
@pytest.mark.parametrize("niter", [1, 3])
def test_replays(p2z, ctx, form, niter):
    import torch
    counts = np.array([9600, 33, 4000, 700, 1, 5000], dtype=np.int64)
    shape = dict(nevts=3, ntrks=3200) if form == "uniform" else dict(nevts=len(counts), event_ntrks=counts)
    cfg = p2z.make_config(bsize=32, nlayer=6, niter=niter, **shape)
    t, h, m = p2z.generate_physics(cfg, with_mask=True)
    p2z.mask_layers(m, 6, min_hits=1, max_hits=6, drop_prob=0.2, seed=3)
    dt, dh = torch.from_numpy(t).cuda(), torch.from_numpy(h).cuda()
    dm = None if form == "uniform" else torch.from_numpy(m.view(np.int32)).cuda()
    calls = {"uniform": [("flat", 0), ("flat", 0), ("per_event", 0)],
             "masked": [("auto", 0), ("flat", p2z.FLAG_SORT_WINDOWS), ("persistent", 0), ("flat", 0)],
             "mixed": [("flat", 0), ("per_event", p2z.FLAG_PER_EVENT_STREAMS), ("flat", 0), ("per_event", 0),
                       ("per_event", p2z.FLAG_PER_EVENT_STREAMS), ("per_event", p2z.FLAG_PER_EVENT_STREAMS)]}[form]

    def run_all(outs, stream):
        # each pass but the first reads the tracks the one before it wrote
        src = dt
        for (schedule, flags), o in zip(calls, outs):
            cfg.schedule, cfg.flags = p2z.SCHED_NAMES[schedule], flags
            ctx.run_device(cfg, src, dh, o, d_mask=dm, stream=stream, stats=False)
            src = o

    s = torch.cuda.Stream()
    outs = [torch.empty_like(dt) for _ in calls]
    run_all(outs, s)  # (creates the context's ten streams)
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        run_all(outs, s)
    for shift in (0.0, 0.25):
        dt[:, 0] += shift
        want = [torch.empty_like(dt) for _ in calls]
        torch.cuda.synchronize()
        run_all(want, s)
        s.synchronize()
        for o in outs:
            o.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert torch.equal(o.view(torch.int32), w.view(torch.int32))
    del graph
