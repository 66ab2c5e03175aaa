"""Measured cases of the propagate-to-z + Kalman-update library, through its public entry points.

A case is one call as a user's program makes it: tracks and hits are at hand (on the device, or in
page-locked host memory for the host entry point), one context serves the whole process, output and
work buffers are allocated once.  Inputs are drawn from the physics distribution the benchmark runs:
pT log-uniform 0.5-20 GeV, phi uniform, eta 1.6-2.5, a correlated covariance around the true state,
and hits on planes between z = 30 and 270 cm at the true helix point plus 30 um / 1 um noise.
"""
import importlib.util
import math
import pathlib
import random
import sys

import numpy as np
import torch

KFACT = float(np.float32(100.0 / (-0.299792458 * 3.8112)))
SCRATCH = {}  # the process's context


def _p2z():
    name = "p2z_b200"
    if name not in sys.modules:
        pkg = pathlib.Path("p2z-tests_b200").resolve()
        spec = importlib.util.spec_from_file_location(name, pkg / "__init__.py", submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _context():
    if "ctx" not in SCRATCH:
        SCRATCH["ctx"] = _p2z().Context(0)
    return SCRATCH["ctx"]


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------

def _case(kind, nevts, ntrks, nlayer=20, bsize=32, update="v2", **more):
    """kind: "uniform" (nevts events of ntrks tracks), "ragged" (event sizes from ntrks_min to ntrks, every
    track with all layers), "masked" (the same with missing layers), "packed" (masked, packed by hit count
    first), "host" (uniform, from host memory), "prepare" (the reference's input preparation)."""
    c = {"kind": kind, "nevts": nevts, "ntrks": ntrks, "nlayer": nlayer, "bsize": bsize, "update": update,
         "layout": "aosoa", "flags": 0, "ntrks_min": ntrks}
    c.update(more)
    return c


REFERENCE_ROUNDING = 0x20


def listed():
    return [
        # one small event, as an online caller hands them over: latency and launches
        dict(_case("uniform", 1, 1024), name="event_1k"),
        # one event of the reference's size
        dict(_case("uniform", 1, 9600), name="event_9600"),
        # the reference's default run: 100 events of 9600 tracks
        dict(_case("uniform", 100, 9600), name="events_100"),
        # the benchmark's sample
        dict(_case("uniform", 1000, 9600), name="events_1000"),
        # uneven events whose tracks miss layers (5-20 hits each), as reconstruction meets them
        dict(_case("masked", 500, 20011, ntrks_min=1003), name="masked_500"),
        # events of odd sizes, every layer present, another detector and batch width
        dict(_case("ragged", 61, 20011, nlayer=13, bsize=16, ntrks_min=251), name="ragged_61"),
        # a serving group: uneven events through the 3-D update with its double-precision inversion
        dict(_case("masked", 60, 20011, update="3x3_f64", ntrks_min=1003), name="masked_3x3"),
        # the reference's own rounding, for callers who compare with its printed results
        dict(_case("uniform", 10, 9600, flags=REFERENCE_ROUNDING), name="reference_rounding"),
        # one array per element instead of batches
        dict(_case("uniform", 64, 4096, layout="soa"), name="soa_64"),
        # masked events whose caller packs them by hit count, runs, and wants its own order back
        dict(_case("packed", 500, 20011, ntrks_min=1003), name="packed_500"),
        # the reference's prepareTracks and prepareHits, on the device
        dict(_case("prepare", 10, 9600), name="prepare_10"),
        # a whole pass from page-locked host memory
        dict(_case("host", 16, 9600), name="host_16"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["uniform"] * 4 + ["masked"] * 3 + ["ragged", "packed", "prepare", "host"])
    bsize = rng.choice([8, 16, 32, 32, 64])
    nlayer = rng.randint(5, 32)
    update, flags, layout = "v2", 0, "aosoa"
    most = 9.6e6 * min(20 / nlayer, 704 / (224 + 24 * nlayer))  # tracks: neither more updates nor more bytes than the largest listed
    if kind in ("uniform", "masked"):
        update = rng.choice(["v2"] * 4 + ["3x3_f64"])
        if update == "v2" and kind == "uniform":
            flags = rng.choice([0, 0, 0, REFERENCE_ROUNDING])
            layout = rng.choice(["aosoa", "aosoa", "soa"])
        most = most / 10 if update != "v2" or flags else most
    if kind == "packed":
        most /= 3
    if kind in ("prepare", "host"):
        most = 1.5e5 * min(1, 20 / nlayer)
    total = _log(rng, 1024, most)
    if kind in ("masked", "ragged", "packed"):
        hi = min(20011, max(600, int(total)))
        lo = rng.randint(100, 500)
        nevts = max(1, int(total / ((hi - lo) / math.log(hi / lo))))
        return _case(kind, nevts, hi, nlayer, bsize, update, ntrks_min=lo, layout=layout, flags=flags)
    ntrks = int(_log(rng, min(256, total), min(20000, total)))
    ntrks = max(1, ntrks // bsize) * bsize
    return _case(kind, max(1, int(total / ntrks)), ntrks, nlayer, bsize, update, layout=layout, flags=flags)


def _counts(case):
    """Tracks per event.  Uneven events: spread over the logarithm of [ntrks_min, ntrks], in mixed order."""
    n = case["nevts"]
    if case["kind"] not in ("ragged", "masked", "packed"):
        return [case["ntrks"]] * n
    lo, hi = case["ntrks_min"], case["ntrks"]
    counts = [int(round(lo * (hi / lo) ** ((i + 0.5) / n))) for i in range(n)]
    random.Random(n).shuffle(counts)
    return counts


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

SYM = [(i, j) for i in range(6) for j in range(i + 1)]  # packed lower triangle


def _generator(seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _present(case, counts, g, device):
    """Per slot the layers with a hit, as bits (int32); 0 for the padding slots at an event's end."""
    B, nl = case["bsize"], case["nlayer"]
    n = torch.tensor(counts, device=device)
    room = (n + B - 1) // B * B
    first = torch.cumsum(room, 0) - room
    ns = int(room.sum())
    slot = torch.arange(ns, device=device)
    event = torch.repeat_interleave(torch.arange(len(counts), device=device), room, output_size=ns)
    real = slot - first[event] < n[event]
    if case["kind"] == "ragged":
        m = torch.full((ns,), (1 << nl) - 1, dtype=torch.int64, device=device)
    else:
        # a run of layers from the first on, at least a quarter of them, one in ten of them missing
        least = max(1, nl // 4)
        length = torch.randint(least, nl + 1, (ns,), generator=g, device=device)
        m = torch.zeros(ns, dtype=torch.int64, device=device)
        for l in range(nl):
            has = (l < length) & ((l < least) | (torch.rand(ns, generator=g, device=device) >= 0.1))
            m |= has.to(torch.int64) << l
    m = torch.where(real, m, torch.zeros_like(m))
    return torch.where(m >= 2 ** 31, m - 2 ** 32, m).to(torch.int32)


def _inputs(case, seed, device):
    """(tracks, hits, mask) in the case's layout: AOSOA (nbatches, 28, B) and (nbatches, nlayer, 9, B), or SoA
    (28, slots) and (nlayer, 9, slots); the charge is an int32 in the tracks' last word."""
    B, nl = case["bsize"], case["nlayer"]
    g = _generator(seed, device)
    counts = _counts(case)
    nb = sum((n + B - 1) // B for n in counts)
    ns = nb * B
    soa = case["layout"] == "soa"
    trk = torch.empty((28, ns) if soa else (nb, 28, B), dtype=torch.float32, device=device)
    hits = torch.empty((nl, 9, ns) if soa else (nb, nl, 9, B), dtype=torch.float32, device=device)
    mask = _present(case, counts, g, device) if case["kind"] in ("ragged", "masked", "packed") else None

    def put(e, v):
        if soa:
            trk[e] = v
        else:
            trk[:, e] = v.view(nb, B)

    def put_hit(l, e, v):
        if soa:
            hits[l, e] = v
        else:
            hits[:, l, e] = v.view(nb, B) if torch.is_tensor(v) else v

    def uniform(lo, hi):
        return lo + (hi - lo) * torch.rand(ns, generator=g, device=device, dtype=torch.float64)

    def normal():
        return torch.randn(ns, generator=g, device=device, dtype=torch.float64)

    q = torch.where(uniform(0, 1) < 0.5, -1.0, 1.0).double()
    ipt = torch.exp(-uniform(math.log(0.5), math.log(20.0)))
    phi = uniform(-math.pi, math.pi)
    theta = 2.0 * torch.atan(torch.exp(-uniform(1.6, 2.5)))
    vz = 5.0 * normal()
    # covariance D L L^T D, L a unit-row lower triangle near the identity
    low = [[None] * 6 for _ in range(6)]
    for i in range(6):
        row = [uniform(-0.2, 0.2) for _ in range(i)] + [torch.ones_like(q)]
        norm = torch.sqrt(sum(v * v for v in row))
        for j, v in enumerate(row):
            low[i][j] = v / norm
    sigma = [0.01, 0.01, 0.05, 0.01 * ipt, 1e-3, 1e-3]
    noise = [normal() for _ in range(6)]
    truth = [torch.zeros_like(q), torch.zeros_like(q), vz, ipt, phi, theta]
    for i in range(6):
        put(i, truth[i] + sigma[i] * sum(low[i][j] * noise[j] for j in range(i + 1)))
    for e, (i, j) in enumerate(SYM):
        put(6 + e, sigma[i] * sigma[j] * sum(low[i][k] * low[j][k] for k in range(j + 1)))
    put(27, q.to(torch.int32).view(torch.float32))
    del low, noise
    k = q * KFACT
    cp, sp, tan = torch.cos(phi), torch.sin(phi), torch.tan(theta)
    for l in range(nl):
        z = 30.0 + 240.0 * l / max(1, nl - 1)
        alpha = (z - vz) * tan * ipt / k
        sa, va = torch.sin(alpha), 2.0 * torch.sin(0.5 * alpha) ** 2
        put_hit(l, 0, k / ipt * (cp * sa - sp * va) + 30e-4 * normal())
        put_hit(l, 1, k / ipt * (sp * sa + cp * va) + 30e-4 * normal())
        put_hit(l, 2, z + 1e-4 * normal())
        put_hit(l, 3, 9e-6)
        put_hit(l, 4, 9e-6 * uniform(-0.2, 0.2))
        put_hit(l, 5, 9e-6)
        put_hit(l, 6, 3e-7 * uniform(-0.2, 0.2))
        put_hit(l, 7, 3e-7 * uniform(-0.2, 0.2))
        put_hit(l, 8, 1e-8)
    if mask is not None:  # padding slots hold zeros
        pad = mask == 0
        trk.masked_fill_(pad.view(nb, 1, B), 0.0)
        hits.masked_fill_(pad.view(nb, 1, 1, B), 0.0)
    return trk, hits, mask


def _seed_words(case, seed):
    """One seed track and a hit per layer, as the reference's programs hold them in their source."""
    r = np.random.default_rng(seed)
    track = ([-12.8, -7.7, 38.2, 0.23 * r.uniform(0.9, 1.1), -2.61, 0.35],
             [float(v) for v in 1e-4 * r.uniform(0.5, 1.5, 21)], 1)
    hits = [([float(v) for v in r.uniform(-60, 60, 2)] + [30.0 + 12.0 * l], [float(v) for v in 1e-5 * r.uniform(0.5, 1.5, 6)])
            for l in range(case["nlayer"])]
    return track, hits


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def _views(out, case):
    """The output tracks by quantity: positions, 1/pT, phi, theta, the covariance's rows and the charge."""
    e = out if case["layout"] == "soa" else out.transpose(0, 1)
    return {"xy": e[0:2], "z": e[2], "ipt": e[3], "phi": e[4], "theta": e[5], "cov_xy": e[6:9], "cov_z": e[9:12],
            "cov_ipt": e[12:16], "cov_phi": e[16:21], "cov_theta": e[21:27], "charge": e[27]}


def prepare(case, seed):
    p2z, ctx = _p2z(), _context()
    s = {"kind": case["kind"], "ctx": ctx}
    if case["kind"] == "prepare":
        track, hits = _seed_words(case, seed)
        nb = case["nevts"] * (case["ntrks"] // case["bsize"])
        s["args"] = (p2z.make_atrk(*track), p2z.make_ahits(hits), case["bsize"], case["nevts"], case["ntrks"], case["nlayer"])
        trk = torch.empty((nb, 28, case["bsize"]), dtype=torch.float32, device="cuda")
        hit = torch.empty((nb, case["nlayer"], 9, case["bsize"]), dtype=torch.float32, device="cuda")
        s["trk"], s["hits"] = trk, hit
        s["outputs"] = {"par": trk[:, :6], "cov": trk[:, 6:27], "charge": trk[:, 27].view(torch.int32), "hits": hit}
        return s
    counts = _counts(case)
    uneven = case["kind"] in ("ragged", "masked", "packed")
    s["cfg"] = p2z.make_config(bsize=case["bsize"], nevts=case["nevts"], ntrks=None if uneven else case["ntrks"],
                               nlayer=case["nlayer"], update=case["update"], flags=case["flags"], layout=case["layout"],
                               event_ntrks=np.array(counts, dtype=np.int64) if uneven else None)
    trk, hits, mask = _inputs(case, seed, "cuda")
    if case["kind"] == "ragged":
        mask = None  # every layer present: the event sizes say all
    if case["kind"] == "host":
        trk, hits = (torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for t in (trk, hits))
        out = torch.empty(trk.shape, dtype=trk.dtype, pin_memory=True)
    else:
        out = torch.empty_like(trk)
    s.update(trk=trk, hits=hits, mask=mask, out=out, outputs=_views(out, case))
    s["outputs"]["charge"] = s["outputs"]["charge"].view(torch.int32)
    if case["kind"] == "packed":
        s["perm"] = torch.empty(2 * mask.numel(), dtype=torch.int64, device="cuda")
        s["packed"] = (torch.empty_like(trk), torch.empty_like(hits), torch.empty_like(mask), torch.empty_like(trk))
        s["outputs"] = dict(s["outputs"], perm=s["perm"])
    return s


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "prepare":
        ctx.prepare_device(*s["args"], s["trk"], s["hits"])
    elif kind == "host":
        ctx.run(s["cfg"], s["trk"], s["hits"], s["out"])
    elif kind == "packed":
        trk, hits, mask, out = s["packed"]
        ctx.pack_by_hits_device(s["cfg"], s["trk"], s["hits"], trk, hits, s["perm"], d_mask_in=s["mask"], d_mask_out=mask)
        ctx.run_device(s["cfg"], trk, hits, out, d_mask=mask, stats=False)
        ctx.unpack_tracks_device(s["cfg"], s["perm"], out, s["out"])
    else:
        ctx.run_device(s["cfg"], s["trk"], s["hits"], s["out"], d_mask=s["mask"], stats=False)
    return s["outputs"]


def work(case):
    """One read of each input word the pass needs, one write of each output word; floating-point operations of the
    update in its reduced form (349 for a propagation and a 2-D update, 227 and 374 with the 3-D update)."""
    B, nl, counts = case["bsize"], case["nlayer"], _counts(case)
    ns = sum((n + B - 1) // B * B for n in counts)
    tracks = sum(counts)
    if case["kind"] == "prepare":
        return {"bytes": 4.0 * tracks * (28 + 9 * nl), "flops": 20.0 * tracks * (27 + 9 * nl)}
    layers = float(nl)
    if case["kind"] in ("masked", "packed"):
        least = max(1, nl // 4)  # mean of the mask's distribution
        layers = sum(least + 0.9 * (n - least) for n in range(least, nl + 1)) / (nl + 1 - least)
    hit_words, flops = (9, 601) if case["update"].startswith("3x3") else (6, 349)
    moved = 4.0 * (2 * 28 * ns + hit_words * layers * tracks + (ns if case["kind"] in ("masked", "packed") else 0))
    if case["kind"] == "packed":  # the packed copy: every word read and written once more, the permutation twice
        moved += 4.0 * (2 * 28 * ns + 2 * 9 * nl * ns + 2 * ns + 2 * 28 * ns) + 8.0 * 4 * ns
    return {"bytes": moved, "flops": flops * layers * tracks}


# ---------------------------------------------------------------------------
# The same in double precision
# ---------------------------------------------------------------------------

def _propagate_and_update(par, C, k, hit, three):
    """One layer for n tracks: par (n, 6), C (n, 6, 6), k (n,), hit (n, 9)."""
    n = par.shape[0]
    x, y, z, ipt, phi, theta = par.unbind(1)
    dz, pt = hit[:, 2] - z, 1.0 / ipt
    cp, sp, st, ct = torch.cos(phi), torch.sin(phi), torch.sin(theta), torch.cos(theta)
    alpha = dz * st * ipt / (ct * k)
    sa, ca, va = torch.sin(alpha), torch.cos(alpha), 2.0 * torch.sin(0.5 * alpha) ** 2
    sc, vc = torch.sin(cp * sa), 2.0 * torch.sin(0.5 * cp * sa) ** 2
    J = torch.zeros(n, 6, 6, dtype=par.dtype, device=par.device)
    for i in (0, 1, 3, 4, 5):
        J[:, i, i] = 1.0
    J[:, 0, 2] = cp * st * (sp * ca * sc - ca) / ct
    J[:, 0, 3] = cp * st * dz * ca * (1.0 - sp * sc) * pt / ct - k * (cp * sa - sp * vc) * pt * pt
    J[:, 0, 4] = k * pt * (-sp * sa + sp * sp * sa * sc - cp * vc)
    J[:, 0, 5] = cp * dz * ca * (1.0 - sp * sc) / ct ** 2
    J[:, 1, 2] = ca * st * (cp * cp * sc - sp) / ct
    J[:, 1, 3] = st * dz * ca * (cp * cp * sc + sp) * pt / ct - k * (sp * sa + cp * vc) * pt * pt
    J[:, 1, 4] = k * pt * (-sp * vc - sp * cp * sa * sc + cp * sa)
    J[:, 1, 5] = dz * ca * (cp * cp * sc + sp) / ct ** 2
    J[:, 4, 2] = -ipt * st / (ct * k)
    J[:, 4, 3] = st * dz / (ct * k)
    J[:, 4, 5] = ipt * dz / (ct * ct * k)
    new = torch.stack([x + k * pt * (cp * sa - sp * va), y + k * pt * (sp * sa + cp * va), hit[:, 2], ipt, phi + alpha, theta], 1)
    C = J @ C @ J.transpose(1, 2)
    d = 3 if three else 2
    V = torch.empty(n, d, d, dtype=par.dtype, device=par.device)
    for i in range(d):
        for j in range(i + 1):
            V[:, i, j] = V[:, j, i] = hit[:, 3 + i * (i + 1) // 2 + j]
    K = torch.linalg.solve(C[:, :d, :d] + V, C[:, :d, :]).transpose(1, 2)
    new = new + (K @ (hit[:, :d] - new[:, :d]).unsqueeze(2)).squeeze(2)
    return new, C - K @ C[:, :d, :]


def exact(case, seed):
    if case["kind"] == "prepare":
        return None  # the C library's rand() stream is sequential: minutes in plain code, and the words are exact
    device = "cuda" if torch.cuda.is_available() else "cpu"
    trk, hits, mask = _inputs(case, seed, device)
    soa, nl, B = case["layout"] == "soa", case["nlayer"], case["bsize"]
    nb = trk.shape[1] // B if soa else trk.shape[0]
    out = torch.empty(trk.shape, dtype=torch.float64, device=device)
    step = max(1, (1 << 18) // B)
    for b in range(0, nb, step):
        at = slice(b * B, min(nb, b + step) * B)
        if soa:
            w, h = trk[:, at].T, hits[:, :, at].permute(2, 0, 1)
        else:
            w = trk[b:b + step].transpose(1, 2).reshape(-1, 28)
            h = hits[b:b + step].permute(0, 3, 1, 2).reshape(-1, nl, 9)
        m = None if mask is None else mask[at].to(torch.int64)
        k = w[:, 27].contiguous().view(torch.int32).double() * KFACT
        par, C = w[:, :6].double(), torch.empty(w.shape[0], 6, 6, dtype=torch.float64, device=device)
        for e, (i, j) in enumerate(SYM):
            C[:, i, j] = C[:, j, i] = w[:, 6 + e].double()
        for l in range(nl):
            on = slice(None) if m is None else ((m >> l) & 1).nonzero()[:, 0]
            par[on], C[on] = _propagate_and_update(par[on], C[on], k[on], h[on, l].double(), case["update"].startswith("3x3"))
        o = torch.cat([par] + [C[:, i, j].unsqueeze(1) for i, j in SYM] + [k.unsqueeze(1)], 1)
        if soa:
            out[:, at] = o.T
        else:
            out[b:b + step] = o.view(-1, B, 28).transpose(1, 2)
    return dict(_views(out, case), charge=None, **({"perm": None} if case["kind"] == "packed" else {}))
