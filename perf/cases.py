"""The work a user of this library has it do, as timed cases over its public entry points.

Every case runs synthetic helices through one entry point: the fused forward, the reference's
per-layer call shape, the host-buffer pipeline, the work queue for uneven batches, and the adjoint
(direct, through torch autograd, and over the queue). Truth is in FP64, hits are smeared by 10 um,
seeds by their covariance and kept within two sigma of it, |eta| < 1 as barrel cylinders see them.
`listed()` names the cases, `draw()` gives more of the same ranges, `prepare()` makes
what a caller has in hand, `run()` is one pass, `work()` its necessary bytes and operations,
`exact()` the same results in 64-bit torch, from the formulas alone.
"""
import math

import numpy as np
import torch

import p2r_tests_b200 as p2r

FLOP_PER_UPDATE = 1272  # one propagateToR + KalmanUpdate of one track at one layer (FMA = 2)


# ------------------------------------------------------------------ the cases
def _case(kind, bsize=32, nb=1, nevts=1, nlayer=20, bz=3.8, **more):
    c = {"kind": kind, "bsize": bsize, "nb": nb, "nevts": nevts, "nlayer": nlayer, "bz": bz, "pt": 4.0, "r_first": 20.0,
         "r_last": 100.0, "chi2": False, "dr": False, "squash": False, "ordered": False, "lay_lo": 0, "layout": 1}
    c.update(more)
    return c


def listed():
    return [
        # a handful of seeds refitted on their own, chi2 wanted: latency and the launch
        _case("forward", nb=8, chi2=True, name="forward_256"),
        # one event as it arrives: 9600 tracks do not fill the chip
        _case("forward", nb=300, name="forward_event"),
        # the headline batch: 9600 tracks x 100 events x 20 layers
        _case("forward", nb=300, nevts=100, name="forward_full"),
        # a caller with its own block width and layer count, alignment offsets, chi2 and wrapped phi
        _case("forward", bsize=20, nb=331, nevts=13, nlayer=17, bz=3.8112, chi2=True, dr=True, squash=True,
              name="forward_ragged"),
        # the reference's stock loop (every layer restarts from the input track)
        _case("restart", nb=300, nevts=100, name="restart_full"),
        # the reference's per-layer call shape, 9600 tracks x 10 events x 20 layers
        _case("layers", nb=300, nevts=10, name="layers_10ev"),
        # the same batch from pinned host buffers and back
        _case("host", nb=300, nevts=10, name="host_10ev"),
        # 40-layer calibration sample: 20 to 40 layers per track, radius offsets, chi2
        _case("masked", nb=3125, nevts=10, nlayer=40, r_first=4.0, r_last=110.0, lay_lo=20, chi2=True, dr=True,
              ordered=True, name="masked_40_layers"),
        # uneven events (log-normal, median 2000 tracks, 10 to 25 layers) as one captured queue launch
        _case("queue", bsize=64, nevts=1000, nlayer=25, lay_lo=10, ordered=True, name="queue_uneven"),
        # forward + adjoint of the headline batch, gradients per event
        _case("adjoint", nb=300, nevts=100, dr=True, name="adjoint_full"),
        # one event's differentiable fit step through torch autograd
        _case("autograd", nb=300, dr=True, name="autograd_event"),
        # per-event calibration gradients of an uneven 40-layer batch in one captured queue launch
        _case("queue_adjoint", nb=125, nevts=100, nlayer=40, r_first=4.0, r_last=110.0, lay_lo=20, dr=True, ordered=True,
              name="queue_adjoint_40_layers"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "restart", "layers", "host", "masked", "queue", "adjoint", "adjoint",
                       "autograd", "queue_adjoint"])
    # tracks in all, log-uniform up to the largest listed batch of that path
    most = {"forward": 960000, "restart": 960000, "layers": 96000, "host": 96000, "masked": 400000, "queue": 1000000,
            "adjoint": 900000, "autograd": 96000, "queue_adjoint": 300000}[kind]
    ntrk = _log(rng, 256, most)
    queue = kind in ("queue", "queue_adjoint")
    bsize = rng.choice([32, 64, 128] if queue or kind == "masked" else [32, 32, 64, 128, rng.randint(1, 100)])
    nevts = min(_log(rng, 1, 200), max(1, ntrk // (64 if queue else bsize)))
    nb = max(1, round(ntrk / nevts / bsize))
    nlayer = rng.randint(10, 40) if kind in ("masked", "queue_adjoint") else rng.randint(8, 25)
    if kind in ("adjoint", "autograd", "queue_adjoint"):
        nlayer = min(nlayer, max(8, int(1.8e7 / max(1, nb * nevts * bsize))))
    if kind in ("adjoint", "autograd"):
        bsize = 32 * max(1, bsize // 32)  # per-event gradients need whole warps
        nb = max(1, round(ntrk / nevts / bsize))
    lay_lo = max(1, nlayer // 2) if kind in ("masked", "queue", "queue_adjoint") else 0
    chained = kind in ("forward", "masked")
    return _case(kind, bsize=bsize, nb=nb, nevts=nevts, nlayer=nlayer, bz=rng.choice([3.8, 3.8112, 3.0]),
                 pt=round(rng.uniform(2.0, 8.0), 3), chi2=kind in ("forward", "restart", "masked", "queue") and rng.random() < 0.5,
                 dr=(chained or kind in ("adjoint", "autograd", "queue_adjoint")) and rng.random() < 0.5,
                 squash=kind == "forward" and rng.random() < 0.25, ordered=lay_lo > 0 and rng.random() < 0.5,
                 lay_lo=lay_lo, layout=rng.randint(1, 10**6))


# ------------------------------------------------------------------ sizes and inputs
def _layout(case):
    """Blocks per event and layers per track (numpy): the batch's shape, from the case alone."""
    rng = np.random.default_rng(case["layout"])
    bs, nl = case["bsize"], case["nlayer"]
    counts = np.full(case["nevts"], case["nb"] * bs, np.int64)
    if case["kind"] == "queue":  # log-normal track counts; the listed batch: median 2000 in [50, 20000]
        median = 2000.0 if case["nb"] == 1 else float(case["nb"] * bs)
        counts = np.clip(np.round(median * np.exp(rng.standard_normal(case["nevts"]))), max(1, median / 40), 10 * median).astype(np.int64)
    nb = (counts + bs - 1) // bs
    off = np.concatenate([[0], np.cumsum(nb)]).astype(np.int64)
    nlay = np.full(int(off[-1]) * bs, nl, np.int32)
    if case["lay_lo"]:
        nlay = rng.integers(case["lay_lo"], nl + 1, len(nlay)).astype(np.int32)
    lane = np.arange(len(nlay)) - np.repeat(off[:-1] * bs, nb * bs)
    nlay[lane >= np.repeat(counts, nb * bs)] = 0  # padding lanes of an event's last block
    return off, nlay


def _nblocks(case):
    return int(_layout(case)[0][-1]) if case["kind"] == "queue" else case["nb"] * case["nevts"]


def _inputs(case, seed):
    """Matriplex tracks (nblocks, 28, bsize) and hits (nblocks, nlayer, 9, bsize) on the GPU."""
    dev, bs, nl, nblk = "cuda", case["bsize"], case["nlayer"], _nblocks(case)
    g = torch.Generator(dev).manual_seed(1000003 * int(seed) + 17)
    shape = (nblk, bs)

    def rand():
        return torch.rand(shape, dtype=torch.float64, device=dev, generator=g)

    def gauss():
        return torch.randn(shape, dtype=torch.float64, device=dev, generator=g)

    phi0 = (2 * rand() - 1) * math.pi
    theta = 0.7 + 1.74 * rand()  # beyond, seeds leave the filter's linear regime and gradients lose their digits
    pt = case["pt"] * (1 + 0.1 * gauss().clamp(-4, 4))
    r_seed = 15.0 * (1 + 0.1 * gauss().clamp(-4, 4))
    q = torch.where(rand() < 0.5, -1.0, 1.0).double()
    R = 100.0 * pt / (0.299792458 * case["bz"])  # bending radius, cm
    cot = torch.cos(theta) / torch.sin(theta)

    def helix(rho):
        s = 2 * R * torch.asin(rho / (2 * R))
        a = phi0 - q * s / R
        return -R * q * (torch.sin(a) - torch.sin(phi0)), R * q * (torch.cos(a) - torch.cos(phi0)), s * cot, a

    x, y, z, a = helix(r_seed)
    var = [1e-4, 1e-4, 1e-4, 1e-3, 1e-3, 1e-3]
    trk = torch.zeros(nblk, 28, bs, dtype=torch.float32, device=dev)
    for i, v in enumerate((x, y, z, 1 / pt, a, theta)):
        trk[:, i] = v + math.sqrt(var[i]) * gauss().clamp(-2, 2)
        trk[:, 6 + i * (i + 1) // 2 + i] = var[i]
    trk.view(torch.int32)[:, 27] = q.to(torch.int32)
    hit = torch.zeros(nblk, nl, 9, bs, dtype=torch.float32, device=dev)
    for lay in range(nl):
        rho = case["r_first"] + (case["r_last"] - case["r_first"]) * lay / max(1, nl - 1)
        for i, v in enumerate(helix(torch.full_like(R, rho))[:3]):
            hit[:, lay, i] = v + 1e-3 * gauss()
        for i in (3, 5, 8):
            hit[:, lay, i] = 1e-6
    dr = (torch.rand(nl, device=dev, generator=g) * 0.02 - 0.01).contiguous() if case["dr"] else None  # +-100 um
    # cotangents of a fit: the summed chi2 and the final parameters
    w = torch.zeros_like(trk) if case["kind"] in ("adjoint", "autograd") else None
    if w is not None:
        w[:, :6] = torch.randn(nblk, 6, bs, device=dev, generator=g)
    return trk, hit, dr, w


# ------------------------------------------------------------------ what a caller keeps
def prepare(case, seed):
    kind = case["kind"]
    trk, hit, dr, w = _inputs(case, seed)
    flags = (p2r.FLAG_SQUASH_PHI if case["squash"] else 0) | (p2r.FLAG_ORDER_BY_LAYERS if case["ordered"] else 0)
    cfg = p2r.Config(bsize=case["bsize"], nlayer=case["nlayer"], nevts=case["nevts"], nb=case["nb"], bz=case["bz"],
                     mode=p2r.MODE_RESTART if kind == "restart" else p2r.MODE_CHAINED, flags=flags)
    s = {"kind": kind, "cfg": cfg, "trk": trk, "hit": hit, "dr": dr, "out": torch.empty_like(trk), "chi2": None}
    ntrk = trk.shape[0] * case["bsize"]
    if case["chi2"]:
        s["chi2"] = torch.empty(ntrk, dtype=torch.float32, device="cuda")
    if kind == "masked":
        s["nlay"] = torch.from_numpy(_layout(case)[1]).cuda()
    elif kind == "host":
        s["host"] = [torch.empty(t.shape, dtype=torch.float32, pin_memory=True) for t in (trk, hit, trk)]
        s["host"][0].copy_(trk)
        s["host"][1].copy_(hit)
        s["host_np"] = [t.numpy() for t in s["host"]]
    elif kind in ("queue", "queue_adjoint"):
        off, nlay = _layout(case)
        batch = {"event_block_offset": off, "nlay_lane": nlay, "nblocks": int(off[-1]), "bsize": case["bsize"],
                 "nlayer": case["nlayer"], "bz": case["bz"]}
        s["queue"] = p2r.Queue(batch, blocks_per_item=4, block_threads=128, flags=flags)
        if kind == "queue":
            s["queue"].capture(trk, hit, s["out"], chi2=s["chi2"])
        else:
            s["seed_chi2"] = torch.ones(ntrk, dtype=torch.float32, device="cuda")
            s["grads"] = s["queue"].capture_adjoint(trk, hit, dr=dr, grad_chi2=s["seed_chi2"])
    elif kind == "adjoint":
        s["w"], s["seed_chi2"] = w, torch.ones(ntrk, dtype=torch.float32, device="cuda")
        s["grads"] = {}
    elif kind == "autograd":
        s["w"] = w[:, :6].contiguous()
        s["leaves"] = [trk.view(-1).requires_grad_(), hit.view(-1).requires_grad_(),
                       (dr if dr is not None else torch.zeros(case["nlayer"], device="cuda")).requires_grad_(),
                       torch.tensor(case["bz"], dtype=torch.float64, requires_grad=True)]
    return s


def _tracks(out):
    """A Matriplex track array as its parameter, covariance and charge rows (views of the whole)."""
    return {"par": out[:, :6], "cov": out[:, 6:27], "q": out.view(torch.int32)[:, 27]}


def run(s):
    kind, cfg = s["kind"], s["cfg"]
    if kind in ("forward", "restart"):
        p2r.forward(cfg, s["trk"], s["hit"], s["out"], chi2=s["chi2"], dr=s["dr"])
    elif kind == "masked":
        p2r.forward(cfg, s["trk"], s["hit"], s["out"], chi2=s["chi2"], dr=s["dr"], nlay_lane=s["nlay"])
    elif kind == "layers":
        p2r.run_layers(cfg, s["trk"], s["hit"], s["out"])
    elif kind == "host":
        p2r.forward_host(cfg, *s["host_np"], s["trk"], s["hit"], s["out"])
        return _tracks(s["host"][2])
    elif kind == "queue":
        s["queue"].replay()
    elif kind == "queue_adjoint":
        s["queue"].replay()
        return _gradients(s, s["grads"])
    elif kind == "adjoint":
        return _gradients(s, p2r.forward_backward(cfg, s["trk"], s["hit"], dr=s["dr"], grad_trk_out=s["w"],
                                                  grad_chi2=s["seed_chi2"], per_event=True, out=s["grads"]))
    elif kind == "autograd":
        out, chi2 = p2r.P2RChain.apply(*s["leaves"], cfg)
        out = out.view(s["trk"].shape)
        loss = chi2.sum() + (out[:, :6] * s["w"]).sum()
        g = torch.autograd.grad(loss, s["leaves"])
        return {**_tracks(out.detach()), "chi2": chi2.detach(), "g_trk": g[0], "g_hits": g[1], "g_dr": g[2], "g_bz": g[3]}
    return {**_tracks(s["out"]), **({} if s["chi2"] is None else {"chi2": s["chi2"]})}


def _gradients(s, o):
    return {**_tracks(o["trk_out"].view(s["trk"].shape)), "chi2": o["chi2"], "g_trk": o["grad_trk_in"].view(-1),
            "g_hits": o["grad_hits"].view(-1), "g_dr": o["grad_dr"], "g_bz": o["grad_bz"],
            "g_dr_event": o["grad_dr_event"], "g_bz_event": o["grad_bz_event"]}


def work(case):
    kind = case["kind"]
    nblk, bs, nl = _nblocks(case), case["bsize"], case["nlayer"]
    ntrk = nblk * bs
    updates = ntrk if kind == "restart" else int(_layout(case)[1].sum())  # restart: only the last layer is computed
    nbytes = 36 * updates + 224 * ntrk + (4 * ntrk if case["chi2"] else 0) + (4 * ntrk if case["lay_lo"] else 0)
    flops = FLOP_PER_UPDATE * updates
    if kind in ("adjoint", "autograd", "queue_adjoint"):
        # chi2 and its cotangent, the gradients of tracks and hits; a reverse sweep costs about twice its forward
        nbytes += 8 * ntrk + 112 * ntrk + 36 * updates + (112 * ntrk if kind != "queue_adjoint" else 0)
        flops *= 3
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ the same results in 64 bits
def _f(v):
    """A literal of the path in single precision, widened."""
    return float(np.float32(v))


def _sincos4(x):
    x2 = x * x
    omc = 0.5 * x2 - _f(0.04166667) * x2 * x2
    return x - _f(0.16666667) * x * x2, 1.0 - omc, omc


def _propagate(p, C, k, r):
    x, y, z, ipt, phi, theta = p
    r0, pt = torch.sqrt(x * x + y * y), 1.0 / ipt
    cP, sP = torch.cos(phi), torch.sin(phi)
    px, py = cP * pt, sP * pt
    Dx, Dy, Dipt, Dphi, D = -x / r0, -y / r0, 0.0, 0.0, 0.0
    xo, yo = x, y
    for i in range(5):
        r0 = torch.sqrt(xo * xo + yo * yo)
        step = r - r0
        D = D + step
        t = step * ipt / k
        sa, ca, omc = _sincos4(t)
        a1, a2 = px * ca - py * sa, py * ca + px * sa
        if i < 4:  # path derivatives once the step is below a micrometre
            o = (step.detach().abs() < _f(0.0001)).to(x.dtype) / r0
            g = (1.0 - ipt * o * (xo * a1 + yo * a2)) * o
            Dx, Dy = Dx - xo * g, Dy - yo * g
            Dipt = Dipt - k * (xo * (a1 * t - a2 + py) + yo * (a2 * t + a1 - px)) * pt * o
            Dphi = Dphi + k * (xo * (py * sa + px * ca - px) - yo * (a2 - py)) * o
        xo, yo = xo + k * (px * sa - py * omc), yo + k * (py * sa + px * omc)
        px, py = a1, a2
    al = D * ipt / k
    ax, ay, aphi, aipt = Dx * ipt / k, Dy * ipt / k, Dphi * ipt / k, (ipt * Dipt + D) / k
    sa, ca, omc = _sincos4(al)
    cT, sT = torch.cos(theta), torch.sin(theta)
    U, V, w, kp = cP * ca - sP * sa, sP * ca + cP * sa, ipt * aipt, k * pt
    G = kp * cT / sT
    O, I = torch.zeros_like(x), torch.ones_like(x)
    J = [1 + ax * U * kp, ay * U * kp, O, (w * U - V + sP) * kp * pt, ((aphi + 1) * U - cP) * kp, O,
         ax * V * kp, 1 + ay * V * kp, O, (w * V + U - cP) * kp * pt, ((aphi + 1) * V - sP) * kp, O,
         G * ax, G * ay, I, G * pt * (w - al), G * aphi, -kp * al / (sT * sT),
         O, O, O, I, O, O,
         ax, ay, O, aipt, 1 + aphi, O,
         O, O, O, O, O, I]
    J = torch.stack(J, 1).view(-1, 6, 6)
    return (xo, yo, z + G * al, ipt, phi + al, theta), J @ C @ J.transpose(1, 2)


def _update(p, C, hp, hc):
    x, y, z = p[0], p[1], p[2]
    hx, hy, hz = hp
    r2 = 2 * torch.sqrt(hx * hx + hy * hy)
    R0, R1 = -(hy + y) / r2, (hx + x) / r2
    a0, a1, a2, a3, a4 = C[:, 0, 0] + hc[0], C[:, 1, 0] + hc[1], C[:, 1, 1] + hc[2], C[:, 2, 0] + hc[3], C[:, 2, 1] + hc[4]
    e0, e1, e2 = R0 * R0 * a0 + 2 * R0 * R1 * a1 + R1 * R1 * a2, R0 * a3 + R1 * a4, C[:, 2, 2] + hc[5]
    det = e0 * e2 - e1 * e1
    i0, i1, i2 = e2 / det, -e1 / det, e0 / det
    u = R0[:, None] * C[:, :, 0] + R1[:, None] * C[:, :, 1]
    v = C[:, :, 2]
    K0, K1 = u * i0[:, None] + v * i1[:, None], u * i1[:, None] + v * i2[:, None]
    s0, s1 = R0 * (hx - x) + R1 * (hy - y), hz - z
    chi2 = i0 * s0 * s0 + 2 * i1 * s0 * s1 + i2 * s1 * s1
    pn = tuple(p[m] + K0[:, m] * s0 + K1[:, m] * s1 for m in range(6))
    return pn, C - K0[:, :, None] * u[:, None, :] - K1[:, :, None] * v[:, None, :], chi2


def _chain(trk, hit, q, dr, bz, nlay, squash, restart, kround):
    """trk (n, 27), hit (n, L, 9), q (n,), dr (n or 1, L), bz (n or 1,), nlay (n,), all FP64 but nlay."""
    kf = 100.0 / (-0.299792458 * bz)
    k = q * (kf.float().double() if kround else kf)
    i, j = np.tril_indices(6)
    full = np.zeros((6, 6), int)
    full[i, j] = full[j, i] = np.arange(21)
    p0, C0 = tuple(trk[:, m] for m in range(6)), trk[:, 6:][:, torch.from_numpy(full.reshape(-1)).to(trk.device)].view(-1, 6, 6)
    p, C, chi2 = p0, C0, torch.zeros_like(q)
    for lay in range(hit.shape[1]):
        if restart and lay < hit.shape[1] - 1:
            continue
        h = hit[:, lay]
        hp, hc = (h[:, 0], h[:, 1], h[:, 2]), tuple(h[:, 3 + m] for m in range(6))
        r = torch.sqrt(hp[0] * hp[0] + hp[1] * hp[1]) + dr[:, lay]
        pn, Cn = _propagate(p, C, k, r)
        pn, Cn, c2 = _update(pn, Cn, hp, hc)
        if squash:
            pn = pn[:4] + (pn[4] - 2 * math.pi * torch.round(pn[4] / (2 * math.pi)), pn[5])
        on = lay < nlay
        p = tuple(torch.where(on, a, b) for a, b in zip(pn, p))
        C = torch.where(on[:, None, None], Cn, C)
        chi2 = chi2 + torch.where(on, c2, 0.0)
    cov = C.reshape(-1, 36)[:, torch.from_numpy(i * 6 + j).to(trk.device)]
    return torch.cat([torch.stack(p, 1), cov], 1), chi2


def exact(case, seed):
    kind = case["kind"]
    grads = kind in ("adjoint", "autograd", "queue_adjoint")
    trk, hit, dr, w = _inputs(case, seed)
    off, nlay = _layout(case)
    nblk, bs, nl = trk.shape[0], case["bsize"], case["nlayer"]
    nlay = torch.from_numpy(nlay).cuda()
    ev = torch.from_numpy(np.repeat(np.arange(case["nevts"]), np.diff(off) * bs)).cuda()
    q = trk.view(torch.int32)[:, 27].reshape(-1).double()
    tracks = trk[:, :27].permute(0, 2, 1).reshape(-1, 27)
    hits = hit.permute(0, 3, 1, 2).reshape(-1, nl, 9)
    cot = None if w is None else w[:, :6].permute(0, 2, 1).reshape(-1, 6)
    n = nblk * bs
    step = max(1, int(3.2e6 / nl)) if grads else 400000
    dev = trk.device
    out, chi2 = torch.empty(n, 27, dtype=torch.float64, device=dev), torch.empty(n, dtype=torch.float64, device=dev)
    if grads:
        g_trk, g_hit = torch.zeros(n, 28, dtype=torch.float64, device=dev), torch.empty(n, nl, 9, dtype=torch.float64, device=dev)
        g_dr = torch.zeros(case["nevts"], nl, dtype=torch.float64, device=dev)
        g_bz = torch.zeros(case["nevts"], dtype=torch.float64, device=dev)
    for a in range(0, n, step):
        b = min(n, a + step)
        t, h = tracks[a:b].double(), hits[a:b].double()
        d = torch.zeros(1, nl, dtype=torch.float64, device=dev) if dr is None else dr.detach().double()[None]
        z = torch.full((1,), case["bz"], dtype=torch.float64, device=dev)
        with torch.set_grad_enabled(grads):
            if grads:  # offsets and field of each event on their own
                d, z = d.repeat(case["nevts"], 1), z.repeat(case["nevts"])
                leaves = [v.requires_grad_() for v in (t, h, d, z)]
                d, z = d[ev[a:b]], z[ev[a:b]]
            o, c = _chain(t, h, q[a:b], d, z, nlay[a:b], case["squash"], kind == "restart", not grads)
            if grads:
                loss = c.sum() if cot is None else c.sum() + (o[:, :6] * cot[a:b]).sum()
                g = torch.autograd.grad(loss, leaves)
                g_trk[a:b, :27], g_hit[a:b] = g[0], g[1]
                g_dr += g[2]
                g_bz += g[3]
            out[a:b], chi2[a:b] = o.detach(), c.detach()
            del o, c

    def matriplex(v, rows):  # (n, ..., rows) back to (nblocks, ..., rows, bsize)
        return v.view(nblk, bs, -1, rows).permute(0, 2, 3, 1).contiguous()

    m = matriplex(out, 27)[:, 0]
    res = {"par": m[:, :6], "cov": m[:, 6:], "q": None}
    if case["chi2"] or grads:
        res["chi2"] = chi2
    if grads:
        res |= {"g_trk": matriplex(g_trk, 28).view(-1), "g_hits": matriplex(g_hit, 9).view(-1), "g_dr": g_dr.sum(0)}
        res["g_bz"] = g_bz.sum() if kind == "autograd" else g_bz.sum().view(1)
        if kind != "autograd":
            res |= {"g_dr_event": g_dr, "g_bz_event": g_bz}
    return res
