"""The work that users of this engine have it do, as measurable cases.

Six listed cases trace rooms through the array API (single rooms from a 12-triangle shoebox preview to
the 500k-triangle arena, a hall with an audience map, a batch of rooms); the others are the steps around
a trace: parameter maps of a finished run, receiver filters (one receiver, a hall from host arrays, an
arena on the device) and the emission proposal's network (inference for one room, training).

A trace's room is a model that its user has; what changes from call to call are the random streams and
the places of sources and receivers, which are drawn from the seed.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from pachydermacoustic_universal_gb300 import _capi, proposal, rooms, tracer

BANDS = 8
DIR_BINS = 1536                                            # emission directions of the proposal's targets
LAYERS = ((256, 12), (256, 256), (256, 256), (160, 256))   # its network: (out, in)
CARRIER = 16384
CUT = 4096
# Octave-ray segments that one primary leaves behind in each kind of room (sound decays over the same
# 60 dB whatever the engine does): used by work() only.
SEGMENTS = {"shoebox": 139400.0, "hall": 14400.0, "arena": 2910.0, "batch": 131500.0}


def listed():
    return [
        # a quick look while a shoebox room is being edited: latency of one call
        {"name": "preview_shoebox", "kind": "shoebox", "rays": 1003},
        # the shoebox at its full ray count
        {"name": "shoebox_100k", "kind": "shoebox", "rays": 100_000},
        # a design run of the 20k-triangle hall, 2 sources, 16 receivers
        {"name": "hall_20k_rays", "kind": "hall", "tris": 20_000, "rays": 20_000},
        # the 500k-triangle arena, 4 sources, 64 receivers, into pinned arrays that the caller keeps
        {"name": "arena_60k_rays", "kind": "arena", "tris": 500_000, "rays": 60_000},
        # the hall with its 608-receiver audience map, from the trace to the parameter maps
        {"name": "hall_audience_map", "kind": "hall_map", "tris": 20_000, "rays": 2500},
        # eight rooms of 500 to 50k triangles in one batch run
        {"name": "batch_8_rooms", "kind": "batch", "rooms": 8, "rays": 500},
        # parameter maps of a finished map run: decay times, clarity, definition of every receiver and band
        {"name": "map_parameters", "kind": "parameters", "rays": 1000, "depth": 30, "clarity": 80},
        # one receiver's band envelopes to a filter
        {"name": "filter_one_receiver", "kind": "etc_filter", "n": 1, "bins": 2000},
        # a hall's 16 receivers with their directional filters, host arrays in and out
        {"name": "filters_hall", "kind": "filters", "receivers": 16, "bins": 3000},
        # an arena's 64 receivers, histograms and filters on the device
        {"name": "filters_arena", "kind": "filters_device", "receivers": 64, "bins": 3500},
        # the proposal for one room's 12 receivers
        {"name": "proposal_room", "kind": "proposal", "rows": 12},
        # fitting the proposal to 100 rooms of 12 receivers
        {"name": "proposal_train", "kind": "train", "rows": 1200, "steps": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["shoebox", "hall", "hall", "arena", "hall_map", "batch", "parameters", "etc_filter", "filters",
                       "filters_device", "proposal", "train"])
    if kind == "shoebox":
        return {"kind": kind, "rays": _log(rng, 700, 100_000)}
    if kind == "hall":
        return {"kind": kind, "tris": _log(rng, 2500, 60_000), "rays": _log(rng, 500, 20_000)}
    if kind == "arena":
        return {"kind": kind, "tris": _log(rng, 100_000, 500_000), "rays": _log(rng, 4000, 60_000)}
    if kind == "hall_map":
        return {"kind": kind, "tris": _log(rng, 2500, 20_000), "rays": _log(rng, 300, 2500)}
    if kind == "batch":
        return {"kind": kind, "rooms": rng.randint(2, 8), "rays": _log(rng, 100, 500)}
    if kind == "parameters":
        return {"kind": kind, "rays": _log(rng, 300, 1000), "depth": rng.choice([15, 20, 30]),
                "clarity": rng.choice([50, 80])}
    if kind == "etc_filter":
        return {"kind": kind, "n": rng.randint(1, 12), "bins": _log(rng, 300, 20_000)}
    if kind == "filters":
        return {"kind": kind, "receivers": rng.randint(1, 16), "bins": _log(rng, 500, 4000)}
    if kind == "filters_device":
        return {"kind": kind, "receivers": rng.randint(8, 64), "bins": _log(rng, 1000, 16_000)}
    if kind == "proposal":
        return {"kind": kind, "rows": _log(rng, 1, 2000)}
    return {"kind": kind, "rows": _log(rng, 100, 2400), "steps": rng.randint(2, 20)}


# ------------------------------------------------------------------------------------------ rooms
@functools.lru_cache(maxsize=None)
def _room(kind, tris):
    if kind == "shoebox":
        return rooms.shoebox_c1()
    if kind == "arena":
        return rooms.arena_c5(target_tris=tris)
    return rooms.irregular_hall_c2(target_tris=tris)


@functools.lru_cache(maxsize=None)
def _rooms(n):
    return rooms.batched_rooms_c3(n_rooms=n)


def _places(rng, scene, n, margin):
    lo, hi = scene.bounds()
    m = np.minimum(margin, 0.3 * (hi - lo))
    return [tuple(float(x) for x in lo + m + (hi - lo - 2 * m) * rng.random(3)) for _ in range(n)]


def _workload(kind, tris, seed):
    """The room with sources and receivers placed by the seed."""
    w = _room(kind, tris)
    rng = np.random.default_rng(seed)
    margin = 1.0 if kind == "shoebox" else 4.0
    src = [rooms.SourceSpec(p) for p in _places(rng, w.scene, len(w.sources), margin)]
    rec = [rooms.ReceiverSpec(p) for p in _places(rng, w.scene, len(w.receivers), margin)]
    return rooms.Workload(w.name, w.scene, src, rec, w.rays, w.cutoff_s)


def _pinned(shape):
    return torch.zeros(shape, dtype=torch.float64, pin_memory=True).numpy()


def _audience():
    """The hall's 608 audience squares of 1 m."""
    return rooms.audience_plane((4.0, 3.0), (36.0, 22.0), 1.0, 1.0)


# ------------------------------------------------------------------------------------ histograms
def _histograms(rng, R, T):
    """Scaled histograms as a trace leaves them: exponential decay, sparse late bins, arrival
    directions that split each bin's energy."""
    t = np.arange(T)
    tau = 0.15 * T * (0.5 + rng.random((R, BANDS, 1)))
    E = np.exp(-t / tau) * rng.gamma(0.7, 1.0, (R, BANDS, T)) * 1e-6
    E[rng.random(E.shape) < 0.5 * t / T] = 0.0
    E[:, :, : T // 50] = 0.0
    P = np.sqrt(E * 411.6)
    d = rng.normal(size=(R, 3, BANDS, T))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    share = rng.random((R, 3, BANDS, T))
    return E, P, np.abs(d) * E[:, None] * share, -np.abs(d) * E[:, None] * (1.0 - share)


def _swl(rng):
    return np.round(95.0 + 30.0 * rng.random(BANDS), 1)


def _network(seed, rows):
    """Flat weights of a network with the usual fan-in scale (log kappa bias 1), and conditions (source,
    receiver, room bounds in metres) of `rows` receivers in shoebox rooms."""
    rng = np.random.default_rng(seed)
    flat = []
    for k, (n, m) in enumerate(LAYERS):
        flat.append(rng.uniform(-1.0, 1.0, n * m) * (math.sqrt(6.0 / m) if k < 3 else 0.5 / math.sqrt(m)))
        flat.append(np.where(np.arange(n) % 5 == 3, 1.0, 0.0) if k == 3 else np.zeros(n))
    size = rng.uniform([8, 6, 3], [12, 10, 5], (rows, 3))
    cond = np.concatenate([size * rng.uniform(0.1, 0.9, (rows, 3)), size * rng.uniform(0.1, 0.9, (rows, 3)),
                           np.zeros((rows, 3)), size], axis=1)
    return rng, np.concatenate(flat).astype(np.float32), cond.astype(np.float32)


def _targets(rng, rows):
    """Captured energy shares: a few strong directions over a broad floor."""
    t = rng.gamma(0.3, 1.0, (rows, DIR_BINS))
    t[np.arange(rows), rng.integers(0, DIR_BINS, rows)] += 60.0
    return (t / t.sum(axis=1, keepdims=True)).astype(np.float32)


# ------------------------------------------------------------------------------------------ cases
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case, seed=seed % (1 << 31) + 1)
    if kind in ("shoebox", "hall", "arena"):
        w = _workload(kind, case.get("tris", 12), seed)
        s.update(w=w, scene=tracer.DeviceScene(w.scene))
        if kind == "arena":
            R, T = len(w.receivers), int(w.cutoff_s * w.sample_rate)
            s["out"] = {"energy": _pinned((R, 8, T)), "pressure": _pinned((R, 8, T)), "dir_pos": _pinned((R, 3, 8, T)),
                        "dir_neg": _pinned((R, 3, 8, T)), "analysis": _pinned((R, 3, 8, T))}
    elif kind in ("hall_map", "parameters"):
        w = _workload("hall", case.get("tris", 20_000), seed)
        m = tracer.MapReceivers(_audience(), 1.0, w.cutoff_s * 1000.0)
        s.update(w=w, map=m)
        scene = tracer.DeviceScene(w.scene)
        if kind == "parameters":  # the run goes into the state before its scene, which has to outlive it
            s["run"] = _map_run(dict(s, scene=scene))
            s["run"].wait()
        s["scene"] = scene
    elif kind == "batch":
        ws = _rooms(case["rooms"])
        s.update(ws=ws, scenes=tracer.DeviceScene.many([w.scene for w in ws]))
    elif kind == "etc_filter":
        rng = np.random.default_rng(seed)
        s.update(prms=_histograms(rng, case["n"], case["bins"])[1], swl=_swl(rng))
    elif kind == "filters":
        rng = np.random.default_rng(seed)
        s.update(h=_histograms(rng, case["receivers"], case["bins"]), swl=_swl(rng))
    elif kind == "filters_device":
        rng = np.random.default_rng(seed)
        R, T = case["receivers"], case["bins"]
        n = _capi.lib().pach_filters_workspace_bytes(7 * R, T)
        s.update(h=[torch.from_numpy(x).cuda() for x in _histograms(rng, R, T)], swl=_swl(rng),
                 out=torch.zeros((R, 7, T + CARRIER - 1 - CUT), dtype=torch.float64, device="cuda"),
                 ws=torch.empty(n, dtype=torch.uint8, device="cuda"))
    elif kind == "proposal":
        _, params, cond = _network(seed, case["rows"])
        net = proposal.ProposalNet(max_rows=case["rows"])
        net.set_params(params)
        s.update(net=net, cond=cond)
    elif kind == "train":
        rng, params, cond = _network(seed, case["rows"])
        net = proposal.ProposalNet(max_rows=case["rows"])
        net.set_data(cond, _targets(rng, case["rows"]))
        s.update(net=net, params=params)
    return s


def _map_run(s):
    w = s["w"]
    p = tracer.make_params(rays=s["rays"], cutoff_length_m=w.cutoff_length_m, hist_cotime_ms=w.cutoff_s * 1000.0,
                           seed=s["seed"], sample_rate=w.sample_rate, map_receivers=s["map"])
    return tracer.Run(s["scene"], w.sources, w.receivers, p)


def run(s):
    kind = s["kind"]
    if kind in ("shoebox", "hall", "arena"):
        return tracer.trace(s["w"], dscene=s["scene"], rays=s["rays"], seed=s["seed"], scaled=True,
                            out=s.get("out"))[0]
    if kind == "hall_map":
        r = _map_run(s)
        try:
            r.wait()
            return {"receivers": r.histograms(scaled=True), "map": r.map_parameters()}
        finally:
            r.close()
    if kind == "batch":
        return tracer.trace_batch(s["ws"], dscenes=s["scenes"], rays=[s["rays"]] * len(s["ws"]), seed=s["seed"],
                                  scaled=True)[0]
    if kind == "parameters":
        return s["run"].map_parameters(decay_depth=s["depth"], clarity_ms=s["clarity"])
    if kind == "etc_filter":
        return tracer.etc_to_filter(s["prms"], swl=s["swl"])
    if kind == "filters":
        E, P, Dp, Dn = s["h"]
        return tracer.receiver_filters(P, E, Dp, Dn, swl=s["swl"])
    if kind == "filters_device":
        E, P, Dp, Dn = (x.data_ptr() for x in s["h"])
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        _capi.check(_capi.lib().pach_filters_device(E, P, Dp, Dn, None, s["receivers"], s["bins"], 7, 1000,
                                                    _capi.dptr(s["swl"]), CUT, s["out"].data_ptr(),
                                                    s["ws"].data_ptr(), s["ws"].numel(), stream))
        return s["out"]
    if kind == "proposal":
        return s["net"].forward(s["cond"])
    s["net"].set_params(s["params"])
    curve = s["net"].train(s["steps"], lr=1e-3)
    return {"loss": curve, "params": s["net"].params()}


def work(case):
    kind = case["kind"]
    if kind in ("shoebox", "hall", "arena", "hall_map"):
        shape = {"shoebox": (12, 3, 2000), "arena": (case.get("tris"), 64, 3500)}.get(kind, (case.get("tris"), 16, 3000))
        tris, R, T = shape
        seg = case["rays"] * SEGMENTS[kind.split("_")[0]]
        tests = R + (60 if kind == "hall_map" else 0)
        # triangles (three float4) and materials once; histograms of 11 lanes once; per segment one
        # triangle test, the sphere tests and the surface interaction with its Philox block
        b = tris * (48 + 16 + 128) + R * 11 * BANDS * T * 8 + (608 * BANDS * T * 16 if kind == "hall_map" else 0)
        return {"bytes": b, "flops": seg * (60 + 20 * tests + 150)}
    if kind == "batch":
        R, T, tris = 18 * case["rooms"], 2000, 8000 * case["rooms"]
        return {"bytes": tris * 192 + R * 11 * BANDS * T * 8,
                "flops": case["rooms"] * case["rays"] * SEGMENTS["batch"] * (60 + 20 * 18 + 150)}
    if kind == "parameters":
        n, T = 608 * BANDS, 3000
        return {"bytes": n * T * 8 + n * 40, "flops": n * T * 12}
    if kind in ("etc_filter", "filters", "filters_device"):
        T = case["bins"]
        R = case.get("n") or case["receivers"]
        kinds = 1 if kind == "etc_filter" else 7
        lanes = 1 if kind == "etc_filter" else 8
        L = T + CARRIER - 1 - (0 if kind == "etc_filter" else CUT)
        W = 1 << (T + CARRIER - 2).bit_length()
        fft = 2.5 * W * math.log2(W)
        return {"bytes": R * lanes * BANDS * T * 8 + R * kinds * L * 8, "flops": R * kinds * (10 * fft + 9 * 4 * W)}
    n = sum(a * b + a for a, b in LAYERS)
    rows = case["rows"]
    if kind == "proposal":
        return {"bytes": 2 * n + rows * (12 + 160) * 4, "flops": 2.0 * n * rows}
    # per step: weights, moments and gradients, the target read once; forward, input and weight gradients,
    # and the loss over 1536 bins x 32 lobes
    return {"bytes": case["steps"] * (28 * n + rows * 1536 * 4),
            "flops": case["steps"] * rows * (6.0 * n + 1536 * 32 * 20)}


# ------------------------------------------------------------------------------------------ exact
def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "etc_filter":
        prms, swl = _histograms(rng, case["n"], case["bins"])[1], _swl(rng)
        return _filters(prms, swl)
    if kind in ("filters", "filters_device"):
        E, P, Dp, Dn = _histograms(rng, case["receivers"], case["bins"])
        swl = _swl(rng)
        R, T = case["receivers"], case["bins"]
        if R * T > 64 * 4000:
            return None
        env = np.zeros((R, 7, BANDS, T))
        env[:, 0] = P
        with np.errstate(divide="ignore", invalid="ignore"):
            for d in range(3):
                env[:, 1 + 2 * d] = np.where(E == 0, 0.0, P * Dn[:, d] / E)
                env[:, 2 + 2 * d] = np.where(E == 0, 0.0, P * Dp[:, d] / E)
        out = _filters(env.reshape(R * 7, BANDS, T), swl)
        return out[:, :-CUT].reshape(R, 7, -1)
    if kind == "proposal":
        _, params, cond = _network(seed, case["rows"])
        return _forward(_layers(params), torch.from_numpy(cond).double()).numpy()
    if kind == "train":
        rng, params, cond = _network(seed, case["rows"])
        return _train(params, cond, _targets(rng, case["rows"]), case["steps"])
    return None


def _air(f, tk=293.15, pa=101.325 * 1000, hr=50.0):
    """ISO 9613-1 attenuation, dB/m, with the reference's integer exponents."""
    h = hr * 10 ** (-6.8346 * (273.16 / tk) ** 1.261 + 4.6151) / (pa / 101.325)
    fr_o = (pa / 101.325) * (24 + 4.04e4 * h * ((0.02 + h) / (0.391 + h)))
    fr_n = (pa / 101.325) * (9 + 280 * h)
    z = 0.1068 * math.exp(-3352 / tk) / (fr_n + f * f / fr_n)
    y = (tk / 293.15) ** -2 * (0.01275 * math.exp(-2239.1 / tk) / (fr_o + f * f / fr_o) + z)
    return 8.686 * f * f * (1.84e-11 / (pa / 101.325) + y)


def _filters(prms, swl, fs=1000):
    """[n][8][T] envelopes to [n][T + 16383] filters: nine band-limited pulses, each convolved with its
    band's envelope (16 kHz: the 8 kHz one under the extra air attenuation), summed."""
    n, _, T = prms.shape
    t = (np.arange(CARRIER) - (CARRIER - 1) / 2.0) / fs
    W = 1 << (T + CARRIER - 2).bit_length()
    env = np.abs(prms) * (10.0 ** ((120.0 - swl) / 20.0))[:, None]
    ramp = 10.0 ** (-(_air(16000.0) - _air(8000.0)) * (np.arange(T) / fs) * 343.0 / 20.0)
    spec = np.zeros((n, W // 2 + 1), dtype=np.complex128)
    for b in range(9):
        centre = 62.5 * 2.0 ** b
        lo, hi = centre / math.sqrt(2.0), centre * math.sqrt(2.0)
        x = math.pi * (hi - lo) * t
        c = np.sin(x) / x * np.cos(2 * math.pi * (lo + hi) / 2.0 * t)
        c *= 2.0 / (np.abs(c).sum() * CARRIER)
        e = env[:, b] if b < 8 else env[:, 7] * ramp
        spec += np.fft.rfft(e, W) * np.fft.rfft(c, W)
    return np.fft.irfft(spec, W)[:, : T + CARRIER - 1]


def _layers(p):
    """Flat parameters -> [(W, b)] in 64 bits."""
    out, k = [], 0
    p = torch.from_numpy(np.asarray(p, dtype=np.float64))
    for n, m in LAYERS:
        out.append([p[k:k + n * m].view(n, m).clone(), p[k + n * m:k + n * m + n].clone()])
        k += n * m + n
    return out


def _forward(layers, cond):
    x = cond * 0.1
    for i, (w, b) in enumerate(layers):
        x = x @ w.T + b
        if i < 3:
            x = torch.nn.functional.gelu(x)
    return x


def _bin_centres():
    d = np.zeros((DIR_BINS, 3))
    for f in range(6):
        for j in range(16):
            for i in range(16):
                u, v = (i + 0.5) / 8.0 - 1.0, (j + 0.5) / 8.0 - 1.0
                s = -1.0 if f & 1 else 1.0
                c = (s, u, v) if f < 2 else ((u, s, v) if f < 4 else (u, v, s))
                d[f * 256 + j * 16 + i] = np.array(c) / np.linalg.norm(c)
    return torch.from_numpy(d)


def _loss(out, target, bins):
    """Cross-entropy of the targets against the von Mises-Fisher mixture at the bin centres."""
    o = out.view(out.shape[0], 32, 5)
    mu = o[:, :, :3] / o[:, :, :3].norm(dim=2, keepdim=True).clamp_min(1e-6)
    kappa = o[:, :, 3].clamp(-3.0, 6.0).exp()
    lw = torch.log_softmax(o[:, :, 4], dim=1) + torch.log(kappa / (2 * math.pi * -torch.expm1(-2 * kappa)))
    x = lw[:, None, :] + kappa[:, None, :] * (torch.einsum("mkc,bc->mbk", mu, bins) - 1.0)
    return -(target * torch.logsumexp(x, dim=2)).sum(dim=1)


def _train(params, cond, target, steps, lr=1e-3):
    """Adam on the mean loss in 64 bits: the loss of every step and the weights after the last."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    layers = [[x.to(dev).requires_grad_(True) for x in wb] for wb in _layers(params)]
    flat = [x for wb in layers for x in wb]
    c, t = torch.from_numpy(cond).double().to(dev), torch.from_numpy(target).double().to(dev)
    bins = _bin_centres().to(dev)
    m1, m2 = [torch.zeros_like(x) for x in flat], [torch.zeros_like(x) for x in flat]
    curve = []
    for step in range(1, steps + 1):
        total = 0.0
        for x in flat:
            x.grad = None
        for k in range(0, c.shape[0], 256):
            part = _loss(_forward(layers, c[k:k + 256]), t[k:k + 256], bins).sum() / c.shape[0]
            part.backward()
            total += float(part.detach())
        curve.append(total)
        with torch.no_grad():
            for x, a, b in zip(flat, m1, m2):
                a.mul_(0.9).add_(x.grad, alpha=0.1)
                b.mul_(0.999).addcmul_(x.grad, x.grad, value=0.001)
                x -= lr * (a / (1 - 0.9 ** step)) / ((b / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return {"loss": np.array(curve), "params": torch.cat([x.detach().reshape(-1) for x in flat]).cpu().numpy()}
