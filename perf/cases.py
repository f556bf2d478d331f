"""Performance cases of the photon-transport engine: what its users have it do,
through the package's public entry points, from the smallest calls to the largest.

The setups are those of ``params.py`` (the polished cube, the wrapped Lambertian
cube with Rayleigh scattering, the long bar with a black -z face), the batch of
uneven events and the genstep tracks of the package's own generators. `exact`
transports the same photons in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

from gpu_optical_photons_b200 import backend, gensteps, params, wavefront

# Steps per photon and scalar operations per step (additions, products,
# comparisons, Philox and library calls, emission included) of each setup.
STEPS_OPS = {"cube": (4.32, 185.1), "lambert": (5.16, 268.6), "bar": (18.2, 149.1), "batch": (4.27, 250.2)}
SETUPS = {"cube": params.config1, "lambert": params.config2, "bar": params.config3}
BATCH_TALLY = (100, 50.0, 10)  # time bins, window (ns), hit-map bins per axis
THETA = (1000.0, 700.0, 0.95, 4.0)  # where the calibration starts


def listed():
    return [
        # The shortest call: one setup probed with a thousand photons (scans, tests).
        {"name": "tally cube 1k", "kind": "tally", "setup": "cube", "n": 1000, "math": "fast"},
        # An ordinary validation run; a size that is no multiple of anything.
        {"name": "tally lambert 300k", "kind": "tally", "setup": "lambert", "n": 300_007, "math": "fast"},
        # The long bar at its specified statistics, the largest run here.
        {"name": "tally bar 100M", "kind": "tally", "setup": "bar", "n": 100_000_000, "math": "fast"},
        # Per-photon records for the analysis scripts, in host arrays that the program reuses.
        {"name": "records cube 1M", "kind": "records", "setup": "cube", "n": 1_000_003, "math": "fast"},
        # Records that stay on the GPU (the history kernel), for a consumer there.
        {"name": "device records lambert 2.5M", "kind": "device_records", "setup": "lambert", "n": 2_500_001,
         "math": "fast"},
        # The device tally (the history kernel) added to a buffer of the caller's.
        {"name": "device tally bar 10M", "kind": "device_tally", "setup": "bar", "n": 10_000_000, "math": "fast"},
        # The benchmark's batch of uneven events with the autotuner's settings.
        {"name": "batch 4096", "kind": "batch", "events": 4096, "median": 10_000, "math": "fast", "tuned": True},
        # A few small events, bit-reproducible arithmetic, default engine settings.
        {"name": "batch 48 exact", "kind": "batch", "events": 48, "median": 300, "math": "exact", "tuned": False},
        # Gensteps that a producer on the GPU hands over in device memory.
        {"name": "gensteps 512", "kind": "gensteps", "events": 512, "yield": 200, "math": "fast"},
        # One gradient step of a calibration: forward run, loss, adjoint replay.
        {"name": "response 1M", "kind": "response", "n": 1_000_000},
        # One Fisher-scoring step: histogram and Jacobian from one replay.
        {"name": "fisher 3M", "kind": "fisher", "n": 3_000_001},
        # The event backend's records with a forced compaction every 8 steps.
        {"name": "event records lambert 300k k8", "kind": "event_records", "setup": "lambert", "n": 300_000, "k": 8,
         "math": "fast"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tally", "records", "device_records", "device_tally", "batch", "gensteps", "response",
                       "fisher", "event_records"])
    case = {"kind": kind}
    if kind in ("tally", "records", "device_records", "device_tally", "event_records"):
        hi = {"tally": 60_000_000, "records": 3_000_000, "event_records": 3_000_000}.get(kind, 20_000_000)
        case.update(setup=rng.choice(sorted(SETUPS)), n=_log(rng, 1000, hi) | 1,
                    math=rng.choice(["fast", "fast", "exact", "approx"]))
        if kind == "event_records":
            case["k"] = rng.choice([1, 2, 4, 8, 20_000])
    elif kind == "batch":
        case.update(events=_log(rng, 2, 4000), median=_log(rng, 100, 8000),
                    math=rng.choice(["fast", "fast", "exact", "approx"]), tuned=rng.random() < 0.5)
    elif kind == "gensteps":
        case.update(events=_log(rng, 4, 600), math=rng.choice(["fast", "exact"]))
        case["yield"] = _log(rng, 10, 300)
    else:
        case["n"] = _log(rng, 10_000, 10_000_000) | 1
    return case


def _photons(case):
    if case["kind"] == "batch":  # mean of the lognormal counts
        return case["events"] * case["median"] * math.exp(0.5)
    if case["kind"] == "gensteps":  # mean chord of random tracks in the 50 mm cube
        return case["events"] * case["yield"] * 45.0
    return float(case["n"])


def work(case):
    kind = case["kind"]
    setup = {"batch": "batch"}.get(kind, case.get("setup", "lambert"))
    n = _photons(case)
    steps, ops = STEPS_OPS[setup]
    flops = n * steps * ops
    if kind in ("records", "device_records", "event_records"):
        nbytes = n * 29
    elif kind in ("tally", "device_tally"):
        nbytes = 8.0 * SETUPS[setup]()[1].length
    elif kind == "batch":
        nbytes = case["events"] * (72 + 8 + 8.0 * params.TallyConfig(*BATCH_TALLY).length)
    elif kind == "gensteps":
        nbytes = case["events"] * (45 * 40 + 72 + 8.0 * params.TallyConfig(*BATCH_TALLY).length)
    elif kind == "fisher":
        nbytes = 501 * 5 * 8.0
    else:  # a forward run and its replay
        nbytes = 501 * 8.0 * 3
        flops *= 2
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---- inputs ------------------------------------------------------------------

def _single(case, seed):
    """(SimParams, TallyConfig, first photon id) of a single-setup case."""
    rng = np.random.default_rng([seed, 1])
    p, c = SETUPS[case["setup"]]()
    p = p.replace(seed=int(rng.integers(1 << 62)))
    if p.source == params.POINT:
        h = np.array([p.hx, p.hy, p.hz])
        at = np.array([p.src_x, p.src_y, p.src_z]) + rng.uniform(-0.1, 0.1, 3) * h
        p = p.replace(**{k: float(np.float32(v)) for k, v in zip(("src_x", "src_y", "src_z"), at)})
    return p, c, int(rng.integers(1 << 40))


def _calibration(case, seed):
    """(base SimParams, theta, target histogram, first photon id) of a calibration step."""
    rng = np.random.default_rng([seed, 2])
    p = params.config2()[0].replace(seed=int(rng.integers(1 << 62)))
    theta = [float(np.float32(t * s)) for t, s in zip(THETA, rng.uniform(0.9, 1.0, 4))]
    at = (np.arange(500) + 0.5) * 0.1
    shape = np.exp(-at / 4.3) * (1 - np.exp(-at / 0.3))
    target = rng.poisson(0.45 * case["n"] * shape / shape.sum()).astype(np.float64)
    return p, theta, target, int(rng.integers(1 << 40))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("tally", "records", "device_records", "device_tally", "event_records"):
        s["p"], s["c"], s["first"] = _single(case, seed)
        if kind == "records":
            s["out"] = backend.Records.empty(case["n"])
        elif kind == "device_records":
            s["out"] = backend.device_records(case["n"])
        elif kind == "device_tally":
            s["out"] = torch.zeros(s["c"].length, dtype=torch.int64, device="cuda")
    elif kind == "batch":
        events, counts = wavefront.batched_events(case["events"], seed=int(seed), median=float(case["median"]),
                                                  photon_seed=int(seed) + 12345)
        cfg = wavefront.WaveConfig(math=case["math"])
        if case["tuned"]:
            cfg = wavefront.WaveConfig(math=case["math"], blocks_per_sm=7, threshold=32)
        s["events"], s["counts"] = wavefront.EventTable(events), counts
        s["engine"] = wavefront.WavefrontEngine(params.TallyConfig(*BATCH_TALLY), case["events"],
                                                int(counts.sum()), cfg)
    elif kind == "gensteps":
        events, g = gensteps.muon_events(case["events"], seed=int(seed), photons_per_mm=float(case["yield"]))
        events = [e.replace(seed=int(seed) + 12345) for e in events]
        s["events"], s["gensteps"] = wavefront.EventTable(events), gensteps.to_device(g)
        s["engine"] = wavefront.WavefrontEngine(params.TallyConfig(*BATCH_TALLY), case["events"],
                                                gensteps.photons_of(g),
                                                wavefront.WaveConfig(math=case["math"], max_gensteps=len(g)))
    else:
        from gpu_optical_photons_b200 import adjoint
        p, s["theta"], target, first = _calibration(case, seed)
        s["model"] = adjoint.ResponseModel(p, case["n"], first_id=first)
        s["target"] = torch.as_tensor(target)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "tally":
        _, flat, _ = backend.run_gpu_tally(s["p"], s["c"], case["n"], first_id=s["first"], math=case["math"])
        return flat.view(np.int64)
    if kind == "records":
        rec, _ = backend.run_gpu_records(s["p"], case["n"], first_id=s["first"], math=case["math"], out=s["out"])
        return dict(rec)
    if kind == "event_records":
        rec, _, _ = backend.run_gpu_records_event(s["p"], case["n"], case["k"], first_id=s["first"],
                                                  math=case["math"])
        return dict(rec)
    if kind == "device_records":
        return backend.records_device(s["p"], case["n"], s["first"], out=s["out"], math=case["math"])
    if kind == "device_tally":
        return backend.tally_device(s["p"], s["c"], case["n"], s["first"], out=s["out"].zero_(), math=case["math"])
    if kind == "batch":
        return s["engine"].run_batch(s["events"], s["counts"])[0].view(np.int64)
    if kind == "gensteps":
        s["engine"].set_gensteps_device(s["events"], s["gensteps"])
        s["engine"].run_tally()
        return s["engine"].tallies().view(np.int64)
    if kind == "fisher":
        hist, jac = s["model"].score_moments(s["theta"])
        return {"hist": hist, "jac": jac}
    from gpu_optical_photons_b200 import adjoint
    theta = torch.tensor(s["theta"], dtype=torch.float64, requires_grad=True)
    loss = adjoint.loss_fn(theta, s["model"], s["target"])
    loss.backward()
    return {"loss": loss.detach(), "grad": theta.grad}


# ---- the same photons in 64 bits, with plain torch -------------------------------

_M32 = 0xFFFFFFFF


def _philox(block, lo, hi, key):
    """Philox4x32-10 of counters {block, 0, lo, hi} (int64 tensors holding 32-bit words)."""
    c = [block, torch.zeros_like(block), lo, hi]
    k0, k1 = key & _M32, (key >> 32) & _M32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # the low 64 bits; the sign does not matter
        c = [((p1 >> 32) & _M32) ^ c[1] ^ k0, p1 & _M32, ((p0 >> 32) & _M32) ^ c[3] ^ k1, p0 & _M32]
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return torch.stack(c)


def _uniforms(draws, ids, key, count):
    """The next `count` (<= 5) uniforms of each photon's stream after `draws` words."""
    lo, hi = ids & _M32, (ids >> 32) & _M32
    w = torch.cat([_philox(draws // 4, lo, hi, key), _philox(draws // 4 + 1, lo, hi, key)])
    at = draws % 4
    return [((torch.gather(w, 0, (at + j)[None])[0] >> 8) + 1).double() / 16777216.0 for j in range(count)]


def _rotate(a, ct, u):
    """Unit vectors at polar cosine ct and azimuth 2 pi u about the axes a (3 x n)."""
    ax, ay, az = a
    sg = torch.copysign(torch.ones_like(az), az)
    k = -1.0 / (sg + az)
    b = ax * ay * k
    st = torch.sqrt(torch.clamp(1 - ct * ct, min=0))
    cp, sp = st * torch.cos(2 * math.pi * u), st * torch.sin(2 * math.pi * u)
    d = torch.stack([cp * (1 + sg * ax * ax * k) + sp * b + ct * ax,
                     cp * sg * b + sp * (sg + ay * ay * k) + ct * ay, -cp * sg * ax - sp * ay + ct * az])
    return d / d.norm(dim=0)


def _transport(p, n, first, dev):
    f = lambda v: float(np.float32(v))  # noqa: E731  the C structure holds floats
    h = torch.tensor([f(p.hx), f(p.hy), f(p.hz)], dtype=torch.float64, device=dev)[:, None]
    n1, nd, no, la, ls = (f(v) for v in (p.n_scint, p.n_det, p.n_out, p.abs_length, p.scat_length))
    tau, key = f(p.tau), p.seed
    faces = list(p.face_surface or [p.surface] * 6)[:5] + [params.POLISHED]
    model = torch.tensor(faces, device=dev)
    refl = torch.tensor([f(r) for r in (p.face_reflectivity or [p.reflectivity] * 6)], dtype=torch.float64, device=dev)
    z = lambda: torch.zeros(n, dtype=torch.float64, device=dev)  # noqa: E731
    out = {k: z() for k in ("t", "x", "y", "z", "path", "t_emit")}
    out.update({k: torch.zeros(n, dtype=torch.int64, device=dev) for k in ("n_boundary", "n_scatter", "refl")})
    out["fate"] = torch.full((n,), params.MAX_STEPS, dtype=torch.int64, device=dev)

    me = torch.arange(n, device=dev)
    ids = me + first
    draws = torch.zeros_like(me)
    if p.source == params.VOLUME:
        pos = h * (2 * torch.stack(_uniforms(draws, ids, key, 3)) - 1)
        draws = draws + 3
    else:
        pos = torch.tensor([f(p.src_x), f(p.src_y), f(p.src_z)], dtype=torch.float64, device=dev)[:, None].repeat(1, n)
    ua, ub, ue = _uniforms(draws, ids, key, 3)
    draws = draws + 3
    ct = 2 * ua - 1
    st = torch.sqrt(torch.clamp(1 - ct * ct, min=0))
    d = torch.stack([st * torch.cos(2 * math.pi * ub), st * torch.sin(2 * math.pi * ub), ct])
    t = -tau * torch.log(ue) if tau > 0 else torch.zeros_like(ue)
    out["t_emit"] = t.clone()
    path, nb, ns, nr = torch.zeros_like(t), torch.zeros_like(me), torch.zeros_like(me), torch.zeros_like(me)
    for _ in range(p.max_steps):
        if me.numel() == 0:
            break
        u = _uniforms(draws, ids, key, 5)
        far = torch.full_like(t, math.inf)
        sa = -la * torch.log(u[0]) if math.isfinite(la) else far
        ss = -ls * torch.log(u[1]) if math.isfinite(ls) else far
        tt = torch.where(d != 0, (torch.where(d > 0, h, -h) - pos) / d, math.inf)
        dist, axis = tt.min(dim=0)
        dist = dist.clamp(min=0)
        face = 2 * axis + (torch.gather(d, 0, axis[None])[0] > 0).long()
        ab = (sa < dist) & (sa <= ss)
        sc = ~ab & (ss < dist)
        hit = ~ab & ~sc
        s = torch.where(ab, sa, torch.where(sc, ss, dist))
        pos = pos + s * d
        on = (torch.arange(3, device=dev)[:, None] == axis) & hit
        pos = torch.where(on, torch.where((face & 1) == 1, h, -h), torch.where(hit, torch.clamp(pos, -h, h), pos))
        t = t + s * (n1 / params.SPEED_OF_LIGHT)
        path = path + s
        nb, ns = nb + hit.long(), ns + sc.long()
        ci = torch.gather(d, 0, axis[None])[0].abs()
        pol = hit & (model[face] == params.POLISHED)
        n2 = torch.where(face == params.READOUT_FACE, nd, no).double()
        s2 = (n1 / n2) ** 2 * torch.clamp(1 - ci * ci, min=0)
        c2 = torch.sqrt(torch.clamp(1 - s2, min=0))
        rs, rp = (n1 * ci - n2 * c2) / (n1 * ci + n2 * c2), (n2 * ci - n1 * c2) / (n2 * ci + n1 * c2)
        R = torch.where(n1 == n2, 0.0, torch.where(s2 >= 1, 1.0, 0.5 * (rs * rs + rp * rp)))
        painted = hit & ~pol & (model[face] != params.BLACK)
        bounce = painted & (u[2] <= refl[face])
        mirror = pol & (u[2] <= R) | bounce & (model[face] == params.SPECULAR)
        lam = bounce & (model[face] == params.LAMBERTIAN)
        nr = nr + bounce.long()
        q = 4 * u[2] - 2
        c3 = (q.abs() + torch.sqrt(q * q + 1)) ** (1 / 3)
        c3 = torch.where(q >= 0, c3, 1 / c3)
        inward = torch.where(torch.arange(3, device=dev)[:, None] == axis, torch.where((face & 1) == 1, -1.0, 1.0), -0.0)
        turned = _rotate(torch.where(sc, d, inward.double()), torch.where(sc, torch.clamp(c3 - 1 / c3, -1, 1),
                                                                        torch.sqrt(u[3])), torch.where(sc, u[3], u[4]))
        d = torch.where(mirror & on, -d, torch.where(sc | lam, turned, d))
        live = sc | mirror | lam
        fate = torch.where(ab, params.ABSORBED_BULK, torch.where(pol & ~mirror, torch.where(
            face == params.READOUT_FACE, params.DETECTED, params.ESCAPED), params.ABSORBED_SURFACE))
        end = ~live
        for k, v in (("t", t), ("x", pos[0]), ("y", pos[1]), ("z", pos[2]), ("path", path), ("n_boundary", nb),
                     ("n_scatter", ns), ("refl", nr), ("fate", fate)):
            out[k][me[end]] = v[end].to(out[k].dtype)
        draws = draws + torch.where(sc, 4, torch.where(lam, 5, 3))
        me, ids, draws, t, path, nb, ns, nr = (v[live] for v in (me, ids, draws, t, path, nb, ns, nr))
        pos, d = pos[:, live], d[:, live]
    for k, v in (("t", t), ("x", pos[0]), ("y", pos[1]), ("z", pos[2]), ("path", path), ("n_boundary", nb),
                 ("n_scatter", ns), ("refl", nr)):
        out[k][me] = v
    return out


def _moments(p, theta, n, first, dev):
    """Arrival-time histogram (500 bins of 0.1 ns and the overflow), the score sums
    per bin (501 x 4) and the detected fraction, at theta."""
    la, ls, R, tau = theta
    r = _transport(p.replace(abs_length=la, scat_length=ls, reflectivity=R, tau=tau), n, first, dev)
    det = r["fate"] == params.DETECTED
    tb = torch.clamp((r["t"][det] * 10.0).long(), max=500)
    path, ns, nr, te = (r[k][det].double() for k in ("path", "n_scatter", "refl", "t_emit"))
    S = torch.stack([path / la ** 2, path / ls ** 2 - ns / ls, nr / R, te / tau ** 2 - 1 / tau], dim=1)
    hist = torch.bincount(tb, minlength=501).double()
    jac = torch.zeros(501, 4, dtype=torch.float64, device=dev).index_add_(0, tb, S)
    return hist, jac, det.double().mean()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("tally", "device_tally", "batch", "gensteps") or case["n"] > 4_000_000:
        return None  # whole numbers; or too many photons for this
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind in ("response", "fisher"):
        p, theta, target, first = _calibration(case, seed)
        hist, jac, frac = _moments(p, theta, case["n"], first, dev)
        if kind == "fisher":
            return {"hist": hist, "jac": jac}
        lam, k = hist[:500] + 1.0, torch.as_tensor(target, device=dev)
        loss = (lam - k * torch.log(lam)).sum() / case["n"] + frac
        w = torch.zeros(501, dtype=torch.float64, device=dev)
        w[:500] = (1.0 - k / lam) / case["n"]
        return {"loss": loss, "grad": ((w + 1.0 / case["n"])[:, None] * jac).sum(0)}
    p, _, first = _single(case, seed)
    r = _transport(p, case["n"], first, dev)
    return {k: (r[k] if k in ("t", "x", "y", "z", "path") else None) for k in backend.Records.FIELDS}
