"""The timed cases of this framework: what its users run, through the entry points they call.

``listed()`` names the standing cases, ``draw(rng)`` gives another one of the same ranges,
``prepare(case, seed)`` makes a case's inputs, ``run(state)`` is one pass, ``work(case)`` the bytes
and operations a pass cannot do without and ``exact(case, seed)`` its result in 64 bits.

Scenes are those of the repository's benchmark workloads: a planar scan of a 3 TX x 4 RX array
(1 mm pitch, 77.3704 GHz, 4 GHz swept in S samples at 5 Msps) looking at a scene around
(0, 0, 0.4) m; tracer points are samples along rays through a bumpy sphere of 0.1 m radius, whose
normals and alpha-composited amplitudes are distributed like those of a freshly initialised NeuS
field (about one pair in ten specular).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "geraf-sens_b200"))

from geraf_b200.bank import AntennaBank  # noqa: E402
from geraf_b200.model_utils import base_matched_filter, bilinear_ray_sampler, lensless_ray_tracer  # noqa: E402
from geraf_b200.ops.RFSignalTracer.ragged import signal_tracer_ragged  # noqa: E402
from geraf_b200.stage1 import stage1_rf_prediction  # noqa: E402

MF_CARRIER = 773.704  # 1e8 Hz, the matched filter's fixed carrier
TRACER_CARRIER = 770.0
CENTER = (0.0, 0.0, 0.4)
NEAR, FAR = 0.22, 0.58


def listed():
    return [
        # Matched filter at a handful of points (a probe, a unit test, an interactive cursor): launch latency.
        dict(name="mf_few_points", op="mf", scan=2, S=64, N=343, precision="mixed", backward=False),
        # The small imaging workload: 3072 channels onto 48^3 voxels, as mf_small_workload.
        dict(name="mf_image_48", op="mf", scan=16, S=128, N=48 ** 3, precision="mixed", backward=False),
        # One voxel chunk of an image of the full 49152-channel array.
        dict(name="mf_image_80_full_array", op="mf", scan=64, S=256, N=80 ** 3, precision="mixed", backward=False),
        # A reconstruction step through the matched filter at odd sizes: forward and adjoint.
        dict(name="mf_step_odd", op="mf", scan=9, S=201, N=37 ** 3, precision="mixed", backward=True),
        # The bit-faithful form, forward and adjoint, as a user checks against the reference.
        dict(name="mf_step_plain", op="mf", scan=5, S=128, N=24 ** 3, precision="plain", backward=True),
        # The fast approximate form on a mid-size image, forward and adjoint.
        dict(name="mf_step_nufft", op="mf", scan=16, S=256, N=64 ** 3, precision="nufft", backward=True),
        # Signal tracer at the benchmark's training size with position gradients.
        dict(name="tracer_step", op="tracer", A=64, rays=4096, T=128, S=128, precision="mixed"),
        # A small odd tracer call (few antennas, few rays): latency and remainders.
        dict(name="tracer_step_small", op="tracer", A=13, rays=300, T=33, S=101, precision="mixed"),
        # The fast approximate form of the tracer on a chunk of a step.
        dict(name="tracer_step_nufft", op="tracer", A=32, rays=2048, T=128, S=256, precision="nufft"),
        # Every antenna with its own uneven set of points, in one batched call.
        dict(name="ragged_step", op="ragged", A=64, rays=2304, T=128, S=256),
        # Coarse-to-target resampling along rays, forward and adjoint.
        dict(name="resample_step", op="resample", A=1, rays=4096, T=128, S=128),
        # The RF part of a stage-1 training step: resample, trace, antenna bank, matched filter, adjoints.
        dict(name="stage1_step", op="stage1", A=128, bank=2, rays=2048, T=128, coarse=128, S=256),
    ]


def draw(rng):
    """One more case of the listed ranges: the sizes log-uniform, odd ones among them."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["mf", "mf", "mf", "tracer", "tracer", "ragged", "resample", "stage1"])
    if op == "mf":
        precision = rng.choice(["mixed", "mixed", "nufft", "plain"])
        backward = rng.random() < 0.5
        scan, S, N = size(2, 64), size(60, 256), size(343, 64 ** 3)
        # a plain triple costs ten mixed ones; a drawn case stays well under the largest listed one
        most = {"mixed": 1.5e12, "nufft": 3e12, "plain": 2e10}[precision]
        N = max(343, min(N, int(most / (12.0 * scan * scan * S))))
        if 12.0 * scan * scan * S * N > most:
            scan = max(2, int(math.sqrt(most / (12.0 * S * N))))
        return dict(op="mf", scan=scan, S=S, N=N, precision=precision, backward=backward)
    if op == "tracer":
        return dict(op="tracer", A=size(8, 64), rays=size(200, 4096), T=size(32, 128), S=size(64, 256),
                    precision=rng.choice(["mixed", "mixed", "nufft"]))
    if op == "ragged":
        return dict(op="ragged", A=size(8, 64), rays=size(300, 2304), T=size(64, 128), S=size(64, 256))
    if op == "resample":
        return dict(op="resample", A=rng.choice([1, 1, 2, 8]), rays=size(500, 4096), T=size(32, 128), S=size(32, 128))
    bank = rng.choice([1, 2, 4])
    return dict(op="stage1", A=bank * size(8, 128 // bank), bank=bank, rays=size(300, 2048), T=size(32, 128),
                coarse=size(32, 128), S=size(64, 256))


# ---- inputs -----------------------------------------------------------------------------------

def _cfg(S, carrier):
    fs = 5e6
    return {"numADCSample": S, "adcSampleRate": fs, "As_sci": 4e9 * fs / S / 1e8, "fc_start": carrier}


def _array(scan):
    lam = 2.9979 / MF_CARRIER
    c = (np.arange(scan) - (scan - 1) / 2.0) * 1e-3
    gy, gx = np.meshgrid(c, c, indexing="ij")
    pos = np.stack([gx.ravel(), gy.ravel(), np.zeros(gx.size)], 1)
    tx = np.stack([np.arange(3) * 2.0 * lam, np.zeros(3), np.zeros(3)], 1)
    rx = np.stack([np.arange(4) * 0.5 * lam + 2.0 * lam, np.full(4, 2.0 * lam), np.zeros(4)], 1)
    tx = np.broadcast_to(pos[:, None, None] + tx[None, :, None], (pos.shape[0], 3, 4, 3)).reshape(-1, 3)
    rx = np.broadcast_to(pos[:, None, None] + rx[None, None], (pos.shape[0], 3, 4, 3)).reshape(-1, 3)
    return torch.tensor(tx, dtype=torch.float32, device="cuda"), torch.tensor(rx, dtype=torch.float32, device="cuda")


def _pick_antennas(A, gen):
    tx, rx = _array(16)
    keep = torch.randperm(tx.shape[0], generator=gen, device="cuda")[:A].sort().values
    return tx[keep].contiguous(), rx[keep].contiguous()


def _if_samples(tx, rx, cfg, gen, scatterers=12):
    """IF of point scatterers in a 0.2 m cube at 20 dB SNR."""
    S = cfg["numADCSample"]
    pos = (torch.rand(scatterers, 3, generator=gen, device="cuda") - 0.5) * 0.2 + torch.tensor(CENTER, device="cuda")
    amp = torch.randn(scatterers, 2, generator=gen, device="cuda")
    tau = (torch.cdist(tx.double(), pos.double()) + torch.cdist(rx.double(), pos.double()) + 0.15) / 2.9979
    w = 2 * math.pi * (MF_CARRIER + cfg["As_sci"] / cfg["adcSampleRate"] * torch.arange(S, device="cuda", dtype=torch.float64))
    out = torch.zeros(tx.shape[0], S, dtype=torch.complex64, device="cuda")
    for k in range(scatterers):
        ph = (tau[:, k:k + 1] * w).remainder_(2 * math.pi).float()
        out += torch.polar(torch.ones_like(ph), ph) * torch.complex(amp[k, 0], amp[k, 1])
    sigma = (out.abs().square().mean() / 100.0 / 2.0).sqrt()
    re = out.real + sigma * torch.randn(out.shape, generator=gen, device="cuda")
    im = out.imag + sigma * torch.randn(out.shape, generator=gen, device="cuda")
    return re.contiguous(), im.contiguous()


def _voxels(N, edge):
    """The first N points of the regular grid that holds at least N, over a cube."""
    n = int(math.ceil(round(N ** (1 / 3), 6)))
    ax = torch.linspace(-edge / 2, edge / 2, n, dtype=torch.float64)
    gz, gy, gx = torch.meshgrid(ax + CENTER[2], ax + CENTER[1], ax + CENTER[0], indexing="ij")
    return torch.stack([gx, gy, gz], -1).reshape(-1, 3)[:N].float().cuda().contiguous()


def _rays(R, T, gen):
    """Points [R,T,3] and depths [R,T] of samples along rays through a disk around the scene."""
    u, th = torch.rand(R, generator=gen, device="cuda"), 2 * math.pi * torch.rand(R, generator=gen, device="cuda")
    aim = torch.stack([0.2 * u.sqrt() * th.cos(), 0.2 * u.sqrt() * th.sin(), torch.zeros_like(u)], -1)
    aim = aim + torch.tensor(CENTER, device="cuda")
    dirs = aim / aim.norm(dim=-1, keepdim=True)
    step = (FAR - NEAR) / T
    z = NEAR + step * (torch.arange(T, device="cuda") + torch.rand(R, T, generator=gen, device="cuda"))
    return dirs[:, None, :] * z[..., None], z.contiguous()


def _field(pts):
    """Signed distance, gradient of a bumpy sphere of 0.1 m radius at points [..., 3]."""
    q = pts - torch.tensor(CENTER, device="cuda")
    r = q.norm(dim=-1, keepdim=True).clamp_min(1e-6)
    k = torch.tensor([[70.0, 20.0, -30.0], [-25.0, 60.0, 45.0]], device="cuda")
    ph = q @ k.t()
    sdf = r[..., 0] - 0.1 - 0.004 * ph.sin().sum(-1)
    return sdf, q / r - 0.004 * ph.cos() @ k


def _amplitudes(sdf, gen):
    """Alpha-composited weights along each ray [R,T] times a reflectance in [0, 1]."""
    cdf = torch.sigmoid(sdf * 100.0)
    alpha = ((cdf[:, :-1] - cdf[:, 1:]) / (cdf[:, :-1] + 1e-5)).clamp(0.0, 1.0)
    alpha = torch.cat([alpha, alpha[:, -1:]], 1)
    trans = torch.cumprod(torch.cat([torch.ones_like(alpha[:, :1]), 1.0 - alpha + 1e-7], 1), 1)[:, :-1]
    return alpha * trans * torch.sigmoid(torch.randn(sdf.shape, generator=gen, device="cuda"))


def _ragged_points(case, gen):
    """Points of every antenna: rays U[1/4, 7/4] x rays, samples U[1/2, 3/2] x T, antenna by antenna
    (the counts are the case's own, the same for every seed)."""
    A = case["A"]
    g = torch.Generator().manual_seed(A)
    rays = (case["rays"] * (0.25 + 1.5 * torch.rand(A, generator=g))).long().clamp_min(1).tolist()
    samples = (case["T"] * (0.5 + torch.rand(A, generator=g))).long().clamp_min(2).tolist()
    pts, nrm, sig = [], [], []
    for r, t in zip(rays, samples):
        p, _ = _rays(r, t, gen)
        sdf, grad = _field(p)
        pts.append(p.reshape(-1, 3))
        nrm.append((grad / grad.norm(dim=-1, keepdim=True)).reshape(-1, 3))
        sig.append(_amplitudes(sdf, gen).reshape(-1))
    counts = torch.tensor([p.shape[0] for p in pts])
    offsets = torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)]).cuda()
    return torch.cat(pts), torch.cat(nrm), torch.cat(sig), offsets


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    st = {"case": case}
    op, S = case["op"], case["S"]
    if op == "mf":
        cfg = st["cfg"] = _cfg(S, MF_CARRIER)
        st["tx"], st["rx"] = _array(case["scan"])
        st["re"], st["im"] = _if_samples(st["tx"], st["rx"], cfg, gen)
        st["vox"] = _voxels(case["N"], 0.32 if case["scan"] > 16 else 0.2)
        if case["backward"]:
            st["gr"], st["gi"] = torch.randn(2, case["N"], generator=gen, device="cuda").unbind(0)
            st["re"].requires_grad_(True)
            st["im"].requires_grad_(True)
        return st
    if op == "tracer":
        st["cfg"] = _cfg(S, TRACER_CARRIER)
        st["tx"], st["rx"] = _pick_antennas(case["A"], gen)
        pts, _ = _rays(case["rays"], case["T"], gen)
        sdf, grad = _field(pts)
        st["points"] = pts.reshape(-1, 3).contiguous().requires_grad_(True)
        st["normals"] = (grad / grad.norm(dim=-1, keepdim=True)).reshape(-1, 3).contiguous().requires_grad_(True)
        sig = _amplitudes(sdf, gen).reshape(1, -1)
        st["sigmas"] = sig.repeat(case["A"], 1).contiguous().requires_grad_(True)
        st["inb"] = torch.rand(sig.shape[1], generator=gen, device="cuda") < 0.97
    elif op == "ragged":
        st["cfg"] = _cfg(S, TRACER_CARRIER)
        st["tx"], st["rx"] = _pick_antennas(case["A"], gen)
        pts, nrm, sig, st["offsets"] = _ragged_points(case, gen)
        st["points"], st["normals"], st["sigmas"] = (t.requires_grad_(True) for t in (pts, nrm, sig))
    elif op == "resample":
        A, R, T = case["A"], case["rays"], case["T"]
        pts, st["z"] = _rays(R, S, gen)
        sdf, grad = _field(pts)
        st["normals"] = (grad / grad.norm(dim=-1, keepdim=True)).contiguous().requires_grad_(True)
        st["sigmas"] = _amplitudes(sdf, gen).repeat(A, 1, 1).contiguous().requires_grad_(True)
        _, st["tz"] = _rays(R, T, gen)
        st["gn"] = torch.randn(R, T, 3, generator=gen, device="cuda")
        st["gs"] = torch.randn(A, R, T, generator=gen, device="cuda")
        return st
    else:  # stage1
        R, T = case["rays"], case["T"]
        cfg = st["cfg"] = _cfg(S, MF_CARRIER)
        tx, rx = _pick_antennas(case["A"], gen)
        st["bank"] = AntennaBank(tx, rx, case["bank"], S)
        scale = 1e-2  # the size of a rendered chunk's samples
        st["bank"].fill(lambda t, r: tuple(scale * x for x in _if_samples(t, r, cfg, gen)))
        z = (NEAR + (FAR - NEAR) * torch.rand(R, case["coarse"], generator=gen, device="cuda")).sort(1).values
        tgt, tz = _rays(R, T, gen)
        dirs = tgt / tgt.norm(dim=-1, keepdim=True)
        sdf, grad = _field(dirs[:, :1] * z[..., None])
        st["z"], st["tz"], st["tgt"] = z.contiguous(), tz, tgt.contiguous()
        st["gradients"] = grad.contiguous().requires_grad_(True)
        st["sigmas"] = _amplitudes(sdf, gen).contiguous().requires_grad_(True)
        st["cot"] = torch.randn(R * T, generator=gen, device="cuda")
        return st
    st["gr"], st["gi"] = torch.randn(2, case["A"], S, generator=gen, device="cuda").unbind(0)
    return st


# ---- one pass ---------------------------------------------------------------------------------

def run(st):
    case, op = st["case"], st["case"]["op"]
    if op == "mf":
        y = base_matched_filter(st["re"], st["im"], st["tx"], st["rx"], st["vox"], st["cfg"],
                                precision=case["precision"])
        if not case["backward"]:
            return y
        return y + torch.autograd.grad(y, (st["re"], st["im"]), (st["gr"], st["gi"]))
    if op == "tracer":
        x = lensless_ray_tracer(st["normals"], st["sigmas"], st["points"], st["tx"], st["rx"], st["cfg"],
                                inbounds=st["inb"], precision=case["precision"])
        return x + torch.autograd.grad(x, (st["normals"], st["sigmas"], st["points"]), (st["gr"], st["gi"]))
    if op == "ragged":
        cfg = st["cfg"]
        x = signal_tracer_ragged(st["normals"], st["sigmas"], st["points"], st["offsets"], st["tx"], st["rx"],
                                 cfg["numADCSample"], cfg["adcSampleRate"], cfg["fc_start"], cfg["As_sci"])
        return x + torch.autograd.grad(x, (st["normals"], st["sigmas"], st["points"]), (st["gr"], st["gi"]))
    if op == "resample":
        n, s, inb = bilinear_ray_sampler(st["normals"], st["sigmas"], st["z"], st["tz"])
        return (n, s, inb) + torch.autograd.grad((n, s), (st["normals"], st["sigmas"]), (st["gn"], st["gs"]))
    pred, inb = stage1_rf_prediction(st["gradients"], st["sigmas"], st["z"], st["tz"], st["tgt"], st["bank"],
                                     st["cfg"])
    return (pred, inb) + torch.autograd.grad(pred, (st["gradients"], st["sigmas"]), st["cot"])


def work(case):
    """Per (point, antenna) pair: two path lengths, the phase, its phasor and one complex
    multiply-add onto an interpolated sample sum (40 operations); per specular pair of the tracer
    (one in ten) the specular geometry and its gradients (200)."""
    S = case["S"]
    if case["op"] == "mf":
        A, N = 12 * case["scan"] ** 2, case["N"]
        passes = 2 if case["backward"] else 1
        return {"bytes": passes * (8 * A * S + 24 * A + 20 * N), "flops": passes * (40 * A * N + 8 * A * S)}
    if case["op"] in ("tracer", "ragged"):
        A = case["A"]
        P = case["rays"] * case["T"] * (A if case["op"] == "ragged" else 1)
        pairs = P if case["op"] == "ragged" else A * P
        # sigmas in and their gradients out; points and normals in, twice, and their gradients out
        return {"bytes": 8 * pairs + 73 * P + 16 * A * S, "flops": 30 * pairs + 0.1 * pairs * 300}
    if case["op"] == "resample":
        per_s, per_t = case["rays"] * S, case["rays"] * case["T"]
        channels = 3 + case["A"]
        return {"bytes": 4 * (channels * 2 * (per_s + per_t) + 2 * per_s + 2 * per_t) + per_t,
                "flops": 8 * channels * per_t}
    A, C = case["A"], case["A"] // case["bank"]
    P, Q = case["rays"] * case["T"], case["rays"] * case["coarse"]
    pairs = A * P + 3 * C * P  # matched filter, its adjoint for the chunk, tracer, its adjoint
    return {"bytes": 16 * A * S + 40 * Q + 60 * P, "flops": 40 * pairs}


# ---- the same in 64 bits ----------------------------------------------------------------------

def _f(x):
    return float(np.float32(x))


def _rates(cfg, carrier):
    w0 = 2.0 * _f(np.pi) * _f(carrier)
    w1 = 2.0 * _f(np.pi) * _f(cfg["As_sci"]) / _f(cfg["adcSampleRate"])
    return w0, w1


def _delay(tx, rx, pts):
    d = (tx - pts).norm(dim=-1) + (rx - pts).norm(dim=-1)
    return d, (d + _f(0.15)) / _f(2.9979)


def _cis(x):
    return torch.polar(torch.ones_like(x), x)


def _mf_exact(re, im, tx, rx, vox, cfg, cot=None, cot_antennas=None):
    """y [N] complex, and the adjoint [A, S] of `cot` over the first `cot_antennas` antennas."""
    w0, w1 = _rates(cfg, MF_CARRIER)
    s = torch.complex(re.detach().double(), im.detach().double())
    tx, rx, vox = tx.double(), rx.double(), vox.double()
    A, S = s.shape
    y = torch.zeros(vox.shape[0], dtype=torch.complex128, device="cuda")
    g = torch.zeros_like(s) if cot is not None else None
    step = max(1, int(2e7 // vox.shape[0]))
    for a in range(0, A, step):
        e = slice(a, min(A, a + step))
        _, tau = _delay(tx[e, None], rx[e, None], vox[None])
        base, z = _cis(w0 * tau), _cis(w1 * tau)
        acc = torch.zeros_like(base)
        zc = z.conj().resolve_conj()
        for n in range(S - 1, -1, -1):
            acc.mul_(zc).add_(s[e, n:n + 1])
        y += (acc * base.conj()).sum(0)
        if cot is not None:
            w = base * cot
            for n in range(S):
                g[e, n] = w.sum(1)
                w.mul_(z)
    return y / A, g


def _tracer_exact(nrm, sig, pts, inb, tx, rx, cfg, gr, gi, count):
    """One antenna: x [S] complex and the gradients of Re(conj(gr + j gi) x) over its points."""
    w0, w1 = _rates(cfg, cfg["fc_start"])
    S = cfg["numADCSample"]
    nrm, sig, pts = (t.detach().double().requires_grad_(True) for t in (nrm, sig, pts))

    def unit(v):
        return v / (v.norm(dim=-1, keepdim=True) + _f(1e-7))

    inc = unit(pts - tx)
    idn = (inc * nrm).sum(-1)
    rho = (unit(rx - pts) * unit(inc - 2 * idn[:, None] * nrm)).sum(-1)
    d, tau = _delay(tx, rx, pts)
    live = (inb & ~(rho < _f(1e-6)) & ~(idn > 0)).nonzero()[:, 0]
    amp, tau = (sig * rho / (d * d))[live], tau[live]
    t = torch.arange(S, device="cuda", dtype=torch.float64)
    x = torch.zeros(S, dtype=torch.complex128, device="cuda")
    g = torch.complex(gr.double(), gi.double()) / count
    d_amp, d_tau = torch.zeros_like(amp), torch.zeros_like(tau)
    with torch.no_grad():
        for i in range(0, live.numel(), 1 << 17):
            e = slice(i, i + (1 << 17))
            ph = _cis(tau[e, None] * (w0 + w1 * t))
            x += (amp[e, None] * ph).sum(0)
            gp = g.conj() * ph
            d_amp[e] = gp.real.sum(1)
            d_tau[e] = -amp[e] * (gp.imag * (w0 + w1 * t)).sum(1)
    grads = torch.autograd.grad((amp, tau), (nrm, sig, pts), (d_amp, d_tau))
    return x / count, grads


def exact(case, seed):
    op = case["op"]
    if op == "mf" and 12.0 * case["scan"] ** 2 * case["N"] * case["S"] * (2 if case["backward"] else 1) > 6e11:
        return None
    st = prepare(case, seed)
    cfg = st.get("cfg")
    if op == "mf":
        cot = torch.complex(st["gr"], st["gi"]).to(torch.complex128) if case["backward"] else None
        y, g = _mf_exact(st["re"], st["im"], st["tx"], st["rx"], st["vox"], cfg, cot)
        out = (y.real, y.imag)
        return out if g is None else out + (g.real / g.shape[0], g.imag / g.shape[0])
    if op == "tracer":
        P = st["points"].shape[0]
        x = torch.zeros(case["A"], case["S"], dtype=torch.complex128, device="cuda")
        gn, gp = (torch.zeros(P, 3, dtype=torch.float64, device="cuda") for _ in range(2))
        gs = torch.zeros(case["A"], P, dtype=torch.float64, device="cuda")
        for a in range(case["A"]):
            x[a], g = _tracer_exact(st["normals"], st["sigmas"][a], st["points"], st["inb"], st["tx"][a].double(),
                                    st["rx"][a].double(), cfg, st["gr"][a], st["gi"][a], P)
            gn += g[0]
            gs[a] = g[1]
            gp += g[2]
        return x.real, x.imag, gn, gs, gp
    if op == "ragged":
        off = st["offsets"].tolist()
        x = torch.zeros(case["A"], case["S"], dtype=torch.complex128, device="cuda")
        grads = [], [], []
        for a in range(case["A"]):
            e = slice(off[a], off[a + 1])
            n, s, p = st["normals"][e], st["sigmas"][e], st["points"][e]
            x[a], g = _tracer_exact(n, s, p, torch.ones_like(s, dtype=torch.bool), st["tx"][a].double(),
                                    st["rx"][a].double(), cfg, st["gr"][a], st["gi"][a], p.shape[0])
            for k in range(3):
                grads[k].append(g[k])
        return (x.real, x.imag) + tuple(torch.cat(g) for g in grads)
    if op == "resample":
        n, s = (st[k].detach().double().requires_grad_(True) for k in ("normals", "sigmas"))
        on, os_, inb = _resample_exact(n, s, st["z"], st["tz"])
        return (on.detach(), os_.detach(), inb) + torch.autograd.grad((on, os_), (n, s), (st["gn"].double(),
                                                                                         st["gs"].double()))
    # stage1: the prediction; its gradients are sums through every operator above, each exact on its own
    bank, unit = st["bank"], torch.nn.functional.normalize
    with torch.no_grad():
        on, os_, inb = _resample_exact(unit(st["gradients"].double(), dim=-1), st["sigmas"].double()[None], st["z"],
                                       st["tz"])
        on, sig, inb, pts = unit(on, dim=-1).reshape(-1, 3), os_.reshape(-1), inb.reshape(-1), st["tgt"].reshape(-1, 3)
    re, im = bank.real.double(), bank.imag.double()
    zero = torch.zeros(case["S"], device="cuda")
    for a in bank.sel_idx.tolist():
        x, _ = _tracer_exact(on, sig, pts, inb, bank.tx[a].double(), bank.rx[a].double(), cfg, zero, zero, sig.numel())
        re[a], im[a] = x.real, x.imag
    y, _ = _mf_exact(re, im, bank.tx, bank.rx, pts, cfg)
    return torch.sqrt(y.abs().square() + 1e-20), inb, None, None


def _resample_exact(n, s, z, tz):
    lo = (torch.searchsorted(z, tz, right=True) - 1).clamp(0, z.shape[1] - 2)
    z0, z1 = z.gather(1, lo).double(), z.gather(1, lo + 1).double()
    t = tz.double()
    inb = (t >= z0) & (t <= z1)
    wu = torch.where(inb, (t - z0) / (z1 - z0).clamp_min(_f(1e-6)), 0.0)
    wl = torch.where(inb, 1 - wu, 0.0)

    def at_n(i):
        return n.gather(1, i[..., None].expand(-1, -1, 3))

    def at_s(i):
        return s.gather(2, i[None].expand(s.shape[0], -1, -1))

    on = wl[..., None] * at_n(lo) + wu[..., None] * at_n(lo + 1)
    os_ = wl[None] * at_s(lo) + wu[None] * at_s(lo + 1)
    return on, os_, inb
