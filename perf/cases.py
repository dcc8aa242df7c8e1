"""The work a user of this framework has it do, as timed cases through its public entry points.

Families (``kind``):

* ``line``    one 1D program (``Sim1D.step``): the reference's fd1d scripts
* ``slabs``   a batch of uneven layered 1D runs with DFT probes (``BatchRunner``)
* ``tm``      one 2D TM program with a point source (``SimTM2D.step``)
* ``tfsf``    the 2D program with plane wave and running DFT (fd2d_3_4)
* ``adjoint`` objective and gradient of a 2D design box (``AdjointProblem``)
* ``serve``   transmission spectra from the neural operator (``FNO.spectrum``)
* ``train``   one minibatch step of the neural operator (loss, gradients, Adam)

A pass restarts a program's clock (``t = 0``) and runs its time loop on the
fields that the last pass left, as a program does that sends one pulse after
another.  ``exact`` restates every family in 64 bits with plain torch/numpy.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from simulation_gb300 import adjoint as A
from simulation_gb300 import batch1d as B1
from simulation_gb300 import fd1d as G1
from simulation_gb300 import fd2d as G2
from simulation_gb300 import surrogate as S

EPS0 = 8.854e-12
DT = 0.01 / 6e8
DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a short teaching line: 200 cells with a dielectric half, 1000 steps; the smallest call there is
        dict(name="line_200", kind="line", cells=200, steps=1000, form="cb", source="hard", freqs=0),
        # the fd1d_2_2 program: D form with the running DFT at every cell and an input probe
        dict(name="line_512_dft", kind="line", cells=512, steps=740, form="dform", source="soft", freqs=3),
        # the line length of the reference's own 1D benchmark programs
        dict(name="line_38000", kind="line", cells=38000, steps=4000, form="cb", source="soft", freqs=0),
        # spectra sweep: thousands of uneven slab runs, 64 frequencies at two probes
        dict(name="slabs_4096", kind="slabs", runs=4096, steps=2000, freqs=64),
        # the fd2d_3_2 program at its own size
        dict(name="tm_100", kind="tm", nx=100, ny=100, npml=8, lossy=False, steps=120),
        # the grid and layer of the reference's own 2D benchmark programs
        dict(name="tm_1024", kind="tm", nx=1024, ny=1024, npml=80, lossy=False, steps=300),
        # a grid cut to the object: neither side a multiple of anything, lossy material
        dict(name="tm_1501x1203", kind="tm", nx=1501, ny=1203, npml=20, lossy=True, steps=100),
        # the large lossy-cylinder benchmark grid
        dict(name="tm_8192", kind="tm", nx=8192, ny=8192, npml=32, lossy=True, steps=100),
        # plane wave on a lossy cylinder with a 3-frequency DFT of the whole field (fd2d_3_4, scaled up)
        dict(name="tfsf_2048", kind="tfsf", nx=2048, ny=2048, npml=8, freqs=3, steps=100),
        # permittivity gradient of a 256 x 256 design box
        dict(name="adjoint_1024", kind="adjoint", nx=1024, ny=1024, npml=16, box=256, off=40, sigma=0.0,
             steps=1500, checkpoint=64),
        # a request of 4096 profiles to the surrogate: inputs from the layer tables, network, frame
        dict(name="serve_4096", kind="serve", profiles=4096),
        # one training step of the surrogate at its own minibatch size
        dict(name="train_256", kind="train", batch=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["line", "line", "slabs", "slabs", "tm", "tm", "tm", "tfsf", "tfsf", "adjoint", "serve", "train"])
    if kind == "line":
        cells = _log(rng, 60, 60000)
        form = rng.choice(["cb", "cacb", "dform", "debye"])
        return dict(kind=kind, cells=cells, steps=rng.randint(300, 3000), form=form,
                    source=rng.choice(["hard", "soft"]), freqs=rng.choice([0, 0, 3, 5]) if cells < 4000 else 0)
    if kind == "slabs":
        return dict(kind=kind, runs=_log(rng, 16, 3000), steps=rng.randint(500, 2000), freqs=rng.choice([16, 33, 64]))
    if kind == "tm":
        nx, ny = _log(rng, 60, 7000), _log(rng, 60, 7000)
        nx, ny = max(nx, ny // 4), max(ny, nx // 4)
        ny = ny if rng.random() < 0.3 else max(60, 4 * (ny // 4))
        npml = rng.choice([0, 8, 16, 25])
        return dict(kind=kind, nx=nx, ny=ny, npml=npml, lossy=rng.random() < 0.6,
                    steps=max(30, min(rng.randint(80, 400), int(3e9 / (nx * ny)))))
    if kind == "tfsf":
        nx, ny = _log(rng, 80, 2000), _log(rng, 80, 2000)
        nx, ny = max(nx, ny // 4), max(ny, nx // 4)
        ny = ny if rng.random() < 0.3 else max(80, 4 * (ny // 4))
        return dict(kind=kind, nx=nx, ny=ny, npml=rng.choice([8, 12]), freqs=rng.choice([0, 1, 3, 6]),
                    steps=rng.randint(50, 100))
    if kind == "adjoint":
        nx, ny = rng.randint(300, 1000), 4 * rng.randint(75, 250)
        return dict(kind=kind, nx=nx, ny=ny, npml=rng.choice([8, 16]), box=rng.randint(40, 120),
                    off=rng.randint(15, 40), sigma=rng.choice([0.0, 0.01]), steps=rng.randint(600, 1000),
                    checkpoint=rng.choice([25, 32, 64]))
    if kind == "serve":
        return dict(kind=kind, profiles=_log(rng, 16, 4000))
    return dict(kind="train", batch=rng.randint(32, 255))


# ------------------------------------------------------------------ inputs
def _line_inputs(case, seed):
    """Coefficients (float64), source and wave of one 1D program."""
    r = np.random.default_rng(seed)
    n, form = case["cells"], case["form"]
    start = int(r.integers(n // 3, 2 * n // 3))
    epsr, sigma = float(r.uniform(1.5, 6.0)), float(r.uniform(0.0, 0.04))
    hi = np.arange(n) >= start
    nb = sigma * DT / EPS0
    co = {}
    if form == "cb":
        co["cb"] = np.where(hi, 0.5 / epsr, 0.5)
    elif form == "cacb":
        eaf = DT * sigma / (2 * EPS0 * epsr)
        co["ca"] = np.where(hi, (1 - eaf) / (1 + eaf), 1.0)
        co["cb"] = np.where(hi, 0.5 / (epsr * (1 + eaf)), 0.5)
    elif form == "dform":
        co["nax"] = np.where(hi, 1 / (epsr + nb), 1.0)
        co["nbx"] = np.where(hi, nb, 0.0)
    else:
        chi, tau = float(r.uniform(1.0, 3.0)), 1e-9
        co["nax"] = np.where(hi, 1 / (epsr + nb + chi * DT / tau), 1.0)
        co["nbx"] = np.where(hi, nb, 0.0)
        co["ncx"] = np.where(hi, math.exp(-DT / tau), 0.0)
        co["ndx"] = np.where(hi, chi * DT / tau, 0.0)
    wave = ("gauss", float(r.uniform(35, 55)), float(r.uniform(9, 14)))
    src_k = 5 if case["source"] == "hard" else int(r.integers(1, 6))
    freq = np.sort(r.uniform(50e6, 700e6, size=case["freqs"])) if case["freqs"] else None
    return co, wave, src_k, freq


def _tm_material(case, seed):
    """(naz, nbz) float32 maps of a lossy or lossless cylinder."""
    r = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    rad = float(r.uniform(0.12, 0.22)) * min(nx, ny)
    ci, cj = nx / 2 + float(r.uniform(-0.05, 0.05)) * nx, ny / 2 + float(r.uniform(-0.05, 0.05)) * ny
    epsr, sigma = float(r.uniform(4, 30)), float(r.uniform(0.1, 0.3))
    i = torch.arange(nx, dtype=F64, device=DEV)[:, None]
    j = torch.arange(ny, dtype=F64, device=DEV)[None, :]
    inside = ((i - ci) ** 2 + (j - cj) ** 2 <= rad * rad).to(F64)
    nb = sigma * DT / EPS0 if case.get("lossy", True) else 0.0
    naz = (1.0 / (1.0 + (epsr - 1.0) * inside + nb * inside)).float()
    nbz = (nb * inside).float() if case.get("lossy", True) else None
    return naz, nbz


def _tm_start(case, seed):
    """A smooth initial Dz (float32) and the point source of a 2D program."""
    r = np.random.default_rng([seed, 1])
    nx, ny = case["nx"], case["ny"]
    i = torch.arange(nx, dtype=F64, device=DEV)[:, None] / nx
    j = torch.arange(ny, dtype=F64, device=DEV)[None, :] / ny
    dz = torch.zeros((nx, ny), dtype=F64, device=DEV)
    for _ in range(3):
        a, fi, fj, pi, pj = (float(v) for v in r.uniform([0.02, 1, 1, 0, 0], [0.05, 6, 6, 6.28, 6.28]))
        dz += a * torch.cos(2 * math.pi * fi * i + pi) * torch.cos(2 * math.pi * fj * j + pj)
    si, sj = nx // 2 + int(r.integers(-4, 5)), ny // 2 + int(r.integers(-4, 5))
    wave = ("gauss", 20.0, float(r.uniform(5, 8))) if case.get("lossy", True) else ("sin", 0.01, float(r.uniform(1.0e9, 1.5e9)))
    return dz.float(), si, sj, wave


def _tfsf_freq(case, seed):
    r = np.random.default_rng([seed, 2])
    return np.sort(r.uniform(50e6, 700e6, size=case["freqs"])) if case["freqs"] else None


def _model_params(seed):
    """Network parameters as after some training: a nonzero output layer."""
    g = torch.Generator().manual_seed(1000 + seed)
    m = S.FNO(seed=seed % 1000, device=DEV)
    p = m.state_dict()
    p["H2"] = (torch.rand(p["H2"].shape, generator=g) * 2 - 1) / math.sqrt(p["H2"].shape[1])
    p["hb2"] = (torch.rand(p["hb2"].shape, generator=g) * 2 - 1) * 0.5
    return m, p


def _train_target(frame, seed):
    """Spectra like the frame's, off by the interfaces a network has to learn."""
    g = torch.Generator().manual_seed(2000 + seed)
    n = frame.shape[0]
    f = frame.cpu()
    re = 0.6 + 0.3 * torch.randn((n, 1), generator=g)
    im = 0.3 * torch.randn((n, 1), generator=g)
    a, b = f[:, :S.NFREQ], f[:, S.NFREQ:]
    return torch.cat([re * a - im * b, re * b + im * a], dim=1).to(DEV)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "line":
        co, wave, src_k, freq = _line_inputs(case, seed)
        extra = dict(freq=freq, dt=DT, probes=(10,), full_dft=True) if freq is not None else {}
        return case, G1.Sim1D(case["cells"], case["form"], src_kind=case["source"], src_k=src_k, wave=wave,
                              ns=case["steps"], device=DEV, **co, **extra)
    if kind == "slabs":
        batch = B1.slab_batch(case["runs"], seed=seed)
        freqs = np.linspace(100e6, 3e9, case["freqs"])
        return case, B1.BatchRunner(batch, nsteps=case["steps"], freqs=freqs, device=DEV)
    if kind == "tm":
        naz, nbz = _tm_material(case, seed)
        dz, si, sj, wave = _tm_start(case, seed)
        pml = G2.pmlparam(case["nx"], case["ny"], case["npml"], device=DEV) if case["npml"] else None
        sim = G2.SimTM2D(case["nx"], case["ny"], pml=pml, naz=naz, nbz=nbz, lossy=case["lossy"],
                         source=G2.PointSource(si, sj, wave, "hard"), ns=case["steps"], device=DEV)
        sim.dz.copy_(dz)
        return case, sim
    if kind == "tfsf":
        naz, nbz = _tm_material(case, seed)
        pml = G2.pmlparam(case["nx"], case["ny"], case["npml"], device=DEV)
        sim = G2.SimTM2D(case["nx"], case["ny"], pml=pml, naz=naz, nbz=nbz, lossy=True, tfsf_npml=case["npml"],
                         freq=_tfsf_freq(case, seed), dt=DT, ns=case["steps"], device=DEV)
        sim.dz.copy_(_tm_start(case, seed)[0])
        return case, sim
    if kind == "adjoint":
        off = case["off"]
        pr = A.AdjointProblem(nx=case["nx"], ny=case["ny"], npml=case["npml"], box=(case["box"], case["box"]),
                              src_offset=off, probe_offset=off, ns=case["steps"], checkpoint=case["checkpoint"],
                              sigma_box=case["sigma"], device=DEV)
        return case, (pr, _adjoint_eps(case, seed))
    if kind == "serve":
        model, p = _model_params(seed)
        model.load_state_dict(p)
        return case, (model, B1.slab_batch(case["profiles"], seed=seed))
    model, p = _model_params(seed)
    model.load_state_dict(p)
    x = S.device_features(B1.slab_batch(case["batch"], seed=seed), device=DEV)
    frame = S.propagation(x)
    return case, (model, x, frame, _train_target(frame, seed))


def _adjoint_eps(case, seed):
    rng = np.random.default_rng(seed)
    return torch.as_tensor(rng.uniform(1.0, 4.0, size=(case["box"], case["box"])), dtype=F64)


# ------------------------------------------------------------------ one pass
def run(state):
    case, s = state
    kind = case["kind"]
    if kind == "line":
        s.t = 0
        s.step(case["steps"])
        names = ("ex", "hy", "r_pt", "i_pt", "r_pr", "i_pr") if case["freqs"] else ("ex", "hy")
        return {k: getattr(s, k) for k in names}
    if kind == "slabs":
        s.run()
        return {"spec": s.spec, "T": s.spectrum()}
    if kind in ("tm", "tfsf"):
        s.t = 0
        s.step(case["steps"])
        names = ("dz", "ez", "iz", "hx", "hy", "ihx", "ihy", "ezi", "r_pt", "i_pt", "r_in", "i_in")
        return {k: getattr(s, k) for k in names if getattr(s, k) is not None}
    if kind == "adjoint":
        pr, eps = s
        pr.set_eps(eps)
        J = pr.forward()
        return {"J": J, "trace": pr.trace, "grad": pr.gradient_naz()}
    if kind == "serve":
        model, batch = s
        return {"T": model.spectrum(S.device_features(batch, device=DEV))}
    model, x, frame, target = s
    loss = model.loss_and_grad(x, target, relative=True, frame=frame)
    model.adam_step(lr=1e-5)
    return {"loss": loss, "grads": dict(model.g)}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "line":
        n, form, nf = case["cells"], case["form"], case["freqs"]
        coef, state, ops = {"cb": (1, 2, 5), "cacb": (2, 2, 6), "dform": (2, 4, 9), "debye": (4, 5, 13)}[form]
        return {"bytes": 4 * n * (coef + 2 * state + 4 * nf) + 4 * case["steps"] * (1 + 2 * nf),
                "flops": n * case["steps"] * (ops + 4 * nf)}
    if kind == "slabs":
        cells = case["runs"] * 10250  # mean length of the seeded runs
        return {"bytes": case["runs"] * (4.5 * 24 + 16 + 24 * case["freqs"]) + case["steps"] * 4 * (1 + 2 * case["freqs"]),
                "flops": case["steps"] * (cells * 6 + case["runs"] * 8 * case["freqs"])}
    if kind in ("tm", "tfsf"):
        n = case["nx"] * case["ny"]
        lossy, pml, nf = case.get("lossy", True), case["npml"] > 0, case.get("freqs", 0)
        fields = 3 + lossy + 2 * pml
        ops = 5 + (4 if lossy else 1) + (8 if pml else 6) + 4 * nf
        return {"bytes": 4 * n * (1 + lossy + 2 * fields + 1 + 4 * nf), "flops": n * case["steps"] * ops}
    if kind == "adjoint":
        n, b = case["nx"] * case["ny"], case["box"] ** 2
        ops = 14 + 2 * (case["sigma"] > 0)
        return {"bytes": b * (8 + 4) + 4 * n + 4 * case["steps"], "flops": case["steps"] * (3 * n * ops + 2 * b)}
    N, C, M, H, D = S.NBINS, S.WIDTH, S.MODES, S.HIDDEN, S.OUT
    layer = 2 * N * C * 2 * M + 2 * M * (2 * C) * (2 * C) + 2 * N * C * (C + 2 * M)
    flops = S.LAYERS * layer + 2 * N * C * S.CIN + 2 * C * H + 2 * H * D
    weights = S.LAYERS * (C * C + C + 2 * M * C * C) + C * (S.CIN + 1) + H * (C + 1) + D * (H + 1)
    if kind == "serve":
        n = case["profiles"]
        return {"bytes": n * (4 * D + 4.5 * 24) + 4 * weights, "flops": n * flops}
    n = case["batch"]
    return {"bytes": n * 4 * (N * S.CIN + 2 * D) + 4 * weights * 8, "flops": 3 * n * flops}


# ------------------------------------------------------------------ the same in 64 bits
def _wave(wave, t):
    if wave[0] == "gauss":
        return math.exp(-0.5 * ((t - wave[1]) / wave[2]) ** 2)
    return math.sin(2 * math.pi * wave[2] * (wave[1] / 6e8) * t)


def _line_exact(case, seed):
    co, wave, k, freq = _line_inputs(case, seed)
    n, form = case["cells"], case["form"]
    ex, hy, dx, ix, sx = (np.zeros(n) for _ in range(5))
    bc = [0.0, 0.0, 0.0, 0.0]
    if freq is not None:
        r_pt, i_pt = np.zeros((freq.size, n)), np.zeros((freq.size, n))
        r_pr, i_pr = np.zeros((1, freq.size)), np.zeros((1, freq.size))
    for t in range(1, case["steps"] + 1):
        f = ex if form in ("cb", "cacb") else dx
        curl = hy[:-1] - hy[1:]
        if form == "cb":
            f[1:] += co["cb"][1:] * curl
        elif form == "cacb":
            f[1:] = co["ca"][1:] * f[1:] + co["cb"][1:] * curl
        else:
            f[1:] += 0.5 * curl
        f[k] = _wave(wave, t) + (0.0 if case["source"] == "hard" else f[k])
        if form == "dform":
            ex[1:] = co["nax"][1:] * (dx[1:] - ix[1:])
            ix[1:] += co["nbx"][1:] * ex[1:]
        elif form == "debye":
            ex[1:] = co["nax"][1:] * (dx[1:] - ix[1:] - co["ncx"][1:] * sx[1:])
            ix[1:] += co["nbx"][1:] * ex[1:]
            sx[1:] = co["ncx"][1:] * sx[1:] + co["ndx"][1:] * ex[1:]
        if freq is not None:
            c, s = np.cos(2 * np.pi * freq * DT * t), np.sin(2 * np.pi * freq * DT * t)
            r_pr[0] += c * ex[10]
            i_pr[0] -= s * ex[10]
            r_pt += c[:, None] * ex
            i_pt -= s[:, None] * ex
        ex[0], bc[0], bc[1] = bc[0], bc[1], ex[1]
        ex[-1], bc[3], bc[2] = bc[3], bc[2], ex[-2]
        hy[:-1] += 0.5 * (ex[:-1] - ex[1:])
    out = {"ex": ex, "hy": hy}
    if freq is not None:
        out.update(r_pt=r_pt, i_pt=i_pt, r_pr=r_pr, i_pr=i_pr)
    return out


def _slabs_exact(case, seed):
    b = B1.slab_batch(case["runs"], seed=seed)  # the layer tables are the inputs
    # nothing moves more than one cell a step: cells beyond that are still zero
    W = int(min(b.ke.max(), b.src_k + case["steps"] + 8))
    R = b.nruns
    ca, cb = np.ones((R, W)), np.full((R, W), 0.5)
    for r in range(R):
        for q in range(b.layer_off[r], b.layer_off[r + 1]):
            eaf = DT * b.sigma[q] / (2 * EPS0 * b.epsr[q])
            lo, hi = int(b.layer_start[q]), int(b.layer_end[q])
            ca[r, lo:hi], cb[r, lo:hi] = (1 - eaf) / (1 + eaf), 0.5 / (b.epsr[q] * (1 + eaf))
    d = lambda a: torch.as_tensor(a, device=DEV)  # noqa: E731
    ke = d(np.minimum(b.ke, W))
    col = torch.arange(W, device=DEV)[None, :]
    live = col < ke[:, None]
    ca, cb = d(ca) * live, d(cb) * live
    hc = 0.5 * (col < ke[:, None] - 1).to(F64)
    hc[d(b.ke) > W] = 0.5
    last = d(np.nonzero(b.ke <= W)[0])
    lk = ke[last]
    rows = torch.arange(R, device=DEV)
    pin, pout = d(np.minimum(b.probe_in, W - 1)), d(np.minimum(b.probe_out, W - 1))
    seen = d((b.probe_out < W).astype(np.float64))
    freqs = d(np.linspace(100e6, 3e9, case["freqs"]))
    ex, hy = torch.zeros((R, W), dtype=F64, device=DEV), torch.zeros((R, W), dtype=F64, device=DEV)
    spec = torch.zeros((R, 4, case["freqs"]), dtype=F64, device=DEV)
    b0 = b1 = torch.zeros(R, dtype=F64, device=DEV)
    b2 = b3 = torch.zeros(last.numel(), dtype=F64, device=DEV)
    for t in range(1, case["steps"] + 1):
        ex[:, 1:] = ca[:, 1:] * ex[:, 1:] + cb[:, 1:] * (hy[:, :-1] - hy[:, 1:])
        ex[:, b.src_k] += math.exp(-0.5 * ((t - 50) / 10.0) ** 2)
        arg = 2 * math.pi * freqs * DT * t
        w = torch.stack([torch.cos(arg), -torch.sin(arg)])
        spec[:, :2] += ex[rows, pin][:, None, None] * w
        spec[:, 2:] += (ex[rows, pout] * seen)[:, None, None] * w
        e1 = ex[:, 1].clone()
        ex[:, 0] = b0
        b0, b1 = b1, e1
        if last.numel():
            e2 = ex[last, lk - 2].clone()
            ex[last, lk - 1] = b3
            b3, b2 = b2, e2
        hy[:, :-1] += hc[:, :-1] * (ex[:, :-1] - ex[:, 1:])
    T = torch.complex(spec[:, 2], spec[:, 3]) / torch.complex(spec[:, 0], spec[:, 1])
    return {"spec": spec, "T": torch.cat([T.real, T.imag], dim=1)}


def _pml64(nx, ny, npml):
    """The ten layer vectors (grade 0.33), rounded to the float32 values the program holds."""
    v = dict(fx1=np.zeros(nx), fx2=np.ones(nx), fx3=np.ones(nx), fy1=np.zeros(ny), fy2=np.ones(ny), fy3=np.ones(ny),
             gx2=np.ones(nx), gx3=np.ones(nx), gy2=np.ones(ny), gy3=np.ones(ny))
    for q in range(npml):
        xm, xn = 0.33 * ((npml - q) / npml) ** 3, 0.33 * ((npml - q - 0.5) / npml) ** 3
        for ax, n in (("x", nx), ("y", ny)):
            for at in (q, n - 2 - q):
                v["f%s1" % ax][at], v["f%s2" % ax][at], v["f%s3" % ax][at] = xn, 1 / (1 + xn), (1 - xn) / (1 + xn)
            for at in (q, n - 1 - q):
                v["g%s2" % ax][at], v["g%s3" % ax][at] = 1 / (1 + xm), (1 - xm) / (1 + xm)
    t = {k: torch.as_tensor(a.astype(np.float32).astype(np.float64), device=DEV) for k, a in v.items()}
    return {k: (a[:, None] if k[1] == "x" else a[None, :]) for k, a in t.items()}


def _tm_exact(case, seed):
    nx, ny, npml, ns = case["nx"], case["ny"], case["npml"], case["steps"]
    tfsf = case["kind"] == "tfsf"
    lossy = True if tfsf else case["lossy"]
    naz, nbz = _tm_material(case, seed)
    naz, nbz = naz.to(F64), None if nbz is None else nbz.to(F64)
    z = lambda *sh: torch.zeros(sh or (nx, ny), dtype=F64, device=DEV)  # noqa: E731
    dz, ez, hx, hy = z(), z(), z(), z()
    iz = z() if lossy else None
    p = _pml64(nx, ny, npml) if npml else None
    ihx, ihy = (z(), z()) if npml else (None, None)
    freq = _tfsf_freq(case, seed) if tfsf else None
    if tfsf:
        ezi, hxi, bc = z(ny), z(ny), [0.0, 0.0, 0.0, 0.0]
        lo, ihi, jhi = npml - 1, nx - npml, ny - npml
    dz0, si, sj, wave = _tm_start(case, seed)
    dz += dz0.to(F64)
    if freq is not None:
        r_pt, i_pt, r_in, i_in = z(freq.size, nx, ny), z(freq.size, nx, ny), z(freq.size), z(freq.size)
    if p is not None:
        gd, gc = (p["gx3"] * p["gy3"])[1:, 1:], 0.5 * (p["gx2"] * p["gy2"])[1:, 1:]
    for t in range(1, ns + 1):
        if tfsf:
            ezi[1:] += 0.5 * (hxi[:-1] - hxi[1:])
            e1, e2 = ezi[1].clone(), ezi[-2].clone()
            ezi[0], ezi[-1] = bc[0], bc[3]
            bc = [bc[1], e1, e2, bc[2]]
        curl = hy[1:, 1:] - hy[:-1, 1:] - hx[1:, 1:] + hx[1:, :-1]
        if p is not None:
            dz[1:, 1:] = gd * dz[1:, 1:] + gc * curl
        else:
            dz[1:, 1:] += 0.5 * curl
        if tfsf:
            ezi[3] = math.exp(-0.5 * ((t - 20) / 8.0) ** 2)
            dz[lo:ihi + 1, lo] += 0.5 * hxi[npml - 2]
            dz[lo:ihi + 1, jhi] -= 0.5 * hxi[jhi]
        else:
            dz[si, sj] = _wave(wave, t)
        if lossy:
            ez = naz * (dz - iz)
            iz += nbz * ez
        else:
            ez = naz * dz
        if freq is not None:
            for q, f in enumerate(freq):
                c, s = math.cos(2 * math.pi * f * DT * t), math.sin(2 * math.pi * f * DT * t)
                r_in[q] += c * ezi[6]
                i_in[q] -= s * ezi[6]
                r_pt[q] += c * ez
                i_pt[q] -= s * ez
        if tfsf:
            hxi[:-1] += 0.5 * (ezi[:-1] - ezi[1:])
        cx, cy = ez[:-1, :-1] - ez[:-1, 1:], ez[:-1, :-1] - ez[1:, :-1]
        hxv, hyv = hx[:-1, :-1], hy[:-1, :-1]
        if p is not None:
            ihx[:-1, :-1] += cx
            ihy[:-1, :-1] += cy
            fy1, fy2, fy3 = (p[k][:, :-1] for k in ("fy1", "fy2", "fy3"))
            fx1, fx2, fx3 = (p[k][:-1] for k in ("fx1", "fx2", "fx3"))
            hx[:-1, :-1] = fy3 * hxv + fy2 * (0.5 * cx + fx1 * ihx[:-1, :-1])
            hy[:-1, :-1] = fx3 * hyv - fx2 * (0.5 * cy + fy1 * ihy[:-1, :-1])
        else:
            hxv += 0.5 * cx
            hyv -= 0.5 * cy
        if tfsf:
            hx[lo:ihi + 1, npml - 2] += 0.5 * ezi[lo]
            hx[lo:ihi + 1, jhi] -= 0.5 * ezi[jhi]
            hy[npml - 2, lo:jhi + 1] -= 0.5 * ezi[lo:jhi + 1]
            hy[ihi, lo:jhi + 1] += 0.5 * ezi[lo:jhi + 1]
    out = dict(dz=dz, ez=ez, iz=iz, hx=hx, hy=hy, ihx=ihx, ihy=ihy)
    if tfsf:
        out["ezi"] = ezi
    if freq is not None:
        out.update(r_pt=r_pt, i_pt=i_pt, r_in=r_in, i_in=i_in)
    return {k: v for k, v in out.items() if v is not None}


def _adjoint_exact(case, seed):
    """Objective, probe trace and gradient by autograd through the update, one
    recomputed segment at a time."""
    nx, ny, ns, nb_ = case["nx"], case["ny"], case["steps"], case["box"]
    i0, j0 = nx // 2 - nb_ // 2, ny // 2 - nb_ // 2
    off = case["off"]
    si, sj, pi, pj = i0 - off, ny // 2, i0 + nb_ - 1 + off, ny // 2
    p = _pml64(nx, ny, case["npml"])
    gd, gc = (p["gx3"] * p["gy3"])[1:, 1:], 0.5 * (p["gx2"] * p["gy2"])[1:, 1:]
    fy1, fy2, fy3 = (p[k][:, :-1] for k in ("fy1", "fy2", "fy3"))
    fx1, fx2, fx3 = (p[k][:-1] for k in ("fx1", "fx2", "fx3"))
    nb = case["sigma"] * DT / EPS0
    box = (1.0 / (_adjoint_eps(case, seed).to(DEV) + nb)).float().to(F64).requires_grad_(True)
    nbz = torch.zeros((nx, ny), dtype=F64, device=DEV)
    nbz[i0:i0 + nb_, j0:j0 + nb_] = float(np.float32(nb))
    pad = (j0, ny - j0 - nb_, i0, nx - i0 - nb_)
    at_src = torch.zeros((nx, ny), dtype=F64, device=DEV)
    at_src[si, sj] = 1.0
    P = torch.nn.functional.pad

    def step(naz, s, t):
        dz, iz, hx, hy, ihx, ihy = s
        curl = hy[1:, 1:] - hy[:-1, 1:] - hx[1:, 1:] + hx[1:, :-1]
        dz = P(gd * dz[1:, 1:] + gc * curl, (1, 0, 1, 0)) + _wave(("gauss", 40, 12.0), t) * at_src
        ez = naz * (dz - iz) if case["sigma"] > 0 else naz * dz
        iz = iz + nbz * ez if case["sigma"] > 0 else iz
        cx, cy = ez[:-1, :-1] - ez[:-1, 1:], ez[:-1, :-1] - ez[1:, :-1]
        a, b = ihx[:-1, :-1] + cx, ihy[:-1, :-1] + cy
        hx = P(fy3 * hx[:-1, :-1] + fy2 * (0.5 * cx + fx1 * a), (0, 1, 0, 1))
        hy = P(fx3 * hy[:-1, :-1] - fx2 * (0.5 * cy + fy1 * b), (0, 1, 0, 1))
        return (dz, iz, hx, hy, P(a, (0, 1, 0, 1)), P(b, (0, 1, 0, 1))), ez[pi, pj]

    def whole(b):
        return 1.0 + P(b - 1.0, pad)

    seg = 20
    zero = torch.zeros((nx, ny), dtype=F64, device=DEV)
    s, kept, trace = (zero,) * 6, [], []
    with torch.no_grad():
        naz = whole(box)
        for t in range(1, ns + 1):
            if (t - 1) % seg == 0:
                kept.append(s)
            s, e = step(naz, s, t)
            trace.append(e)
    grad, back = torch.zeros_like(box), None
    for k in reversed(range(len(kept))):
        start = [x.detach().clone().requires_grad_(True) for x in kept.pop()]
        naz, s, J = whole(box), tuple(start), 0.0
        for t in range(k * seg + 1, min(ns, (k + 1) * seg) + 1):
            s, e = step(naz, s, t)
            J = J + e * e
        L = J if back is None else J + sum((x * g).sum() for x, g in zip(s, back))
        got = torch.autograd.grad(L, [box] + start, allow_unused=True)
        grad += got[0]
        back = [torch.zeros_like(x) if g is None else g for x, g in zip(start, got[1:])]
    trace = torch.stack(trace)
    return {"J": (trace * trace).sum(), "trace": trace, "grad": grad}


def _frame64(batch):
    """exp(-i sum of the complex wavenumbers from the entry to the exit probe), [n][2 nf]."""
    w = 2 * np.pi * S.FREQS * DT
    s, c = np.sin(w / 2), np.cos(w / 2)

    def wavenumber(epsr, sigma):
        eaf = DT * sigma / (2 * EPS0 * epsr)
        ca, cb = np.float32((1 - eaf) / (1 + eaf)).astype(float), np.float32(0.5 / (epsr * (1 + eaf))).astype(float)
        q = ((c + 1j * s) - ca * (c - 1j * s)) * s / (1j * cb)
        k = 2 * np.arcsin(np.sqrt(q + 0j))
        return np.where(k.real < 0, -k, k)

    k0 = wavenumber(1.0, 0.0)
    K = np.zeros((batch.nruns, S.NFREQ), dtype=complex)
    for r in range(batch.nruns):
        a, b = batch.layer_off[r], batch.layer_off[r + 1]
        inside = 0
        for q in range(a, b):
            d = int(batch.layer_end[q] - batch.layer_start[q])
            # the network's inputs hold the material in float32
            e = 1 + S.EPS_SCALE * float(np.float32((batch.epsr[q] - 1) / S.EPS_SCALE))
            g = S.SIG_SCALE * float(np.float32(batch.sigma[q] / S.SIG_SCALE))
            K[r] += d * wavenumber(e, g)
            inside += d
        K[r] += (int(batch.layer_end[b - 1]) + S.PROBE_GAP - S.PROBE_IN - inside) * k0
    P = np.exp(-1j * K)
    return torch.as_tensor(np.concatenate([P.real, P.imag], axis=1), device=DEV)


def _net64(p, x):
    N, M = S.NBINS, S.MODES
    th = 2 * math.pi * torch.arange(M, dtype=F64, device=DEV)[:, None] * torch.arange(N, dtype=F64, device=DEV) / N
    phi = torch.cat([torch.cos(th), -torch.sin(th)])
    a = torch.full((M, 1), 2.0 / N, dtype=F64, device=DEV)
    a[0] = 1.0 / N
    psi = (phi * torch.cat([a, a])).T
    gelu = lambda z: 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))  # noqa: E731
    x = x @ p["P"].T + p["pb"]
    for l in range(S.LAYERS):
        F = phi @ x  # [B][2M][C]
        Fr, Fi = F[:, :M].transpose(0, 1), F[:, M:].transpose(0, 1)  # [M][B][C]
        Rr, Ri = p["L%d.Rr" % l].transpose(1, 2), p["L%d.Ri" % l].transpose(1, 2)
        G = torch.cat([Fr @ Rr - Fi @ Ri, Fr @ Ri + Fi @ Rr]).transpose(0, 1)
        x = gelu(x @ p["L%d.W" % l].T + p["L%d.b" % l] + psi @ G)
    h = gelu(x.mean(dim=1) @ p["H1"].T + p["hb1"])
    return h @ p["H2"].T + p["hb2"]


def _product(P, y):
    n = S.NFREQ
    return torch.cat([P[:, :n] * y[:, :n] - P[:, n:] * y[:, n:], P[:, :n] * y[:, n:] + P[:, n:] * y[:, :n]], dim=1)


def _features64(batch):
    """(eps_r - 1)/8 of cells 2b-1, 2b, 2b+1, then sigma/0.05 of the same, as float32 values."""
    n = 2 * S.NBINS
    m = np.zeros((batch.nruns, 2, n + 2), dtype=np.float32)
    for r in range(batch.nruns):
        for q in range(batch.layer_off[r], batch.layer_off[r + 1]):
            lo, hi = int(batch.layer_start[q]) + 1, min(int(batch.layer_end[q]), n) + 1
            m[r, 0, lo:hi] = (batch.epsr[q] - 1) / S.EPS_SCALE
            m[r, 1, lo:hi] = batch.sigma[q] / S.SIG_SCALE
    m = torch.as_tensor(m, device=DEV)
    return torch.stack([m[:, c, j:j + n:2] for c in (0, 1) for j in (0, 1, 2)], dim=2)


def _serve_exact(case, seed):
    _, p = _model_params(seed)
    p = {k: v.to(DEV).to(F64) for k, v in p.items()}
    batch = B1.slab_batch(case["profiles"], seed=seed)
    x, P = _features64(batch), _frame64(batch)
    y = torch.cat([_net64(p, x[i:i + 128].to(F64)) for i in range(0, batch.nruns, 128)])
    return {"T": _product(P, y)}


def _train_exact(case, seed):
    _, p = _model_params(seed)
    p = {k: v.to(DEV).to(F64).requires_grad_(True) for k, v in p.items()}
    batch = B1.slab_batch(case["batch"], seed=seed)
    x, P = _features64(batch), _frame64(batch)
    tgt = _train_target(P.float(), seed).to(F64)
    floor2 = S.SPECTRUM_FLOOR ** 2 * S.NFREQ
    w = 1.0 / torch.clamp((tgt ** 2).sum(1), min=floor2) / batch.nruns
    loss, grads = 0.0, {k: torch.zeros_like(v) for k, v in p.items()}
    for i in range(0, batch.nruns, 32):
        o = _product(P[i:i + 32], _net64(p, x[i:i + 32].to(F64)))
        L = (w[i:i + 32] * ((o - tgt[i:i + 32]) ** 2).sum(1)).sum()
        for k, g in zip(p, torch.autograd.grad(L, list(p.values()))):
            grads[k] += g
        loss += L.detach()
    # the imaginary mode weights of the last layers have gradients that are small differences of
    # large terms: 16-bit activations leave too little of them to be held against 64 bits
    for l in range(2, S.LAYERS):
        grads["L%d.Ri" % l] = None
    return {"loss": loss.reshape(1), "grads": grads}


def exact(case, seed):
    return {"line": _line_exact, "slabs": _slabs_exact, "tm": _tm_exact, "tfsf": _tm_exact, "adjoint": _adjoint_exact,
            "serve": _serve_exact, "train": _train_exact}[case["kind"]](case, seed)
