"""Performance cases: what a program does with this framework, through its
public entry points, over the range of sizes it is used at.

Kinds of case (``case["kind"]``):

* ``step``     one time step of an equation module (``equations2d.*._time_step``)
               and its backward: what a program with a time loop of its own calls;
* ``forward``  a whole forward modelling, ``build_model -> WaveRNN.forward``;
* ``gradient`` an FWI / LSRTM gradient: ``WaveRNN.forward -> L2 -> backward``;
* ``uneven``   several grids of different shapes, shots and trace lengths
               replayed as one plan (``engine.UnevenBatch``);
* ``net``      the learned preconditioner, one prediction or one training step
               (``learned.PrecondNet``).

Models are smooth random fields of the values the equations are used with,
observed data are band-limited direct arrivals plus noise, sources and
receivers lie on row 2 of the interior.  ``exact`` restates every path in
float64 with plain torch.
"""
import math

import numpy as np
import torch

DEV = "cuda"
W = 50  # boundary width of every configuration

# The C1-C5 shapes of the benchmark, at trace lengths of a fraction of a second
_LISTED = [
    # a program with a time loop of its own: one HABC step and its VJP, small grid, two shots
    dict(name="step_habc", kind="step", eq="acoustic_habc", nz=128, nx=256, shots=2, order=2, multiple=False),
    # forward modelling of a small survey (benchmark configuration 1): latency and launches count
    dict(name="forward_small", kind="forward", eq="acoustic", nz=128, nx=256, shots=8, nt=1000, order=4,
         multiple=False, rec_step=1),
    # viscoacoustic modelling, the spectral damping term on a large grid with a prime factor in its width
    dict(name="forward_viscoacoustic", kind="forward", eq="vacoustic_habc", nz=400, nx=1000, shots=16, nt=60, order=2,
         multiple=False, rec_step=1),
    # a batch of uneven grids and trace lengths (benchmark configuration 4, fewer shots), replayed plan
    dict(name="forward_uneven", kind="uneven", nz=200, nx=400, shots=16, nt=240, order=8),
    # the benchmark's headline: L2 gradient of 64 shots, 8th order, boundary saving (configuration 2)
    dict(name="gradient_pml", kind="gradient", eq="acoustic", nz=400, nx=1000, shots=64, nt=160, order=8,
         multiple=False, rec_step=1, illum=False),
    # the FWI loop's gradient with source illumination (configuration 5's survey)
    dict(name="gradient_illumination", kind="gradient", eq="acoustic", nz=256, nx=512, shots=32, nt=200, order=4,
         multiple=False, rec_step=1, illum=True),
    # one shot on an odd grid with a free surface: the smallest gradient of an inversion
    dict(name="gradient_one_shot", kind="gradient", eq="acoustic", nz=151, nx=301, shots=1, nt=400, order=4,
         multiple=True, rec_step=3, illum=False),
    # elastic gradient in (vp, vs, rho), two-component receivers (configuration 3)
    dict(name="gradient_elastic", kind="gradient", eq="elastic", nz=300, nx=800, shots=32, nt=80, order=2,
         multiple=False, rec_step=1, illum=False),
    # acoustic gradient with the hybrid absorbing boundary
    dict(name="gradient_habc", kind="gradient", eq="acoustic_habc", nz=400, nx=1000, shots=64, nt=100, order=2,
         multiple=False, rec_step=1, illum=False),
    # LSRTM gradient (Born modelling), half the shots, an odd grid
    dict(name="gradient_born", kind="gradient", eq="acoustic_lsrtm_habc", nz=333, nx=901, shots=24, nt=100, order=2,
         multiple=False, rec_step=2, illum=False),
    # the preconditioner inside an inversion: one prediction on the inversion grid
    dict(name="net_predict", kind="net", train=False, nz=256, nx=512, shots=1),
    # one training step of the preconditioner, batch 8
    dict(name="net_train", kind="net", train=True, nz=256, nx=512, shots=8),
]

# inverted parameters, fields and receiver channels of each equation
_EQS = {
    "acoustic": dict(models=("vp",), inv=("vp",), src=["h1"], rec=["h1"]),
    "acoustic_habc": dict(models=("vp",), inv=("vp",), src=["h1"], rec=["h1"]),
    "acoustic_lsrtm_habc": dict(models=("vp", "m"), inv=("m",), src=["h1"], rec=["sh1"]),
    "vti_habc2": dict(models=("vp", "epsilon", "delta"), inv=("vp", "epsilon", "delta"), src=["p1"], rec=["p1"]),
    "acoustic_rho_habc": dict(models=("vp", "rho"), inv=("vp", "rho"), src=["h1"], rec=["h1"]),
    "vacoustic_habc": dict(models=("vp", "Q"), inv=(), src=["h1"], rec=["h1"]),
    "elastic": dict(models=("vp", "vs", "rho"), inv=("vp", "vs", "rho"), src=["txx", "tzz"], rec=["vx", "vz"]),
}
_SECOND_ORDER = ("vti_habc2", "acoustic_rho_habc", "elastic", "acoustic_lsrtm_habc")  # used at order 2


def listed():
    return [dict(c) for c in _LISTED]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "forward", "forward", "gradient", "gradient", "gradient", "uneven", "net"])
    if kind == "net":
        return dict(kind="net", train=rng.random() < 0.5, nz=8 * rng.randint(8, 48), nx=rng.choice([512, 1024]),
                    shots=rng.choice([1, 2, 3, 4]))
    if kind == "uneven":
        return dict(kind="uneven", nz=rng.randint(90, 260), nx=rng.randint(150, 520), shots=_log(rng, 2, 24),
                    nt=rng.randint(60, 240), order=rng.choice([2, 4, 6, 8]))
    nz, nx = _log(rng, 60, 450), _log(rng, 110, 1200)
    if kind == "step":
        eq = rng.choice(["acoustic", "acoustic_habc", "vti_habc2", "acoustic_rho_habc", "vacoustic_habc", "elastic"])
    elif kind == "forward":
        eq = rng.choice(["acoustic", "acoustic_habc", "vacoustic_habc", "vti_habc2", "elastic"])
    else:
        eq = rng.choice(["acoustic", "acoustic", "acoustic_habc", "acoustic_lsrtm_habc", "vti_habc2",
                         "acoustic_rho_habc", "elastic"])
    shots = _log(rng, 1, 4 if kind == "step" else 64)
    order = 2 if eq in _SECOND_ORDER or kind == "step" else rng.choice([2, 4, 6, 8])
    c = dict(kind=kind, eq=eq, nz=nz, nx=nx, shots=shots, order=order, multiple=rng.random() < 0.3)
    if kind != "step":
        pts = shots * (nz + 2 * W) * (nx + 2 * W)
        top = {"elastic": 6e8, "vacoustic_habc": 4e8}.get(eq, 2e9)
        c.update(nt=max(40, min(_log(rng, 60, 600), int(top / pts))), rec_step=rng.choice([1, 1, 2, 5]))
        if kind == "gradient":
            c["illum"] = eq in ("acoustic", "elastic") and rng.random() < 0.5
    return c


# ------------------------------------------------------------------ inputs ---

def _smooth_field(gen, nz, nx, sigma):
    """Gaussian-smoothed white noise scaled to [0, 1] (float64, CPU)."""
    f = torch.fft.rfft2(torch.randn(nz, nx, generator=gen, dtype=torch.float64))
    kz = torch.fft.fftfreq(nz, dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(nx, dtype=torch.float64)[None]
    f = f * torch.exp(-2.0 * (math.pi * sigma) ** 2 * (kz ** 2 + kx ** 2))
    f = torch.fft.irfft2(f, s=(nz, nx))
    return (f - f.min()) / (f.max() - f.min())


def _sampling(case):
    """(dt, h, peak frequency) of the equation's configurations."""
    return (0.0005, 5.0, 40.0) if case["eq"] == "elastic" else (0.001, 10.0, 20.0)


def _models(case, gen):
    nz, nx, eq = case["nz"], case["nx"], case["eq"]
    f = _smooth_field(gen, nz, nx, 12.0)
    if eq == "elastic":
        vp = 2000.0 + 2600.0 * f
        return {"vp": vp, "vs": vp / 1.73, "rho": 310.0 * vp ** 0.25}
    vp = 1500.0 + (3000.0 if eq.startswith("acoustic") else 2000.0) * f
    out = {"vp": vp}
    if eq == "acoustic_lsrtm_habc":
        out["m"] = 0.2 * (_smooth_field(gen, nz, nx, 4.0) - 0.5)
    if eq == "vti_habc2":
        out["epsilon"] = 0.05 + 0.15 * _smooth_field(gen, nz, nx, 12.0)
        out["delta"] = 0.02 + 0.08 * _smooth_field(gen, nz, nx, 12.0)
    if eq == "acoustic_rho_habc":
        out["rho"] = 310.0 * vp ** 0.25
    if eq == "vacoustic_habc":
        out["Q"] = 40.0 + 100.0 * f
    return out


def _ricker(fm, dt, nt):
    c = np.pi * fm * (np.arange(nt) * dt - int(1.0 / fm / dt) * dt)
    return torch.from_numpy(((1 - 2 * c ** 2) * np.exp(-c ** 2)).astype(np.float32))


def _survey(case):
    """Interior grid columns of the sources and of the receivers, and their row."""
    xs = np.linspace(0, case["nx"] - 1, case["shots"] + 2)[1:-1].round().astype(int).tolist()
    return xs, list(range(0, case["nx"], case["rec_step"])), 2


def _observed(case, gen, nch):
    """Direct arrivals at one velocity per shot, and noise: (shots, nt, nrec, nch) float32 on the CPU."""
    dt, h, fm = _sampling(case)
    xs, rx, _ = _survey(case)
    t = torch.arange(case["nt"], dtype=torch.float64) * dt
    out = torch.empty(len(xs), case["nt"], len(rx), nch)
    v = 1600.0 + 800.0 * torch.rand(len(xs), generator=gen, dtype=torch.float64)
    r = torch.tensor(rx, dtype=torch.float64)
    for b, x in enumerate(xs):
        d = (r - x).abs() * h
        arg = (math.pi * fm) ** 2 * (t[:, None] - 1.0 / fm - d[None] / v[b]) ** 2
        w = (1 - 2 * arg) * torch.exp(-arg) / torch.sqrt(1.0 + d / h)[None]
        out[b] = w[..., None].float()
    return out + 0.01 * torch.randn(out.shape, generator=gen)


def _fields(case, gen, n):
    """Smooth wavefields of unit size, (n, shots, padded grid) float32 on the CPU."""
    nz, nx = _padded(case)
    f = torch.empty(n, case["shots"], nz, nx)
    for k in range(n):
        for b in range(case["shots"]):
            f[k, b] = (2.0 * _smooth_field(gen, nz, nx, 2.0) - 1.0).float()
    return f


def _padded(case):
    return case["nz"] + (W if case["multiple"] else 2 * W), case["nx"] + 2 * W


def _pad(case, m):
    """Edge padding by the boundary width (none on top with ``multiple``)."""
    return torch.nn.functional.pad(m[None, None], (W, W, 0 if case["multiple"] else W, W), mode="replicate")[0, 0]


def _gen(seed):
    return torch.Generator().manual_seed(1000003 * (seed % 1000003) + 17)


def _uneven_groups(case):
    """Four grids of growing size, shots and trace length."""
    return [(case["nz"] * s // 4, case["nx"] * s // 4, max(1, case["shots"] * k // 4), case["nt"] * n // 8)
            for s, k, n in ((4, 4, 4), (6, 4, 6), (7, 3, 7), (9, 2, 8))]


def _uneven_case(case, nz, nx, shots, nt):
    return dict(eq="acoustic", nz=nz, nx=nx, shots=shots, nt=nt, order=case["order"], multiple=False, rec_step=1)


def _net_inputs(case, gen):
    """Normalised gradient and illumination panels and model updates: (x, target) float32 on the CPU."""
    B, nz, nx = case["shots"], case["nz"], case["nx"]
    x, y = torch.empty(B, 2, nz, nx), torch.empty(B, nz, nx)
    depth = torch.linspace(1.0, 0.02, nz, dtype=torch.float64)[:, None]
    for b in range(B):
        g = (2.0 * _smooth_field(gen, nz, nx, 3.0) - 1.0) * depth
        p = depth ** 2 * (0.5 + _smooth_field(gen, nz, nx, 10.0))
        x[b, 0], x[b, 1] = (g / g.abs().max()).float(), (p / p.max()).float()
        y[b] = (0.6 * (_smooth_field(gen, nz, nx, 6.0) - 0.5)).float()
    return x, y


# ----------------------------------------------------------------- the work ---

def _damping(case):
    from seistorch_gb300.habc import generate_habc_coefficients_2d
    from seistorch_gb300.pml import generate_pml_coefficients_2d
    make = generate_habc_coefficients_2d if case["eq"].endswith(("habc", "habc2")) else generate_pml_coefficients_2d
    return make(_padded(case), W, multiple=case["multiple"]).to(DEV, torch.float32)


def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "net":
        from seistorch_gb300.learned import PrecondNet
        x, y = _net_inputs(case, gen)
        return dict(case=case, x=x.to(DEV), y=y.to(DEV), net=PrecondNet(torch.device(DEV), seed=seed % 997))
    if kind == "uneven":
        from seistorch_gb300 import engine
        dt, h, fm = 0.001, 10.0, 20.0
        groups = []
        for nz, nx, shots, nt in _uneven_groups(case):
            c = _uneven_case(case, nz, nx, shots, nt)
            vp = _pad(c, _models(c, gen)["vp"]).float().to(DEV)
            xs, rx, row = _survey(c)
            prop = engine.AcousticPropagator(*_padded(c), dt, h, c["order"], "pml", W, False, DEV)
            acq = engine.Acquisition(*_padded(c), [[(row + W, x + W)] for x in xs],
                                     [([row + W] * len(rx), [x + W for x in rx])] * len(xs), _ricker(fm, dt, nt), DEV)
            groups.append((prop, vp, _damping(c), acq))
        return dict(case=case, batch=engine.UnevenBatch(groups).plan())
    eq = _EQS[case["eq"]]
    dt, h, fm = _sampling(case)
    if kind == "step":
        import importlib
        module = importlib.import_module("seistorch_gb300.equations2d." + case["eq"])
        models = {k: _pad(case, v).float().to(DEV).requires_grad_(True) for k, v in _models(case, gen).items()}
        nf = 5 if case["eq"] == "elastic" else 2
        f = _fields(case, gen, 2 * nf).to(DEV)
        habcs = None
        if case["eq"] != "elastic" and case["eq"] != "acoustic":
            from seistorch_gb300.habc import bound_mask
            habcs = bound_mask(*_padded(case), W, DEV, case["shots"], return_idx=True, multiple=case["multiple"])
        return dict(case=case, step=module._time_step, models=list(models.values()),
                    fields=[f[i].contiguous().requires_grad_(True) for i in range(nf)],
                    cot=[f[nf + i].contiguous() for i in range(nf)], dt=torch.tensor(dt), h=torch.tensor(h),
                    d=_damping(case), habcs=habcs)
    from seistorch_gb300 import build_model
    models = {k: v.numpy() for k, v in _models(case, gen).items()}
    inv = eq["inv"] if kind == "gradient" else ()
    cfg = {"equation": case["eq"], "dtype": "float32",
           "geom": {"dt": dt, "h": h, "nt": case["nt"],
                    "boundary": {"type": "habc" if case["eq"].endswith(("habc", "habc2")) else "pml", "width": W},
                    "multiple": case["multiple"], "boundary_saving": True, "source_type": eq["src"],
                    "receiver_type": eq["rec"], "spatial_order": case["order"],
                    "source_illumination": bool(case.get("illum", False)), "invlist": {k: k in inv for k in models}}}
    _, model = build_model(cfg, device=DEV, mode="inversion" if inv else "forward", models=models)
    xs, rx, row = _survey(case)
    model.reset_geom(list(range(len(xs))), [[x, row] for x in xs], [[rx, [row] * len(rx)]] * len(xs), cfg)
    s = dict(case=case, model=model, wav=_ricker(fm, dt, case["nt"])[None].to(DEV))
    if kind == "gradient":
        s["obs"] = _observed(case, gen, len(eq["rec"])).to(DEV)
        s["params"] = [getattr(model.cell.geom, k) for k in inv]
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "net":
        net = state["net"]
        if not case["train"]:
            return {"pred": net.predict(state["x"])}
        loss = net.train_batch(state["x"], state["y"], 1e-4)
        return {"loss": loss, "grads": net.grads, "params": net.params}
    if kind == "uneven":
        return state["batch"].replay()
    if kind == "step":
        ins = state["models"] + state["fields"]
        out = state["step"](*ins, state["dt"], state["h"], state["d"], habcs=state["habcs"])
        n = 5 if case["eq"] == "elastic" else 1
        grads = torch.autograd.grad(out[:n], ins, state["cot"][:n], allow_unused=True)
        return {"out": [o.detach() for o in out[:n]], "grads": [g for g in grads if g is not None]}
    model = state["model"]
    if kind == "forward":
        with torch.no_grad():
            y = model(state["wav"])
        return {"records": torch.stack(list(y.data))}
    from seistorch_gb300.postprocess import L2
    for p in state["params"]:
        p.grad = None
    y = model(state["wav"])
    syn = torch.stack(list(y.data))
    loss = L2()(syn, state["obs"])
    loss.backward()
    out = {"records": syn.detach(), "loss": loss.detach(), "grads": [p.grad for p in state["params"]]}
    if case["illum"]:
        out["illum"] = model.precondition
    return out


def work(case):
    kind = case["kind"]
    if kind == "net":
        layers = [(2, 32, 0), (32, 32, 0), (32, 64, 1), (64, 64, 1), (64, 128, 2), (128, 128, 2), (128, 256, 3),
                  (384, 128, 2), (192, 64, 1), (96, 32, 0), (32, 1, 0)]
        pix = case["shots"] * case["nz"] * case["nx"]
        fl = sum(18.0 * ci * co * pix / 4 ** l for ci, co, l in layers)
        by = sum(2.0 * (ci + co) * pix / 4 ** l for ci, co, l in layers)  # bf16 activations in and out
        if not case["train"]:
            return {"bytes": by, "flops": fl}
        return {"bytes": 3.0 * by, "flops": 3.0 * fl}  # data and weight gradients read them again
    if kind == "uneven":
        pts = sum(s * (z + 2 * W) * (x + 2 * W) * t for z, x, s, t in _uneven_groups(case))
        return {"bytes": 12.0 * pts, "flops": (4.5 * case["order"] + 4) * pts}
    nz, nx = _padded(case)
    plane, pts = nz * nx, case["shots"] * nz * nx
    lap = 4.5 * case["order"] + 4  # Laplacian and update
    # per point and step: bytes of the fields read and written, flops; coefficient planes
    fwd, ffl, coef = {"acoustic": (12, lap, 2), "acoustic_habc": (12, lap, 1), "vti_habc2": (12, lap + 2, 2),
                      "acoustic_rho_habc": (12, 18, 5), "acoustic_lsrtm_habc": (24, 2 * lap, 2),
                      "vacoustic_habc": (12, lap + 10 * math.log2(plane), 2), "elastic": (40, 40, 6)}[case["eq"]]
    if kind == "step":
        nm = len(_EQS[case["eq"]]["models"])
        n = 5 if case["eq"] == "elastic" else 2
        # forward: fields in, new fields out; backward: fields and cotangents in, gradients out
        by = 4.0 * (pts * (3 * n + (5 if n == 5 else 1) + (5 if n == 5 else 1)) + plane * (2 * coef + nm))
        return {"bytes": by, "flops": 3.0 * ffl * pts}
    nrec = len(range(0, case["nx"], case["rec_step"])) * case["shots"] * len(_EQS[case["eq"]]["rec"])
    by, fl = (fwd * pts + 4 * coef * plane + 4 * nrec) * case["nt"], ffl * pts * case["nt"]
    if kind == "gradient":
        # reconstruction and adjoint: each field's two (elastic: one) old states in, the new one out
        by += ({"elastic": 80}.get(case["eq"], 24) * pts + 4 * coef * plane + 8 * nrec) * case["nt"]
        fl += 2.5 * ffl * pts * case["nt"]
    return {"bytes": float(by), "flops": float(fl)}


# ------------------------------------------------------- the same in 64 bits ---

class _Shift(torch.autograd.Function):
    """y[i] = x[i + n] along ``dim`` with zeros outside; the adjoint shifts back."""

    @staticmethod
    def forward(ctx, x, dim, n):
        ctx.dim, ctx.n = dim, n
        y = torch.zeros_like(x)
        L = x.shape[dim]
        if abs(n) < L:
            y.narrow(dim, max(0, -n), L - abs(n)).copy_(x.narrow(dim, max(0, n), L - abs(n)))
        return y

    @staticmethod
    def backward(ctx, g):
        return _Shift.apply(g, ctx.dim, -ctx.n), None, None


def _weights(order):
    return {2: [1.0], 4: [4 / 3, -1 / 12], 6: [3 / 2, -3 / 20, 1 / 90], 8: [8 / 5, -1 / 5, 8 / 315, -1 / 560]}[order]


def _second(x, dim, order):
    c = _weights(order)
    y = (-2.0 * sum(c)) * x
    L = x.shape[dim]
    for j, w in enumerate(c, 1):
        if j < L:
            y.narrow(dim, 0, L - j).add_(x.narrow(dim, j, L - j), alpha=w)
            y.narrow(dim, j, L - j).add_(x.narrow(dim, 0, L - j), alpha=w)
    return y


class _Second(torch.autograd.Function):
    """Central second difference with zeros outside (its own transpose)."""

    @staticmethod
    def forward(ctx, x, dim, order):
        ctx.dim, ctx.order = dim, order
        return _second(x, dim, order)

    @staticmethod
    def backward(ctx, g):
        return _second(g, ctx.dim, ctx.order), None, None


def _lap(u, order):
    return _Second.apply(u, -2, order) + _Second.apply(u, -1, order)


def _pml64(case):
    nz, nx = _padded(case)
    d0 = (1.5 * 1500.0 / W) * 4.0
    ramp = d0 * (1.0 - torch.arange(W + 1, dtype=torch.float64) / W) ** 2
    dz, dx = torch.zeros(nz, nx, dtype=torch.float64), torch.zeros(nz, nx, dtype=torch.float64)
    dx[:, :W + 1] = ramp
    dx[:, nx - W - 1:] = ramp.flip(0)
    if not case["multiple"]:
        dz[:W + 1] = ramp[:, None]
    dz[nz - W - 1:] = ramp.flip(0)[:, None]
    return torch.sqrt(dz ** 2 + dx ** 2).to(DEV)


def _habc64(case):
    """Blend weight b and the four sides' shares (top, bottom, left, right) of every cell."""
    nz, nx = _padded(case)
    mult = case["multiple"]
    z, x = torch.arange(nz)[:, None].expand(nz, nx), torch.arange(nx)[None].expand(nz, nx)
    dT, dB, dL, dR = z, nz - 1 - z, x, nx - 1 - x
    top = (dT < W) & (dT <= dL) & (dT <= dR) & (not mult)
    bot = (dB < W) & (dB <= dL) & (dB <= dR)
    side = lambda d: (d < W) & ((mult & (z < W)) | (((z >= W) | (d <= z)) & ((dB >= W) | (d <= dB))))
    lft, rgt = side(dL), side(dR)
    b = torch.zeros(nz, nx, dtype=torch.float64)
    for m, d in ((top, dT), (bot, dB), (lft, dL), (rgt, dR)):
        b = torch.where(m, (W - 1 - d).double() / (W - 1), b)
    one = lambda *v: torch.tensor(v, dtype=torch.float64)[:, None, None]
    S = torch.zeros(4, nz, nx, dtype=torch.float64)
    rules = [(top, (1, 0, 0, 0)), (bot, (0, 1, 0, 0)), (lft, (0, 0, 1, 0)), (rgt, (0, 0, 0, 1)),
             ((z < W) & (x == z) & (not mult), (.5, 0, .5, 0)), ((z < W) & (x == nx - W + z) & (not mult), (.5, 0, 0, .5)),
             ((z >= nz - W) & (x == z - (nz - W)), (0, .5, .5, 0)),
             ((z >= nz - W) & (x == nx - W + z - (nz - W)), (0, .5, 0, .5))]
    for m, v in rules:
        S = torch.where(m, one(*v), S)
    return b.to(DEV), S.to(DEV)


class _Habc:
    """The one-way blend of the four strips (depth k cells use their two inward neighbours; the last one the edge cell)."""

    def __init__(self, case, dt, h):
        self.b, self.S = _habc64(case)
        self.l, self.m = 2.0 * dt / h, dt * dt / (h * h)
        self.wi = 1.0 - self.b * self.S.sum(0)

    def __call__(self, y, u, um, vp):
        nz, nx = y.shape[-2:]
        out = self.wi * y
        for s, (dim, n, last) in enumerate(((-2, nz, 0), (-2, nz, 1), (-1, nx, 0), (-1, nx, 1))):
            if not bool((self.S[s] != 0).any()):
                continue
            ax = lambda t: (t.flip(dim) if last else t).narrow(dim, 0, W + 1)
            U, P, c = ax(u), ax(um), ax(vp).narrow(dim, 0, W)
            U0, U1 = U.narrow(dim, 0, W), U.narrow(dim, 1, W)
            U2 = torch.cat([U.narrow(dim, 2, W - 1), U.narrow(dim, 0, 1)], dim)
            P0, P1 = P.narrow(dim, 0, W), P.narrow(dim, 1, W)
            lam, mu = c * self.l, c * c * self.m
            o = (2.0 - lam - mu) * U0 + (lam + 2.0 * mu) * U1 - mu * U2 + (lam - 1.0) * P0 - lam * P1
            o = ax(self.b * self.S[s]).narrow(dim, 0, W) * o
            pad = (0, 0, 0, n - W) if dim == -2 else (0, n - W)
            o = torch.nn.functional.pad(o, pad)
            out = out + (o.flip(dim) if last else o)
        return out


class _Exact:
    """One equation's step in float64: state tuple -> state tuple; ``src`` / ``rec``: indices of its fields."""

    def __init__(self, case, models, dt, h):
        self.eq, self.order, self.dt, self.h = case["eq"], case["order"], dt, h
        self.v = {k: m for k, m in models.items()}
        vp, r2 = self.v["vp"], (dt / h) ** 2
        nz, nx = _padded(case)
        self.nf, self.src, self.rec = 2, (0,), (0,)
        if self.eq == "acoustic":
            d = _pml64(case)
            self.g, self.k = 2.0 / (1.0 + d * dt), vp ** 2 * r2 / (1.0 + d * dt)
        elif self.eq == "elastic":
            self.nf, self.src, self.rec = 5, (2, 3), (0, 1)
            c = 0.5 * dt * _pml64(case)
            self.q, e = (1.0 - c) / (1.0 + c), dt / (h * (1.0 + c))
            vs, rho = self.v["vs"], self.v["rho"]
            lam, mu = rho * (vp ** 2 - 2 * vs ** 2), rho * vs ** 2
            self.pa, self.la, self.ma, self.bv = e * (lam + 2 * mu), e * lam, e * mu, e / rho
        else:
            self.blend = _Habc(case, dt, h)
            self.k = vp ** 2 * r2
        if self.eq == "acoustic_lsrtm_habc":
            self.nf, self.rec = 4, (2,)
        if self.eq == "vti_habc2":
            fx = torch.fft.fftfreq(nz, d=h, dtype=torch.float64, device=DEV)[:, None]
            fz = torch.fft.fftfreq(nx, d=h, dtype=torch.float64, device=DEV)[None]
            e, dl = self.v["epsilon"], self.v["delta"]
            sk = -2.0 * (e - dl) * fx ** 2 * fz ** 2 / ((1 + 2 * e) * fx ** 4 + fz ** 4 + 2 * (1 + dl) * fx ** 2 * fz ** 2
                                                        + 1e-26)
            self.kx, self.kz = self.k * (1 + 2 * e + sk), self.k * (1 + sk)
        if self.eq == "acoustic_rho_habc":
            rho = self.v["rho"]
            b = 1.0 / rho
            self.C = r2 * rho * vp ** 2
            self.bh = [(b + _Shift.apply(b, dim, n)) / 2 for dim, n in ((-1, 1), (-1, -1), (-2, 1), (-2, -1))]
        if self.eq == "vacoustic_habc":
            Q, om = self.v["Q"], 16.5
            ts = (torch.sqrt(1.0 + Q ** -2) - Q ** -1) / om
            t = (om ** 2 * ts) ** -1 / (ts - 1e-8) - 1.0
            self.k = self.k * (1.0 - (1.0 - torch.sqrt(Q ** 2 + 1.0)) * Q ** -2)
            self.an = -dt * t * vp / 2.0
            kz = torch.fft.fftfreq(nz, d=h, dtype=torch.float64, device=DEV)[:, None]
            kx = torch.fft.fftfreq(nx, d=h, dtype=torch.float64, device=DEV)[None]
            self.kk = torch.sqrt(kz ** 2 + kx ** 2)

    def _edge(self, f, dim, n):
        """f[i + 1] - f[i] (n = 1) or f[i] - f[i - 1] (n = -1), zero where the neighbour is outside."""
        L = f.shape[dim]
        d = (f.narrow(dim, 1, L - 1) - f.narrow(dim, 0, L - 1))
        return torch.nn.functional.pad(d, ((0, 1) if n == 1 else (1, 0)) if dim == -1 else
                                       ((0, 0, 0, 1) if n == 1 else (0, 0, 1, 0)))

    def __call__(self, s):
        if self.eq == "elastic":
            vx, vz, txx, tzz, txz = s
            E, F = self._edge(vx, -1, -1), self._edge(vz, -2, 1)
            xx = self.q * txx + self.pa * E + self.la * F
            zz = self.q * tzz + self.la * E + self.pa * F
            xz = self.q * txz + self.ma * (self._edge(vz, -1, 1) + self._edge(vx, -2, -1))
            vx = self.q * vx + self.bv * (self._edge(xx, -1, 1) + self._edge(xz, -2, 1))
            vz = self.q * vz + self.bv * (self._edge(xz, -1, -1) + self._edge(zz, -2, -1))
            return vx, vz, xx, zz, xz
        u, um = s[0], s[1]
        if self.eq == "acoustic":
            return self.g * (u - um) + um + self.k * _lap(u, self.order), u
        if self.eq == "vti_habc2":
            y = 2.0 * u - um + self.kx * _Second.apply(u, -1, 2) + self.kz * _Second.apply(u, -2, 2)
        elif self.eq == "acoustic_rho_habc":
            sh = [_Shift.apply(u, dim, n) for dim, n in ((-1, 1), (-1, -1), (-2, 1), (-2, -1))]
            y = 2.0 * u - um + self.C * sum(b * (t - u) for b, t in zip(self.bh, sh))
        else:
            lap = _lap(u, self.order)
            y = 2.0 * u - um + self.k * lap
            if self.eq == "vacoustic_habc":
                y = y + self.an * torch.fft.ifft2(self.kk * torch.fft.fft2(u - um)).real
        y = self.blend(y, u, um, self.v["vp"])
        if self.eq != "acoustic_lsrtm_habc":
            return y, u
        sc, scm = s[2], s[3]
        z = 2.0 * sc - scm + self.k * _lap(sc, self.order) + self.v["m"] * (self.k * lap)
        return y, u, self.blend(z, sc, scm, self.v["vp"]), sc


def _exact_loop(case, gen, wav, want_grad):
    eq = _EQS[case["eq"]]
    dt, h, _ = _sampling(case)
    plain = {k: _pad(case, v).float().double().to(DEV) for k, v in _models(case, gen).items()}
    inv = eq["inv"] if want_grad else ()
    xs, rx, row = _survey(case)
    top = 0 if case["multiple"] else W
    nz, nx = _padded(case)
    obs = _observed(case, gen, len(eq["rec"])) if want_grad else None
    wav = wav.double().tolist()
    rz, rxx = row + top, torch.tensor(rx, device=DEV) + W
    grads, recs, loss, illum = None, [], 0.0, torch.zeros(nz, nx, dtype=torch.float64, device=DEV)
    # shots in chunks: the graph keeps about this many bytes per point and step
    keep = {"elastic": 260.0, "acoustic": 30.0}.get(case["eq"], 110.0) if want_grad else 1.0
    chunk = max(1, min(case["shots"], int(6e10 / (keep * nz * nx * case["nt"] + 1)), int(6e9 / (nz * nx * 80))))
    for b0 in range(0, case["shots"], chunk):
        sx = torch.tensor(xs[b0:b0 + chunk], device=DEV) + W
        B = len(sx)
        m = {k: (v.clone().requires_grad_(True) if k in inv else v) for k, v in plain.items()}
        with torch.set_grad_enabled(want_grad):
            step = _Exact(case, m, dt, h)
            s = tuple(torch.zeros(B, nz, nx, dtype=torch.float64, device=DEV) for _ in range(step.nf))
            out = []
            for t in range(case["nt"]):
                s = list(step(s))
                for f in step.src:
                    inj = torch.zeros_like(s[f])
                    inj[torch.arange(B, device=DEV), row + top, sx] = wav[t]
                    s[f] = s[f] + inj
                if case.get("illum"):
                    illum += (s[step.src[-1]].detach() ** 2).sum(0)
                out.append(torch.stack([s[f][:, rz, :].index_select(-1, rxx) for f in step.rec], -1))
            r = torch.stack(out, 1)
            recs.append(r.detach())
            if want_grad:
                L = ((r - obs[b0:b0 + chunk].double().to(DEV)) ** 2).sum()
                g = torch.autograd.grad(L, [m[k] for k in inv])
                loss += float(L.detach())
                grads = list(g) if grads is None else [a + c for a, c in zip(grads, g)]
        del s, out, r, step, m
    res = {"records": torch.cat(recs)}
    if want_grad:  # gradients are those of the undamped interior, 0 in the boundary
        box = torch.zeros(nz, nx, dtype=torch.bool, device=DEV)
        box[top:nz - W, W:nx - W] = True
        res.update(loss=loss, grads=[torch.where(box, g, 0.0) for g in grads])
        if case.get("illum"):
            res["illum"] = illum
    return res


def _exact_step(case, gen):
    dt, h, _ = _sampling(case)
    models = {k: _pad(case, v).float().double().to(DEV).requires_grad_(True) for k, v in _models(case, gen).items()}
    nf = 5 if case["eq"] == "elastic" else 2
    f = _fields(case, gen, 2 * nf).double().to(DEV)
    fields = [f[i].clone().requires_grad_(True) for i in range(nf)]
    n = 5 if nf == 5 else 1
    out = _Exact(case, models, dt, h)(tuple(fields))
    grads = torch.autograd.grad(out[:n], list(models.values()) + fields, [f[nf + i] for i in range(n)],
                                allow_unused=True)
    return {"out": [o.detach() for o in out[:n]], "grads": [g for g in grads if g is not None]}


# name, input channels, output channels
_NET = [("e1a", 2, 32), ("e1b", 32, 32), ("e2a", 32, 64), ("e2b", 64, 64), ("e3a", 64, 128), ("e3b", 128, 128),
        ("b4", 128, 256), ("d3", 384, 128), ("d2", 192, 64), ("d1", 96, 32), ("out", 32, 1)]


class _Round(torch.autograd.Function):
    """bfloat16 storage of an activation, and of the gradient that flows back through it."""

    @staticmethod
    def forward(ctx, x, grad):
        ctx.grad = grad
        return x.float().bfloat16().double()

    @staticmethod
    def backward(ctx, g):
        return (g.float().bfloat16().double() if ctx.grad else g), None


def _exact_net(case, gen, seed):
    """The network with the bfloat16 roundings that its storage types define, everything between them in float64."""
    F = torch.nn.functional
    x, y = (t.double().to(DEV) for t in _net_inputs(case, gen))
    rng = np.random.default_rng(seed % 997)
    P = {}
    for name, ci, co in _NET:  # He initialisation; a small last layer; zero biases
        std = math.sqrt(2.0 / (ci * 9)) if name != "out" else math.sqrt(1.0 / (ci * 9)) * 0.1
        w = torch.from_numpy((rng.standard_normal(ci * co * 9) * std).astype(np.float32)).double().to(DEV)
        P[name] = (w.view(co, ci, 3, 3).requires_grad_(True),
                   torch.zeros(co, dtype=torch.float64, device=DEV, requires_grad=True))

    def conv(name, t):
        w, b = P[name]
        if name not in ("e1a", "out"):
            w = _Round.apply(w, False)
        o = torch.cat([F.conv2d(t[k:k + 1], w, b, padding=1) for k in range(t.shape[0])])
        # the gradient is rounded where it is stored: after the ReLU's mask
        return o if name == "out" else _Round.apply(F.relu(_Round.apply(o, True)), False)

    up = lambda t: F.interpolate(t, scale_factor=2, mode="nearest")
    pool = lambda t: _Round.apply(F.avg_pool2d(t, 2), False)
    with torch.set_grad_enabled(case["train"]):
        s1 = conv("e1b", conv("e1a", x))
        s2 = conv("e2b", conv("e2a", pool(s1)))
        s3 = conv("e3b", conv("e3a", pool(s2)))
        t = conv("b4", pool(s3))
        t = conv("d3", torch.cat([up(t), s3], 1))
        t = conv("d2", torch.cat([up(t), s2], 1))
        t = conv("d1", torch.cat([up(t), s1], 1))
        pred = conv("out", t)[:, 0]
        if not case["train"]:
            return {"pred": pred}
        loss = ((pred - y) ** 2).mean()
        flat = [q for name, _, _ in _NET for q in P[name]]
        g = torch.autograd.grad(loss, flat)
    # the first Adam step divides a gradient by its own size: no 64-bit value for the weights near 0
    return {"loss": loss.detach().reshape(1), "grads": torch.cat([q.reshape(-1) for q in g]),
            "params": None}


def exact(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "net":
        return _exact_net(case, gen, seed)
    if kind == "uneven":
        out = []
        for nz, nx, shots, nt in _uneven_groups(case):
            c = _uneven_case(case, nz, nx, shots, nt)
            r = _exact_loop(c, gen, _ricker(20.0, 0.001, nt), False)["records"]
            out.append(r[..., 0].permute(1, 0, 2).reshape(nt, -1, 1))
        return out
    if kind == "step":
        return _exact_step(case, gen)
    dt, _, fm = _sampling(case)
    return _exact_loop(case, gen, _ricker(fm, dt, case["nt"]), kind == "gradient")
