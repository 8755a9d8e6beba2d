"""Cases for timing the framework: the calls its users make, through its public entry points.

  step       one accepted time step of a large simulation that is under way (Context.run), the
             state read back on the device: the reference's Air-driven model, the flow-through
             model with acid flowing in, a fractured geometry
  run        a whole short simulation from a label image: upload, start, steps, read-back; on a
             context that a study of many samples keeps, or (fresh) with the context made and freed
  pressure   a cold pressure solve (assembly and solve from zero), as at a run's first step
  transport  the conc + acid solve on given fields, two species at once
  net        the learned pressure network, forward
  train      one training step of that network, with its gradients and updated weights
  geometry   the preparation of a grey-level image: classify, clean, fracture, coarsen

Geometries are seeded Gaussian random fields made on the GPU (Pore below a quantile, mineral from
a second field), as leachingsim_gb300.geometry makes them on the CPU.
"""
import ctypes

import numpy as np
import torch

from leachingsim_gb300 import _abi, learned
from leachingsim_gb300 import runtime as rt

AIR, PORE, ROCK, SULPHIDE, PRECIPITATE = 1, 2, 3, 4, 5
DT = 1.0


def _sim(kind, name, shape, **kw):
    c = dict(name=name, kind=kind, I=shape[0], J=shape[1], K=shape[2], label_bytes=1, flow=False, implicit=False,
             fractured=False, solver="mixed", porosity=0.25, corr=6.0, press_rtol=1e-8, conc_rtol=1e-12)
    c.update(kw)
    if kind == "run":
        c.setdefault("steps", 10)
        c.setdefault("fresh", False)
    return c


def listed():
    return [
        # the smallest domain that the accuracy tests run whole (tmax 10): launches and read-backs are all there is
        _sim("run", "run_small", (32, 40, 40), porosity=0.30, corr=4.0),
        # the plain-method configuration (64^3, flow-through, acid flowing in, tmax 10)
        _sim("run", "run_flow_64", (64, 64, 64), flow=True, porosity=0.30, corr=4.0, press_rtol=1e-12),
        # a ragged grid with an odd row length, uint16 labels and the implicit saturation (--implicit_sat)
        _sim("run", "run_implicit_odd", (61, 83, 101), label_bytes=2, implicit=True, press_rtol=1e-12, steps=6),
        # one sample from start to end with the plain FP64 solver, the context's own start-up included
        _sim("run", "run_fp64_fresh", (48, 64, 64), solver="fp64", porosity=0.30, corr=4.0, press_rtol=1e-12, steps=5,
             fresh=True),
        # the benchmark's workload: Air inlet, 32 M voxels
        _sim("step", "step_air_large", (283, 338, 338)),
        # the same size flow-through: every step dissolves mineral and solves a changed pressure system
        _sim("step", "step_flow_large", (283, 338, 338), flow=True, press_rtol=1e-12),
        # fractured uint16 geometry (permeability contrast 1e4), flow-through with acid
        _sim("step", "step_fractured", (224, 320, 320), label_bytes=2, flow=True, fractured=True, press_rtol=1e-12),
        # the first pressure solve of a run, from zero
        dict(name="pressure_cold", kind="pressure", I=160, J=256, K=256, label_bytes=1, solver="mixed",
             porosity=0.25, corr=6.0, press_rtol=1e-8),
        # the two species of a leaching run, odd row length
        dict(name="transport_two", kind="transport", I=97, J=128, K=121, label_bytes=1, theta=1.0, porosity=0.25,
             corr=6.0, conc_rtol=1e-12),
        # the network at the half resolution of the benchmark's workload
        dict(name="net_forward", kind="net", D=144, H=176, W=176),
        # one training sample: a half-resolution column crop
        dict(name="net_train", kind="train", D=144, H=32, W=32),
        # a grey-level image on its way to a label image
        dict(name="geometry_prepare", kind="geometry", I=400, J=400, K=400, corr=6.0),
    ]


def _extents(rng, lo, hi, step=1):
    """Extents of a box of lo..hi voxels (log-uniform), up to a factor 3 from a cube, multiples of step."""
    n = lo * (hi / lo) ** rng.random()
    f = [3.0 ** rng.uniform(-0.5, 0.5) for _ in range(3)]
    s = (n / (f[0] * f[1] * f[2])) ** (1.0 / 3.0)
    return [max(2 * step, int(round(s * v / step)) * step) for v in f]


def draw(rng):
    kind = rng.choice(["step", "step", "run", "run", "pressure", "transport", "transport", "net", "train", "geometry"])
    if kind in ("step", "run"):
        i, j, k = _extents(rng, *((2e6, 2e7) if kind == "step" else (3e4, 2e6)))
        flow = rng.random() < 0.5
        implicit = kind == "run" and not flow and rng.random() < 0.3
        fresh = kind == "run" and rng.random() < 0.4
        fractured = kind == "step" and flow and rng.random() < 0.5
        c = _sim(kind, "", (i, j, k), label_bytes=rng.choice([1, 2]), flow=flow, implicit=implicit, fractured=fractured,
                 porosity=round(rng.uniform(0.22, 0.35), 3), corr=round(rng.uniform(3.0, 7.0), 2),
                 press_rtol=1e-12 if flow or implicit else 1e-8)
        if kind == "run":
            c.update(fresh=fresh, solver="fp64" if fresh and i * j * k < 3e5 else "mixed", steps=rng.randint(3, 6))
        del c["name"]
        return c
    if kind == "pressure":
        i, j, k = _extents(rng, 3e4, 1.2e7)
        return dict(kind=kind, I=i, J=j, K=k, label_bytes=rng.choice([1, 2]),
                    solver=rng.choice(["mixed", "mixed", "fp64"]), porosity=round(rng.uniform(0.22, 0.35), 3),
                    corr=round(rng.uniform(3.0, 7.0), 2), press_rtol=1e-8)
    if kind == "transport":
        i, j, k = _extents(rng, 3e4, 6e6)
        return dict(kind=kind, I=i, J=j, K=k, label_bytes=rng.choice([1, 2]), theta=rng.choice([1.0, 1.0, 0.5]),
                    porosity=round(rng.uniform(0.22, 0.35), 3), corr=round(rng.uniform(3.0, 7.0), 2), conc_rtol=1e-12)
    if kind in ("net", "train"):
        d, h, w = _extents(rng, 8e3, 4e6 if kind == "net" else 1.5e5, 8)
        return dict(kind=kind, D=d, H=h, W=w)
    i, j, k = _extents(rng, 3e4, 6e7, 2)
    return dict(kind=kind, I=i, J=j, K=k, corr=round(rng.uniform(3.0, 7.0), 2))


# ---------------------------------------------------------------------------
# inputs


def _shape(case):
    return tuple(int(case[q]) for q in ("I", "J", "K"))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _smooth(shape, sigma, gen):
    """Periodic Gaussian-smoothed white noise (float32, unit scale up to a constant)."""
    f = torch.fft.rfftn(torch.randn(shape, generator=gen, device="cuda"))
    for ax, n in enumerate(shape):
        q = torch.fft.rfftfreq(n, device="cuda") if ax == 2 else torch.fft.fftfreq(n, device="cuda")
        g = torch.exp(-2.0 * (np.pi * sigma * q) ** 2)
        f *= g.reshape([-1 if a == ax else 1 for a in range(3)])
    return torch.fft.irfftn(f, s=shape)


def _quantile(v, q):
    v = v.reshape(-1)
    v = v[:: max(1, v.numel() // 2_000_000)]
    return torch.sort(v).values[min(v.numel() - 1, int(q * v.numel()))]


def _labels(case, gen, air):
    """Label image (torch, on the GPU): Pore below the porosity quantile, 15 % of the solid mineral."""
    shape = _shape(case)
    f = _smooth(shape, case["corr"], gen)
    pore = f <= _quantile(f, case["porosity"])
    g = _smooth(shape, max(case["corr"] / 2.0, 1.0), gen)
    lab = torch.full(shape, ROCK, dtype=torch.uint8, device="cuda")
    lab[g <= _quantile(g[~pore], 0.15)] = SULPHIDE
    lab[pore] = PORE
    if air:
        lab[:2] = AIR
    return lab


def _fractures(shape, gen, count=4):
    """Mask of planar fractures of 1-3 voxel aperture and random orientation."""
    grids = [torch.arange(n, device="cuda", dtype=torch.float32) - n / 2.0 for n in shape]
    mask = torch.zeros(shape, dtype=torch.bool, device="cuda")
    for _ in range(count):
        n = torch.randn(3, generator=gen, device="cuda")
        n = (n / n.norm()).tolist()
        u = torch.rand(2, generator=gen, device="cuda").tolist()
        d = grids[0][:, None, None] * n[0] + grids[1][None, :, None] * n[1] + grids[2][None, None, :] * n[2]
        mask |= (d - (0.6 * u[0] - 0.3) * min(shape)).abs() <= (1 + int(3 * u[1])) / 2.0
    return mask


def _host_labels(case, lab):
    return lab.cpu().numpy().astype(np.uint8 if case["label_bytes"] == 1 else np.uint16)


def _params(case):
    kw = dict(c_sat=1.0, press_rtol=case["press_rtol"], conc_rtol=case["conc_rtol"], sat_rtol=case["conc_rtol"],
              press_solver=_abi.PRESS_FP64 if case["solver"] == "fp64" else _abi.PRESS_MIXED)
    if case["flow"]:
        kw.update(bc_mode=_abi.BC_FLOW_I, p_inlet=1.0, p_outlet=0.0, acid_inlet=1.0)
    if case["implicit"]:
        kw.update(use_implicit_saturation=1)
    return _abi.default_params(**kw)


def _simulation_inputs(case, seed):
    gen = _gen(seed)
    lab = _labels(case, gen, not case["flow"])
    kmult = None
    if case["fractured"]:
        cut = _fractures(_shape(case), gen)
        lab[cut] = PORE
        kmult = torch.where(cut, 1e4, 1.0).to(torch.float32).cpu().numpy()
    return _host_labels(case, lab), kmult


def _context(case):
    return rt.Context(_shape(case), label_bytes=case["label_bytes"], params=_params(case))


def _start(ctx, lab, kmult):
    ctx.upload("label", lab)
    if kmult is not None:
        ctx.upload("kmult", kmult)
    ctx.init_all()


STATE = ["label", "frac", "pressure", "saturation", "conc", "acid", "precipitate"]
_TORCH = {np.uint8: torch.uint8, np.uint16: torch.int16, np.float32: torch.float32, np.float64: torch.float64}


def _buffers(ctx, names):
    return {n: torch.empty(ctx.NP, dtype=_TORCH[ctx._dtype(_abi.FIELDS[n])], device="cuda") for n in names}


def _move(ctx, bufs, up):
    """Fields of a context from / into device tensors (padded arrays), through the C entry points."""
    fn = rt.load().ls_upload_field_device if up else rt.load().ls_download_field_device
    for n, b in bufs.items():
        ctx._check(fn(ctx.h, _abi.FIELDS[n], ctypes.c_void_p(b.data_ptr()), b.numel(), 1))


TMAX_STEPS = 50  # the benchmark's run; the simulation starts again after it


def _restart(s):
    """The simulation from its label image up to its third step."""
    _start(s["ctx"], s["lab"], s["kmult"])
    log = s["ctx"].run(1e30, DT, max_steps=2)
    s["t"], s["n"] = log[-1]["t"] + log[-1]["dt"], 2


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "run"):
        lab, kmult = _simulation_inputs(case, seed)
        s = {"case": case, "lab": lab, "kmult": kmult}
        if kind == "step" or not case["fresh"]:
            s["ctx"] = _context(case)
            s["out"] = _buffers(s["ctx"], STATE)
        if kind == "step":
            _restart(s)
    elif kind == "pressure":
        c = dict(case, flow=False, implicit=False, conc_rtol=1e-12)
        ctx = _context(c)
        _start(ctx, _host_labels(case, _labels(case, _gen(seed), True)), None)
        s = {"case": case, "ctx": ctx, "zero": torch.zeros(_shape(case), device="cuda"),
             "out": _buffers(ctx, ["pressure"])}
    elif kind == "transport":
        lab, fields = _transport_inputs(case, seed)
        ctx = rt.Context(_shape(case), label_bytes=case["label_bytes"], params=_transport_params(case))
        ctx.upload("label", _host_labels(case, lab))
        _move(ctx, {n: fields[n] for n in ("flux_x", "flux_y", "flux_z")}, True)
        s = {"case": case, "ctx": ctx, "in": {n: fields[n] for n in ("conc", "acid")},
             "out": _buffers(ctx, ["conc", "acid"])}
    elif kind in ("net", "train"):
        net = rt.LPNet((case["D"], case["H"], case["W"]), seed=0)
        net.set_params(learned.load_weights())
        s = {"case": case, "net": net, "in": _net_inputs(case, seed)}
    else:
        f = _smooth(_shape(case), case["corr"], _gen(seed))
        lo, hi = f.min(), f.max()
        grey = ((f - lo) / (hi - lo) * 65535.0).to(torch.int32)
        thr = [int(_quantile(grey, 0.20)), int(_quantile(grey, 0.88))]
        return {"case": case, "grey": grey.cpu().numpy().astype(np.uint16), "thr": thr}
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "step":
        ctx = s["ctx"]
        if s["n"] >= TMAX_STEPS:
            _restart(s)
        log = ctx.run(1e30, DT, t0=s["t"], n0=s["n"], max_steps=1)
        s["t"] += log[-1]["dt"]
        s["n"] += 1
        _move(ctx, s["out"], False)
        return s["out"]
    if kind == "run":
        fresh = s["case"]["fresh"]
        ctx = _context(s["case"]) if fresh else s["ctx"]
        out = _buffers(ctx, STATE) if fresh else s["out"]
        _start(ctx, s["lab"], s["kmult"])
        ctx.run(1e30, DT, max_steps=s["case"]["steps"])
        _move(ctx, out, False)
        if fresh:
            ctx.close()
        return out
    if kind == "pressure":
        ctx = s["ctx"]
        ctx.pressure_setup(0.0)
        ctx.pressure_solve_start(s["zero"], 0.0)
        _move(ctx, s["out"], False)
        return s["out"]
    if kind == "transport":
        ctx = s["ctx"]
        _move(ctx, s["in"], True)
        ctx.transport(DT)
        _move(ctx, s["out"], False)
        return s["out"]
    if kind == "net":
        return s["net"].forward(*s["in"][:3])
    if kind == "train":
        loss = s["net"].train_step(*s["in"], lr=2e-3)
        return {"loss": loss, "grads": s["net"].get_grads(), "weights": s["net"].get_params()}
    lab = rt.geom_classify(s["grey"], s["thr"], [PORE, ROCK, SULPHIDE], 2)
    cleaned, removed = rt.geom_clean(lab, "core_sample")
    drilled, n_drilled, n_encapsulated = rt.geom_fracture(cleaned)
    coarse = rt.geom_coarsen(drilled)
    images = {"cleaned": cleaned, "drilled": drilled, "coarse": coarse}
    return {**{n: a.view(np.int16) for n, a in images.items()}, "counts": [removed, n_drilled, n_encapsulated]}


# ---------------------------------------------------------------------------
# transport: fields and the exact solution


def _transport_params(case):
    return _abi.default_params(c_sat=1.0, theta=case["theta"], alpha_transfer=0.05, Dpore_fac=0.8,
                               conc_rtol=case["conc_rtol"])


def _transport_inputs(case, seed):
    gen = _gen(seed)
    shape = _shape(case)
    lab = _labels(case, gen, True)
    lab[(lab == PORE) & (torch.rand(shape, generator=gen, device="cuda") < 0.02)] = PRECIPITATE
    pad = (shape[0] + 1, shape[1], shape[2])
    pore = torch.zeros(pad, dtype=torch.bool, device="cuda")
    pore[:-1] = lab == PORE
    fields = {}
    for n in ("flux_x", "flux_y", "flux_z"):
        fields[n] = (0.3 * torch.randn(pad, generator=gen, device="cuda", dtype=torch.float64) * pore).reshape(-1)
    for n in ("conc", "acid"):
        f = torch.rand(pad, generator=gen, device="cuda", dtype=torch.float64)
        fields[n] = (f * pore if n == "acid" else 0.2 + 0.8 * f).reshape(-1)
    return lab, fields


def _shifted(a, ax, d):
    """a at the neighbour along axis ax in direction d (+1 / -1); 0 outside."""
    out = torch.zeros_like(a)
    n = a.shape[ax]
    out.narrow(ax, 0 if d > 0 else 1, n - 1).copy_(a.narrow(ax, 1 if d > 0 else 0, n - 1))
    return out


def _transport_exact(case, seed):
    """The implicit upwind system of the two species in 64 bits, solved by Jacobi-BiCGStab to rounding."""
    lab, fields = _transport_inputs(case, seed)
    shape, n = _shape(case), int(np.prod(_shape(case)))
    lab = lab.to(torch.int32)
    alpha, D, Dp, th, idt = 0.05, 1.0, 0.8, case["theta"], 1.0 / DT
    flux = [fields[f][:n].reshape(shape) for f in ("flux_x", "flux_y", "flux_z")]
    ident, rock = lab == PRECIPITATE, lab == ROCK
    diag = torch.full(shape, idt, dtype=torch.float64, device="cuda")
    diag[ident] = 1.0
    expl = torch.zeros(shape, dtype=torch.float64, device="cuda")  # explicit part of the diagonal
    offs, xoffs = [], []
    for ax in range(3):
        for d in (1, -1):
            nl = _shifted(lab, ax, d)
            inside = nl > 0
            q = flux[ax] if d > 0 else -_shifted(flux[ax], ax, -1)
            q = torch.where((nl == PRECIPITATE) | (nl == SULPHIDE), torch.zeros_like(q), q)
            dc = -D - (Dp - D) * (nl == PORE).double()
            self_c, nb_c = -dc + q.clamp(min=0), dc - q.clamp(max=0)
            to_rock = ~ident & ~rock & (nl == ROCK)
            from_rock = rock & (nl == PORE)
            flow = ~ident & ~rock & inside & (nl != ROCK)
            off = torch.where(flow, th * nb_c, 0.0)
            off[to_rock | from_rock] = -alpha
            diag += torch.where(flow, th * self_c, 0.0) + alpha * (to_rock | from_rock).double()
            expl += torch.where(flow, (1 - th) * self_c, 0.0)
            offs.append((ax, d, off))
            xoffs.append((ax, d, torch.where(flow, (1 - th) * nb_c, 0.0)))

    def apply(c0, links, x):
        y = c0 * x
        for ax, d, o in links:
            y += o * _shifted(x, ax, d)
        return y

    def mul(x):
        return apply(diag, offs, x) / diag

    out = {}
    for name in ("conc", "acid"):
        old = fields[name].reshape(shape[0] + 1, shape[1], shape[2])
        b = torch.where(ident, old[:-1], old[:-1] * idt) - apply(expl, xoffs, old[:-1])
        b = b / diag
        x = b.clone()
        for _ in range(6):  # restarted BiCGStab until the residual stops falling
            r = b - mul(x)
            if float(r.norm()) <= 2e-16 * float(b.norm()):
                break
            rh, p = r.clone(), r.clone()
            rho = (rh * r).sum()
            target = 1e-9 * float(r.norm())
            for _ in range(200):
                v = mul(p)
                a = rho / (rh * v).sum()
                s = r - a * v
                t = mul(s)
                w = (t * s).sum() / (t * t).sum()
                x += a * p + w * s
                r = s - w * t
                if float(r.norm()) <= target:
                    break
                new = (rh * r).sum()
                p = r + (new / rho) * (a / w) * (p - w * v)
                rho = new
        res = old.clone()  # the solution lands one plane up
        res[1:] = x
        out[name] = res.reshape(-1)
    return out


# ---------------------------------------------------------------------------
# network: inputs and the same network in 64 bits


def _net_inputs(case, seed):
    gen = _gen(seed)
    shape = (case["D"], case["H"], case["W"])
    f = _smooth(shape, 3.0, gen)
    mask = (f <= _quantile(f, 0.35)).float()
    logk = mask * (1.0 + 0.05 * torch.randn(shape, generator=gen, device="cuda"))
    depth = torch.arange(shape[0], device="cuda", dtype=torch.float32)[:, None, None].expand(shape) / 100.0
    target = mask * (depth + 0.1 * _smooth(shape, 2.0, gen))
    return [t.contiguous() for t in (mask, logk, depth, target, mask)]


def _net64(p, x):
    """The U-shaped network with every value in 64 bits; x (D, H, W, 16), p a dict of tensors."""
    def conv(a, name, relu=True):
        D, H, W, _ = a.shape
        pad = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1, 1, 1))
        o = p[name + "_b"].expand(D, H, W, -1)
        for t in range(27):
            z, y, w = t // 9, (t // 3) % 3, t % 3
            o = o + pad[z:z + D, y:y + H, w:w + W] @ p[name][t].T
        return torch.relu(o) if relu else o

    def pool(a):
        D, H, W, C = a.shape
        return a.reshape(D // 2, 2, H // 2, 2, W // 2, 2, C).mean(dim=(1, 3, 5))

    def up(a):
        return a.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)

    s0 = conv(conv(x, "W0a"), "W0b")
    s1 = conv(pool(s0), "W1")
    s2 = conv(pool(s1), "W2")
    b2 = conv(up(conv(pool(s2), "W3")) + s2, "U2")
    b1 = conv(up(b2) + s1, "U1")
    return conv(up(b1) + s0, "U0", relu=False)[..., 0]


def _net_exact(case, seed):
    w = rt.lpnet_unflatten(np.asarray(learned.load_weights(), np.float32))
    p = {k: torch.from_numpy(np.array(v, np.float64)).cuda() for k, v in w.items()}
    mask, logk, depth, target, _ = _net_inputs(case, seed)
    x = torch.zeros(mask.shape + (16,), dtype=torch.float64, device="cuda")
    for q, f in enumerate((mask, logk, depth)):
        x[..., q] = f
    if case["kind"] == "net":
        with torch.no_grad():
            return _net64(p, x)
    for v in p.values():
        v.requires_grad_(True)
    loss = ((_net64(p, x) - target) ** 2 * mask).sum() / mask.sum()
    loss.backward()
    grads = rt.lpnet_flatten({k: v.grad.cpu().numpy() for k, v in p.items()})
    return {"loss": float(loss), "grads": grads.astype(np.float64), "weights": None}


def exact(case, seed):
    if case["kind"] == "transport":
        return _transport_exact(case, seed)
    if case["kind"] in ("net", "train"):
        return _net_exact(case, seed)
    return None  # whole steps and pressure solves take minutes in plain torch; geometry is whole numbers


# ---------------------------------------------------------------------------


def work(case):
    """Each input of a pass read once and each output written once; the arithmetic that no
    algorithm for the path goes without."""
    kind = case["kind"]
    if kind in ("net", "train"):
        n = case["D"] * case["H"] * case["W"]
        flops = 2.0 * 27 * n * (3 * 16 + 16 * 16 + 16 * 32 / 8 + 32 * 64 / 64 + 64 * 64 / 512 + 64 * 32 / 64
                                + 32 * 16 / 8 + 16)
        return {"bytes": n * (16 if kind == "net" else 24) + 4.0 * 27e4 * (1 if kind == "net" else 3),
                "flops": flops * (1 if kind == "net" else 3)}
    n = float(np.prod(_shape(case)))
    if kind == "geometry":  # grey in, labels out and in between the three stages, the coarse image
        return {"bytes": n * 2.0 * (2 + 2 + 2 + 1 + 0.125), "flops": 0.0}
    lb = case["label_bytes"]
    if kind == "pressure":  # label, permeability, viscosity -> pressure
        return {"bytes": n * (lb + 16 + 8), "flops": n * 30}
    if kind == "transport":  # label, three fluxes, two species in and out
        return {"bytes": n * (lb + 24 + 32), "flops": n * 60}
    state = lb + 4 + 5 * 8
    if kind == "run":  # the label image in, then every step's state
        return {"bytes": n * (lb + case["steps"] * 2.0 * state), "flops": n * 200.0 * case["steps"]}
    return {"bytes": n * (2.0 * state + 24), "flops": n * 200.0}
