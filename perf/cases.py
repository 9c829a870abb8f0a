"""Measured workloads of the SRC/MPCD step on one GPU, through the package's public entry points.

``listed()`` are the named cases, ``draw(rng)`` gives further ones of the same ranges. A case is a
plain dict; ``kind`` says which part of the framework it drives:

    step     native.Context.step in a state form ("f64", "f32", "fast"), then the state in
             particle-id order: a run that advances to its next dump or metrics row. The state
             stays on the device and every pass continues the run, as a driver's loop does.
    batch    native.Batch.step of independent channels, then every replica's state
    phases   one step through the phase functions (the reference drivers' call sequence), on a
             state the caller owns and hands over on every pass
    learned  the learned closure's network: inference, full-batch gradient, one epoch of training
"""
import math

import numpy as np
import torch

from src_incompressible_openmp_b200 import native
from src_incompressible_openmp_b200.cases import ensemble_family, poiseuille_params

DEVICE = "cuda:0"

# Walls of a closed box with a moving lid (the four wall modes); a channel is the default.
BOX = dict(boundary_left="bounceback", boundary_right="specular", boundary_bottom="thermalize",
           boundary_top="thermalize", Utop=0.05)


def listed():
    return [
        # The reference's own benchmark case (25,000 particles): a metrics row every ten steps.
        # Latency and launches decide it.
        dict(name="f64_50x50_metrics", kind="step", form="f64", Nx=50, Ny=50, ppc=10, steps=10, metrics=True),
        # A parameter study's odd box: no size a multiple of the tiles, walls all round, a state
        # whose density is far from even, so that many cells are redistributed.
        dict(name="f64_333x97_box", kind="step", form="f64", Nx=333, Ny=97, ppc=7, steps=8, box=True, amp=0.5),
        # The large channel of the plain form, ten particles per cell.
        dict(name="f64_2048x512", kind="step", form="f64", Nx=2048, Ny=512, ppc=10, steps=4),
        # The headline channel (84 M particles) in the plain form.
        dict(name="f64_4096x1024", kind="step", form="f64", Nx=4096, Ny=1024, ppc=20, steps=4),
        # The FP32 precision form, where the state's memory matters, on an uneven channel.
        dict(name="f32_1501x333", kind="step", form="f32", Nx=1501, Ny=333, ppc=15, steps=4),
        # The fast form on the reference's case, with its metrics row.
        dict(name="fast_50x50_metrics", kind="step", form="fast", Nx=50, Ny=50, ppc=10, steps=10, metrics=True),
        # The fast form with the plain closure.
        dict(name="fast_2048x512", kind="step", form="fast", Nx=2048, Ny=512, ppc=10, steps=16),
        # The headline channel in the chosen form: fast, with the learned closure.
        dict(name="fast_4096x1024_learned", kind="step", form="fast", Nx=4096, Ny=1024, ppc=20, steps=8, learned=True),
        # Ensembles of uneven channels: the plain form, and the fast form at the size of the
        # named ensemble workload.
        dict(name="batch_f64_64", kind="batch", form="f64", replicas=64, family=20, steps=8),
        dict(name="batch_fast_256", kind="batch", form="fast", replicas=256, family=20, steps=16),
        # A driver of the reference on the drop-in phase functions.
        dict(name="phases_400x200", kind="phases", Nx=400, Ny=200, ppc=10),
        # Training and use of the learned closure's network.
        dict(name="learned_32k", kind="learned", rows=32768, batch=512),
    ]


def _log_int(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["f64", "f64", "f64", "f32", "fast", "fast", "fast", "batch", "phases", "learned"])
    if kind == "learned":
        return dict(kind="learned", rows=_log_int(rng, 1000, 200000), batch=rng.choice([128, 256, 512, 1000]))
    if kind == "batch":
        form = rng.choice(["f64", "fast"])
        return dict(kind="batch", form=form, replicas=_log_int(rng, 4, 64 if form == "f64" else 256),
                    family=rng.randrange(1, 1000), steps=rng.randint(2, 12))
    Nx, Ny, ppc = _log_int(rng, 24, 3000), _log_int(rng, 16, 800), rng.randint(5, 20)
    if kind == "phases":
        Nx, Ny = min(Nx, 800), min(Ny, 400)
        return dict(kind="phases", Nx=Nx, Ny=Ny, ppc=ppc)
    c = dict(kind="step", form=kind, Nx=Nx, Ny=Ny, ppc=ppc, steps=rng.randint(2, 12), metrics=rng.random() < 0.3)
    if rng.random() < 0.3:
        c["box"] = True
    if rng.random() < 0.3:
        c["amp"] = round(rng.uniform(0.1, 0.5), 3)
    if kind == "fast" and not c.get("box") and rng.random() < 0.4:
        c["learned"] = True
    return c


def _params(case):
    return poiseuille_params(case["Nx"], case["Ny"], case["ppc"], **(BOX if case.get("box") else {}))


def _state(p, seed, amp=0.0):
    """Seeded positions (uniform, or with the density modulated along x by up to amp) and
    Maxwellian velocities with the mean removed: two (n, 2) tensors in particle-id order."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    n = p["n"]
    x = torch.rand((n, 2), generator=g, device=DEVICE, dtype=torch.float64)
    if amp:
        x[:, 0] += amp / (2.0 * math.pi) * torch.sin(2.0 * math.pi * x[:, 0])
        x[:, 0].clamp_(0.0, 1.0 - 1e-12)
    x[:, 0] *= p["Lx"]
    x[:, 1] *= p["Ly"]
    v = torch.randn((n, 2), generator=g, device=DEVICE, dtype=torch.float64)
    v *= math.sqrt(p["kBT"])
    v -= v.mean(dim=0)
    return x, v


def _network(seed):
    """A network of the learned closure with kicks of the plain closure's size."""
    net = native.learned_init(seed)
    net[-1] = 1e-3
    return net


def _learned_rows(case, seed):
    """Feature rows and targets with the magnitudes that the step's samples have."""
    rng = np.random.default_rng(seed)
    rows = case["rows"]
    X = 0.3 * rng.standard_normal((rows, native.LEARNED_FEATURES), dtype=np.float32)
    W = rng.standard_normal((native.LEARNED_FEATURES, native.LEARNED_OUTPUTS), dtype=np.float32)
    Y = 0.01 * np.tanh(X @ W / math.sqrt(native.LEARNED_FEATURES))
    return X, Y.astype(np.float32), native.learned_init(seed)


def _set_state(ctx, x, v):
    ctx.set_state_device(x.data_ptr(), v.data_ptr())


def prepare(case, seed):
    kind = case["kind"]
    if kind == "learned":
        X, Y, net = _learned_rows(case, seed)
        net[-1] = 0.01
        return dict(kind=kind, X=X, Y=Y, net=net, batch=case["batch"], seed=seed)
    if kind == "batch":
        family = [p for p, _ in ensemble_family(case["replicas"], case["family"])]
        batch = native.Batch(family, form=case["form"])
        # all replicas' particles in two tensors, one replica after another
        X, V = (torch.empty((sum(p["n"] for p in family), 2), dtype=torch.float64, device=DEVICE) for _ in range(2))
        at = np.cumsum([0] + [p["n"] for p in family])
        out = [(X[a:b], V[a:b]) for a, b in zip(at[:-1], at[1:])]
        for r, p in enumerate(family):
            for to, made in zip(out[r], _state(p, seed * 1000 + r)):
                to.copy_(made)
        torch.cuda.synchronize()
        for r, (x, v) in enumerate(out):
            _set_state(batch.member(r), x, v)
        return dict(kind=kind, batch=batch, X=X, V=V, out=out, steps=case["steps"], step=0)
    p = _params(case)
    x, v = _state(p, seed, case.get("amp", 0.0))
    torch.cuda.synchronize()
    if kind == "phases":
        return dict(kind=kind, ctx=native.Context(p), x=x, v=v, out=(torch.empty_like(x), torch.empty_like(v)),
                    rho=p["gamma"] / (p["a0"] * p["a0"]), seed=seed)
    ctx = native.Context(p, form=case["form"])
    _set_state(ctx, x, v)
    if case.get("learned"):
        ctx.learned_set(_network(7), 0.25)
    # the initial state's tensors receive the states that the run returns
    return dict(kind=kind, ctx=ctx, out=(x, v), steps=case["steps"], metrics=bool(case.get("metrics")), step=0)


def _numbers(d):
    """The values of a metrics row without its wall-clock times."""
    return {k: (_numbers(u) if isinstance(u, dict) else u) for k, u in d.items()
            if not k.startswith("time") and not k.startswith("reserved")}


def _get_state(ctx, out):
    ctx.get_state_device(out[0].data_ptr(), out[1].data_ptr())


def run(state):
    kind = state["kind"]
    if kind == "step":
        ctx = state["ctx"]
        row = ctx.step(state["step"], state["steps"], metrics=state["metrics"])
        state["step"] += state["steps"]
        _get_state(ctx, state["out"])
        return {"x": state["out"][0], "v": state["out"][1], "row": _numbers(row) if row else None}
    if kind == "batch":
        batch = state["batch"]
        batch.step(state["step"], state["steps"])
        state["step"] += state["steps"]
        for r, out in enumerate(state["out"]):
            _get_state(batch.member(r), out)
        return {"x": state["X"], "v": state["V"]}
    if kind == "phases":
        ctx, s = state["ctx"], state["seed"] % 1000
        _set_state(ctx, state["x"], state["v"])
        fields = ctx.cell_fields(state["rho"])
        ctx.stream()
        wall = ctx.apply_bc(104729 + 10007 * s)
        cells = ctx.srd_shift_cells(130363 + 10007 * s)
        ctx.srd_collide(433494437 + 10007 * s)
        ctx.save_ref()
        base = ctx.zone_pass("base", 88172645463325252 + 10007 * s)
        shifted = ctx.zone_pass("shifted", 88172645463325252 + 4099 + 10007 * s)
        closure = ctx.liquid_closure()
        _get_state(ctx, state["out"])
        return {"fields": {k: fields[k] for k in ("N", "Ux", "Uy", "T", "rho", "P")}, "wall": _numbers(wall), "cells": cells,
                "base": _numbers(base), "shifted": _numbers(shifted), "closure": _numbers(closure), "x": state["out"][0],
                "v": state["out"][1]}
    kick = native.learned_predict(state["X"], state["net"])
    grad, loss = native.learned_grad(state["X"], state["Y"], state["net"])
    net, losses = native.learned_train(state["X"], state["Y"], state["net"], epochs=1, batch=state["batch"], seed=state["seed"])
    return {"kick": kick, "grad": grad, "loss": loss, "net": net, "losses": losses}


# bytes of a particle's state in each form (position, velocity; the fast form's and the FP32
# form's cell) and of its copy in particle-id order
STATE_BYTES = {"f64": 32, "f32": 20, "fast": 20}
# additions and multiplications of a particle's step: streaming, rotation and thermostat, cell
# sums of the reference and the red state, momentum correction, kick
STEP_FLOPS = 100


def work(case):
    kind = case["kind"]
    if kind == "learned":
        rows, mlp = case["rows"], 2 * (75 * 64 + 64 * 64 + 64 * 2)
        # inference, gradient and training each read the rows once
        return {"bytes": rows * (3 * 300 + 3 * 8), "flops": rows * mlp * (1 + 3 + 3)}
    if kind == "batch":
        n = sum(p["n"] for p, _ in ensemble_family(case["replicas"], case["family"]))
    else:
        n = _params(case)["n"]
    if kind == "phases":
        return {"bytes": n * (32 + 32 + 4), "flops": n * STEP_FLOPS}
    per = STATE_BYTES[case["form"]]
    # every step reads and writes the state; the last one's result goes out in id order
    return {"bytes": n * (2 * per * case["steps"] + 32), "flops": n * STEP_FLOPS * case["steps"]}


def _gelu(z):
    c = math.sqrt(2.0 / math.pi)
    t = torch.tanh(c * (z + 0.044715 * z ** 3))
    return 0.5 * z * (1.0 + t), 0.5 * (1.0 + t) + 0.5 * z * (1.0 - t * t) * c * (1.0 + 3 * 0.044715 * z * z)


def _exact_learned(case, seed):
    """The network's kick, and the gradient and value of its mean squared error, in 64 bits."""
    X, Y, net = _learned_rows(case, seed)
    X, Y = torch.from_numpy(X).double(), torch.from_numpy(Y).double()
    w = torch.from_numpy(net).double()
    scale = 0.01
    W1, b1 = w[:4800].view(64, 75), w[4800:4864]
    W2, b2 = w[4864:8960].view(64, 64), w[8960:9024]
    W3, b3 = w[9024:9152].view(2, 64), w[9152:9154]
    a1, g1 = _gelu(X @ W1.T + b1)
    a2, g2 = _gelu(a1 @ W2.T + b2)
    out = a2 @ W3.T + b3
    err = out - Y / scale
    loss = float((err * err).mean())
    d3 = 2.0 * err / err.numel()
    d2 = (d3 @ W3) * g2
    d1 = (d2 @ W2) * g1
    grad = torch.cat([(d1.T @ X).reshape(-1), d1.sum(0), (d2.T @ a1).reshape(-1), d2.sum(0),
                      (d3.T @ a2).reshape(-1), d3.sum(0), torch.zeros(1, dtype=torch.float64)])
    return {"kick": out * scale, "grad": grad, "loss": loss, "net": None, "losses": None}


def _exact_fields(case, seed):
    """The cell fields of the initial state in 64 bits."""
    p = _params(case)
    x, v = _state(p, seed)
    Nc, Ny = p["Nc"], p["Ny"]
    dx, dy = p["Lx"] / p["Nx"], p["Ly"] / p["Ny"]
    c = (x[:, 1] / dy).floor().long().clamp_(0, Ny - 1) + Ny * (x[:, 0] / dx).floor().long().clamp_(0, p["Nx"] - 1)
    zero = torch.zeros(Nc, dtype=torch.float64, device=DEVICE)
    N = torch.bincount(c, minlength=Nc)
    m = N.clamp(min=1).double()
    ux, uy = (zero.index_add(0, c, v[:, k]) / m for k in (0, 1))
    pec = zero.index_add(0, c, (v[:, 0] - ux[c]) ** 2 + (v[:, 1] - uy[c]) ** 2)
    dof = 2 * (N - 1).clamp(min=0)
    T = torch.where(dof > 0, pec / dof.clamp(min=1), zero)
    rho = N / (dx * dy)
    P = rho * T + p["Kvirial"] * (rho - p["gamma"] / (p["a0"] * p["a0"]))
    return {"fields": {"N": N.to(torch.int32), "Ux": ux, "Uy": uy, "T": T, "rho": rho, "P": P}}


def exact(case, seed):
    """The outputs that plain 64-bit arithmetic gives. The steps themselves have no such value:
    their trajectories follow the framework's random streams."""
    if case["kind"] == "learned":
        return _exact_learned(case, seed)
    if case["kind"] == "phases":
        return _exact_fields(case, seed)
    return None
