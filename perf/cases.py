"""The work that users of the library have it do, as cases that can be timed and checked.

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare` makes what a
program holds before the call, `run` is one pass through the package's public entry points,
`work` what a pass cannot do without, and `exact` the same outputs in 64 bits from plain torch.

Kinds of work:
  stepwise  a consumer that calls step() once per lattice step and then reads the fields (the
            member-by-member use of the drop-in solver class);
  job       upload a state from pinned host memory, run, read rho / u_x / u_y into pinned memory
            (the end-to-end form of the benchmark);
  wake      cylinder wake: run a few steps, sample the force on the disc, repeat, read the fields;
  probe     open cylinder: timed chunks with a velocity probe between them, read the fields (the
            command-line driver's loop);
  strips    the strip engine's run with the populations read back;
  batch     an ensemble of uneven closed channels, run and read back instance by instance;
  adjoint   one iteration of an optimisation over a drag field: set it, forward, backward.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

PKG = "simulation-de-fluide-par-la-m-thode-de-boltzmann-sur-r-seau-lbm-du-cpu-au-multi-gpu_gb300"

CX = (0, 1, 0, -1, 0, 1, -1, -1, 1)
CY = (0, 0, 1, 0, -1, 1, 1, -1, -1)
OPP = (0, 3, 4, 1, 2, 7, 8, 5, 6)
W = (4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4
HOST_BYTES = {"fp32": 4, "fp16": 4, "bf16": 4, "fp64": 8}
STORE_BYTES = {"fp32": 4, "fp16": 2, "bf16": 2, "fp64": 8}
FLOPS_PER_CELL = 200  # moments, equilibrium, Guo source and relaxation of one cell
ON_CHIP_BYTES = 100e6  # two states below this stay in the on-chip memories between steps


def _pkg():
    return importlib.import_module(PKG)


def listed():
    return [
        # The smallest calls: the 53 x 31 obstacle channel of the reference's own tests, stepped
        # one call at a time.
        {"name": "stepwise_fp32", "kind": "stepwise", "precision": "fp32", "nx": 53, "ny": 31, "discs": 1, "tau": 0.8,
         "fx": 1e-5, "steps": 16},
        # A small validation run: Poiseuille channel of the accuracy study, 16-bit storage.
        {"name": "poiseuille_fp16", "kind": "job", "precision": "fp16", "nx": 128, "ny": 66, "discs": 0, "tau": 0.8,
         "fx": 1.2e-5, "steps": 400},
        # The cylinder wake's inner loop: 50 steps between two samples of the force on the disc.
        {"name": "wake_fp32", "kind": "wake", "precision": "fp32", "nx": 1024, "ny": 256, "discs": 1, "tau": 0.548,
         "fx": 6.784303312490499e-07, "every": 50, "samples": 8},
        # The reference's Strouhal case: open cylinder, probed every 200 steps as its driver does.
        {"name": "probe_fp32", "kind": "probe", "precision": "fp32", "nx": 1000, "ny": 320, "discs": 1, "tau": 0.56,
         "u_in": 0.05, "every": 200, "samples": 2},
        # A mid-size study at a ragged width, 16-bit storage.
        {"name": "channel_fp16", "kind": "job", "precision": "fp16", "nx": 1021, "ny": 700, "discs": 3, "tau": 0.6,
         "fx": 1e-6, "steps": 200},
        # The headline grid end to end, plain FP32 and 16-bit storage.
        {"name": "large_fp32", "kind": "job", "precision": "fp32", "nx": 4096, "ny": 4096, "discs": 0, "tau": 0.6,
         "fx": 1e-6, "steps": 100},
        {"name": "large_fp16", "kind": "job", "precision": "fp16", "nx": 4096, "ny": 4096, "discs": 0, "tau": 0.6,
         "fx": 1e-6, "steps": 100},
        # A double-precision validation run.
        {"name": "channel_fp64", "kind": "job", "precision": "fp64", "nx": 1024, "ny": 512, "discs": 2, "tau": 0.6,
         "fx": 1e-6, "steps": 40},
        # The decomposed lattice: five strips of a ragged grid.
        {"name": "strips_fp32", "kind": "strips", "precision": "fp32", "nx": 2047, "ny": 1025, "discs": 4, "tau": 0.6,
         "fx": 1e-6, "strips": 5, "steps": 100},
        # Ensembles of uneven channels: the workload's sizes, and one of small channels.
        {"name": "batch_fp32", "kind": "batch", "precision": "fp32", "count": 48, "nx_lo": 64, "nx_hi": 1024,
         "ny_lo": 32, "ny_hi": 512, "steps": 400},
        {"name": "batch_fp16", "kind": "batch", "precision": "fp16", "count": 24, "nx_lo": 64, "nx_hi": 256,
         "ny_lo": 32, "ny_hi": 128, "steps": 500},
        # Forward and backward of the adjoint workload's batch of drag fields.
        {"name": "adjoint_fp32", "kind": "adjoint", "precision": "fp32", "nx": 512, "ny": 128, "batch": 32, "tau": 0.6,
         "fx": 5e-6, "steps": 300, "window": 100, "every": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stepwise", "job", "job", "job", "wake", "probe", "strips", "batch", "adjoint"])
    precision = rng.choice(["fp32", "fp32", "fp16", "bf16", "fp64"])
    tau = round(rng.uniform(0.54, 0.95), 4)
    fx = float("%.3g" % (10 ** rng.uniform(-6.5, -5.0)))
    cap = 2.0e7 if precision == "fp64" else 1.2e9  # cell updates of a pass
    if kind == "stepwise":
        return {"kind": kind, "precision": precision, "nx": _log_int(rng, 24, 400), "ny": _log_int(rng, 20, 200),
                "discs": 1, "tau": tau, "fx": fx, "steps": rng.randint(4, 40)}
    if kind == "job":
        nx, ny = _log_int(rng, 60, 4000), _log_int(rng, 40, 4000)
        steps = max(4, int(min(_log_int(rng, 20, 400), cap / (nx * ny))))
        return {"kind": kind, "precision": precision, "nx": nx, "ny": ny, "discs": rng.randint(0, 3), "tau": tau,
                "fx": fx, "steps": steps}
    if kind == "wake":
        nx, ny = _log_int(rng, 200, 2000), _log_int(rng, 80, 500)
        every = rng.choice([20, 50, 100])
        return {"kind": kind, "precision": precision, "nx": nx, "ny": ny, "discs": 1, "tau": tau, "fx": fx,
                "every": every, "samples": max(1, int(min(8, cap / (nx * ny * every))))}
    if kind == "probe":
        nx, ny = _log_int(rng, 120, 2000), _log_int(rng, 48, 600)
        every = 200 if precision != "fp64" else 20
        return {"kind": kind, "precision": precision, "nx": nx, "ny": ny, "discs": 1, "tau": tau, "u_in": 0.05,
                "every": every, "samples": max(1, int(min(4, cap / (nx * ny * every))))}
    if kind == "strips":
        nx, ny = _log_int(rng, 100, 3000), _log_int(rng, 60, 2000)
        return {"kind": kind, "precision": precision, "nx": nx, "ny": ny, "discs": rng.randint(0, 4), "tau": tau,
                "fx": fx, "strips": rng.randint(1, 16), "steps": max(4, int(min(100, cap / (nx * ny))))}
    if kind == "batch":
        big = rng.random() < 0.4
        return {"kind": kind, "precision": precision, "count": rng.randint(3, 48), "nx_lo": 64,
                "nx_hi": 1024 if big else 256, "ny_lo": 32, "ny_hi": 512 if big else 128,
                "steps": (5 if precision == "fp64" else rng.randint(50, 300))}
    precision = rng.choice(["fp32", "fp32", "fp64"])
    steps = rng.randint(10, 40) if precision == "fp64" else rng.randint(40, 240)
    return {"kind": kind, "precision": precision, "nx": _log_int(rng, 100, 512), "ny": _log_int(rng, 40, 128),
            "batch": rng.randint(1, 4 if precision == "fp64" else 24), "tau": tau, "fx": fx, "steps": steps,
            "window": max(1, steps // 3), "every": rng.randint(10, 100)}


# ------------------------------------------------------------------------------------- inputs


def _rng(seed, salt=0):
    return np.random.RandomState((int(seed) * 1000003 + 7919 * salt + 12345) % (2 ** 32 - 1))


def _mask(nx, ny, discs, r, inlet=False):
    """Walled channel with `discs` discs clear of the walls (and of an open inlet and outlet)."""
    m = np.zeros((ny, nx), np.uint8)
    m[0] = m[-1] = 1
    y, x = np.arange(ny)[:, None], np.arange(nx)[None, :]
    for _ in range(discs):
        rad = min(ny / 8.0, nx / 12.0, 24.0) * (0.7 + 0.3 * r.rand())
        cx = nx * (0.25 + 0.1 * r.rand() if inlet or discs == 1 else 0.1 + 0.8 * r.rand())
        cy = rad + 2 + (ny - 2 * rad - 4) * (0.45 + 0.1 * r.rand() if inlet else r.rand())
        m |= ((x - cx) ** 2 + (y - cy) ** 2 <= rad * rad).astype(np.uint8)
    return m


def _state(mask, seed, dtype, device):
    """Post-streaming populations f_i - w_i (ny, nx, 9) near the equilibrium of a slow flow, with
    a perturbation of every population: a developing channel flow."""
    ny, nx = mask.shape
    gen = torch.Generator(device=device).manual_seed(int(seed) * 7 + 1)
    x = torch.arange(nx, device=device, dtype=torch.float32) * (2 * math.pi / nx)
    y = torch.arange(ny, device=device, dtype=torch.float32) / max(ny - 1, 1)
    ph = torch.rand(4, generator=gen, device=device) * 6.28
    prof = (4 * y * (1 - y))[:, None]
    ux = 0.03 * prof * (1 + 0.2 * torch.sin(2 * x + ph[0])[None])
    uy = 0.004 * prof * torch.sin(3 * x + ph[1])[None]
    dr = 1e-3 * torch.sin(x + ph[2])[None] * torch.cos(3.1 * y + ph[3])[:, None]
    out = torch.empty(ny, nx, 9, device=device, dtype=dtype)
    for i in range(9):
        cu = CX[i] * ux + CY[i] * uy
        g = W[i] * (dr + (1 + dr) * (3 * cu + 4.5 * cu * cu - 1.5 * (ux * ux + uy * uy)))
        g = g + 2e-4 * W[i] * (torch.rand(ny, nx, generator=gen, device=device) - 0.5)
        out[..., i] = g.to(dtype)
    out[torch.from_numpy(mask).to(device) != 0] = 0
    return out


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _dtype(case):
    return torch.float64 if case["precision"] == "fp64" else torch.float32


def _inputs(case, seed, device):
    """mask(s), initial state(s) and per-case parameters, from the seed alone."""
    kind = case["kind"]
    if kind == "batch":
        r = _rng(seed, 3)
        specs = []
        # Sizes come from the case alone (the same work for every seed), discs from the seed.
        rs = _rng(11, 5)
        for k in range(case["count"]):
            nx = case["nx_lo"] + int(rs.rand() * (case["nx_hi"] - case["nx_lo"] + 1))
            ny = case["ny_lo"] + int(rs.rand() * (case["ny_hi"] - case["ny_lo"] + 1))
            specs.append({"nx": nx, "ny": ny, "mask": _mask(nx, ny, 1 + int(4 * r.rand()), r),
                          "tau": 0.52 + 0.48 * r.rand(), "fx": 1e-6 + 9e-6 * r.rand(), "fy": 0.0})
        states = [_state(s["mask"], seed * 64 + k, _dtype(case), device) for k, s in enumerate(specs)]
        return specs, states
    if kind == "adjoint":
        mask = _mask(case["nx"], case["ny"], 0, _rng(seed))
        r = _rng(seed, 9)
        b, nx, ny = case["batch"], case["nx"], case["ny"]
        y, x = np.arange(ny)[:, None], np.arange(nx)[None, :]
        alpha = np.zeros((b, ny, nx))
        for k in range(b):  # smooth random drag fields in [0, 0.1]
            for _ in range(6):
                cx, cy, w, a = r.rand() * nx, r.rand() * ny, 8 + 24 * r.rand(), 0.5 + 0.5 * r.rand()
                dx = np.abs(x - cx)
                dx = np.minimum(dx, nx - dx)
                alpha[k] += a * np.exp(-dx * dx / (2 * w * w)) * np.exp(-(y - cy) ** 2 / (2 * w * w))
            alpha[k] *= 0.1 / alpha[k].max()
        alpha[:, mask != 0] = 0.0
        return mask, alpha.reshape(b, -1)
    mask = _mask(case["nx"], case["ny"], case["discs"], _rng(seed), inlet=kind == "probe")
    if kind in ("probe", "wake", "stepwise"):
        return mask, None
    return mask, _state(mask, seed, _dtype(case), device)


def _u0(case, seed):
    """Start velocity of the runs that begin from a uniform equilibrium."""
    return 0.05 * (1.0 + 0.1 * (_rng(seed, 2).rand() - 0.5))


def prepare(case, seed):
    L = _pkg()
    kind, p = case["kind"], case["precision"]
    if kind == "batch":
        specs, states = _inputs(case, seed, "cuda")
        b = L.Batch(specs, precision=p)
        for k, s in enumerate(states):
            b.set_populations(k, s.cpu().numpy())
        return {"case": case, "h": b}
    if kind == "adjoint":
        mask, alpha = _inputs(case, seed, "cuda")
        a = L.Adjoint(case["nx"], case["ny"], case["tau"], case["fx"], 0.0, mask, precision=p, batch=case["batch"],
                      checkpoint_every=case["every"])
        return {"case": case, "h": a, "alpha": alpha}
    mask, s0 = _inputs(case, seed, "cuda")
    nx, ny, tau, fx = case["nx"], case["ny"], case["tau"], case.get("fx", 0.0)
    if kind == "strips":
        h = L.Strips(nx, ny, tau, fx, 0.0, mask, case["strips"], precision=p)
        h.set_populations(s0.cpu().numpy())
        return {"case": case, "h": h}
    h = L.Solver(nx, ny, tau, fx, 0.0, mask, precision=p)
    st = {"case": case, "h": h}
    if kind == "job":
        st["in"] = _pinned(s0)
        st["out"] = [torch.empty(ny * nx, dtype=_dtype(case), pin_memory=True) for _ in range(3)]
        st["in_np"], st["out_np"] = st["in"].numpy(), tuple(t.numpy() for t in st["out"])
        return st
    u = _u0(case, seed)
    if kind == "probe":
        h.set_inflow_outflow(case["u_in"])
        u = case["u_in"] * u / 0.05
    h.init_equilibrium(1.0, u, 0.0)
    if kind == "wake":
        disc = mask.copy()
        disc[0] = disc[-1] = 0
        h.set_body(disc)
    return st


def _probe_at(case):
    return int(0.7 * case["nx"]), case["ny"] // 2


def run(state):
    case, h = state["case"], state["h"]
    kind = case["kind"]
    if kind == "stepwise":
        for _ in range(case["steps"]):
            h.step()
        return list(h.macroscopic())
    if kind == "job":
        h.set_populations(state["in_np"])
        h.run(case["steps"])
        h.macroscopic(out=state["out_np"])
        return state["out"]
    if kind == "wake":
        force = []
        for _ in range(case["samples"]):
            h.run(case["every"])
            force.append(h.body_force())
        return [np.array(force), *h.macroscopic()]
    if kind == "probe":
        x, y = _probe_at(case)
        seen = []
        for _ in range(case["samples"]):
            h.timed_run(case["every"])
            seen.append(h.populations_at(x, y))
        return [np.array(seen), *h.macroscopic()]
    if kind == "strips":
        h.run(case["steps"])
        return h.populations()
    if kind == "batch":
        h.run(case["steps"])
        return [h.populations(k) for k in range(case["count"])]
    h.set_alpha(state["alpha"])
    j = h.forward(case["steps"], case["window"])
    g = h.backward()
    return {"J": j, "tau": g["tau"], "fx": g["fx"], "fy": g["fy"], "alpha": g["alpha"]}


def _cells(case):
    if case["kind"] == "batch":
        rs = _rng(11, 5)
        n = 0
        for _ in range(case["count"]):
            nx = case["nx_lo"] + int(rs.rand() * (case["nx_hi"] - case["nx_lo"] + 1))
            ny = case["ny_lo"] + int(rs.rand() * (case["ny_hi"] - case["ny_lo"] + 1))
            n += nx * ny
        return n
    return case["nx"] * case["ny"] * case.get("batch", 1)


def work(case):
    """Bytes: every population read and written once per step where two states do not fit on the
    chip, once per pass where they do; plus the uploads and the fields read back. A backward step
    reads the state and the next adjoint, writes the adjoint and updates the drag's gradient."""
    n, kind = _cells(case), case["kind"]
    steps = case["steps"] if "steps" in case else case["every"] * case["samples"]
    state, host = 9 * STORE_BYTES[case["precision"]] * n, HOST_BYTES[case["precision"]] * n
    moved = 2 * state * (steps if 2 * state > ON_CHIP_BYTES else 1)
    flops = FLOPS_PER_CELL * n * steps
    if kind == "adjoint":
        elem = STORE_BYTES[case["precision"]]
        # Forward, then per step the adjoint (3 states and 3 fields); recomputation is not counted.
        return {"bytes": steps * n * elem * (18 + 1 + 27 + 3) + 16 * n, "flops": 3 * flops}
    if kind == "job":
        moved += 9 * host + 3 * host
    elif kind in ("strips", "batch"):
        moved += 9 * host
    else:
        moved += 3 * host
    return {"bytes": moved, "flops": flops}


# ------------------------------------------------------------------------------ 64-bit answers


class _Pull(torch.autograd.Function):
    """y = x[..., idx] over the flat (direction, cell) axis; idx reads each fluid slot once, so
    the transpose is a gather by the inverse index."""

    @staticmethod
    def forward(ctx, x, idx, inv):
        ctx.save_for_backward(inv)
        return x.index_select(1, idx)

    @staticmethod
    def backward(ctx, g):
        (inv,) = ctx.saved_tensors
        pad = torch.cat([g, torch.zeros_like(g[:, :1])], 1)
        return pad.index_select(1, inv), None, None


def _links(masks, open_x, dev):
    """Flat index (9 n) of the slot each population is pulled from, over the concatenated cells of
    all masks: the neighbour's, or the opposite slot of the cell itself behind a solid."""
    total = sum(m.size for m in masks)
    rows = []
    for i in range(9):
        off, parts = 0, []
        for m in masks:
            ny, nx = m.shape
            s = torch.from_numpy(m).to(dev) != 0
            y = torch.arange(ny, device=dev)[:, None].expand(ny, nx)
            x = torch.arange(nx, device=dev)[None, :].expand(ny, nx)
            xc = torch.where(x == nx - 1, torch.full_like(x, nx - 2), x) if open_x and CX[i] == -1 else x
            xs, ys = (xc - CX[i]) % nx, (y - CY[i]) % ny
            src, own = i * total + off + ys * nx + xs, OPP[i] * total + off + y * nx + xc
            parts.append(torch.where(s[ys, xs], own, src).reshape(-1))
            off += m.size
        rows.append(torch.cat(parts))
    return torch.cat(rows)


def _moments(s, fx, fy, kf=1.0):
    rho = 1 + s.sum(1)
    ux = (s[:, 1] - s[:, 3] + s[:, 5] - s[:, 6] - s[:, 7] + s[:, 8] + 0.5 * fx) / (rho * kf)
    uy = (s[:, 2] - s[:, 4] + s[:, 5] + s[:, 6] - s[:, 7] - s[:, 8] + 0.5 * fy) / (rho * kf)
    return rho, ux, uy


def _collide(s, tau, fx, fy, alpha=None):
    """Post-collision populations of s (batch, 9, cells)."""
    rho, ux, uy = _moments(s, fx, fy, 1.0 if alpha is None else 1 + 0.5 * alpha)
    if alpha is not None:
        fx, fy = fx - alpha * rho * ux, fy - alpha * rho * uy
    om = 1 / tau
    usq, uf = 1.5 * (ux * ux + uy * uy), ux * fx + uy * fy
    out = []
    for i in range(9):
        cu, cf = CX[i] * ux + CY[i] * uy, CX[i] * fx + CY[i] * fy
        geq = W[i] * ((rho - 1) + rho * (3 * cu + 4.5 * cu * cu - usq))
        out.append(s[:, i] - om * (s[:, i] - geq) + (1 - 0.5 * om) * W[i] * (3 * (cf - uf) + 9 * cu * cf))
    return torch.stack(out, 1)


def _step(s, idx, tau, fx, fy, inlet):
    r = _collide(s, tau, fx, fy)
    y = r.reshape(r.shape[0], -1).index_select(1, idx).reshape(s.shape)
    if inlet is not None:
        at, eq = inlet
        for i in (1, 5, 8):
            y[0, i, at] = eq[i]
    return y


def _equilibrium(rho, ux, uy):
    return [W[i] * ((rho - 1) + rho * (3 * (CX[i] * ux + CY[i] * uy) + 4.5 * (CX[i] * ux + CY[i] * uy) ** 2
                                       - 1.5 * (ux * ux + uy * uy))) for i in range(9)]


def _exact_adjoint(case, seed, dev):
    mask, alpha = _inputs(case, seed, dev)
    b, n = case["batch"], mask.size
    fluid = torch.from_numpy(mask.reshape(-1)).to(dev) == 0
    idx = _links([mask], False, dev)
    inv = torch.full((9 * n,), 9 * n, dtype=torch.int64, device=dev)
    keep = fluid.repeat(9)
    inv[idx[keep]] = torch.arange(9 * n, device=dev)[keep]
    leaf = [torch.full((b, 1), v, dtype=torch.float64, device=dev, requires_grad=True)
            for v in (case["tau"], case["fx"], 0.0)]
    al = torch.from_numpy(alpha).to(dev).requires_grad_(True)
    s = torch.zeros(b, 9, n, dtype=torch.float64, device=dev)
    steps, window = case["steps"], case["window"]
    nf = int(fluid.sum())

    def objective(s, fx, al):
        u = (s[:, 1] - s[:, 3] + s[:, 5] - s[:, 6] - s[:, 7] + s[:, 8] + 0.5 * fx) / ((1 + s.sum(1)) * (1 + 0.5 * al))
        return torch.where(fluid, u, torch.zeros_like(u)).sum(1) / (nf * window)

    def one(s, tau, fx, fy, al):
        r = _collide(s, tau, fx, fy, al)
        return _Pull.apply(r.reshape(b, -1), idx, inv).reshape(b, 9, n)

    total = torch.zeros(b, dtype=torch.float64, device=dev)
    for t in range(steps + 1):
        if t >= steps - window + 1:
            total = total + checkpoint(objective, s, leaf[1], al, use_reentrant=False)
        if t < steps:
            s = checkpoint(one, s, *leaf, al, use_reentrant=False)
    total.sum().backward()
    return {"J": total.detach(), "tau": leaf[0].grad[:, 0], "fx": leaf[1].grad[:, 0], "fy": leaf[2].grad[:, 0],
            "alpha": al.grad}


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "adjoint":
        return _exact_adjoint(case, seed, dev)
    with torch.no_grad():
        inlet = None
        if kind == "batch":
            specs, states = _inputs(case, seed, dev)
            masks = [sp["mask"] for sp in specs]
            s = torch.cat([st.reshape(-1, 9) for st in states]).double().t()[None].contiguous()
            per = [torch.full((sp["mask"].size,), sp[k], dtype=torch.float64, device=dev)
                   for k in ("tau", "fx") for sp in specs]
            tau, fx, fy = torch.cat(per[:len(specs)]), torch.cat(per[len(specs):]), 0.0
        else:
            mask, s0 = _inputs(case, seed, dev)
            masks, tau, fx, fy = [mask], case["tau"], case.get("fx", 0.0), 0.0
            if s0 is None:
                u = _u0(case, seed)
                if kind == "probe":
                    u = case["u_in"] * u / 0.05
                eq = torch.tensor(_equilibrium(1.0, u, 0.0), dtype=torch.float64, device=dev)
                s = eq[None, :, None].repeat(1, 1, mask.size)
            else:
                s = s0.reshape(-1, 9).double().t()[None].contiguous()
            del s0
        flat = np.concatenate([m.reshape(-1) for m in masks])
        solid = torch.from_numpy(flat).to(dev) != 0
        idx = _links(masks, kind == "probe", dev)
        if kind == "probe":
            ny, nx = masks[0].shape
            at = torch.arange(ny, device=dev) * nx
            inlet = (at, _equilibrium(1.0, case["u_in"], 0.0))
            s[:, :, solid] = 0
            for i in (1, 5, 8):
                s[0, i, at] = inlet[1][i]
        if kind == "batch":
            for _ in range(case["steps"]):
                s = _step(s, idx, tau, fx, fy, inlet)
            s[:, :, solid] = 0
            out, off = [], 0
            for m in masks:
                out.append(s[0, :, off:off + m.size].t().reshape(-1))
                off += m.size
            return out
        seen = []
        if kind in ("wake", "probe"):
            if kind == "wake":
                ny, nx = masks[0].shape
                body = masks[0].copy()
                body[0] = body[-1] = 0
                bt = torch.from_numpy(body).to(dev) != 0
                fl = torch.from_numpy(masks[0]).to(dev) == 0
            for _ in range(case["samples"]):
                for _ in range(case["every"]):
                    s = _step(s, idx, tau, fx, fy, inlet)
                if kind == "probe":
                    x, y = _probe_at(case)
                    seen.append(s[0, :, y * case["nx"] + x].clone())
                    continue
                g, f = s[0].reshape(9, ny, nx), [0.0, 0.0]
                for i in range(1, 9):
                    link = fl & torch.roll(bt, (-CY[i], -CX[i]), (0, 1))
                    v = ((g[OPP[i]] + W[i]) * link).sum()
                    f = [f[0] + 2 * CX[i] * v, f[1] + 2 * CY[i] * v]
                seen.append(torch.stack(f))
        else:
            for _ in range(case["steps"]):
                s = _step(s, idx, tau, fx, fy, inlet)
        if kind == "strips":
            s[:, :, solid] = 0
            return s[0].t().reshape(-1)
        m = [torch.where(solid, torch.zeros_like(v[0]), v[0]) for v in _moments(s, fx, fy)]
        return ([torch.stack(seen)] if seen else []) + m
