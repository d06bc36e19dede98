"""Workloads of the advection library, as a user's program runs them: whole
RK runs on a resident state, the tendency on device arrays, RK steps on a
state that lives on the host, the derivative operators and batched ensembles.

A case is a dict of plain values; `prepare` builds what the program holds
before the call, `run` is one pass through the public entry points, `exact`
the same result in plain float64 torch operations.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "scale-dg-kernel-extraction_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import sdg_b200 as sdg  # noqa: E402

_FLAGS = {
    "GPU": 0,
    "OPT1": sdg.FLAG_EXACT,
    "GENERAL": sdg.FLAG_EXACT | sdg.FLAG_ORDER_GENERAL,
    "MIXED": sdg.FLAG_MIXED,
}


def _steps(name, box, p, form, vel, steps, log):
    c = {"kind": "steps", "nex": box[0], "ney": box[1], "nez": box[2], "p": p, "form": form,
         "vel": vel, "steps": steps, "log": log}
    return dict(c, name=name) if name else c


def listed():
    return [
        # The reference's own input.conf: 4^3 elements, p = 7, OPT1, a min/max
        # line after every 100 steps.
        _steps("input_conf_4c_p7", (4, 4, 4), 7, "OPT1", "constant", 100, True),
        # The plain GENERAL run: 8^3 elements, p = 3, 100 steps.
        _steps("general_8c_p3", (8, 8, 8), 3, "GENERAL", "constant", 100, True),
        # Production size in FP64 (the headline mesh) and in the mixed form,
        # at p = 7 and with the same number of nodes at p = 15.
        _steps("fp64_32c_p7", (32, 32, 32), 7, "GPU", "constant", 5, False),
        _steps("mixed_32c_p7", (32, 32, 32), 7, "MIXED", "divfree", 5, False),
        _steps("mixed_16c_p15", (16, 16, 16), 15, "MIXED", "divfree", 5, False),
        # A ragged box of high order, the size of one served request.
        _steps("fp64_13x11x9_p11", (13, 11, 9), 11, "GPU", "constant", 20, False),
        # A ragged box of low order: many small elements.
        _steps("fp64_36x30x25_p2", (36, 30, 25), 2, "GPU", "constant", 10, False),
        # One small tendency call on device arrays with its halo update, as a
        # program with a time loop of its own makes it (latency).
        {"name": "tend_5x4x3_p4", "kind": "tend", "nex": 5, "ney": 4, "nez": 3, "p": 4,
         "form": "GPU"},
        # A host program that hands its state over for one RK step at a time.
        {"name": "host_24c_p7", "kind": "host", "nex": 24, "ney": 24, "nez": 24, "p": 7,
         "form": "GPU", "steps": 1},
        # The five-field derivative of the Euler fluxes, and the gradient of
        # one field.
        {"name": "divlike_20c_p7", "kind": "deriv", "ne": 8000, "p": 7, "nvar": 5,
         "form": "GPU"},
        {"name": "gradlike_7429_p9", "kind": "deriv", "ne": 7429, "p": 9, "nvar": 0,
         "form": "GPU"},
        # An ensemble of uneven boxes and orders, results fetched at the end.
        {"name": "batch_12_fp64", "kind": "batch", "count": 12, "lo": 6, "hi": 16,
         "orders": "3,5,7,9", "mixed": False, "steps": 50, "draw": 4},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, p, dofs):
    """A box of about `dofs` nodes whose three extents differ by up to 2x."""
    ne = max(1.0, dofs / (p + 1) ** 3)
    s = [rng.uniform(0.7, 1.4) for _ in range(3)]
    f = (ne / (s[0] * s[1] * s[2])) ** (1.0 / 3.0)
    return tuple(max(2, int(round(x * f))) for x in s)


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["tend", "tend", "host", "deriv", "deriv", "batch"])
    p = rng.randint(1, 15)
    if kind == "steps":
        dofs = _log_uniform(rng, 4000, 16_000_000)
        box = _box(rng, p, dofs)
        n = box[0] * box[1] * box[2] * (p + 1) ** 3
        most = max(1, min(100, 80_000_000 // n))
        form = rng.choice(["GPU", "GPU", "GPU", "MIXED", "MIXED", "OPT1", "GENERAL"])
        return _steps(None, box, p, form, rng.choice(["constant", "divfree"]),
                      _log_uniform(rng, 1, most), rng.random() < 0.3)
    if kind == "tend":
        box = _box(rng, p, _log_uniform(rng, 4000, 16_000_000))
        return {"kind": "tend", "nex": box[0], "ney": box[1], "nez": box[2], "p": p,
                "form": rng.choice(["GPU", "GPU", "GPU", "OPT1", "GENERAL"])}
    if kind == "host":
        box = _box(rng, p, _log_uniform(rng, 20_000, 8_000_000))
        return {"kind": "host", "nex": box[0], "ney": box[1], "nez": box[2], "p": p,
                "form": rng.choice(["GPU", "GPU", "MIXED", "OPT1"]), "steps": rng.randint(1, 5)}
    if kind == "deriv":
        nvar = rng.choice([0, 1, 3, 5, 5])
        ne = max(1, _log_uniform(rng, 4000, 20_000_000) // ((p + 1) ** 3 * max(1, nvar)))
        return {"kind": "deriv", "ne": ne, "p": p, "nvar": nvar,
                "form": rng.choice(["GPU", "GPU", "OPT1", "GENERAL"])}
    lo = rng.randint(3, 6)
    return {"kind": "batch", "count": rng.randint(2, 12), "lo": lo, "hi": rng.randint(lo, 14),
            "orders": rng.choice(["3,5,7,9", "3,5,7,9", "2,4,6,8", "3,4,5,6,7,8,9,10,11"]),
            "mixed": rng.random() < 0.5, "steps": rng.randint(5, 50),
            "draw": rng.randint(0, 1 << 20)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _lgl(p):
    """Node coordinates, D(i,l) and Lift(n,f) of the operator file, as read."""
    path = os.path.join(_ROOT, "operator_data", "p%d.dat" % p)
    with open(path) as f:
        v = np.array(f.read().split(), dtype=np.float64)
    nq = p + 1
    x, d, lift = v[:nq], v[nq:nq + nq * nq], v[nq + nq * nq:nq + nq * nq + 6 * nq ** 3]
    return x, d.reshape(nq, nq).T.copy(), lift.reshape(6, nq, nq, nq)  # lift[f][k][j][i]


def _fields(box, p, vel, seed):
    """q, u, v, w on the GPU, shaped (NeZ, NeY, NeX, k, j, i): a Gaussian bump
    and eight Fourier modes; a constant velocity or a divergence-free one."""
    rng = np.random.default_rng([seed, p, *box])
    x = torch.tensor((_lgl(p)[0] + 1.0) / 2.0, device="cuda")
    nq = p + 1
    axes = []
    for d in range(3):  # x, y, z
        c = (torch.arange(box[d], device="cuda", dtype=torch.float64)[:, None] + x[None, :]) / box[d]
        shape = [1] * 6
        shape[2 - d], shape[5 - d] = box[d], nq
        axes.append(c.reshape(shape))
    X, Y, Z = axes
    g = lambda c: torch.exp(-(c - 0.5) ** 2 / (2 * 0.1 ** 2))  # noqa: E731
    q = g(X) * g(Y) * g(Z)
    for _ in range(8):
        k = rng.integers(1, 5, 3)
        a, ph = rng.normal(0.0, 0.01), rng.uniform(0.0, 2 * math.pi, 3)
        s = [torch.sin(2 * math.pi * int(k[d]) * axes[d] + float(ph[d])) for d in range(3)]
        q = q + float(a) * s[0] * s[1] * s[2]
    q = q.contiguous()
    if vel == "divfree":
        ph = rng.uniform(0.0, 2 * math.pi, 3)
        w3 = [torch.sin(2 * math.pi * c + float(f)) for c, f in zip((Y, Z, X), ph)]
        u, v, w = (f.expand(q.shape).contiguous() for f in w3)
    else:
        u, v, w = (torch.full_like(q, float(c)) for c in rng.uniform(-1.0, 1.0, 3))
    return q, u, v, w


def _dt(box, p):
    return 0.1 / max(box) / (p + 1) ** 2


def _host(t):
    return t.reshape(-1).cpu().numpy()


def _box_of(case):
    return case["nex"], case["ney"], case["nez"]


@functools.lru_cache(maxsize=4)
def _mesh(box, p):
    ops = sdg.read_operators(p)
    return ops, sdg.mesh_setup(*box, p, ops.x1D)


def _members(case):
    """Extents and order of each instance of an ensemble."""
    rng = np.random.default_rng(case["draw"])
    orders = [int(x) for x in case["orders"].split(",")]
    return [((int(n),) * 3, int(rng.choice(orders)))
            for n in rng.integers(case["lo"], case["hi"] + 1, case["count"])]


def _deriv_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["ne"] * max(1, case["nvar"]) * (case["p"] + 1) ** 3
    return [torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
            for _ in range(3 if case["nvar"] else 1)]


def prepare(case, seed):
    if case["kind"] == "deriv":
        ins = _deriv_inputs(case, seed)
        return {"case": case, "D": sdg.read_operators(case["p"]).D1D, "ins": ins,
                "outs": [torch.empty_like(ins[0]) for _ in range(3)]}
    if case["kind"] == "batch":
        b = sdg.Batch(sdg.FLAG_MIXED if case["mixed"] else 0)
        for m, (box, p) in enumerate(_members(case)):
            f = _fields(box, p, "constant", seed + 7919 * m)
            b.add(*box, p, sdg.read_operators(p), *[_host(t) for t in f], _dt(box, p))
        b.commit()
        return {"case": case, "batch": b}
    box, p = _box_of(case), case["p"]
    ops, mesh = _mesh(box, p)
    h = sdg.Handle(ops, mesh, _FLAGS[case["form"]])
    if case["kind"] == "tend":
        stream = torch.cuda.Stream()
        n, full = mesh.Np * mesh.Ne, mesh.Np * mesh.NeA
        arrs = []
        for f in _fields(box, p, "divfree", seed):
            a = torch.zeros(full, device="cuda", dtype=torch.float64)
            a[:n] = f.reshape(-1)
            arrs.append(a)
        torch.cuda.synchronize()
        for a in arrs[1:]:
            h.update_halo_dev(a, stream.cuda_stream)
        return {"case": case, "h": h, "stream": stream, "arrs": arrs,
                "dqdt": torch.zeros(full, device="cuda", dtype=torch.float64), "n": n}
    fields = _fields(box, p, case.get("vel", "constant"), seed)
    for which, f in zip((sdg.FIELD_Q, sdg.FIELD_U, sdg.FIELD_V, sdg.FIELD_W), fields):
        h.set_field(which, _host(f))
    s = {"case": case, "h": h, "dt": _dt(box, p), "n": mesh.Np * mesh.Ne}
    if case["kind"] == "host":
        s["pinned"] = fields[0].reshape(-1).cpu().pin_memory()
        s["q"] = s["pinned"].numpy()
    return s


def run(state):
    case = state["case"]
    if case["kind"] == "steps":
        h = state["h"]
        h.rk3_steps(state["dt"], case["steps"])
        # A view of the handle's own array, which lives as long as the handle.
        q = h.resident_array(sdg.FIELD_Q)[:state["n"]]
        q.handle = h
        if case["log"]:
            lo, hi = h.minmax()
            return {"q": q, "min": lo, "max": hi}
        return {"q": q}
    if case["kind"] == "tend":
        h, s = state["h"], state["stream"].cuda_stream
        h.update_halo_dev(state["arrs"][0], s)
        h.cal_tend_dev(state["dqdt"], *state["arrs"], s)
        return state["dqdt"][:state["n"]]
    if case["kind"] == "host":
        return state["h"].rk3_steps_host(state["q"], state["dt"], case["steps"])
    if case["kind"] == "deriv":
        ins, outs = state["ins"], state["outs"]
        flags = _FLAGS[case["form"]]
        if case["nvar"]:
            sdg.divlike_dirXYZ_var_dev(state["D"], case["nvar"], case["ne"], *ins, *outs, flags)
        else:
            sdg.gradlike_dirXYZ_dev(state["D"], case["ne"], ins[0], *outs, flags)
        return list(outs)
    b = state["batch"]
    b.run(case["steps"])
    return [b.get(i) for i in range(case["count"])]


def work(case):
    """Inputs read once, outputs written once; about 6 Nq + 22 operations per
    node and right-hand side."""
    nq = case["p"] + 1 if "p" in case else 0
    if case["kind"] == "deriv":
        n = case["ne"] * max(1, case["nvar"]) * nq ** 3
        return {"bytes": (48 if case["nvar"] else 32) * n, "flops": 6 * nq * n}
    if case["kind"] == "batch":
        size = [(b[0] * b[1] * b[2] * (p + 1) ** 3, p + 1) for b, p in _members(case)]
        per = 28 if case["mixed"] else 40
        return {"bytes": per * sum(n for n, _ in size),
                "flops": sum(3 * case["steps"] * n * (6 * q + 22) for n, q in size)}
    n = case["nex"] * case["ney"] * case["nez"] * nq ** 3
    if case["kind"] == "tend":
        return {"bytes": 40 * n, "flops": (6 * nq + 22) * n}
    per = 28 if case["form"] == "MIXED" else 40
    return {"bytes": per * n, "flops": 3 * case["steps"] * n * (6 * nq + 22)}


# ---------------------------------------------------------------------------
# The same results in plain float64 torch
# ---------------------------------------------------------------------------
def _contract(D, f, axis):
    """sum_l D(i,l) f(..., l, ...) along one of the three node axes."""
    return torch.movedim(torch.movedim(f, axis, -1) @ D.T, -1, axis)


def _rhs(q, vel, D, lift, box):
    """dqdt of linear advection: sum-factorised derivative, upwind face flux
    and its lift, periodic in the three directions."""
    out = torch.zeros_like(q)
    for d in range(3):  # x, y, z
        e_ax, n_ax, un, esc = 2 - d, 5 - d, vel[d], 2.0 * box[d]
        out -= esc * _contract(D, q * un, n_ax)
        last = q.shape[n_ax] - 1
        for side in (0, 1):
            at = last if side else 0
            qm, um = q.select(n_ax, at), un.select(n_ax, at)
            roll = (-1 if side else 1)
            qp = torch.roll(q.select(n_ax, last - at), roll, e_ax)
            up = torch.roll(un.select(n_ax, last - at), roll, e_ax)
            sg = 1.0 if side else -1.0
            vm, vp = um * sg, up * sg
            alpha = 0.5 * (vp + vm).abs()
            flux = 0.5 * esc * (qp * vp - qm * vm - alpha * (qp - qm))
            face = {(0, 0): 3, (0, 1): 1, (1, 0): 0, (1, 1): 2, (2, 0): 4, (2, 1): 5}[d, side]
            out -= lift[face] * flux.unsqueeze(n_ax)
    return out


def _rk3(q, vel, p, box, dt, steps):
    _, D, lift = _lgl(p)
    D, lift = torch.tensor(D, device="cuda"), torch.tensor(lift, device="cuda")
    for _ in range(steps):
        q1 = q + dt * _rhs(q, vel, D, lift, box)
        q2 = 0.75 * q + 0.25 * (q1 + dt * _rhs(q1, vel, D, lift, box))
        q = q / 3.0 + (2.0 / 3.0) * (q2 + dt * _rhs(q2, vel, D, lift, box))
    return q


def exact(case, seed):
    if case["kind"] == "deriv":
        D, nq = torch.tensor(_lgl(case["p"])[1], device="cuda"), case["p"] + 1
        ins = _deriv_inputs(case, seed)
        ins = ins if case["nvar"] else ins * 3
        return [_contract(D, f.view(-1, nq, nq, nq), 3 - d).reshape(-1)
                for d, f in enumerate(ins)]
    if case["kind"] == "batch":
        out = []
        for m, (box, p) in enumerate(_members(case)):
            q, *vel = _fields(box, p, "constant", seed + 7919 * m)
            r = _rk3(q, vel, p, box, _dt(box, p), case["steps"])
            out.append(_host(r).reshape(-1, (p + 1) ** 3).T)
        return out
    box, p = _box_of(case), case["p"]
    if case["kind"] == "tend":
        q, *vel = _fields(box, p, "divfree", seed)
        _, D, lift = _lgl(p)
        return _rhs(q, vel, torch.tensor(D, device="cuda"), torch.tensor(lift, device="cuda"),
                    box).reshape(-1)
    q, *vel = _fields(box, p, case.get("vel", "constant"), seed)
    r = _rk3(q, vel, p, box, _dt(box, p), case["steps"]).reshape(-1)
    if case["kind"] == "host":
        return _host(r)
    if case["log"]:
        return {"q": r, "min": float(r.min()), "max": float(r.max())}
    return {"q": r}
