"""Performance cases: time loops of the engine as a user's program runs them.

A pass is one solve through the public Python entry points: the initial
iterate goes up from (page-locked) host memory, the time loop runs, the
result comes back.  Handles, known fields, border rules and schedules are
kept between passes, as a program that solves many initial states keeps
them.  ``exact`` repeats each solve with plain torch operations in float64.
"""
import math

import numpy as np
import torch

import masterthesis_gb300 as M
from masterthesis_gb300 import workloads as W


# ---- cases --------------------------------------------------------------------

def listed():
    return [
        # The reference's system-test scale: a few thousand nodes, hundreds of
        # steps; launches and latency are the whole cost.
        {"name": "heat_f64_tiny", "kind": "star", "precision": "f64", "border": "dirichlet", "source": "none",
         "nx": 17, "ny": 15, "nz": 16, "steps": 200},
        # The reference's flux-border system tests (source and border field
        # affine in time, rules per border class) on an odd grid.
        {"name": "pennes_neumann_f64_small", "kind": "star", "precision": "f64", "border": "neumann",
         "source": "affine", "nx": 40, "ny": 31, "nz": 27, "steps": 400},
        # The small documented heat workload: 64^3, 200 steps.
        {"name": "heat_f64_64", "kind": "star", "precision": "f64", "border": "dirichlet", "source": "none",
         "nx": 64, "ny": 64, "nz": 64, "steps": 200},
        # The headline path (plain FP64 heat sweep) on a grid far beyond L2.
        {"name": "heat_f64_256", "kind": "star", "precision": "f64", "border": "dirichlet", "source": "none",
         "nx": 256, "ny": 256, "nz": 256, "steps": 600},
        # Compensated FP32 pairs with a heat source, odd sizes.
        {"name": "pennes_f32x2_odd", "kind": "star", "precision": "f32x2", "border": "dirichlet", "source": "static",
         "nx": 201, "ny": 181, "nz": 163, "steps": 800},
        # Plain FP32 on a large grid: the HBM-bound end of the sweep.
        {"name": "heat_f32_large", "kind": "star", "precision": "f32", "border": "dirichlet", "source": "none",
         "nx": 320, "ny": 256, "nz": 256, "steps": 800},
        # The tissue examples: every coefficient a field, one border rule per
        # node (insulated head, convective top face).
        {"name": "tissue_f64", "kind": "tissue", "precision": "f64", "nx": 141, "ny": 121, "nz": 101, "steps": 400},
        # An ensemble of uneven Pennes instances (parameter studies).
        {"name": "ensemble_f64", "kind": "batch", "precision": "f64", "instances": 32, "lo": 32, "hi": 160,
         "steps": 100},
        # Conductivity gradient through the time loop with checkpoints
        # (parameter fitting).
        {"name": "gradient_f64", "kind": "adjoint", "precision": "f64", "nx": 97, "ny": 90, "nz": 83, "steps": 200,
         "snapshots": 16},
        # Elastic wave, three coupled fields with mixed derivatives.
        {"name": "lame_f64", "kind": "lame", "precision": "f64", "nx": 129, "ny": 111, "nz": 101, "steps": 400},
        # Maxwell leapfrog with a point source.
        {"name": "yee_f64", "kind": "yee", "precision": "f64", "nx": 128, "ny": 120, "nz": 113, "steps": 600},
        # Recorded rules of a multi-field problem class (the form the drop-in
        # Problem gives its users' classes): a resonant cavity.
        {"name": "linear_f64", "kind": "linear", "precision": "f64", "nx": 96, "ny": 81, "nz": 73, "steps": 400},
    ]


# kind -> (share of draws, least and most nodes, most node-steps, precisions)
_RANGES = {
    "star": (7, 512, 256 ** 3, 6e9, ("f64", "f64", "f64", "f32x2", "f32")),
    "tissue": (2, 4096, 200 ** 3, 1.5e9, ("f64", "f64", "f32")),
    "batch": (2, 32 ** 3, 96 ** 3, 3e9, ("f64", "f32x2")),
    "adjoint": (2, 4096, 110 ** 3, 1.5e8, ("f64", "f64", "f32x2")),
    "lame": (2, 4096, 144 ** 3, 5e8, ("f64", "f64", "f32x2")),
    "yee": (2, 4096, 144 ** 3, 1e9, ("f64", "f64", "f32", "f32x2")),
    "linear": (1, 4096, 96 ** 3, 2e8, ("f64",)),
}


def draw(rng):
    kinds = [k for k, r in _RANGES.items() for _ in range(r[0])]
    kind = rng.choice(kinds)
    _, lo, hi, budget, precisions = _RANGES[kind]
    case = {"kind": kind, "precision": rng.choice(precisions)}
    if kind == "batch":
        least = rng.randint(8, 48)
        most = rng.randint(least + 8, 160)
        count = rng.randint(4, 40)
        mean = ((least + most) / 2) ** 3
        return {**case, "instances": count, "lo": least, "hi": most,
                "steps": int(min(200, max(10, budget / (count * mean))))}
    nodes = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    side = nodes ** (1 / 3)
    a, b = (math.exp(rng.uniform(-0.4, 0.4)) for _ in range(2))
    n = [max(8, int(v)) for v in (side * a, side * b, side / (a * b))]
    steps = int(min(600, max(10, budget / (n[0] * n[1] * n[2]))) * rng.uniform(0.5, 1.0)) + 1
    case.update({"nx": n[0], "ny": n[1], "nz": n[2], "steps": steps})
    if kind == "star":
        case["border"] = rng.choice(("dirichlet", "dirichlet", "neumann"))
        case["source"] = rng.choice(("none", "static", "affine"))
        if case["border"] == "neumann" and case["source"] == "none":
            case["source"] = "static"  # the flux rules read the source
    if kind == "adjoint":
        case["snapshots"] = rng.randint(4, 40)
    return case


# ---- inputs (host arrays, float64) ------------------------------------------------

def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _to_pinned(a):
    p = _pinned(a.shape)
    p[...] = a
    return p


def _dims(case):
    n = (case["nx"], case["ny"], case["nz"])
    return n, (n[2], n[1], n[0])


def _mesh(n):
    x, y, z = (np.arange(m) / (m - 1) for m in n)
    return x[None, None, :], y[None, :, None], z[:, None, None]


def _star(case, seed):
    """u0, coefficients and known fields of one constant-coefficient problem
    (unit cube, diffusivity 1, perfusion 0.5 with a source)."""
    n, shape = _dims(case)
    rng = np.random.default_rng(seed)
    x, y, z = _mesh(n)
    perf = 0.0 if case["source"] == "none" else 0.5
    tau = 0.9 / (2.0 * sum((m - 1) ** 2 for m in n) + perf)
    cp = [tau * (m - 1) ** 2 for m in n]
    d = {"n": n, "tau": tau, "perf": perf, "cp": cp, "c0": 1.0 - 2.0 * sum(cp) - tau * perf, "cf": tau}
    noise = 1e-3 * (2.0 * rng.random(shape) - 1.0)
    d["fa"] = d["fb"] = d["ga"] = d["gb"] = None
    if case["source"] != "none":
        d["fa"] = 1.0 + x + y + z + 0.1 * rng.random(shape)
        if case["source"] == "affine":
            d["fb"] = 0.5 * (1.0 + x * y + z)
    if case["border"] == "dirichlet":
        u = np.sin(np.pi * x) * np.sin(np.pi * y) * np.sin(np.pi * z) + noise
        u[0], u[-1] = 0.0, 0.0
        u[:, 0], u[:, -1] = 0.0, 0.0
        u[:, :, 0], u[:, :, -1] = 0.0, 0.0
    else:  # Dirichlet at the min faces, a flux condition at the max faces
        u = 1.0 + x + y + z + noise
        flux = np.ones(shape, dtype=bool)
        flux[0] = False
        flux[:, 0] = False
        flux[:, :, 0] = False
        s = 1.0 + x + y + z
        d["ga"] = np.where(flux, -1.0, s)
        d["gb"] = np.where(flux, -0.5, 0.5 * s)
    d["u0"] = u
    return d


def _tissue(case, seed):
    """Seeded tissue coefficients in physiological ranges folded into the
    update's fields; insulated faces, convection at the top (z max)."""
    n, shape = _dims(case)
    rng = np.random.default_rng(seed)

    def field(lo, hi):
        return rng.uniform(lo, hi, shape)

    last = tuple(1e-3 * (m - 1) for m in n)
    rho_c = field(1000.0, 1100.0) * field(3500.0, 3800.0)
    k = field(0.4, 0.6)
    perf = field(1040.0, 1060.0) * field(3700.0, 3900.0) / rho_c * field(0.001, 0.005)
    blood, heat = field(36.5, 37.5), field(1e4, 3e4)
    tau = 0.9 / (6.0 * (0.6 / 3.5e6) / 1e-6)
    d = {"n": n, "last": last, "tau": tau, "cp": [1e6] * 3}
    d["ca"] = tau * k / rho_c
    d["c0"] = 1.0 - 6.0 * 1e6 * d["ca"] - tau * perf
    d["f"] = tau * perf * blood + tau * heat / rho_c
    conv = 2.0 * 1e6 * d["ca"][-1] * 1e-3 / k[-1] * 10.0  # h_conv = 10 W/(m^2 K), 22 degrees outside
    d["u0"] = 37.0 + 0.5 * rng.random(shape)
    # The border nodes' own centre weight and constant.
    cu, cst = d["c0"].copy(), d["f"].copy()
    cu[-1] -= conv
    cst[-1] += 22.0 * conv
    d["cu"], d["cst"] = cu, cst
    return d


def _tissue_rules(d):
    """One rule (cu, cn[6], cst) per border node: the missing neighbour is
    the mirrored inner one."""
    n = d["n"]
    shape = d["u0"].shape
    z, y, x = np.meshgrid(*(np.arange(m) for m in shape), indexing="ij", sparse=True)
    pos = (x, y, z)
    border = np.zeros(shape, dtype=bool)
    cn = []
    for p in range(3):
        s = d["cp"][p] * d["ca"]
        first, final = pos[p] == 0, pos[p] == n[p] - 1
        border |= first | final
        cn.append(np.where(first, 0.0, np.where(final, 2.0 * s, s)))
        cn.append(np.where(final, 0.0, np.where(first, 2.0 * s, s)))
    rules = np.empty((int(border.sum()), 8))
    for i, a in enumerate([d["cu"]] + cn + [d["cst"]]):
        rules[:, i] = a[border]
    return rules


def _ensemble(case, seed):
    # The sizes belong to the case, the data to the seed.
    sizes = np.random.default_rng(case["instances"] * 1009 + case["hi"] * 31 + case["lo"])
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["instances"]):
        n = tuple(int(v) for v in sizes.integers(case["lo"], case["hi"] + 1, 3))
        k, w = rng.uniform(0.4, 0.6), rng.uniform(0.5e-3, 5e-3)
        c, s, amp = rng.uniform(0.3, 0.7, 3), rng.uniform(0.05, 0.15), rng.uniform(1.0, 10.0)
        x, y, z = _mesh(n)
        f = w * 37.0 + amp * np.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / (2.0 * s * s))
        tau = 0.9 / (2.0 * k * sum((m - 1) ** 2 for m in n) + w)
        u = np.full((n[2], n[1], n[0]), 37.0)
        u[1:-1, 1:-1, 1:-1] += 0.5 * rng.random((n[2] - 2, n[1] - 2, n[0] - 2))
        out.append({"n": n, "k": k, "w": w, "tau": tau, "f": f, "u0": u})
    return out


def _gradient(case, seed):
    n, shape = _dims(case)
    rng = np.random.default_rng(seed)
    x, y, z = _mesh(n)
    mode = np.sin(np.pi * x) * np.sin(np.pi * y) * np.sin(np.pi * z)
    return {"n": n, "tau": 0.8 / (2.0 * sum((m - 1) ** 2 for m in n)),
            "k": 0.6 + 0.3 * mode + 0.1 * rng.random(shape),
            "u0": mode + 0.01 * rng.random(shape), "target": 0.8 * mode + 0.01 * rng.random(shape)}


_LAME = (1.0, 0.5, 1.0)  # lambda, mu, rho


def _lame(case, seed):
    n, shape = _dims(case)
    rng = np.random.default_rng(seed)
    x, y, z = _mesh(n)
    c, s = rng.uniform(0.35, 0.65, 3), rng.uniform(0.05, 0.1)
    bump = np.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / (2.0 * s * s))
    for a in (bump[0], bump[-1], bump[:, 0], bump[:, -1], bump[:, :, 0], bump[:, :, -1]):
        a[...] = 0.0
    now = [amp * bump for amp in rng.uniform(-1.0, 1.0, 3)]
    lam, mu, rho = _LAME
    tau = 0.5 / (max(n) - 1) / (math.sqrt((lam + 2.0 * mu) / rho) * math.sqrt(3.0))
    return {"n": n, "tau": tau, "u": now + [0.999 * a for a in now]}


def _cavity(case, seed):
    """Six field components of a few cavity modes plus noise, and the dipole."""
    n, shape = _dims(case)
    rng = np.random.default_rng(seed)
    ax = _mesh(n)
    fields = []
    for f in range(6):
        a = 0.0
        for _ in range(2):
            m = rng.integers(1, 4, 3)
            a = a + rng.uniform(-1.0, 1.0) * np.sin(np.pi * m[0] * ax[0] + f) * np.sin(np.pi * m[1] * ax[1]) * np.cos(
                np.pi * m[2] * ax[2])
        fields.append(a + 1e-3 * rng.random(shape))
    for f in range(3):  # tangential E is zero on the walls
        for p in range(3):
            if p != f:
                view = np.moveaxis(fields[f], 2 - p, 0)
                view[0], view[-1] = 0.0, 0.0
    tau = 0.5 / (n[0] - 1) / math.sqrt(3.0)
    src = tuple(m // 2 for m in n)
    return {"n": n, "tau": tau, "ch": tau * (n[0] - 1), "src": src, "pulse": (1.0, 0.5, 0.25, 4.0), "fields": fields}


# ---- what a program keeps ----------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "steps": case["steps"]}
    if kind == "star":
        d = _star(case, seed)
        border = M.BORDER_DIRICHLET if case["border"] == "dirichlet" else M.BORDER_TABLE
        cfg = M.make_cfg(d["n"], tau=d["tau"], precision=case["precision"], border=border, heat=(1.0, 1.0, d["perf"]))
        p = s["plain"] = M.Plain(cfg)
        if border == M.BORDER_TABLE:
            p.set_border_forms(M.border_forms_flux(cfg, M.FLUX_NEUMANN))
        for slot, key in ((M.FIELD_F_A, "fa"), (M.FIELD_F_B, "fb"), (M.FIELD_G_A, "ga"), (M.FIELD_G_B, "gb")):
            if d[key] is not None:
                p.upload(slot, d[key])
        s["u0"], s["out"] = _to_pinned(d["u0"]), _pinned(d["u0"].shape)
    elif kind == "tissue":
        d = _tissue(case, seed)
        cfg = M.make_cfg(d["n"], last=d["last"], tau=d["tau"], precision=case["precision"], border=M.BORDER_NODES,
                         c0=1.0, cp=d["cp"], cf=1.0)
        p = s["plain"] = M.Plain(cfg)
        p.upload(M.FIELD_C0, d["c0"])
        p.upload(M.FIELD_CA, d["ca"])
        p.upload(M.FIELD_F_A, d["f"])
        p.set_border_node_rules(_tissue_rules(d))
        s["u0"], s["out"] = _to_pinned(d["u0"]), _pinned(d["u0"].shape)
    elif kind == "batch":
        specs = _ensemble(case, seed)
        b = s["batch"] = M.Batch([M.batch_instance(d["n"], d["tau"], d["k"], 1.0, d["w"], 37.0) for d in specs],
                                 case["precision"])
        for i, d in enumerate(specs):
            b.upload(i, M.FIELD_F_A, d["f"])
        s["u0"] = [_to_pinned(d["u0"]) for d in specs]
    elif kind == "adjoint":
        d = _gradient(case, seed)
        a = s["adjoint"] = M.Adjoint(d["n"], d["tau"], case["snapshots"], precision=case["precision"])
        a.set_conductivity(d["k"])
        s["u0"], s["target"] = _to_pinned(d["u0"]), _to_pinned(d["target"])
    elif kind == "lame":
        d = _lame(case, seed)
        s["multi"] = M.MultiField(M.MF_LAME, d["n"], d["tau"], _LAME, case["precision"])
        s["fields"] = [_to_pinned(a) for a in d["u"]]
    elif kind == "yee":
        d = _cavity(case, seed)
        s["multi"] = M.MultiField(M.MF_YEE, d["n"], d["tau"], d["pulse"], case["precision"], src=d["src"])
        s["fields"] = [_to_pinned(a) for a in d["fields"]]
    else:
        d = _cavity(case, seed)
        h = s["multi"] = M.Linear(d["n"], 6, 2)
        for (phase, field, cls), terms in W.yee_linear_rules(d["ch"]).items():
            h.set_rule(phase, field, cls, terms)
        s["fields"] = [_to_pinned(a) for a in d["fields"]]
    return s


def run(s):
    kind = s["kind"]
    if kind in ("star", "tissue"):
        p = s["plain"]
        p.upload(M.FIELD_U, s["u0"])
        p.step(s["steps"])
        return p.download(out=s["out"])
    if kind == "batch":
        b = s["batch"]
        for i, u in enumerate(s["u0"]):
            b.upload(i, M.FIELD_U, u)
        b.step(s["steps"])
        return [b.download(i) for i in range(len(s["u0"]))]
    if kind == "adjoint":
        cost, dk, du0 = s["adjoint"].gradient(s["u0"], s["target"], s["steps"])
        return {"J": cost, "dk": dk, "du0": du0}
    h = s["multi"]
    for f, a in enumerate(s["fields"]):
        h.upload(f, a)
    h.step(s["steps"])
    return [h.download(f) for f in range(6)]


# ---- the least work of a pass ---------------------------------------------------------

def work(case):
    """Each step reads the iterate (and its coefficient fields) once and
    writes the new one once; the host's arrays go up and come back once."""
    kind, steps = case["kind"], case["steps"]
    esz = 4 if case["precision"] == "f32" else 8
    if kind == "batch":
        nodes = sum(d[0] * d[1] * d[2] for d in (
            tuple(int(v) for v in r) for r in np.random.default_rng(
                case["instances"] * 1009 + case["hi"] * 31 + case["lo"]).integers(
                    case["lo"], case["hi"] + 1, (case["instances"], 3))))
        return {"bytes": nodes * (24.0 * steps + 16.0), "flops": 12.0 * nodes * steps}
    nodes = case["nx"] * case["ny"] * case["nz"]
    if kind == "star":
        fields, flops = 2 + {"none": 0, "static": 1, "affine": 2}[case["source"]], 10.0
        return {"bytes": nodes * (fields * esz * steps + 16.0), "flops": flops * nodes * steps}
    if kind == "tissue":
        return {"bytes": nodes * (5.0 * esz * steps + 16.0), "flops": 13.0 * nodes * steps}
    if kind == "adjoint":
        # Forward: u, u', three faces and the diagonal; reverse: lambda in and
        # out, u, the same coefficients, the gradient in and out.
        return {"bytes": nodes * steps * (48.0 + 72.0), "flops": nodes * steps * (13.0 + 35.0)}
    if kind == "lame":
        return {"bytes": nodes * (9.0 * esz * steps + 96.0), "flops": 75.0 * nodes * steps}
    return {"bytes": nodes * (12.0 * esz * steps + 96.0), "flops": 30.0 * nodes * steps}


# ---- the same solves in plain torch, float64 --------------------------------------------

def _dev(a):
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _star_exact(case, seed):
    d = _star(case, seed)
    u, fa, fb, ga, gb = (_dev(d[k]) for k in ("u0", "fa", "fb", "ga", "gb"))
    cx, cy, cz = d["cp"]
    tau, n = d["tau"], d["n"]
    table = case["border"] != "dirichlet"
    if table:
        # Mirrored neighbours beyond the max faces; nodes on a min face are
        # Dirichlet.  Flux term: -cp (2 h / lambda) G(t_old) per max face.
        weight = torch.zeros_like(u)
        for p, (c, m) in enumerate(zip(d["cp"], n)):
            weight.movedim(2 - p, 0)[-1] += c * 2.0 / (m - 1)
        first = torch.zeros_like(u, dtype=torch.bool)
        first[0] = True
        first[:, 0] = True
        first[:, :, 0] = True
    for t in range(case["steps"]):
        old, new = t * tau, (t + 1) * tau
        if table:
            w = torch.nn.functional.pad(u[None, None], (1, 1) * 3, mode="reflect")[0, 0]
        else:
            w = u
        c = w[1:-1, 1:-1, 1:-1]
        v = d["c0"] * c
        v += cx * (w[1:-1, 1:-1, :-2] + w[1:-1, 1:-1, 2:])
        v += cy * (w[1:-1, :-2, 1:-1] + w[1:-1, 2:, 1:-1])
        v += cz * (w[:-2, 1:-1, 1:-1] + w[2:, 1:-1, 1:-1])
        if fa is not None:
            f = fa if fb is None else fa + old * fb
            v += d["cf"] * (f if table else f[1:-1, 1:-1, 1:-1])
        if table:
            v -= weight * (ga + old * gb)
            u = torch.where(first, ga + new * gb, v)
        else:
            u = torch.zeros_like(u)
            u[1:-1, 1:-1, 1:-1] = v
    return u


def _tissue_exact(case, seed):
    d = _tissue(case, seed)
    u, cu, ca, cst = (_dev(d[k]) for k in ("u0", "cu", "ca", "cst"))
    for _ in range(case["steps"]):
        w = torch.nn.functional.pad(u[None, None], (1, 1) * 3, mode="reflect")[0, 0]
        s = d["cp"][0] * (w[1:-1, 1:-1, :-2] + w[1:-1, 1:-1, 2:])
        s += d["cp"][1] * (w[1:-1, :-2, 1:-1] + w[1:-1, 2:, 1:-1])
        s += d["cp"][2] * (w[:-2, 1:-1, 1:-1] + w[2:, 1:-1, 1:-1])
        u = cu * u + cst + ca * s
    return u


def _ensemble_exact(case, seed):
    out = []
    for d in _ensemble(case, seed):
        u, f = _dev(d["u0"]), _dev(d["f"][1:-1, 1:-1, 1:-1])
        cx, cy, cz = (d["tau"] * d["k"] * (m - 1) ** 2 for m in d["n"])
        c0 = 1.0 - 2.0 * (cx + cy + cz) - d["tau"] * d["w"]
        f = d["tau"] * f
        for _ in range(case["steps"]):
            v = c0 * u[1:-1, 1:-1, 1:-1] + f
            v += cx * (u[1:-1, 1:-1, :-2] + u[1:-1, 1:-1, 2:])
            v += cy * (u[1:-1, :-2, 1:-1] + u[1:-1, 2:, 1:-1])
            v += cz * (u[:-2, 1:-1, 1:-1] + u[2:, 1:-1, 1:-1])
            u[1:-1, 1:-1, 1:-1] = v
        out.append(u)
    return out


def _gradient_exact(case, seed):
    d = _gradient(case, seed)
    u, k, target = (_dev(d[v]) for v in ("u0", "k", "target"))
    w = [d["tau"] * (m - 1) ** 2 for m in d["n"]]
    inner = torch.zeros_like(u)
    inner[1:-1, 1:-1, 1:-1] = 1.0

    def up(a, p):    # values at the upper ends of the faces along axis p
        return a.narrow(2 - p, 1, a.shape[2 - p] - 1)

    def down(a, p):  # and at their lower ends
        return a.narrow(2 - p, 0, a.shape[2 - p] - 1)

    faces = [w[p] * 0.5 * (down(k, p) + up(k, p)) for p in range(3)]

    def diffuse(a):
        r = torch.zeros_like(a)
        for p in range(3):
            flux = faces[p] * (up(a, p) - down(a, p))
            down(r, p).add_(flux)
            up(r, p).sub_(flux)
        return r

    states = [u]
    for _ in range(case["steps"]):
        states.append(states[-1] + inner * diffuse(states[-1]))
    lam = states[-1] - target
    cost = float(0.5 * (lam * lam).sum())
    dk = torch.zeros_like(u)
    for t in reversed(range(case["steps"])):
        li, a = inner * lam, states[t]
        for p in range(3):
            g = 0.5 * w[p] * (up(a, p) - down(a, p)) * (down(li, p) - up(li, p))
            down(dk, p).add_(g)
            up(dk, p).add_(g)
        # Border values are held: every step adds their flux into the inner
        # nodes to their cotangent.
        lam = lam + diffuse(li)
    return {"J": cost, "dk": dk, "du0": lam}


def _lame_exact(case, seed):
    d = _lame(case, seed)
    lam, mu, rho = _LAME
    u, old = [_dev(a) for a in d["u"][:3]], [_dev(a) for a in d["u"][3:]]
    h = [1.0 / (m - 1) for m in d["n"]]
    s = d["tau"] ** 2 / rho

    def at(a, *shift):  # inner nodes moved by (dx, dy, dz)
        return a[tuple(slice(1 + o, a.shape[i] - 1 + o) for i, o in enumerate(reversed(shift)))]

    unit = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
    for _ in range(case["steps"]):
        new = []
        for c in range(3):
            v = 2.0 * at(u[c], 0, 0, 0) - at(old[c], 0, 0, 0)
            for p in range(3):
                e = unit[p]
                v += s * (lam + 2.0 * mu if p == c else mu) / h[p] ** 2 * (
                    (at(u[c], *e) + at(u[c], *(-i for i in e))) - 2.0 * at(u[c], 0, 0, 0))
                if p != c:
                    a, b = unit[c], unit[p]
                    pp, pm = [i + j for i, j in zip(a, b)], [i - j for i, j in zip(a, b)]
                    v += s * (lam + mu) / (4.0 * h[c] * h[p]) * (
                        (at(u[p], *pp) - at(u[p], *pm)) - (at(u[p], *(-i for i in pm)) - at(u[p], *(-i for i in pp))))
            r = torch.zeros_like(u[c])
            r[1:-1, 1:-1, 1:-1] = v
            new.append(r)
        old, u = u, new
    return u + old


def _cavity_exact(case, seed):
    d = _cavity(case, seed)
    ex, ey, ez, hx, hy, hz = (_dev(a) for a in d["fields"])
    ch, tau, (i, j, k) = d["ch"], d["tau"], d["src"]
    amp, t0, w, freq = d["pulse"] if case["kind"] == "yee" else (0.0, 0.0, 1.0, 0.0)
    for t in range(case["steps"]):
        hx[:-1, :-1, :] -= ch * ((ez[:-1, 1:, :] - ez[:-1, :-1, :]) - (ey[1:, :-1, :] - ey[:-1, :-1, :]))
        hy[:-1, :, :-1] -= ch * ((ex[1:, :, :-1] - ex[:-1, :, :-1]) - (ez[:-1, :, 1:] - ez[:-1, :, :-1]))
        hz[:, :-1, :-1] -= ch * ((ey[:, :-1, 1:] - ey[:, :-1, :-1]) - (ex[:, 1:, :-1] - ex[:, :-1, :-1]))
        ex[1:-1, 1:-1, :-1] += ch * ((hz[1:-1, 1:-1, :-1] - hz[1:-1, :-2, :-1]) - (hy[1:-1, 1:-1, :-1] - hy[:-2, 1:-1, :-1]))
        ey[1:-1, :-1, 1:-1] += ch * ((hx[1:-1, :-1, 1:-1] - hx[:-2, :-1, 1:-1]) - (hz[1:-1, :-1, 1:-1] - hz[1:-1, :-1, :-2]))
        ez[:-1, 1:-1, 1:-1] += ch * ((hy[:-1, 1:-1, 1:-1] - hy[:-1, 1:-1, :-2]) - (hx[:-1, 1:-1, 1:-1] - hx[:-1, :-2, 1:-1]))
        if amp:
            a = ((t + 1) * tau - t0) / w
            ez[k, j, i] -= tau * amp * math.exp(-a * a) * math.sin(2.0 * math.pi * freq * (t + 1) * tau)
    return [ex, ey, ez, hx, hy, hz]


def exact(case, seed):
    r = {"star": _star_exact, "tissue": _tissue_exact, "batch": _ensemble_exact, "adjoint": _gradient_exact,
         "lame": _lame_exact, "yee": _cavity_exact, "linear": _cavity_exact}[case["kind"]](case, seed)
    if isinstance(r, torch.Tensor):
        return r.cpu().numpy()
    if isinstance(r, dict):
        return {k: v.cpu().numpy() if isinstance(v, torch.Tensor) else v for k, v in r.items()}
    return [v.cpu().numpy() for v in r]
