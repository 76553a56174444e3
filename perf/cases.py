"""The work this framework is used for, as cases with inputs, one timed pass and a 64-bit answer.

Three kinds, each through the package's public entry points:

* ``run``      one simulation on the GPU (``Context``): the initial fields are written into the
               context's device buffers, the explicit steps run, the final fields (and, where a
               program prints progress, the statistics) are read;
* ``sweep``    many independent simulations as one batch (``Batch``): page-locked FP64 fields in,
               steps, fields out;
* ``adjoint``  forward steps with checkpoints and the adjoint sweep of a field-mismatch loss
               (``adjoint.Adjoint``): gradients of four parameters and of the initial fields.

Grids, alloys and step parameters are those of ``microsim_b200.configs`` and of the test fixtures.
The fields are grains with an equilibrium interface in a supersaturated liquid, as they are once seeds
have grown: the seed of a case places the grains and draws its parameters.

``exact`` restates the model in plain torch, 64 bits, vectorised over the grid (one autograd pass
for the adjoint), from the input constants alone.
"""
from __future__ import annotations

import math
import tempfile

import numpy as np
import torch

import microsim_b200 as mb
from microsim_b200 import adjoint, configs

DEV = "cuda"


# ------------------------------------------------------------------------------------- the cases

def _run(name, mx, my, phases, comps, precision, steps, *, aniso=1, well=0, periodic=0, grains=1, gradient=0,
         stats=0, shift=0):
    return {"name": name, "kind": "run", "mx": mx, "my": my, "phases": phases, "comps": comps,
            "precision": precision, "steps": steps, "aniso": aniso, "well": well, "periodic": periodic,
            "grains": grains, "gradient": gradient, "stats": stats, "shift": shift}


def listed():
    return [
        # the smallest configuration: 200x200 isotropic binary alloy, plain FP64, progress printed
        _run("centred_seed_fp64", 200, 200, 2, 1, 64, 64, aniso=0, stats=32),
        # one large 4-fold dendrite in the plain form (the form that equals the reference bit for bit)
        _run("dendrite_fp64", 1024, 1024, 2, 1, 64, 48),
        # the same dendrite in the FP32 form
        _run("dendrite_fp32", 1024, 1024, 2, 1, 32, 100),
        # polycrystalline ternary solidification, the largest single grid, FP32
        _run("ternary_grains_fp32", 2048, 2048, 4, 2, 32, 40, grains=64),
        # a smaller polycrystal of odd sides in the plain form
        _run("ternary_grains_fp64", 611, 500, 4, 2, 64, 16, grains=24),
        # lamellar three-phase eutectic behind a planar front, periodic in x, odd sides
        _run("eutectic_fp32", 517, 333, 3, 1, 32, 60, aniso=0, periodic=1, grains=0),
        # directional solidification in a moving frozen temperature gradient, plain form, progress printed
        _run("frozen_gradient_fp64", 300, 451, 2, 1, 64, 40, gradient=1, stats=20, grains=5),
        # directional growth followed by the moving window: 100 steps, then the front is found and shifted
        _run("moving_window_fp32", 400, 700, 2, 1, 32, 100, shift=1, grains=0),
        # the parameter sweep the framework is quoted on: 256 dendrites of sides 128..512 in one batch
        {"name": "sweep_256_fp32", "kind": "sweep", "n": 256, "lo": 128, "hi": 512, "ragged": 0, "steps": 1000,
         "depth": 2, "comp": 0},
        # a small campaign of odd grids with compensated accumulation, single steps
        {"name": "sweep_ragged_fp32", "kind": "sweep", "n": 12, "lo": 48, "hi": 300, "ragged": 1, "steps": 200,
         "depth": 1, "comp": 1},
        # calibration by gradients: one instance of the 512x512 calibration problem in FP32
        {"name": "calibration_fp32", "kind": "adjoint", "mx": 512, "my": 512, "precision": 32, "steps": 100,
         "aniso": 1, "well": 0, "periodic": 0},
        # the FP64 reference adjoint on a smaller grid of odd sides, well potential
        {"name": "calibration_fp64", "kind": "adjoint", "mx": 255, "my": 190, "precision": 64, "steps": 49,
         "aniso": 1, "well": 1, "periodic": 1},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run", "run", "run", "sweep", "adjoint"])
    if kind == "sweep":
        return {"kind": "sweep", "n": log(2, 48), "lo": 40, "hi": log(120, 512), "ragged": 1,
                "steps": 4 * log(20, 100) + rng.randrange(4), "depth": rng.choice([1, 2]),
                "comp": rng.choice([0, 0, 1])}
    if kind == "adjoint":
        precision = rng.choice([32, 64])
        return {"kind": "adjoint", "mx": log(64, 512), "my": log(64, 512), "precision": precision,
                "steps": log(16, 80), "aniso": rng.choice([0, 1]), "well": rng.choice([0, 1]) if precision == 64 else 0,
                "periodic": rng.choice([0, 1])}
    phases, comps = rng.choice([(2, 1), (2, 1), (2, 1), (3, 1), (4, 2)])
    most = 1500 if phases == 2 else 900
    c = _run("", log(60, most), log(60, most), phases, comps, rng.choice([32, 64]), log(16, 100),
             aniso=1 if phases == 4 else 0 if phases == 3 else rng.choice([0, 1]),
             well=rng.choice([0, 0, 1]) if phases == 2 else 0,
             periodic=rng.choice([0, 0, 1]), grains=log(2, 30), stats=rng.choice([0, 0, 16]))
    if phases == 2 and rng.random() < 0.25:
        c["gradient"] = 1
    del c["name"]
    return c


def _sizes(case):
    """[(mx, my)] of the instances of a sweep: the sweep configuration's own sides, or odd ones."""
    if not case["ragged"]:
        return [(c.mesh_x, c.mesh_y) for c in configs.c4(case["n"])]
    r = np.random.default_rng(17)
    return [tuple(int(v) for v in np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), 2)))
            for _ in range(case["n"])]


def work(case):
    """Bytes: the fields (and what else is returned) in once and out once, at the precision they are handed
    over in.  Flops: the steps' own arithmetic, every cell taken as bulk (two face differences per axis and the
    update per component; the interface cells of a few percent of a grid cost some hundred more)."""
    if case["kind"] == "sweep":
        cells = sum(a * b for a, b in _sizes(case))
        return {"bytes": 2.0 * 24.0 * cells, "flops": 14.0 * cells * case["steps"]}
    cells, size = case["mx"] * case["my"], case["precision"] // 8
    if case["kind"] == "adjoint":  # phi, mu, target in; phi, mu and the adjoints of the initial fields out
        return {"bytes": 11.0 * 8 * cells, "flops": 60.0 * cells * case["steps"]}
    planes = case["phases"] + case["comps"]
    return {"bytes": 2.0 * planes * size * cells,
            "flops": (10.0 * case["comps"] ** 2 + 2 * case["phases"]) * cells * case["steps"]}


def tolerance(case):
    # Measured against exact(), times about four.  FP32: storage rounds every field value at every step.
    # The model's active-phase count makes cells with three or four phases jump between two updates when a
    # vanishing phase rounds to 0, so those differ by more.  FP64: another order differs by roundings.
    # The adjoint passes through the branches of the projection, which cells at phi = 0 and 1 take by a rounding.
    if case["kind"] == "adjoint":
        return {"rel": 2e-3, "max": 0.5} if case["precision"] == 32 else {"rel": 1e-12, "max": 1e-9}
    if case["kind"] == "run" and case["precision"] == 64:
        return {"rel": 1e-12, "max": 1e-9}
    if case["kind"] == "run" and case["phases"] > 2:
        return {"rel": 5e-4, "max": 0.1}
    return {"rel": 2e-5, "max": 2e-3}


# ------------------------------------------------------------------------------- models and fields

def _alloy(case, mx, my, rng):
    """The Input.in description (configs.Case) of one instance, its free parameters drawn from rng."""
    bc = (3, 3, 1, 1) if case.get("periodic") else (1, 1, 1, 1)
    well = 2 if case.get("well") else 1
    if case.get("phases", 2) == 4:
        c = configs.c3(steps=1000, mesh=max(mx, 16), nseeds=4, rng_seed=int(rng.integers(1 << 30)))
        c.mesh_x, c.mesh_y, c.bc_phi, c.bc_mu, c.function_w, c.fills = mx, my, bc, bc, well, []
        return c
    if case.get("phases", 2) == 3:
        eq = [(0, 0, 0.78), (0, 2, 0.5), (2, 0, 0.5), (1, 1, 0.21), (1, 2, 0.5), (2, 1, 0.5)]
        far = round(float(rng.uniform(0.44, 0.47)), 4)
        return configs.Case(
            mesh_x=mx, mesh_y=my, dx=1.0, dt=0.04, N=3, K=2, epsilon=4.0, tau=1.0, gamma=[1.0] * 3,
            tau_ab=[1.5] * 3, aniso=0, dab=[0.0] * 3, function_w=well, gamma_abc=[5.0],
            diffusivity=[(1, 0, 0.0), (1, 1, 0.0), (1, 2, 1.0)], A=[(0, 1.0), (1, 1.0), (2, 1.0)],
            ceq=eq + [(2, 2, 0.5)], cfill=eq + [(2, 2, far)],
            slopes=[(0, 0, 0.45), (0, 2, 0.45), (2, 0, 0.45), (1, 1, -0.45), (1, 2, -0.45), (2, 1, -0.45)],
            T=0.98, bc_phi=bc, bc_mu=bc, solver="BINARY", phases=["alpha", "beta", "liquid"],
            components=["Al", "Cu"])
    eps = float(rng.choice([3.0, 4.0, 5.0])) if case["kind"] == "sweep" else 4.0
    aniso = case.get("aniso", 1)
    c = configs.binary_case(
        mx, my, gap=1.0, supersat=round(float(rng.uniform(0.3, 0.6)), 4), eps=eps,
        delta=round(float(rng.uniform(0.01, 0.05)), 4) if aniso else 0.0,
        theta=round(float(rng.uniform(0.0, 45.0)), 2) if aniso and case["kind"] == "run" else 0.0,
        dt=0.05, tau=round(eps * 0.4444, 4), function_w=well, bc=bc)
    c.fills = []
    if case.get("gradient"):
        c.tempgrady = (0.97, 0.08, float(my), 2.0, 0.5)
    return c


def _model(alloy):
    with tempfile.TemporaryDirectory() as d:
        ip, fp = alloy.write(d)
        return mb.Input(ip, fp).model()


def _fields(case, alloy, k, rng):
    """Grains of the solid phases in a supersaturated liquid: (phi [N, mx, my], mu [K-1, mx, my]) in FP64."""
    mx, my, N = alloy.mesh_x, alloy.mesh_y, alloy.N
    x = torch.arange(mx, device=DEV, dtype=torch.float64)[:, None]
    y = torch.arange(my, device=DEV, dtype=torch.float64)[None, :]
    def edge(d):  # the obstacle potential's equilibrium profile: exactly 1 and 0 outside a compact interface
        return 0.5 - 0.5 * torch.sin(math.pi * torch.clamp(d / (2.4 * alloy.epsilon), -0.5, 0.5))

    if N == 3:  # lamellae of two solids behind a planar front
        near = (y - my / 3.0 - float(rng.uniform(-4, 4))).expand(mx, my)
        pairs = max(1, round((mx - 1) / (2.0 * float(rng.uniform(28, 44)))))
        period = (mx - 1) / pairs
        u = torch.remainder(x + float(rng.uniform(0, period)), period)
        first = edge(torch.maximum(u - 0.75 * period, 0.25 * period - u))
        p = [edge(near) * first, edge(near) * (1.0 - first)]
    else:
        if case.get("shift"):  # a planar front
            grains = [(0, None, 0.0, my / 3.0 + float(rng.uniform(-4, 4)))]
        elif case["kind"] == "adjoint":  # a crystal in the middle, as a filling leaves it: sharp
            grains = [(0, mx // 2, my // 2, float(rng.uniform(8.0, 0.15 * min(mx, my))))]
        elif case["kind"] == "sweep" or case["grains"] < 2:  # a quarter of a crystal in the corner
            grains = [(0, 0.0, 0.0, float(rng.uniform(0.08, 0.2)) * min(mx, my))]
        else:
            grains = _scatter(case["grains"], N - 1, mx, my, 2.4 * alloy.epsilon, rng)
        near = torch.full((mx, my), 1e30, device=DEV, dtype=torch.float64)
        solid = [near] * (N - 1)
        for a, xc, yc, r in grains:
            d = (y - r).expand(mx, my) if xc is None else torch.sqrt((x - xc) ** 2 + (y - yc) ** 2) - r
            near = torch.minimum(near, d)
            solid[a] = torch.minimum(solid[a], d)
        p = [(d < 0).double() if case["kind"] == "adjoint" else edge(d) for d in solid]
    phi = torch.stack(p + [torch.clamp(1.0 - sum(p), min=0.0)])
    # mu from its value at the front (liquid's ceq) to the far field's (cfill), over a diffusion length
    A = k["A"][N - 1]
    mus = []
    for i in range(k["K1"]):
        at = [sum((2.0 if i == j else 1.0) * A[i][j] * c[j] for j in range(k["K1"])) for c in (k["cl"], k["cf"])]
        mus.append(at[0] + (at[1] - at[0]) * (1.0 - torch.exp(-torch.clamp(near, min=0.0) / 18.0)))
    return phi.contiguous(), torch.stack(mus).contiguous()


def _scatter(n, solids, mx, my, gap, rng):
    """Up to n grains [(phase, x, y, radius)] that do not touch (grains before impingement)."""
    top, got = 0.35 * math.sqrt(mx * my / n), []
    for _ in range(40 * n):
        xc, yc, r = float(rng.uniform(0, mx)), float(rng.uniform(0, my)), float(rng.uniform(0.3, 1.0)) * top
        if all(math.hypot(xc - g[1], yc - g[2]) > r + g[3] + 2.0 * gap for g in got):
            got.append((len(got) % solids, xc, yc, r))
        if len(got) == n:
            break
    return got


class _Run:
    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        alloy = _alloy(case, case["mx"], case["my"], rng)
        self.case, self.alloy, self.k = case, alloy, _constants(alloy)
        dt = torch.float64 if case["precision"] == 64 else torch.float32
        self.phi0, self.mu0 = (f.to(dt) for f in _fields(case, alloy, self.k, rng))


def _instances(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for mx, my in _sizes(case):
        alloy = _alloy(case, mx, my, rng)
        k = _constants(alloy)
        out.append((alloy, k) + _fields(case, alloy, k, rng))
    return out


def prepare(case, seed):
    if case["kind"] == "sweep":
        inst = _instances(case, seed)
        batch = mb.Batch([_model(i[0]) for i in inst])
        batch.set_depth(case["depth"])
        if case["comp"]:
            batch.set_compensated(True)
        batch.prepare()
        state = {"case": case, "batch": batch}
        for name, pick in (("phi", 2), ("mu", 3)):
            sizes = [i[pick].numel() for i in inst]
            flat = torch.cat([i[pick].reshape(-1) for i in inst])
            host = torch.empty(flat.numel(), dtype=torch.float64, pin_memory=True).copy_(flat)
            out = torch.zeros(flat.numel(), dtype=torch.float64, pin_memory=True)
            shapes = [tuple(i[pick].shape) for i in inst]
            state[name] = [v.numpy().reshape(s) for v, s in zip(host.split(sizes), shapes)]
            state[name + "_to"] = [v.numpy().reshape(s) for v, s in zip(out.split(sizes), shapes)]
            state[name + "_out"] = out
        return state
    if case["kind"] == "adjoint":
        rng = np.random.default_rng(seed)
        alloy = _alloy(case, case["mx"], case["my"], rng)
        phi, mu = _fields(case, alloy, _constants(alloy), rng)
        model = _model(alloy)
        # the field a calibration compares with: the same crystal, a little larger
        near = torch.roll(phi, (1, 1), (1, 2))
        return {"case": case, "adj": adjoint.Adjoint(model, mb.GP_FP64 if case["precision"] == 64 else mb.GP_FP32),
                "phi0": phi.cpu().numpy(), "mu0": mu.cpu().numpy(), "target": near.cpu().numpy()}
    s = _Run(case, seed)
    s.ctx = mb.Context(_model(s.alloy), mb.GP_FP64 if case["precision"] == 64 else mb.GP_FP32)
    s.stream = torch.cuda.ExternalStream(s.ctx.stream)
    return s


def _pass_run(s):
    case, ctx, my = s.case, s.ctx, s.case["my"]
    main = torch.cuda.current_stream()
    s.stream.wait_stream(main)
    phi, mu = ctx.device_state()
    with torch.cuda.stream(s.stream):
        phi[:, :, :my].copy_(s.phi0)
        mu[:, :, :my].copy_(s.mu0)
    ctx.state_changed()
    if case["gradient"]:
        ctx.set_time_step(0)
    out = {}
    left = case["steps"]
    while left > 0:
        n = min(left, case["stats"] or left)
        ctx.step(n)
        left -= n
        if case["stats"]:
            st = ctx.stats()
            out["progress"] = {name: st[name] for name in ("solute", "phase_fraction", "rel_change_phi",
                                                           "rel_change_mu", "phi_max", "mu_min", "grand_potential")}
    if case["shift"]:
        pos = ctx.interface_y()
        if pos > s.case["my"] // 3:
            ctx.shift_y(pos - s.case["my"] // 3)
        out["front"] = pos
    phi, mu = ctx.device_state()
    main.wait_stream(s.stream)
    out["phi"], out["mu"] = phi[:, :, :my].clone(), mu[:, :, :my].clone()
    return out


def run(state):
    if isinstance(state, _Run):
        return _pass_run(state)
    case = state["case"]
    if case["kind"] == "sweep":
        b = state["batch"]
        b.upload_all(list(zip(state["phi"], state["mu"])))
        b.step(case["steps"])
        b.download_all(list(zip(state["phi_to"], state["mu_to"])))
        b.sync()
        return {"phi": state["phi_out"], "mu": state["mu_out"]}
    adj = state["adj"]
    phi, mu = adj.forward(state["phi0"], state["mu0"], case["steps"])
    grad, lphi, lmu = adj.backward(2.0 * (phi - state["target"]), initial=True)
    return {"phi": phi, "mu": mu, "grad": grad, "lam_phi0": lphi, "lam_mu0": lmu}


# ------------------------------------------------------------------------- the model in 64 bits

def _constants(alloy):
    """Model constants of an input (plain floats), from its text parameters."""
    N, K1 = alloy.N, alloy.K - 1
    A = [[[0.0] * K1 for _ in range(K1)] for _ in range(N)]
    for a, *v in alloy.A:
        off = iter(v[K1:])
        for i in range(K1):
            A[a][i][i] = float(v[i])
        for i in range(K1):
            for j in range(i + 1, K1):
                A[a][i][j] = A[a][j][i] = float(next(off))
    muc = [np.array([[A[a][i][j] * (2.0 if i == j else 1.0) for j in range(K1)] for i in range(K1)]) for a in range(N)]
    cmu = [np.linalg.inv(v).tolist() for v in muc]
    ceq = {(a, b): [float(x) for x in v] for a, b, *v in alloy.ceq}
    cfill = {(a, b): [float(x) for x in v] for a, b, *v in alloy.cfill}
    slope = {(a, b): [float(x) for x in v] for a, b, *v in alloy.slopes}
    Diff = [[[0.0] * K1 for _ in range(K1)] for _ in range(N)]
    for _, a, *v in alloy.diffusivity:
        for i in range(K1):
            Diff[a][i][i] = float(v[i])
    pairs = [(a, b) for a in range(N) for b in range(a + 1, N)]
    triples = [(a, b, c) for a in range(N) for b in range(a + 1, N) for c in range(b + 1, N)]
    k = {"N": N, "K1": K1, "A": A, "cmu": cmu, "Diff": Diff, "dx": alloy.dx, "dt": alloy.dt, "eps": alloy.epsilon,
         "tau": alloy.tau, "T": alloy.T, "Teq": alloy.Teq, "obstacle": alloy.function_w == 1, "aniso": alloy.aniso,
         "bc": alloy.bc_phi, "bc_mu": alloy.bc_mu, "pairs": pairs,
         "Gamma": dict(zip(pairs, alloy.gamma)), "tau_ab": dict(zip(pairs, alloy.tau_ab)),
         "dab": dict(zip(pairs, alloy.dab)), "Gabc": dict(zip(triples, alloy.gamma_abc)),
         "rot": {(a, b): math.radians(th) for a, b, th in alloy.rotations},
         "cl": ceq[(0, N - 1)], "cf": cfill[(N - 1, N - 1)], "gradient": alloy.tempgrady,
         "bc_T": (alloy.bc_T or alloy.bc_mu)[2], "my": alloy.mesh_y, "cs": [], "cls": [], "dC": [], "dTs": [],
         "dTl": [], "dBdT": []}
    L = N - 1
    for a in range(N - 1):
        s, q = ceq[(a, a)], ceq[(a, L)]
        dC = [q[i] - s[i] for i in range(K1)]
        ds = sum(slope[(a, a)][i] * dC[i] for i in range(K1))
        dl = sum(slope[(a, L)][i] * dC[i] for i in range(K1))
        k["cs"].append(s), k["cls"].append(q), k["dC"].append(dC), k["dTs"].append(ds), k["dTl"].append(dl)
        k["dBdT"].append([sum((2.0 if i == j else 1.0) * (A[L][i][j] * dC[j] / dl - A[a][i][j] * dC[j] / ds)
                              for j in range(K1)) for i in range(K1)])
    k["dBdT"].append([0.0] * K1)
    return k


def _BC(k, T):
    """B(T) [N][K-1] and C(T) [N] of the free energies (T: a number or a row of temperatures)."""
    N, K1, L, A = k["N"], k["K1"], k["N"] - 1, k["A"]
    B, C = [], []
    for a in range(N - 1):
        cl = [k["cls"][a][i] - k["dC"][a][i] * (k["Teq"] - T) / k["dTl"][a] for i in range(K1)]
        cs = [k["cs"][a][i] - k["dC"][a][i] * (k["Teq"] - T) / k["dTs"][a] for i in range(K1)]
        B.append([sum((2.0 if i == j else 1.0) * (A[L][i][j] * cl[j] - A[a][i][j] * cs[j]) for j in range(K1))
                  for i in range(K1)])
        C.append(sum(A[a][i][j] * cs[i] * cs[j] - A[L][i][j] * cl[i] * cl[j] for i in range(K1) for j in range(i, K1)))
    return B + [[0.0] * K1], C + [0.0]


def _Beff(k, T):
    Beq = _BC(k, k["Teq"])[0]
    return [[Beq[a][i] + k["dBdT"][a][i] * (T - k["Teq"]) for i in range(k["K1"])] for a in range(k["N"])]


def _ghost(M, n, bc):
    """Source rows of a grid axis padded by n ghosts (mirror about the last cell, or the period M - 1)."""
    v = []
    for i in range(-n, M + n):
        if i < 0:
            i = -i if bc == 1 else M - 1 + i
        elif i >= M:
            i = 2 * M - 2 - i if bc == 1 else 1 + i - M
        v.append(i)
    return torch.tensor(v, device=DEV)


def _pad(f, n, bc):
    return f.index_select(1, _ghost(f.shape[1], n, bc[0])).index_select(2, _ghost(f.shape[2], n, bc[2]))


def _h(p, a):
    N = len(p)
    s = sum(p[b] * p[c] for b in range(N) for c in range(b + 1, N) if a not in (b, c))
    return p[a] ** 2 * (3.0 - 2.0 * p[a]) + 2.0 * p[a] * s


def _dh(p, b, a):
    N = len(p)
    if a == b:
        s = sum(p[e] * p[f] for e in range(N) for f in range(e + 1, N) if b not in (e, f))
        return 6.0 * p[a] * (1.0 - p[a]) + 2.0 * s
    return 2.0 * sum((p[e] for e in range(N) if e not in (a, b)), torch.zeros_like(p[a])) * p[b]


def _bracket(k, pr, Qx, Qy, axis):
    """a_c^2 Q_n + a_c |q|^2 (R^-1 da_c/dq)_n of a face, q = R Q."""
    if not k["aniso"]:
        return (Qx, Qy)[axis]
    c, s = math.cos(k["rot"][pr]), math.sin(k["rot"][pr])
    q0, q1 = c * Qx - s * Qy, s * Qx + c * Qy
    ac, e0, e1 = _aniso(k["dab"][pr], q0, q1)
    return ac * ac * (Qx, Qy)[axis] + ac * ((c * e0 + s * e1), (-s * e0 + c * e1))[axis]


def _aniso(dab, q0, q1):
    q2 = q0 * q0 + q1 * q1
    on = q2 > 1e-15
    s = torch.where(on, q2, torch.ones_like(q2))
    x2, y2 = q0 * q0 / s, q1 * q1 / s
    s4 = x2 * x2 + y2 * y2
    one, nil = torch.ones_like(q2), torch.zeros_like(q2)
    return (torch.where(on, 1.0 - dab * (3.0 - 4.0 * s4), one), torch.where(on, 16.0 * dab * q0 * (x2 - s4), nil),
            torch.where(on, 16.0 * dab * q1 * (y2 - s4), nil))


def _temperatures(k, t):
    """T of ghost-padded columns -1 .. my in the phase-field and the concentration half step of step t."""
    if not k["gradient"]:
        return k["T"], k["T"]
    base, dT, dist, off, v = k["gradient"]
    grad = dT * k["dx"] / dist
    bottom = base - (off / k["dx"] + (v / k["dx"] * (t * k["dt"]) if t else 0.0)) * grad
    row = torch.arange(-1, k["my"] + 1, device=DEV)
    own = bottom + (row + 3).double() * grad
    copy = own[_ghost(k["my"], 1, k["bc_T"]) + 1]
    return (own if t else copy)[None, :], copy[None, :]


def _dphi(k, P, U, T):
    """Delta-phi on the interior plus one ring, from phi padded by 2 and mu padded by 1."""
    N, K1, dx, pairs = k["N"], k["K1"], k["dx"], k["pairs"]
    c = [P[a][1:-1, 1:-1] for a in range(N)]
    xp, xm = [P[a][2:, 1:-1] for a in range(N)], [P[a][:-2, 1:-1] for a in range(N)]
    yp, ym = [P[a][1:-1, 2:] for a in range(N)], [P[a][1:-1, :-2] for a in range(N)]
    div = [((xp[a] - c[a]) - (c[a] - xm[a])) / dx ** 2 + ((yp[a] - c[a]) - (c[a] - ym[a])) / dx ** 2 for a in range(N)]
    act = [d != 0 for d in div]
    cx = [0.5 * ((xp[a] - c[a]) + (c[a] - xm[a])) / dx for a in range(N)]
    cy = [(yp[a] - ym[a]) / (2.0 * dx) for a in range(N)]
    CY = [(P[a][:, 2:] - P[a][:, :-2]) / (2.0 * dx) for a in range(N)]
    CX = [0.5 * ((P[a][2:] - P[a][1:-1]) + (P[a][1:-1] - P[a][:-2])) / dx for a in range(N)]
    g = [torch.zeros_like(c[0]) for _ in range(N)]
    for pr in pairs:
        a, b = pr
        sa, sb = (0.5 * (P[i][1:, 1:-1] + P[i][:-1, 1:-1]) for i in pr)
        ga, gb = ((P[i][1:, 1:-1] - P[i][:-1, 1:-1]) / dx for i in pr)
        Qy = 0.5 * (sa * (CY[b][1:] + CY[b][:-1]) - sb * (CY[a][1:] + CY[a][:-1]))
        Bx = _bracket(k, pr, sa * gb - sb * ga, Qy, 0)
        fa, fb = Bx * sa, Bx * sb
        dab_, dba = (-fb[1:] + fb[:-1]) / dx, (fa[1:] - fa[:-1]) / dx
        sa, sb = (0.5 * (P[i][1:-1, 1:] + P[i][1:-1, :-1]) for i in pr)
        ga, gb = ((P[i][1:-1, 1:] - P[i][1:-1, :-1]) / dx for i in pr)
        Qx = 0.5 * (sa * (CX[b][:, 1:] + CX[b][:, :-1]) - sb * (CX[a][:, 1:] + CX[a][:, :-1]))
        By = _bracket(k, pr, Qx, sa * gb - sb * ga, 1)
        fa, fb = By * sa, By * sb
        dab_, dba = dab_ + (-fb[:, 1:] + fb[:, :-1]) / dx, dba + (fa[:, 1:] - fa[:, :-1]) / dx
        Qx, Qy = c[a] * cx[b] - c[b] * cx[a], c[a] * cy[b] - c[b] * cy[a]
        if k["aniso"]:
            co, si = math.cos(k["rot"][pr]), math.sin(k["rot"][pr])
            q0, q1 = co * Qx - si * Qy, si * Qx + co * Qy
            ac, e0, e1 = _aniso(k["dab"][pr], q0, q1)
            w0, w1 = ac * ac * q0 + ac * e0, ac * ac * q1 + ac * e1
            dA = [w0 * (co * cx[i] - si * cy[i]) + w1 * (si * cx[i] + co * cy[i]) for i in (b, a)]
        else:
            dA = [Qx * cx[i] + Qy * cy[i] for i in (b, a)]
        g2 = 2.0 * k["Gamma"][pr]
        g[a] = g[a] + g2 * (dab_ - dA[0])
        g[b] = g[b] + g2 * (dba + dA[1])
    B, C = _BC(k, T)
    Be = _Beff(k, T)
    psi = []
    for b in range(N):
        cb = [sum(k["cmu"][b][i][j] * (U[j] - Be[b][j]) for j in range(K1)) for i in range(K1)]
        v = sum((B[b][i] - U[i]) * cb[i] for i in range(K1)) + C[b]
        psi.append(v + sum(k["A"][b][i][j] * cb[i] * cb[j] for i in range(K1) for j in range(i, K1)))
    nil = torch.zeros_like(c[0])
    lam = []
    for a in range(N):
        w = nil
        for b in range(N):
            if b == a:
                continue
            G = k["Gamma"][(min(a, b), max(a, b))]
            v = torch.where(c[a] * c[b] >= 0, G * c[b], -G * c[b]) if k["obstacle"] else 2.0 * G * c[b] ** 2 * c[a]
            w = w + torch.where(act[b], v, nil)
        w = w * (16.0 / math.pi ** 2 if k["obstacle"] else 9.0)
        for b in range(N):
            for d in range(b + 1, N):
                if a in (b, d):
                    continue
                v = k["Gabc"][tuple(sorted((a, b, d)))] * c[b] * c[d]
                w = w + torch.where(act[b] & act[d], torch.where(c[a] * c[b] * c[d] >= 0, v, -v), nil)
        dpsi = sum(psi[b] * _dh(c, b, a) for b in range(N))
        lam.append(torch.where(act[a], k["eps"] * g[a] - w / k["eps"] - dpsi, nil))
    n = sum(v.double() for v in act)
    mean = sum(lam) / torch.clamp(n, min=1.0)
    st1 = sum(c[a] * c[b] for a, b in pairs)
    if N == 2:
        tau = torch.where(st1 != 0, nil + k["tau_ab"][(0, 1)], nil + k["tau"])
    else:
        st = sum(k["tau_ab"][p] * c[p[0]] * c[p[1]] for p in pairs)
        tau = torch.where(st1 != 0, st / torch.where(st1 != 0, st1, nil + 1.0), nil + k["tau"])
    dp = [torch.where(act[a], k["dt"] * (lam[a] - mean) / (tau * k["eps"]), nil) for a in range(N)]
    # projection onto the simplex: clamp below 0, share what was added among the phases inside, cap at 1
    v = [c[a] + dp[a] for a in range(N)]
    inside = [act[a] & (v[a] > 0) & (v[a] < 1) for a in range(N)]
    count = sum(i.double() for i in inside)
    share = sum(torch.where(inside[a], c[a], nil) for a in range(N))
    over = sum(torch.where(v[a] < 0, -v[a], nil) for a in range(N))
    dp = [torch.where(v[a] < 0, dp[a] - v[a], dp[a]) for a in range(N)]
    safe, scount = torch.where(share != 0, share, nil + 1.0), torch.clamp(count, min=1.0)
    for a in range(N):
        v2 = c[a] + dp[a]
        on = (over > 0) & act[a] & (v2 > 0) & (v2 < 1)
        dp[a] = torch.where(on, dp[a] - torch.where(share != 0, over * c[a] / safe, over / scount), dp[a])
    hit = torch.full_like(n, -1.0)
    for a in range(N):
        hit = torch.where((hit < 0) & act[a] & (c[a] + dp[a] > 1), nil + a, hit)
    return [torch.where((hit >= 0) & act[a], torch.where(hit == a, 1.0 - c[a], -c[a]), dp[a]) for a in range(N)]


def _face(k, p, n, tc, tn, U, V, dp, dn, Bc, Bn, skip):
    """(diffusion flux, antitrapping current) per component through the faces between cells and neighbours."""
    N, K1, dx, L = k["N"], k["K1"], k["dx"], k["N"] - 1
    DC = [[[sum(k["Diff"][b][i][q] * k["cmu"][b][q][j] for q in range(K1)) for j in range(K1)] for i in range(K1)]
          for b in range(N)]
    F = [sum(0.5 * sum(DC[b][i][j] * (p[b] + n[b]) for b in range(N)) * (V[j] - U[j]) / dx for j in range(K1))
         for i in range(K1)]
    nil = torch.zeros_like(p[0])
    J = [nil] * K1

    def norm(x, y):
        s = x * x + y * y
        return torch.sqrt(torch.where(s != 0, s, nil + 1.0)), s != 0

    def s_of(q, a):
        u = q[a] * (1.0 - q[a])
        return torch.where(u > 0, q[a] * (1.0 - _h(q, a)) / torch.sqrt(torch.where(u > 0, u, nil + 1.0)), nil)

    def gap(W, Be, a, i):
        return (sum(k["cmu"][L][i][j] * (W[j] - Be[L][j]) for j in range(K1))
                - sum(k["cmu"][a][i][j] * (W[j] - Be[a][j]) for j in range(K1)))

    gl, tl = (n[L] - p[L]) / dx, 0.5 * (tc[L] + tn[L])
    nl, nl_on = norm(tl, gl)
    for a in range(N - 1):
        gn, ta = (n[a] - p[a]) / dx, 0.5 * (tc[a] + tn[a])
        ng, on = norm(ta, gn)
        sp = gn * gl + ta * tl
        sp = torch.where(nl_on, sp / nl / ng, sp)
        for i in range(K1):
            un, uc = gap(V, Bn, a, i) * dn[a], gap(U, Bc, a, i) * dp[a]
            s = 0.5 * (s_of(n, a) * un + s_of(p, a) * uc) if k["obstacle"] else 0.5 / math.sqrt(2.0) * (un + uc)
            f = 1.0 - k["Diff"][a][i][i] / k["Diff"][L][i][i]
            J[i] = J[i] + torch.where(on & ~skip, f * torch.abs(sp) * s * gn / ng, nil)
    return F, J


def _step(k, phi, mu, t=0):
    """One explicit step of the grand-potential model: (phi, mu) after it."""
    N, K1, dx, dt = k["N"], k["K1"], k["dx"], k["dt"]
    my = phi.shape[2]
    P, U = _pad(phi, 2, k["bc"]), _pad(mu, 1, k["bc_mu"])
    T0, T1 = _temperatures(k, t)
    R = [P[a][1:-1, 1:-1] for a in range(N)]
    dp = _dphi(k, P, U, T0)
    cy = [(P[a][1:-1, 2:] - P[a][1:-1, :-2]) / (2.0 * dx) for a in range(N)]
    cx = [0.5 * ((P[a][2:, 1:-1] - R[a]) + (R[a] - P[a][:-2, 1:-1])) / dx for a in range(N)]
    Be = _Beff(k, T1)

    def cut(v, sx, sy):
        return [w[sx, sy] for w in v]

    def rows(sl):
        return [[b[:, sl] if torch.is_tensor(b) else b for b in v] for v in Be]

    lo, hi, mid, every = slice(None, -1), slice(1, None), slice(1, -1), slice(None)
    no = torch.zeros((), dtype=torch.bool, device=DEV)
    Fx, Jx = _face(k, cut(R, lo, mid), cut(R, hi, mid), cut(cy, lo, mid), cut(cy, hi, mid), cut(U, lo, mid),
                   cut(U, hi, mid), cut(dp, lo, mid), cut(dp, hi, mid), rows(mid), rows(mid), no)
    skip = (torch.arange(-1, my, device=DEV) == my - 5)[None, :]
    Fy, Jy = _face(k, cut(R, mid, lo), cut(R, mid, hi), cut(cx, mid, lo), cut(cx, mid, hi), cut(U, mid, lo),
                   cut(U, mid, hi), cut(dp, mid, lo), cut(dp, mid, hi), rows(lo), rows(hi), skip)
    js = -0.25 * math.pi * k["eps"] if k["obstacle"] else -k["eps"]
    p, d, Bm = cut(R, mid, mid), cut(dp, mid, mid), rows(mid)
    m0 = [mu[i] for i in range(K1)]
    inc = []
    for i in range(K1):
        inc.append(dt * ((Fx[i][1:] - Fx[i][:-1]) / dx + (Fy[i][:, 1:] - Fy[i][:, :-1]) / dx)
                   - js * ((Jx[i][1:] - Jx[i][:-1]) / dx + (Jy[i][:, 1:] - Jy[i][:, :-1]) / dx))
    c = [[sum(k["cmu"][a][i][j] * (m0[j] - Bm[a][j]) for j in range(K1)) for i in range(K1)] for a in range(N)]
    h = [_h(p, a) for a in range(N)]
    dc = [inc[i] - sum(c[a][i] * sum(_dh(p, a, b) * d[b] for b in range(N)) for a in range(N)) for i in range(K1)]
    D = [[sum(k["cmu"][a][i][j] * h[a] for a in range(N)) for j in range(K1)] for i in range(K1)]
    if K1 == 1:
        new = [m0[0] + dc[0] / D[0][0]]
    else:
        det = D[0][0] * D[1][1] - D[0][1] * D[1][0]
        new = [m0[0] + (D[1][1] * dc[0] - D[0][1] * dc[1]) / det, m0[1] + (D[0][0] * dc[1] - D[1][0] * dc[0]) / det]
    done = torch.zeros_like(p[0], dtype=torch.bool)
    for a in range(N):  # a bulk cell takes mu of its phase's new composition
        here = (p[a] == 1.0) & ~done
        done = done | here
        for i in range(K1):
            v = Bm[a][i] + sum((2.0 if i == j else 1.0) * k["A"][a][i][j] * (c[a][j] + inc[j]) for j in range(K1))
            new[i] = torch.where(here, v, new[i])
    return phi + torch.stack(d), torch.stack(new)


def _sums(k, phi, mu, t):
    Be = _Beff(k, _temperatures(k, t)[1])
    Be = [[b[:, 1:-1] if torch.is_tensor(b) else b for b in v] for v in Be]
    p = [phi[a] for a in range(k["N"])]
    comp = [sum(_h(p, a) * sum(k["cmu"][a][i][j] * (mu[j] - Be[a][j]) for j in range(k["K1"]))
                for a in range(k["N"])).sum().item() for i in range(k["K1"])]
    return np.array(comp), phi.sum((1, 2)).cpu().numpy()


def _exact_run(case, seed):
    s = _Run(case, seed)
    k, phi, mu = s.k, s.phi0.double(), s.mu0.double()
    for t in range(case["steps"]):
        phi, mu = _step(k, phi, mu, t)
    out = {}
    if case["stats"]:
        solute, fraction = _sums(k, phi, mu, case["steps"])
        out["progress"] = {"solute": solute, "phase_fraction": fraction, "rel_change_phi": None,
                           "rel_change_mu": None, "phi_max": None, "mu_min": None, "grand_potential": None}
    if case["shift"]:
        my, L = case["my"], k["N"] - 1
        row = phi[L].index_select(1, _ghost(my, 3, k["bc"][2]))
        up = ((2.0 * row[:, :-1] - 1.0 < 0) & (2.0 * row[:, 1:] - 1.0 > 0)).any(0).nonzero()
        pos = int(up.max()) + 1
        out["front"] = None
        d = pos - my // 3
        if d > 0:
            src = torch.arange(my, device=DEV) + d
            far = [sum((2.0 if i == j else 1.0) * k["A"][L][i][j] * k["cf"][j] for j in range(k["K1"]))
                   for i in range(k["K1"])]
            liquid = torch.tensor([0.0] * L + [1.0], device=DEV, dtype=torch.float64)[:, None, None]
            rows = _ghost(my, 2, k["bc"][2])[torch.clamp(src, max=my + 1) + 2]
            edge = (src > my + 2)[None, None, :]
            last = (src == my + 2)[None, None, :]
            third = 2 * my - 2 - (my + 2) if k["bc"][2] == 1 else 3
            phi, mu = (torch.where(edge, liq, torch.where(last, f[:, :, third:third + 1], f.index_select(2, rows)))
                       for f, liq in ((phi, liquid),
                                      (mu, torch.tensor(far, device=DEV, dtype=torch.float64)[:, None, None])))
    out["phi"], out["mu"] = phi, mu
    return out


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint
    rng = np.random.default_rng(seed)
    alloy = _alloy(case, case["mx"], case["my"], rng)
    k = _constants(alloy)
    phi0, mu0 = _fields(case, alloy, k, rng)
    target = torch.roll(phi0, (1, 1), (1, 2))
    if case["precision"] == 32:
        phi0, mu0 = phi0.float().double(), mu0.float().double()
    par = torch.tensor([1.0 / k["tau_ab"][(0, 1)], k["dab"][(0, 1)] if k["aniso"] else 0.0, k["Gamma"][(0, 1)], k["Diff"][1][0][0]],
                       device=DEV, dtype=torch.float64, requires_grad=True)
    ratio = k["tau"] / k["tau_ab"][(0, 1)]
    if not k["aniso"]:  # the derivative with respect to the strength is taken at 0, in the grid's frame
        k.update(aniso=1, rot={(0, 1): 0.0}, dab={(0, 1): 0.0})

    def one(phi, mu, p):
        q = dict(k, tau_ab={(0, 1): 1.0 / p[0]}, tau=ratio / p[0], dab={(0, 1): p[1]}, Gamma={(0, 1): p[2]},
                 Diff=[k["Diff"][0], [[p[3]]]])
        return _step(q, phi, mu)

    phi0.requires_grad_(True)
    mu0.requires_grad_(True)
    phi, mu = phi0, mu0
    for _ in range(case["steps"]):
        phi, mu = checkpoint(one, phi, mu, par, use_reentrant=False)
    phi.backward(2.0 * (phi.detach() - target))
    return {"phi": phi.detach(), "mu": mu.detach(), "grad": par.grad, "lam_phi0": phi0.grad, "lam_mu0": mu0.grad}


def exact(case, seed):
    if case["kind"] == "run":
        return _exact_run(case, seed)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    if case["n"] * case["steps"] > 6000:  # minutes of small launches
        return None
    phis, mus = [], []
    for _, k, phi, mu in _instances(case, seed):
        phi, mu = phi.float().double(), mu.float().double()
        for _ in range(case["steps"]):
            phi, mu = _step(k, phi, mu)
        phis.append(phi.reshape(-1)), mus.append(mu.reshape(-1))
    return {"phi": torch.cat(phis), "mu": torch.cat(mus)}
