"""Timed cases of the stepper: what a program that uses this library has it do, one pass each.

A case is a dict of plain values. `path` says which calls a pass makes:

* "forward":  a handle set up once (grid, medium, source, receivers); a pass resets it, advances
  `steps` steps and reads the traces, the energies (when on) and, with `state`, the final fields;
* "shot":     a whole shot from the host model in pinned memory: handle, medium, source, receivers,
  steps, traces and energies;
* "batch":    many acoustic shots of uneven sizes advanced together, their traces read;
* "gradient": the misfit gradient of one shot with checkpoints.

`exact` is the same scheme in plain torch in 64 bits (SBP tables, closures, penalties and energy
norms restated here), on the GPU where there is one.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEN_DX = 500      # dx = 1 / DEN_DX, as in the benchmark
F0 = 15.0         # Ricker frequency of the elastic benchmark


def _twave():
    if "twave" not in sys.modules:
        spec = importlib.util.spec_from_file_location("twave", os.path.join(ROOT, "tpu-wave_b200", "__init__.py"))
        mod = importlib.util.module_from_spec(spec)
        sys.modules["twave"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["twave"]


def _case(name, **kw):
    c = {"path": "forward", "physics": "elastic", "bc_x": "free", "sat_y": False, "precision": "f32", "cpst": "00",
         "coef_q16": False, "energy": False, "rcv": 16, "state": True}
    c.update(kw)
    if name:
        c["name"] = name
    return c


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: the size of the smoke run and of most of the test suite, energy on (the default)
        _case("elastic_48x40", Mx=48, My=40, steps=200, energy=True),
        # a small ragged survey grid, energy off
        _case("elastic_509x317", Mx=509, My=317, steps=1000),
        # the headline benchmark: elastic 2048^2 FP32, energy off, final state read
        _case("elastic_2048", Mx=2048, My=2048, steps=2000),
        # the benchmark's end-to-end leg: a whole shot with the discrete energy every step, from the host model
        _case("elastic_2048_shot_energy", path="shot", Mx=2048, My=2048, steps=1000, energy=True, state=False),
        # the large target grid of the benchmark (its state is 2.7 GB of host doubles: traces only)
        _case("elastic_8192", Mx=8192, My=8192, steps=100, rcv=256, state=False),
        # 16-bit coefficient codes, the mixed-precision mode that meets the error bound, on an odd large grid
        _case("elastic_q16_4095x4097", Mx=4095, My=4097, steps=200, coef_q16=True, rcv=64, state=False),
        # FP16 storage as hi + lo pairs
        _case("elastic_fp16_split_1500x1023", Mx=1500, My=1023, steps=400, precision="fp16", cpst="split"),
        # FP64 with the energy record: how a scheme is verified
        _case("elastic_f64_1024_energy", Mx=1024, My=1024, steps=300, precision="f64", energy=True),
        # the compensated time update of the reference ('6C'), FP32
        _case("elastic_6C_1000x1200", Mx=1000, My=1200, steps=400, cpst="6C"),
        # the plain acoustic configuration: 512^2, periodic, 1000 steps
        _case("acoustic_512_periodic", physics="acoustic", bc_x="periodic", Mx=512, My=512, steps=1000),
        # the batched configuration, uneven shots in one launch
        _case("acoustic_batch_24", path="batch", physics="acoustic", bc_x="periodic", Mx=0, My=0, steps=500, shots=24,
              sizes=3, state=False),
        # the gradient configuration: 1024^2 FP32, 256 receivers, checkpoints every 50 steps
        _case("gradient_1024", path="gradient", Mx=1024, My=1024, steps=400, rcv=256, ckpt=50, state=False),
    ]


def draw(rng):
    """One more case of the same ranges: sizes log-uniform from 32^2 to 4096^2 cells, aspect ratios up
    to 3, odd sizes among them, and the storage types, codes and boundaries a handle can have."""
    def size(lo, hi):
        cells, asp = math.exp(rng.uniform(math.log(lo), math.log(hi))), math.exp(rng.uniform(-math.log(3), math.log(3)))
        return max(24, round(math.sqrt(cells * asp))), max(24, round(math.sqrt(cells / asp)))

    kind = rng.choices(["f32", "f32_energy", "shot", "q16", "split", "f64", "cpst", "variant", "acoustic", "batch",
                        "gradient"], [4, 3, 1, 1, 1, 2, 1, 1, 2, 1, 1])[0]
    if kind == "batch":
        return _case(None, path="batch", physics="acoustic", bc_x="periodic", Mx=0, My=0, steps=rng.randint(100, 400),
                     shots=rng.randint(4, 24), sizes=rng.randint(0, 10 ** 6), state=False)
    if kind == "gradient":
        Mx, My = size(64 * 64, 1024 * 1024)
        return _case(None, path="gradient", Mx=Mx, My=My, steps=rng.randint(100, 300), rcv=rng.randint(8, 128),
                     ckpt=rng.choice([10, 50]), precision=rng.choice(["f32", "f32", "f64"]), state=False)
    Mx, My = size(32 * 32, 4096 * 4096)
    kw = {"Mx": Mx, "My": My, "rcv": rng.randint(1, 64)}
    if kind in ("f32_energy", "shot"):
        kw["energy"] = True
    if kind == "shot":
        kw["path"] = "shot"
    if kind == "q16":
        kw.update(coef_q16=True, My=max(My, 200))
    if kind == "split":
        kw.update(precision=rng.choice(["bf16", "fp16"]), cpst="split")
    if kind == "f64":
        kw.update(precision="f64", energy=rng.random() < 0.5)
    if kind == "cpst":
        kw.update(cpst=rng.choice(["-3C", "-3R", "3C", "3R", "6C", "6R"]))
    if kind == "variant":
        kw.update(bc_x=rng.choice(["free", "interface"]), sat_y=True)
    if kind == "acoustic":
        kw.update(physics="acoustic", bc_x=rng.choice(["free", "periodic"]))
    c = _case(None, steps=0, **kw)
    c["state"] = c["path"] == "forward" and kw["Mx"] * kw["My"] <= 1 << 22
    c["steps"] = int(min(rng.randint(100, 1000), max(20, 2e11 / (_bytes_per_update(c) * kw["Mx"] * kw["My"]))))
    return c


def _bytes_per_update(c):
    """HBM bytes one cell-update cannot do without: each field read and written, each coefficient read."""
    nf = 5 if c["physics"] == "elastic" else 3
    e = {"f64": 8, "f32": 4, "bf16": 2, "fp16": 2}[c["precision"]]
    comp = 0 if c["cpst"] == "00" else 2 * e
    coef = 2 if c["coef_q16"] else max(e, 4)
    return nf * (2 * e + comp + coef)


def _sides(c):
    return [int(v) for v in np.random.default_rng(c["sizes"]).choice([256, 512, 1024], c["shots"])]


def work(case):
    c, n = case, case["steps"]
    cells = sum(s * s for s in _sides(c)) if c["path"] == "batch" else c["Mx"] * c["My"]
    out = 8 * 2 * c["rcv"] * n + (8 * 5 * cells if c["state"] else 0)
    if c["path"] == "gradient":
        # per step: the forward step, the step recomputed from its checkpoint, the adjoint state read
        # and written, the coefficients, the forward state read once and the FP64 gradients updated
        e = 8 if c["precision"] == "f64" else 4
        return {"bytes": n * cells * (2 * 15 * e + 20 * e + 80) + 8 * 8 * cells, "flops": n * cells * 350}
    return {"bytes": n * cells * _bytes_per_update(c) + out, "flops": n * cells * (86 if c["physics"] == "elastic" else 36)}


# --------------------------------------------------------------------------- inputs
def _setup(c, seed, side=None):
    """Medium, source, receivers and time step of one shot, from the seed."""
    rng = np.random.default_rng([seed, 0 if side is None else side[1]])
    Mx, My = (c["Mx"], c["My"]) if side is None else (side[0], side[0])
    nl, n = 8, c["steps"]
    vp_l, rho_l = rng.uniform(1.5, 4.5, nl), rng.uniform(1.8, 2.7, nl)
    u = {"Mx": Mx, "My": My, "n": n, "f0": F0, "dx": 1.0 / DEN_DX}
    u["dt"] = 0.4 * u["dx"] / (math.sqrt(2.0) * vp_l.max())
    u["delay"] = min(0.1, 0.4 * n * u["dt"])
    sx, sy = int(rng.integers(Mx // 3, 2 * Mx // 3)), int(rng.integers(My // 3, 2 * My // 3))
    u["src"] = (sx, sy)
    # a line of receivers above the source across the whole width, the first one over the source
    u["rcv"] = (np.full(c["rcv"], max(2, sx - 10)), (sy + np.arange(c["rcv"]) * My // c["rcv"]) % My)
    layer = np.minimum(np.arange(Mx + 2) * nl // (Mx + 1), nl - 1)
    if c["physics"] == "acoustic" and c["bc_x"] == "periodic":
        layer[Mx] = layer[0]   # the seam row repeats row 0
        kap = rho_l * vp_l ** 2
        u["grid"] = (np.repeat(rho_l[layer[:Mx + 1]][:, None], My, 1), np.repeat(rho_l[layer[:Mx]][:, None], My + 1, 1),
                     np.repeat(kap[layer[:Mx]][:, None], My, 1))   # rho of Vx (NM), rho of Vy (MN), kappa
        return u
    vp = np.repeat(vp_l[layer][:, None], My + 2, 1)
    rho = np.repeat(rho_l[layer][:, None], My + 2, 1)
    vs = None if c["physics"] == "acoustic" else vp * (rng.uniform(0.9, 1.1, vp.shape) / math.sqrt(3.0))
    for a in (vp, rho) if vs is None else (vp, rho, vs):   # the reference's zero padding
        a[Mx + 1:, :] = 0.0
        a[:, My + 1:] = 0.0
    u["model"] = (rho, vp, vs)
    return u


def _solver(c, u):
    tw = _twave()
    bc = {"free": tw.SAT_FREE, "periodic": tw.PERIODIC, "interface": tw.SAT_INTERFACE}[c["bc_x"]]
    s = tw.Solver(u["Mx"], u["My"], 1, DEN_DX, u["dt"], physics=tw.ELASTIC if c["physics"] == "elastic" else tw.ACOUSTIC,
                  bc_x=bc, precision=c["precision"], cpst=c["cpst"], central_f=u["f0"], time_delay=u["delay"],
                  max_steps=u["n"], energy=c["energy"], sat_y=c["sat_y"], coef_q16=c["coef_q16"])
    if "grid" in u:
        s.set_material_grid(tw.NM, 0, u["grid"][0])
        s.set_material_grid(tw.MN, 0, u["grid"][1])
        s.set_material_grid(tw.MM, 0, u["grid"][2])
    else:
        s.set_material_model(*u["model"])
    s.set_source(tw.MM, *u["src"])
    s.add_receivers(tw.NM if c["physics"] == "elastic" else tw.MM, *u["rcv"])
    return s


def _perturbed(u):
    """The medium the observed traces come from: 5 % faster in a Gaussian patch under the receivers."""
    rho, vp, vs = u["model"]
    X, Y = np.arange(vp.shape[0])[:, None], np.arange(vp.shape[1])[None, :]
    sx, sy = u["src"]
    w = max(3.0, 0.05 * u["n"])
    bump = 1.0 + 0.05 * np.exp(-((X - sx) ** 2 + (Y - sy) ** 2) / (2 * w * w))
    return rho, vp * bump, vs * bump


def prepare(case, seed):
    tw, c = _twave(), case
    if c["path"] == "batch":
        shots = [_solver(c, _setup(c, seed, (side, k))) for k, side in enumerate(_sides(c))]
        b = tw.Batch(shots)
        b.tune(8)
        return {"case": c, "batch": b, "shots": shots}
    u = _setup(c, seed)
    if c["path"] == "shot":   # the model in pinned memory, as a program that runs many shots keeps it
        pins = []
        for a in u["model"]:
            t = torch.empty(a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
            t.numpy()[...] = a
            pins.append(t)
        u["model"] = tuple(t.numpy() for t in pins)
        return {"case": c, "setup": u, "pins": pins}
    st = {"case": c, "solver": _solver(c, u)}
    if c["path"] == "gradient":
        with torch.no_grad():
            st["obs"] = _simulate(c, u, _coefficients(c, u, _perturbed(u)))["traces"].cpu().numpy()
    return st


# --------------------------------------------------------------------------- one pass
def _read(c, s):
    tw = _twave()
    out = {"traces": s.read_receivers()}
    if c["energy"]:
        out["energy"] = list(s.read_energy())
    if c["state"]:
        slots = [(tw.MN, 0), (tw.NM, 0), (tw.MM, 0)]
        if c["physics"] == "elastic":
            slots = [(tw.NN, 0)] + slots + [(tw.MM, 1)]
        out["state"] = [s.read_field(g, f) for g, f in slots]
    return out


def run(state):
    c = state["case"]
    if c["path"] == "batch":
        for s in state["shots"]:
            s.reset()
        state["batch"].run(c["steps"])
        return [s.read_receivers() for s in state["shots"]]
    if c["path"] == "shot":
        with _solver(c, state["setup"]) as s:
            s.run(c["steps"])
            return _read(c, s)
    s = state["solver"]
    s.reset()
    if c["path"] == "gradient":
        return s.adjoint_gradient(c["steps"], state["obs"], ckpt_every=c["ckpt"])
    s.run(c["steps"])
    return _read(c, s)


# --------------------------------------------------------------------------- the scheme in 64 bits
ST = (1 / 24, -9 / 8, 9 / 8, -1 / 24)
DM_L = ((-2., 3., -1., 0., 0.), (-1., 1., 0., 0., 0.), (1 / 24, -9 / 8, 9 / 8, -1 / 24, 0.),
        (-1 / 71, 6 / 71, -83 / 71, 81 / 71, -3 / 71))
DM_R = ((3 / 71, -81 / 71, 83 / 71, -6 / 71, 1 / 71), (0., 1 / 24, -9 / 8, 9 / 8, -1 / 24), (0., 0., 0., -1., 1.),
        (0., 0., 1., -3., 2.))
DN_L = ((-79 / 78, 27 / 26, -1 / 26, 1 / 78, 0.), (2 / 21, -9 / 7, 9 / 7, -2 / 21, 0.),
        (1 / 75, 0., -27 / 25, 83 / 75, -1 / 25))
DN_R = ((1 / 25, -83 / 75, 27 / 25, 0., -1 / 75), (0., 2 / 21, -9 / 7, 9 / 7, -2 / 21),
        (0., -1 / 78, 1 / 26, -27 / 26, 79 / 78))
A_N = (7 / 18, 9 / 8, 1., 71 / 72)     # norm diagonal next to a left end (mirrored at a right one)
A_M = (13 / 12, 7 / 8, 25 / 24)
P_M = (15 / 8, -5 / 4, 3 / 8)          # projection of three M-type rows onto a left end


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a, np.float64), device=_device())


def _taps(p, dim, m):
    out = ST[0] * p.narrow(dim, 0, m)
    for k in (1, 2, 3):
        out = torch.add(out, p.narrow(dim, k, m), alpha=ST[k])
    return out


def _ends(table, a, dim):
    T = _t(table)
    return T @ a if dim == 0 else a @ T.t()


def _diff(a, from_n, dim, closed):
    """Difference (times dx) along dim of an N-type array at the M-type points (from_n), or the reverse."""
    n = a.shape[dim] - (1 if from_n else 0)   # cells
    if not closed:
        if from_n:   # columns c-1 .. c+2; the seam column is read directly, beyond it the reads wrap
            return _taps(torch.cat([a.narrow(dim, n - 1, 1), a, a.narrow(dim, 1, 1)], dim), dim, n)
        return _taps(torch.cat([a.narrow(dim, n - 2, 2), a, a.narrow(dim, 0, 2)], dim), dim, n + 1)
    if from_n:
        mid = _taps(a.narrow(dim, 2, n - 3), dim, n - 6)
        return torch.cat([_ends(DN_L, a.narrow(dim, 0, 5), dim), mid, _ends(DN_R, a.narrow(dim, n - 4, 5), dim)], dim)
    mid = _taps(a.narrow(dim, 2, n - 4), dim, n - 7)
    return torch.cat([_ends(DM_L, a.narrow(dim, 0, 5), dim), mid, _ends(DM_R, a.narrow(dim, n - 5, 5), dim)], dim)


def _penalty(d, a, from_n, dim, interface):
    """d plus the penalty (times dx) of its end points: the neighbour a projected on the ends."""
    n = a.shape[dim] - (1 if from_n else 0)
    if from_n:
        sL, sR = a.narrow(dim, 0, 1), a.narrow(dim, n, 1)
        wL, wR = [p / q for p, q in zip(P_M, A_M)], [-p / q for p, q in zip(P_M[::-1], A_M[::-1])]
    else:
        sL = sum(p * a.narrow(dim, k, 1) for k, p in enumerate(P_M))
        sR = sum(p * a.narrow(dim, n - 1 - k, 1) for k, p in enumerate(P_M))
        wL, wR = [1 / A_N[0]], [-1 / A_N[0]]
    if interface:
        sL, sR = 0.5 * (sL - sR), 0.5 * (sR - sL)
    shape = (-1, 1) if dim == 0 else (1, -1)
    k, m = len(wL), d.shape[dim]
    return torch.cat([d.narrow(dim, 0, k) + _t(wL).reshape(shape) * sL, d.narrow(dim, k, m - 2 * k),
                      d.narrow(dim, m - k, k) + _t(wR).reshape(shape) * sR], dim)


def _coefficients(c, u, model):
    """mu, 1/rho (MN), 1/rho (NM), lambda, 2mu on the staggered points."""
    if "grid" in u:
        rx, ry, kap = (_t(a) for a in u["grid"])
        return [None, 1 / ry, 1 / rx, kap, None]
    Mx, My = u["Mx"], u["My"]
    r, p, q = ((a if torch.is_tensor(a) else _t(a))[:Mx + 1, :My + 1] if a is not None else None for a in model)
    ax = lambda a: 0.5 * (a[:-1] + a[1:])            # noqa: E731
    ay = lambda a: 0.5 * (a[:, :-1] + a[:, 1:])      # noqa: E731
    if q is None:
        return [None, 1 / ax(r), 1 / ay(r), ax(ay(r * p * p)), None]
    mu = r * q * q
    return [mu.clone(), 1 / ax(r), 1 / ay(r), ax(ay(r * p * p - 2 * mu)), ax(ay(2 * mu))]


def _norm(n, nt, dx, closed):
    """Energy norm along one direction, n cells, N type (n + 1 points) or M type."""
    w = torch.full((n + (1 if nt else 0),), dx, dtype=torch.float64, device=_device())
    if closed:
        a = _t(A_N if nt else A_M)
        w[:len(a)], w[-len(a):] = a * dx, a.flip(0) * dx
    elif nt:
        w[n] = 0.0
    return w


def _step(c, k, co, state):
    """One step; state: NN, MN, NM, MM0, MM1 (acoustic: MN, NM, MM0). k = dt / dx."""
    xc, yc, xi = c["bc_x"] != "periodic", c["sat_y"], c["bc_x"] == "interface"
    mu, im, iv, lam, m2 = co
    if c["physics"] == "acoustic":
        vy, vx, p = state
        d = _diff(p, False, 1, yc)
        vy = vy + k * co[1] * (_penalty(d, p, False, 1, False) if yc else d)
        d = _diff(p, False, 0, xc)
        vx = vx + k * co[2] * (_penalty(d, p, False, 0, xi) if xc else d)
        d = _diff(vx, True, 0, xc)
        d = (_penalty(d, vx, True, 0, True) if xi else d) + _diff(vy, True, 1, yc)
        return [vy, vx, p + k * lam * d]
    nn, mn, nm, s0, s1 = state
    dx_, dy_ = _penalty(_diff(nn, True, 0, True), nn, True, 0, xi), _diff(s1, False, 1, yc)
    mn = mn + k * im * (dx_ + (_penalty(dy_, s1, False, 1, False) if yc else dy_))
    dx_, dy_ = _penalty(_diff(s0, False, 0, True), s0, False, 0, xi), _diff(nn, True, 1, yc)
    nm = nm + k * iv * (dx_ + (_penalty(dy_, nn, True, 1, False) if yc else dy_))
    d = _diff(mn, False, 0, True)
    nn = nn + k * mu * ((_penalty(d, mn, False, 0, True) if xi else d) + _diff(nm, False, 1, yc))
    ex, ey = _diff(nm, True, 0, True), _diff(mn, True, 1, yc)
    ex = _penalty(ex, nm, True, 0, True) if xi else ex
    s = lam * (ex + ey)
    return [nn, mn, nm, s0 + k * (s + m2 * ex), s1 + k * (s + m2 * ey)]


def _source(u, it):
    t = (it + 0.5) * u["dt"] - u["delay"]
    q = (math.pi * u["f0"] * t) ** 2
    return (1 - 2 * q) * math.exp(-q) * u["dt"] / u["dx"] ** 2


def _simulate(c, u, co):
    Mx, My, n = u["Mx"], u["My"], u["n"]
    el = c["physics"] == "elastic"
    z = lambda r, q: torch.zeros(r, q, dtype=torch.float64, device=_device())   # noqa: E731
    state = ([z(Mx + 1, My + 1)] if el else []) + [z(Mx, My + 1), z(Mx + 1, My), z(Mx, My)] + ([z(Mx, My)] if el else [])
    k, (sx, sy) = u["dt"] / u["dx"], u["src"]
    ix, iy = (torch.as_tensor(a, device=_device()) for a in u["rcv"])
    spike = z(Mx, My)
    spike[sx, sy] = 1.0
    stress = (3, 4) if el else (2,)
    energy = []
    if c["energy"]:
        xc, yc, dx = c["bc_x"] != "periodic", c["sat_y"], u["dx"]
        wgt = lambda a, b: _norm(Mx, a, dx, xc)[:, None] * _norm(My, b, dx, yc)[None, :]   # noqa: E731
        den = co[4] * (2 * co[3] + co[4])
        w = [wgt(1, 1) / co[0], wgt(0, 1) / co[1], wgt(1, 0) / co[2], wgt(0, 0) * (co[3] + co[4]) / den,
             wgt(0, 0) * -2 * co[3] / den]
        pot = lambda s: 0.5 * ((w[0] * s[0] ** 2).sum() + (w[3] * (s[3] ** 2 + s[4] ** 2)).sum() +   # noqa: E731
                               (w[4] * s[3] * s[4]).sum())

    def advance(it0, it1, *args):
        st, cf, tr = list(args[:len(state)]), list(args[len(state):]), []
        for it in range(it0, it1):
            p0 = pot(st) if c["energy"] else None
            st = _step(c, k, cf, st)
            for f in stress:
                st[f] = torch.add(st[f], spike, alpha=_source(u, it))
            if c["energy"]:
                energy.append(torch.stack([0.5 * ((w[1] * st[1] ** 2).sum() + (w[2] * st[2] ** 2).sum()), p0, pot(st)]))
            tr.append(st[2][ix, iy])   # NM (elastic) or the pressure (acoustic)
        return (*st, torch.stack(tr, 1))

    grad = any(t is not None and t.requires_grad for t in co)
    seg, traces = 16 if grad else n, []
    for it in range(0, n, seg):
        args = (it, min(n, it + seg), *state, *co)
        *state, tr = checkpoint(advance, *args, use_reentrant=False) if grad else advance(*args)
        traces.append(tr)
    tr = torch.cat(traces, 1)
    out = {"traces": torch.stack([tr, torch.zeros_like(tr)], 1)}
    if c["energy"]:
        out["energy"] = list(torch.stack(energy, 1))
    out["state"] = list(state)
    return out


def _gradient(c, u):
    rho, vp, vs = u["model"]
    with torch.no_grad():
        obs = _simulate(c, u, _coefficients(c, u, _perturbed(u)))["traces"]
    node = [_t(a).requires_grad_() for a in (rho, vp, vs)]
    co = _coefficients(c, u, node)
    for t in co:
        t.retain_grad()
    J = 0.5 * ((_simulate(c, u, co)["traces"] - obs) ** 2).sum()
    J.backward()
    g = [t.grad for t in co]
    grid = {"NN_mu": g[0], "MN_rho": -g[1] * co[1].detach() ** 2, "NM_rho": -g[2] * co[2].detach() ** 2,
            "MM_lambda": g[3], "MM_2mu": g[4]}
    return {"grid": grid, "misfit": J.detach(), "rho": node[0].grad, "vp": node[1].grad, "vs": node[2].grad}


def exact(case, seed):
    c = case
    if c["path"] == "batch":
        us = [_setup(c, seed, (side, k)) for k, side in enumerate(_sides(c))]
        with torch.no_grad():
            return [_simulate(c, u, _coefficients(c, u, None))["traces"].cpu() for u in us]
    u = _setup(c, seed)
    if c["path"] == "gradient":
        out = _gradient(c, u)
        return {k: {q: v.cpu() for q, v in x.items()} if isinstance(x, dict) else x.cpu() for k, x in out.items()}
    with torch.no_grad():
        out = _simulate(c, u, _coefficients(c, u, u.get("model")))
    if not c["state"]:
        del out["state"]
    return {k: [t.cpu() for t in v] if isinstance(v, list) else v.cpu() for k, v in out.items()}
