"""The calls a program makes of this framework, over the sizes it makes them at.

``listed()`` names them; ``draw(rng)`` gives another of the same ranges.  ``prepare`` builds what a
program holds before the call (an evolver with its initial state, a batch, device buffers), ``run`` is one
pass through the public entry points, ``exact`` what that pass computes, in float64 with plain torch
operations, and ``work`` the bytes and operations no implementation of the pass can avoid.

Initial states are those of the simulator's own workloads: chi = 19 + U(-1e-3, 1e-3) and Gaussian packets
of a few cells' width inside the part of the lattice that the sponge leaves free.
"""

import math
import random
import sys
from pathlib import Path

import torch

_SRC = str(Path(__file__).resolve().parents[1] / "lfm-physics_b200")
if _SRC not in sys.path:
    sys.path.insert(0, _SRC)

import lfm_b200  # noqa: E402
from lfm_b200 import adjoint as _adjoint  # noqa: E402
from lfm_b200.batch import BatchedLattices  # noqa: E402
from lfm_b200.split import SplitChiEvolver  # noqa: E402

REAL, COMPLEX, COLOR = 0, 1, 2
DEVICE = "cuda"
CHI0, DT, SPONGE = 19.0, 0.02, 0.3

# couplings of the presets (gravity_only, gravity_em, full_physics), for exact()
KAPPA, LAMBDA_H, EPSILON_W = 1.0 / 63.0, 4.0 / 31.0, 0.1
KAPPA_C = KAPPA_STRING = 1.0 / 189.0
EPSILON_CC, KAPPA_TUBE, SA_GAMMA, SA_D = 2.0 / 17.0, 30.0 / 63.0, 0.1, 4.9


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # A short run on the smallest lattice anybody uses (quick looks, unit checks): each step is
        # a few microseconds, so launches and latency are all there is.
        {"name": "real_32", "kind": "evolve", "level": REAL, "n": 32, "steps": 200},
        # The presets' default lattice, gravity and electromagnetism.
        {"name": "complex_64", "kind": "evolve", "level": COMPLEX, "n": 64, "steps": 100},
        # A lattice edge that is no multiple of four (users type 50, 90, 150 or 250).
        {"name": "real_150", "kind": "evolve", "level": REAL, "n": 150, "steps": 40},
        # An ordinary production run of the complex level.
        {"name": "complex_256", "kind": "evolve", "level": COMPLEX, "n": 256, "steps": 20},
        # The largest: the lattice of the throughput benchmark, state in HBM.
        {"name": "real_512", "kind": "evolve", "level": REAL, "n": 512, "steps": 12},
        # Three colours with every coupling, S_a solved each step: the preset's default lattice ...
        {"name": "color_64", "kind": "evolve", "level": COLOR, "n": 64, "steps": 40},
        # ... and the benchmark's.
        {"name": "color_256", "kind": "evolve", "level": COLOR, "n": 256, "steps": 8},
        # A parameter sweep: many uneven lattices advanced together.
        {"name": "sweep_48", "kind": "sweep", "count": 48, "mix": 5, "steps": 40},
        # One optimisation step through the simulator: forward with checkpoints, and backward.
        {"name": "adjoint_96", "kind": "adjoint", "level": COMPLEX, "n": 96, "steps": 48,
         "split": False},
        # The accurate option: chi held in two floats.
        {"name": "split_256", "kind": "split", "level": REAL, "n": 256, "steps": 16},
        # The report every interval of a run ends with: float64 energies and statistics.
        {"name": "report_256", "kind": "report", "level": COMPLEX, "n": 256},
        # The drop-in Backend protocol, as the reference's own Evolver calls it: A/B buffers and a
        # streamed mask, one call a step.
        {"name": "protocol_128", "kind": "protocol", "level": COMPLEX, "n": 128, "steps": 8},
    ]


def _edge(rng, lo, hi):
    """A lattice edge, spread over the logarithm: mostly multiples of four, often any integer."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.6:
        n = max(lo + (-lo) % 4, n - n % 4)
    return n


def _steps(rng, n, cells, least, most):
    """Steps of a pass that advances about `cells` cells in all."""
    return max(least, int(min(most, cells / n**3) * rng.uniform(0.6, 1.0)))


def draw(rng):
    kind = rng.choice(["evolve", "evolve", "evolve", "color", "sweep", "adjoint", "split", "report",
                       "protocol"])
    level = rng.choice([REAL, COMPLEX])
    if kind == "evolve":
        n = _edge(rng, 16, 400)
        return {"kind": "evolve", "level": level, "n": n, "steps": _steps(rng, n, 4e8, 6, 250)}
    if kind == "color":
        n = _edge(rng, 24, 240)
        return {"kind": "evolve", "level": COLOR, "n": n, "steps": _steps(rng, n, 8e7, 4, 60)}
    if kind == "sweep":
        return {"kind": "sweep", "count": rng.randint(6, 64), "mix": rng.randrange(1 << 16),
                "steps": rng.randint(16, 60)}
    if kind == "adjoint":
        n = _edge(rng, 20, 104)
        return {"kind": "adjoint", "level": level, "n": n, "steps": rng.randint(12, 56),
                "split": rng.random() < 0.3}
    if kind == "split":
        n = _edge(rng, 32, 288)
        return {"kind": "split", "level": level, "n": n, "steps": _steps(rng, n, 2.5e8, 6, 100)}
    if kind == "report":
        return {"kind": "report", "level": rng.choice([REAL, COMPLEX, COLOR]), "n": _edge(rng, 24, 288)}
    n = _edge(rng, 24, 144)
    return {"kind": "protocol", "level": level, "n": n, "steps": rng.randint(2, 12)}


def _sweep(case):
    """(n, level, kappa) of a sweep's lattices: uneven sizes, both levels, kappa swept."""
    r = random.Random(case["mix"])
    return [(r.choice((32, 48, 64, 80, 96)), r.choice((REAL, COMPLEX)), r.uniform(0.5, 2.0) / 63.0)
            for _ in range(case["count"])]


# ------------------------------------------------------------------ initial states
def _packets(n, count, g, parts):
    """`parts` fields (n, n, n): the same packets under independent phases."""
    u = lambda *s: torch.rand(*s, generator=g, device=DEVICE, dtype=torch.float64)  # noqa: E731
    x = torch.arange(n, device=DEVICE, dtype=torch.float64)
    out = [torch.zeros((n, n, n), device=DEVICE) for _ in range(parts)]
    width = min(1.0, n / 40.0)
    for _ in range(count):
        amp, sigma = 2.0 + 4.0 * u(1), (2.0 + 2.0 * u(1)) * width
        centre = n / 2.0 + (2.0 * u(3) - 1.0) * (0.18 * n)
        gx, gy, gz = (torch.exp(-((x - c) ** 2) / (2.0 * sigma * sigma)) for c in centre)
        weight = torch.cos(2.0 * math.pi * u(parts)) if parts > 1 else torch.ones(1, device=DEVICE)
        plane = (amp * gx)[:, None] * gy[None, :]
        env = (plane[:, :, None].float() * gz.float()[None, None, :])
        for p in range(parts):
            out[p].addcmul_(env, weight[p].float().expand_as(env))
    return out


def _state(level, n, seed):
    """psi_r, psi_i (None at REAL; three colours at COLOR) and chi, float32 on the device."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) * 1000003 + n * 17 + level)
    chi = CHI0 + (2e-3 * torch.rand((n, n, n), generator=g, device=DEVICE) - 1e-3)
    count = max(1, min(16, n // 16))
    if level == REAL:
        return _packets(n, count, g, 1)[0], None, chi
    if level == COMPLEX:
        r, i = _packets(n, count, g, 2)
        return r, i, chi
    f = _packets(n, max(2, count // 2), g, 6)
    return torch.stack(f[:3]), torch.stack(f[3:]), chi


def _config(level, n, **kw):
    preset = {REAL: lfm_b200.gravity_only, COMPLEX: lfm_b200.gravity_em, COLOR: lfm_b200.full_physics}
    return preset[level](n, **kw)


def _before(t, seed):
    """A previous field: the current one a step of slow motion ago."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) * 7919 + 11)
    return t * (1.0 - 0.01 * torch.rand(t.shape, generator=g, device=DEVICE))


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        lattices = _sweep(case)
        batch = BatchedLattices([_config(lv, n, kappa=k) for n, lv, k in lattices])
        for i, (n, lv, _) in enumerate(lattices):
            r, im, chi = _state(lv, n, seed * 131 + i)
            batch.set_psi_real(i, r)
            if im is not None:
                batch.set_psi_imag(i, im)
            batch.set_chi(i, chi)
        return {"case": case, "batch": batch}
    level, n = case["level"], case["n"]
    r, im, chi = _state(level, n, seed)
    if kind in ("evolve", "split"):
        ev = (lfm_b200.Evolver if kind == "evolve" else SplitChiEvolver)(_config(level, n))
        ev.set_psi_real(r)
        if im is not None:
            ev.set_psi_imag(im)
        ev.set_chi(chi)
        return {"case": case, "ev": ev}
    if kind == "report":
        ev = lfm_b200.Evolver(_config(level, n))
        ev.set_psi_real(r)
        ev.set_psi_real_prev(_before(r, seed))
        if im is not None:
            ev.set_psi_imag(im)
            ev.set_psi_imag_prev(_before(im, seed + 1))
        ev.set_chi(chi)
        return {"case": case, "ev": ev}
    if kind == "adjoint":
        state = [r, _before(r, seed), im, None if im is None else _before(im, seed + 1), chi,
                 chi.clone()]
        return {"case": case, "config": _config(level, n),
                "state": [None if t is None else t.requires_grad_(True) for t in state],
                "cotangent": _cotangent(level, n, seed, case["split"])}
    be = lfm_b200.get_backend("auto")  # kind == "protocol"
    fields = [r, _before(r, seed)] + ([] if im is None else [im, _before(im, seed + 1)])
    a = [be.from_numpy(t.reshape(-1).cpu().numpy()) for t in fields + [chi, chi]]
    b = [be.from_numpy(torch.zeros(n**3).numpy()) for _ in a]
    return {"case": case, "be": be, "a": a, "b": b, "mask": be.create_boundary_mask(n, SPONGE),
            "config": _config(level, n)}


def _cotangent(level, n, seed, split):
    """d loss / d (psi_r, psi_i, chi) of the final state."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) * 31337 + 5)
    w = lambda: torch.randn((n, n, n), generator=g, device=DEVICE)  # noqa: E731
    r, i, c = w(), w(), w()
    return [r, None if level == REAL else i, c.double() if split else c]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("evolve", "split"):
        state["ev"].evolve(case["steps"])
        out = state["ev"].device_state()
        if kind == "split":
            out.pop("chi")  # chi64 rounded
        return out
    if kind == "sweep":
        batch = state["batch"]
        batch.evolve(case["steps"])
        st = [batch.device_state(i) for i in range(len(batch))]
        keys = sorted({k for s in st for k in s})
        return {k: torch.cat([s[k].reshape(-1) for s in st if k in s]) for k in keys}
    if kind == "report":
        return state["ev"].metrics()
    if kind == "adjoint":
        out = _adjoint.leapfrog(state["config"], state["state"], case["steps"],
                                split_chi=case["split"])
        wrt = [t for t in state["state"] if t is not None]
        pairs = [(out[f], w) for f, w in zip((0, 2, 4), state["cotangent"]) if w is not None]
        grads = torch.autograd.grad([o for o, _ in pairs], wrt, [w for _, w in pairs])
        return {"state": [None if o is None else o.detach() for o in out], "grads": list(grads)}
    be, cfg, n = state["be"], state["config"], case["n"]
    src, dst = state["a"], state["b"]
    dt2 = cfg.dt**2
    for _ in range(case["steps"]):
        if case["level"] == REAL:
            be.step_real(*src, state["mask"], *dst, n, dt2, cfg.kappa, cfg.lambda_self, cfg.chi0,
                         cfg.e0_sq)
        else:
            be.step_complex(*src, state["mask"], *dst, n, dt2, cfg.kappa, cfg.lambda_self, cfg.chi0,
                            cfg.e0_sq, cfg.epsilon_w)
        src, dst = dst, src
    state["a"], state["b"] = src, dst
    return list(src)


# ------------------------------------------------------------------ what cannot be avoided
# Additions and multiplications of one cell's update (one rounding each, nothing fused).
_OPS = {REAL: 65, COMPLEX: 126, COLOR: 345}
_FIELDS = {REAL: 2, COMPLEX: 3, COLOR: 7}
_ON_CHIP = 120e6  # a state that the L2 cache holds need not go through HBM every step


def _step_work(fields, ops, n, steps, streamed=0):
    """`steps` steps of n^3 cells: both time levels read, the new one written."""
    cells = float(n) ** 3
    passes = steps if 8.0 * fields * cells > _ON_CHIP else 1
    return cells * 4.0 * passes * (3.0 * fields + streamed), cells * steps * float(ops)


def _fft_flops(n, transforms):
    return transforms * 2.5 * n**3 * math.log2(n**3)


def work(case):
    kind = case["kind"]
    if kind == "sweep":
        parts = [_step_work(_FIELDS[lv], _OPS[lv], n, case["steps"]) for n, lv, _ in _sweep(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    level, n = case["level"], case["n"]
    f, cells = _FIELDS[level], float(n) ** 3
    if kind == "evolve":
        b, o = _step_work(f, _OPS[level], n, case["steps"])
        return {"bytes": b, "flops": o + (_fft_flops(n, 6 * case["steps"]) if level == COLOR else 0)}
    if kind == "split":
        b, o = _step_work(f + 1, _OPS[level], n, case["steps"])
        return {"bytes": b, "flops": o}
    if kind == "protocol":  # out of place: previous outputs stored too, the mask streamed
        b, o = _step_work(f, _OPS[level], n, case["steps"], streamed=f + 1)
        return {"bytes": b, "flops": o}
    if kind == "report":
        return {"bytes": cells * 4.0 * (2 * f - 1), "flops": cells * (13 * (f - 1) + 15)}
    # adjoint: the state in and out, its cotangent in and its gradient out; forward, recomputed
    # segments and the transposed step
    return {"bytes": cells * 4.0 * (2 * f) * 4, "flops": cells * case["steps"] * 4.0 * _OPS[level]}


# ------------------------------------------------------------------ float64, plain torch
def _lap(f):
    r = lambda t, *sd: torch.roll(t, tuple(s for s, _ in sd), tuple(d for _, d in sd))  # noqa: E731
    faces = sum(r(f, (s, d)) for d in range(3) for s in (1, -1))
    edges = sum(r(f, (s, d), (t, e)) for d in range(3) for e in range(d) for s in (1, -1)
                for t in (1, -1))
    return faces / 3.0 + edges / 6.0 - 4.0 * f


def _sponge(n):
    x = torch.arange(n, device=DEVICE, dtype=torch.float64) - n / 2.0 + 0.5
    r = torch.sqrt(x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2)
    inner = (1.0 - SPONGE) * n / 2.0
    t = torch.clamp((r - inner) / (n / 2.0 - inner), 0.0, 1.0)
    return torch.sin(0.5 * math.pi * t) ** 2


def _smooth(e):
    n = e.shape[-1]
    k = torch.fft.fftfreq(n, device=DEVICE, dtype=torch.float64) * (2.0 * math.pi)
    kz = torch.fft.rfftfreq(n, device=DEVICE, dtype=torch.float64) * (2.0 * math.pi)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
    s = torch.fft.irfftn(SA_GAMMA / (SA_GAMMA + SA_D * k2) * torch.fft.rfftn(e), s=(n, n, n))
    return torch.clamp_min(s, 0.0)


def _exact_step(level, s, mask, kappa):
    """One step of [psi components], [previous], chi, chi_prev."""
    psi, prev, chi, chi_prev = s
    dt2, absorb = DT * DT, 1.0 - mask
    chi2 = chi * chi
    new = [2.0 * p - q + dt2 * (_lap(p) - chi2 * p) for p, q in zip(psi, prev)]
    rho = sum(p * p for p in psi)
    extra = 0.0
    if level != REAL:
        colours = len(psi) // 2
        js = []
        for a in range(colours):
            pr, pi = psi[a], psi[colours + a]
            js.append([pr * (torch.roll(pi, -1, d) - torch.roll(pi, 1, d))
                       - pi * (torch.roll(pr, -1, d) - torch.roll(pr, 1, d)) for d in range(3)])
        rho_j = rho + EPSILON_W * 0.5 * sum(sum(j) for j in js)
    else:
        rho_j = rho
    if level == COLOR:
        for part in (0, 3):
            mean = (psi[part] + psi[part + 1] + psi[part + 2]) / 3.0
            for a in range(part, part + 3):
                new[a] = new[a] - dt2 * EPSILON_CC * chi2 * (psi[a] - mean)
        ea = [psi[a] ** 2 + psi[3 + a] ** 2 for a in range(3)]
        total = rho * rho
        safe = total > 1e-30
        fc = (torch.where(safe, sum(e * e for e in ea) / torch.where(safe, total, 1.0), 0.0)
              - 1.0 / 3.0) * safe
        extra = (KAPPA_C / CHI0) * chi * fc * rho
        ccv = sum(sum(js[a][d] ** 2 for a in range(3)) - sum(js[a][d] for a in range(3)) ** 2 / 3.0
                  for d in range(3))
        sa = [_smooth(e) for e in ea]
        scv = sum(v * v for v in sa) - sum(sa) ** 2 / 3.0
        extra = extra + KAPPA_STRING * ccv + KAPPA_TUBE * scv
    acc = _lap(chi) - (kappa / CHI0) * chi * rho_j - extra
    if level != REAL:
        acc = acc - 4.0 * LAMBDA_H * chi * (chi2 - CHI0 * CHI0)
    chi_new = torch.clamp_min(2.0 * chi - chi_prev + dt2 * acc, -CHI0)
    return ([p * absorb for p in new], [p * absorb for p in psi], mask * CHI0 + absorb * chi_new, chi)


def _exact_run(level, n, psi, prev, chi, chi_prev, steps, kappa=KAPPA):
    mask = _sponge(n)
    s = ([p.double() for p in psi], [p.double() for p in prev], chi.double(), chi_prev.double())
    for _ in range(steps):
        s = _exact_step(level, s, mask, kappa)
    return s


def _parts(level, r, im):
    if level == REAL:
        return [r]
    return [r, im] if level == COMPLEX else [*r, *im]


def _named(level, s):
    psi, prev, chi, _ = s
    if level == REAL:
        return {"psi_r": psi[0], "psi_r_prev": prev[0], "chi": chi}
    if level == COMPLEX:
        return {"psi_r": psi[0], "psi_r_prev": prev[0], "psi_i": psi[1], "psi_i_prev": prev[1],
                "chi": chi}
    return {"psi_r": torch.stack(psi[:3]), "psi_r_prev": torch.stack(prev[:3]),
            "psi_i": torch.stack(psi[3:]), "psi_i_prev": torch.stack(prev[3:]), "chi": chi}


def _exact_report(level, n, seed):
    r, im, chi = _state(level, n, seed)
    cur = [p.double() for p in _parts(level, r, im)]
    old = _parts(level, _before(r, seed), None if im is None else _before(im, seed + 1))
    kin = grad = pot = 0.0
    c64 = chi.double()
    psi2 = sum(p * p for p in cur)
    for p, q in zip(cur, old):
        kin += 0.5 * float((((p - q.double()) / DT) ** 2).sum())
        grad += 0.5 * sum(float((g * g).sum()) for g in torch.gradient(p, edge_order=1))
    pot = 0.5 * float((c64 * c64 * psi2).sum())
    x = torch.arange(n, device=DEVICE, dtype=torch.float64) - n / 2.0
    dist = torch.sqrt(x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2)
    inner = c64[dist <= n / 2.0 * (1.0 - SPONGE)]
    return {"energy_kinetic": kin, "energy_gradient": grad, "energy_potential": pot,
            "energy_total": kin + grad + pot, "chi_min": float(inner.min()),
            "chi_max": float(inner.max()), "chi_mean": float(inner.mean()),
            "chi_std": float(inner.std(unbiased=False)),
            "well_fraction": float((inner < 17.0).double().mean()),
            "void_fraction": float((inner > 18.0).double().mean()),
            "psi_sq_total": float(psi2.sum()), "interior_cells": float(inner.numel()),
            "nonfinite_cells": 0.0}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        outs = []
        for i, (n, lv, kappa) in enumerate(_sweep(case)):
            r, im, chi = _state(lv, n, seed * 131 + i)
            p = _parts(lv, r, im)
            outs.append(_named(lv, _exact_run(lv, n, p, p, chi, chi, case["steps"], kappa)))
        keys = sorted({k for s in outs for k in s})
        return {k: torch.cat([s[k].reshape(-1) for s in outs if k in s]) for k in keys}
    level, n = case["level"], case["n"]
    if kind == "report":
        return _exact_report(level, n, seed)
    r, im, chi = _state(level, n, seed)
    cur = _parts(level, r, im)
    if kind == "evolve":
        return _named(level, _exact_run(level, n, cur, cur, chi, chi, case["steps"]))
    if kind == "split":
        s = _named(level, _exact_run(level, n, cur, cur, chi, chi, case["steps"]))
        s["chi64"] = s.pop("chi").reshape(-1)
        return {k: v.reshape(-1) for k, v in s.items()}
    old = _parts(level, _before(r, seed), None if im is None else _before(im, seed + 1))
    if kind == "protocol":
        psi, prev, c, cp = _exact_run(level, n, cur, old, chi, chi, case["steps"])
        pairs = [t for pq in zip(psi, prev) for t in pq]
        return [t.reshape(-1) for t in pairs + [c, cp]]
    # adjoint: float64 autograd through the steps
    order = [t for pq in zip(cur, old) for t in pq] + [chi, chi]
    leaves = [t.double().requires_grad_(True) for t in order]
    k = len(cur)
    psi, prev, c, cp = leaves[0:2 * k:2], leaves[1:2 * k:2], leaves[-2], leaves[-1]
    psi, prev, c, cp = _exact_run(level, n, psi, prev, c, cp, case["steps"])
    wr, wi, wc = _cotangent(level, n, seed, case["split"])
    loss = (psi[0] * wr.double()).sum() + (c * wc.double()).sum()
    if wi is not None:
        loss = loss + (psi[1] * wi.double()).sum()
    grads = torch.autograd.grad(loss, leaves)
    final = [t for pq in zip(psi, prev) for t in pq]
    final = final + ([None, None] if level == REAL else []) + [c, cp]
    return {"state": [None if t is None else t.detach() for t in final], "grads": list(grads)}
