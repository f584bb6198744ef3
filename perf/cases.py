"""Timed workloads of the public entry points.

Each case is one call sequence that a program equilibrating an actin network
makes, over the sizes of the generator's configurations (``network.CONFIGS``),
the tests and the benchmark:

* ``energy`` / ``forces``: one diagnostic evaluation at coordinates the caller
  holds on the host;
* ``step``: what a controller does after a chemistry step that changed the
  topology: load the network, minimize, read back coordinates, forces,
  linker and motor stretch forces and boundary load forces;
* ``minimize``: the same topology at new coordinates: set them, rebuild the
  neighbor lists, minimize, read the coordinates back;
* ``rebuild``: neighbor lists at new coordinates, and the pair list itself;
* ``ensemble``: independent networks of uneven size minimized together;
* ``second``: a Hessian-vector product and the implicit adjoint of the linker
  parameters;
* ``device_energy``: the filament energy of arrays that already are on the GPU.

Networks start near equilibrium, as between two chemistry steps: overlapping
filaments are pushed apart on the host, then every bead is displaced by a
thermal-size jitter.  A minimization runs for a bounded number of energy calls
(``calls``), which keeps its trajectory reproducible; the iterations are those
of a run to convergence.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from picgo_gb300 import Engine, _lib, cg_params, make_network
from picgo_gb300.network import CONFIGS, CYLINDER_SIZE

JITTER = 0.3          # nm per component
CLEARANCE = 12.0      # nm between segments that started closer
# A solve with the Hessian needs it positive definite, as it is at an equilibrium: away from one, soft contacts and
# the damping of a Levenberg-Marquardt step make it so.
SOFT = 1e-3
SHIFT = 20.0          # pN/nm
C1, C2, C5 = CONFIGS["c1"], CONFIGS["c2"], CONFIGS["c5"]


def _case(name, op, precision, filaments, cylinders, linkers, motors=0, box=0.0, replicas=1, calls=0):
    c = dict(op=op, precision=precision, filaments=filaments, cylinders=cylinders, linkers=linkers, motors=motors,
             box=box, replicas=replicas, calls=calls)
    return dict(c, name=name) if name else c


def listed():
    c1 = (C1["n_filaments"], C1["n_cyl_per_filament"], C1["n_linkers"])
    c2 = (C2["n_filaments"], C2["n_cyl_per_filament"], C2["n_linkers"], C2["n_motors"], C2["box"])
    c5 = (C5["n_filaments"], C5["n_cyl_per_filament"], C5["n_linkers"])
    return [
        # the smallest network of the tests: one energy, all latency
        _case("energy_240_fp64", "energy", "fp64", 24, 10, 40),
        # the example-input size: forces for a diagnostic, single-precision arithmetic
        _case("forces_4k_mixed", "forces", "mixed", *c1),
        # ragged: filament lengths and counts that fill no tile
        _case("forces_21k_fp64", "forces", "fp64", 701, 31, 2617, 263),
        # a chemistry step at the example-input size: topology changes, a short minimization, every read-back
        _case("step_4k_mixed", "step", "mixed", *c1, motors=50, calls=60),
        # the reference's own precision at the example-input size
        _case("minimize_4k_fp64", "minimize", "fp64", *c1, calls=80),
        # the adjoint configuration's size in the production precision
        _case("minimize_60k_mixed", "minimize", "mixed", *c5, calls=120),
        # neighbor lists of the benchmark network, which every chemistry step rebuilds
        _case("rebuild_1M_mixed", "rebuild", "mixed", *c2),
        # the benchmark network, both precisions (the FP64 one is what the mixed one is compared with)
        _case("minimize_1M_mixed", "minimize", "mixed", *c2, calls=120),
        _case("minimize_1M_fp64", "minimize", "fp64", *c2, calls=60),
        # an ensemble of uneven networks minimized together
        _case("ensemble_32_mixed", "ensemble", "mixed", 900, 50, 5600, replicas=32, calls=100),
        # second order: the adjoint's linear solve on its configuration
        _case("second_60k_fp64", "second", "fp64", *c5),
        # arrays on the GPU, nothing allocated
        _case("device_energy_1M_fp64", "device_energy", "fp64", *c2),
    ]


def draw(rng):
    op = rng.choice(["energy", "forces", "forces", "step", "minimize", "minimize", "minimize", "rebuild", "ensemble",
                     "second", "device_energy"])
    precision = "fp64" if op in ("second", "device_energy") else rng.choice(["fp64", "mixed", "mixed"])
    cylinders = rng.randint(8, 50)
    top = 2_000 if op == "ensemble" else 60_000 if op in ("second", "step") else 500_000
    total = math.exp(rng.uniform(math.log(240), math.log(top)))
    filaments = max(5, round(total / cylinders))
    n = filaments * cylinders
    linkers = round(n * rng.uniform(0.05, 0.15))
    motors = rng.choice([0, round(n * 0.01)])
    calls = rng.randint(30, 100) if op in ("step", "minimize", "ensemble") else 0
    replicas = rng.randint(2, 32) if op == "ensemble" else 1
    return _case(None, op, precision, filaments, cylinders, linkers, motors, 0.0, replicas, calls)


# ---------------------------------------------------------------------------
# networks
# ---------------------------------------------------------------------------
def _closest(p1, q1, p2, q2):
    """Parameters (s, t) of the closest points of segments p1-q1 and p2-q2, clamped to the segments."""
    d1, d2, r = q1 - p1, q2 - p2, p1 - p2
    a, e, f = (d1 * d1).sum(1), (d2 * d2).sum(1), (d2 * r).sum(1)
    b, c = (d1 * d2).sum(1), (d1 * r).sum(1)
    den = a * e - b * b
    s = np.clip(np.where(den > 1e-9 * a * e, (b * f - c * e) / np.maximum(den, 1e-30), 0.5), 0.0, 1.0)
    t = np.clip((b * s + f) / e, 0.0, 1.0)
    return np.clip((b * t - c) / a, 0.0, 1.0), t


def _push_apart(net, pairs, sweeps=8):
    """Beads of cylinder pairs whose axes pass closer than CLEARANCE moved apart, each end by its lever arm."""
    x = net.coord.copy()
    a1, a2 = net.cyl_b1[pairs[:, 0]], net.cyl_b2[pairs[:, 0]]
    c1, c2 = net.cyl_b1[pairs[:, 1]], net.cyl_b2[pairs[:, 1]]
    for _ in range(sweeps):
        s, t = _closest(x[a1], x[a2], x[c1], x[c2])
        v = (x[a1] + s[:, None] * (x[a2] - x[a1])) - (x[c1] + t[:, None] * (x[c2] - x[c1]))
        d = np.sqrt((v * v).sum(1))
        k = np.nonzero((d < CLEARANCE) & (d > 1e-6))[0]
        if not k.size:
            break
        u = 0.5 * (CLEARANCE - d[k, None]) * v[k] / d[k, None]
        s, t = s[k, None], t[k, None]
        for bead, move in ((a1[k], (1 - s) * u), (a2[k], s * u), (c1[k], -(1 - t) * u), (c2[k], -t * u)):
            np.add.at(x, bead, move)
    return x


@functools.lru_cache(maxsize=48)
def _base(filaments, cylinders, linkers, motors, box, variant=0):
    """The case's network with its overlaps pushed apart; straight rods where the box holds them, else confined chains."""
    cfg = dict(n_filaments=filaments, n_cyl_per_filament=cylinders, box=box or None, n_linkers=linkers, linker_k=8.0,
               n_motors=motors, motor_l0=C2["motor_l0"], motor_k=C2["motor_k"])
    if not box or box < 1.6 * cylinders * CYLINDER_SIZE:
        cfg["shape"] = "chain"
    if cfg["box"] is None:   # the 2 um density, and room for a chain at the smallest sizes
        cfg["box"] = max(800.0, (filaments * cylinders / (4000 / 2000.0 ** 3)) ** (1 / 3))
    for seed in range(20261300 + 100 * variant, 20261400 + 100 * variant):
        try:
            net = make_network(cfg, seed=seed)
            break
        except RuntimeError:   # no two cylinders within linking range: another placement
            continue
    for _ in range(3):
        net.coord = _push_apart(net, _near_pairs(net))
    return net


def _network(case, seed, variant=0):
    base = _base(case["filaments"], case["cylinders"], case["linkers"], case["motors"], case["box"], variant)
    rng = np.random.default_rng([seed, variant])
    net = base.copy()
    net.coord = net.coord + rng.normal(0.0, JITTER, size=net.coord.shape)
    net.lk_k = rng.uniform(6.0, 10.0, size=net.lk_k.shape)
    if case["op"] == "second":
        net.cyl_kexvol = SOFT * net.cyl_kexvol
    return net


def _ensemble(case, seed):
    """Networks of a tenth to the whole of the case's filament count, in a spread of sizes."""
    nets = []
    for r in range(case["replicas"]):
        f = 0.1 ** (((7 * r) % case["replicas"]) / max(1, case["replicas"] - 1))
        n = max(5, round(case["filaments"] * f))
        one = dict(case, filaments=n, linkers=round(case["linkers"] * n / case["filaments"]),
                   motors=round(case["motors"] * n / case["filaments"]),
                   cylinders=max(4, case["cylinders"] - (5 * r) % max(1, case["cylinders"] // 2)))
        nets.append(_network(one, seed, r + 1))
    return nets


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    op = case["op"]
    s = dict(op=op, single=case["precision"] == "mixed", calls=case["calls"])
    if op == "device_energy":
        return dict(s, **_device_arrays(_network(case, seed)))
    s["engine"] = Engine(case["precision"])
    if op == "ensemble":
        nets = _ensemble(case, seed)
        s["engine"].set_networks(nets)
        return dict(s, replicas=len(nets), params=_params(case))
    s["net"] = _network(case, seed)
    s["engine"].set_network(s["net"])
    if op in ("minimize", "step"):
        s["params"] = _params(case)
    if op == "rebuild":
        s["pairs"] = np.empty((s["net"].n_cyl // 8 + 64, 2), np.int32)
    if op == "second":
        rng = np.random.default_rng([seed, 99])
        s["v"] = rng.normal(size=s["net"].coord.shape)
        s["g"] = rng.normal(size=s["net"].coord.shape)
    return s


def _params(case):
    return cg_params(energy_rel_tol=0.0, energy_call_limit=case["calls"], force_call_limit=100000)


def _device_arrays(net):
    dev = torch.device("cuda", 0)
    put = lambda a, t: torch.from_numpy(np.ascontiguousarray(a, dtype=t)).to(dev)   # noqa: E731
    d = dict(fcs=put(net.fil_cyl_start, np.int32), x=put(net.coord, np.float64), ks=put(net.cyl_kstr, np.float64),
             l0=put(net.cyl_l0, np.float64), kb=put(net.cyl_kbend, np.float64), t0=put(net.cyl_theta0, np.float64))
    return dict(nfil=net.n_filaments, ncyl=net.n_cyl, arrays=d, lib=_lib.load(),
                out=torch.zeros(2, dtype=torch.float64, device=dev))


def _values(state, a):
    """A result as the caller keeps it: the mixed engine's energies and forces carry single precision."""
    return np.asarray(a, dtype=np.float32 if state["single"] else np.float64)


def _outcome(state, results):
    keys = ("status", "error_flags", "num_energy_call", "num_force_call", "num_iter", "num_line_search_trials",
            "num_safe_mode", "num_recover")
    return dict(before=_values(state, [list(r["energies_before"]) for r in results]),
                after=_values(state, [list(r["energies_after"]) for r in results]),
                counts=np.array([[int(r[k]) for k in keys] for r in results], dtype=np.int64))


def run(state):
    op, eng = state["op"], state.get("engine")
    if op == "energy":
        per, total, value = eng.energies(state["net"].coord)
        return _values(state, [*per, total, value])
    if op == "forces":
        return _values(state, eng.forces(state["net"].coord))
    if op == "rebuild":
        eng.set_coords(state["net"].coord)
        info = eng.rebuild()
        pairs = eng.pairs()
        state["pairs"][len(pairs):] = -1
        state["pairs"][:len(pairs)] = pairs
        return dict(pairs=state["pairs"], n_pairs=len(pairs), boundary_beads=int(info["n_boundary_beads"]),
                    boundary_cylinders=int(info["n_boundary_cyl"]))
    if op == "minimize":
        eng.set_coords(state["net"].coord)
        eng.rebuild()
        out = _outcome(state, eng.minimize(state["params"]))
        return dict(out, coords=eng.coords())
    if op == "step":
        eng.set_network(state["net"])
        out = _outcome(state, eng.minimize(state["params"]))
        plus, minus = eng.load_forces()
        linker, motor = eng.stretch_forces()
        return dict(out, coords=eng.coords(), forces=_values(state, eng.last_forces()), plus=plus, minus=minus,
                    linker=_values(state, linker), motor=_values(state, motor))
    if op == "ensemble":
        eng.reset_coords()
        out = _outcome(state, eng.minimize(state["params"]))
        return dict(out, coords=np.concatenate([eng.coords(r) for r in range(state["replicas"])]))
    if op == "second":
        hv = eng.hvp(state["v"])
        # the damped solve of a Levenberg-Marquardt step or a regularised adjoint
        dk, dl0, info = eng.adjoint(state["g"], 0.5, rel_tol=1e-6, max_iter=96, shift=SHIFT)
        return dict(hv=hv, dk=dk, dl0=dl0, iterations=int(info["iterations"]), converged=int(info["converged"]),
                    curvature=int(info["negative_curvature"]))
    if op == "device_energy":
        p = lambda t: ctypes.c_void_p(t.data_ptr())   # noqa: E731
        a = state["arrays"]
        stream = ctypes.c_void_p(torch.cuda.current_stream(0).cuda_stream)
        _lib.check(state["lib"].mech_filament_energy_device(
            state["nfil"], state["ncyl"], p(a["fcs"]), p(a["x"]), p(a["ks"]), p(a["l0"]), p(a["kb"]), p(a["t0"]),
            p(state["out"]), stream))
        return state["out"]
    raise ValueError(op)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Inputs read once and outputs written once; per iteration of a minimization one trial energy, one force
    evaluation and one direction update over the network."""
    op = case["op"]
    ncyl = case["filaments"] * case["cylinders"]
    if op == "ensemble":
        ncyl = 0.4 * ncyl * case["replicas"]   # sizes are spread over a factor of ten
    nb = ncyl * (1 + 1 / case["cylinders"])
    bonds = (case["linkers"] + case["motors"]) * ncyl / (case["filaments"] * case["cylinders"])
    real = 4 if case["precision"] == "mixed" else 8
    energy = nb * (24 + 1 + 4 * real) + bonds * (16 + 4 * real)
    force = energy + nb * 3 * real
    iteration = energy + nb * (3 * real + 24) + force + nb * 3 * real * 3
    host = nb * 24
    flops = {"energy": 60 * nb, "forces": 110 * nb, "device_energy": 60 * nb}.get(op, 0)
    if op == "energy":
        total = host + energy
    elif op == "forces":
        total = 2 * host + force
    elif op == "device_energy":
        total = nb * 24 + ncyl * 32
    elif op == "rebuild":
        total = host + ncyl * (24 + 28)
    elif op == "second":
        total = 3 * host + 24 * nb * 2 + 60 * (force + 8 * 24 * nb)
        flops = 61 * 400 * nb
    else:
        iterations = 0.45 * case["calls"]
        total = 2 * host + (iterations + 2) * iteration + (ncyl * 100 if op == "step" else 0)
        flops = (iterations + 2) * 180 * nb
    return {"bytes": float(total), "flops": float(flops)}


# ---------------------------------------------------------------------------
# 64-bit values from the formulas, in torch
# ---------------------------------------------------------------------------
def _near_pairs(net):
    """Cylinder pairs (c, n), id_c > id_n, midpoints within the cutoff, not within two positions on one filament."""
    mid = 0.5 * (net.coord[net.cyl_b1] + net.coord[net.cyl_b2])
    edge = max(net.exvol_cutoff, net.box / 400)
    cell = np.floor(mid / edge).astype(np.int64) + 1
    g = int(cell.max()) + 2
    key = (cell[:, 0] * g + cell[:, 1]) * g + cell[:, 2]
    order = np.argsort(key, kind="stable")
    skey = key[order]
    rmax2 = float(np.float32(net.exvol_cutoff ** 2))
    found = []
    for off in ((i * g + j) * g for i in (-1, 0, 1) for j in (-1, 0, 1)):   # rows of three cells along z
        lo, hi = np.searchsorted(skey, skey + off - 1, "left"), np.searchsorted(skey, skey + off + 1, "right")
        n = hi - lo
        c = order[np.repeat(np.arange(net.n_cyl), n)]
        m = order[np.arange(int(n.sum())) - np.repeat(np.cumsum(n) - n, n) + np.repeat(lo, n)]
        keep = net.cyl_id[c] > net.cyl_id[m]
        keep &= (net.cyl_fil[c] != net.cyl_fil[m]) | (np.abs(net.cyl_pos[c] - net.cyl_pos[m]) > 2)
        c, m = c[keep], m[keep]
        d = mid[m] - mid[c]
        near = (d * d).sum(1) <= rmax2
        found.append(np.stack([c[near], m[near]], 1))
    return np.concatenate(found)


def _dot(a, b):
    return (a * b).sum(-1)


def _exvol(x, net, pairs, forces):
    """Energies of the double integral of 1/r^4 over cylinder pairs; for forces the nearly coplanar pairs are taken
    with their second bead 0.01 nm off the plane, the move itself not differentiated."""
    c1, c2 = x[net.cyl_b1[pairs[:, 0]]], x[net.cyl_b2[pairs[:, 0]]]
    c3, c4 = x[net.cyl_b1[pairs[:, 1]]], x[net.cyl_b2[pairs[:, 1]]]
    cross = functools.partial(torch.linalg.cross, dim=-1)
    if forces:
        with torch.no_grad():
            n = cross(c2 - c1, c3 - c1)
            n = n / torch.linalg.norm(n, dim=-1, keepdim=True)
            v = c4 - c1
            flat = _dot(n, v / torch.linalg.norm(v, dim=-1, keepdim=True)).abs() < 0.1
            move = torch.where(flat[:, None], 0.01 * n, torch.zeros_like(n))
        c2 = c2 + move
    v12, v34, v31, v14, v32, v24 = c2 - c1, c4 - c3, c1 - c3, c4 - c1, c2 - c3, c4 - c2
    w = cross(v34, v12)
    terms = 0.0
    first = None
    for u, v, p, q, sign in ((v12, v31, v31, v32, 1), (v12, v14, v14, v24, 1), (v34, v31, v31, v14, -1),
                             (v34, v32, v32, v24, -1)):
        k = cross(u, v)
        y = torch.linalg.norm(k, dim=-1)
        num = _dot(k, w)
        if v is v32:
            num = first[0] + first[1] - first[2]
        else:
            first = (first or ()) + (num,)
        terms = terms + num / y * torch.atan2(y, sign * _dot(p, q))
    k = torch.from_numpy(np.maximum(net.cyl_kexvol[pairs[:, 0]], net.cyl_kexvol[pairs[:, 1]]) *
                         net.cyl_l0[pairs[:, 0]] * net.cyl_l0[pairs[:, 1]])
    return 0.5 * k / -(_dot(w, v31) ** 2) * terms


def _fields(x, net, pairs, forces):
    """The six force fields' energies at x, in the library's order."""
    t = torch.from_numpy
    r = x[net.cyl_b2] - x[net.cyl_b1]
    length = torch.linalg.norm(r, dim=-1)
    stretch = (0.5 * t(net.cyl_kstr) * (length - t(net.cyl_l0)) ** 2).sum()
    k = np.nonzero(net.cyl_pos[1:] > 0)[0] + 1    # cylinders that follow one on their filament
    a, b = r[k - 1], r[k]
    c = torch.linalg.cross(a, b, dim=-1)
    ll = length[k - 1] * length[k]
    bend = (t(net.cyl_kbend[k]) * _dot(c, c) / (ll * (ll + _dot(a, b)))).sum()   # k (1 - cos)

    def bonds(cyl, pos, kk, l0):
        if not len(cyl):
            return x.sum() * 0.0
        s, u = t(pos[:, :1]), t(pos[:, 1:])
        p1 = x[net.cyl_b1[cyl[:, 0]]] * (1 - s) + x[net.cyl_b2[cyl[:, 0]]] * s
        p2 = x[net.cyl_b1[cyl[:, 1]]] * (1 - u) + x[net.cyl_b2[cyl[:, 1]]] * u
        return (0.5 * t(kk) * (torch.linalg.norm(p2 - p1, dim=-1) - t(l0)) ** 2).sum()

    exvol = _exvol(x, net, pairs, forces).sum() if len(pairs) else x.sum() * 0.0
    mid = 0.5 * (net.coord[net.cyl_b1] + net.coord[net.cyl_b2])
    wall = x.sum() * 0.0
    for pl, pk, ps in zip(net.planes, net.plane_k, net.plane_slen):
        near = (mid @ pl[:3] + pl[3]) / np.linalg.norm(pl[:3]) < net.boundary_cutoff
        beads = np.concatenate([net.cyl_b1[near & (net.cyl_pos == 0)], net.cyl_b2[near]])
        dist = (x[beads] @ t(pl[:3].copy()) + pl[3]) / float(np.linalg.norm(pl[:3]))
        wall = wall + (pk * torch.exp(-dist / ps)).sum()
    return [stretch, bend, bonds(net.lk_cyl, net.lk_pos, net.lk_k, net.lk_l0),
            bonds(net.mt_cyl, net.mt_pos, net.mt_k, net.mt_l0), exvol, wall]


def _energies(net):
    with torch.no_grad():
        e = [float(v) for v in _fields(torch.from_numpy(net.coord), net, _near_pairs(net), False)]
    return e


def exact(case, seed):
    op = case["op"]
    if op in ("rebuild", "ensemble"):   # whole numbers; and a trajectory, whose start other cases check
        return None
    net = _network(case, seed)
    if op == "device_energy":
        with torch.no_grad():
            e = _fields(torch.from_numpy(net.coord), net, np.zeros((0, 2), np.int64), False)
        return np.array([float(e[0]), float(e[1])])
    if op == "energy":
        e = _energies(net)
        return np.array([*e, sum(e), sum(e)])
    x = torch.from_numpy(net.coord).requires_grad_(True)
    if op == "forces":
        sum(_fields(x, net, _near_pairs(net), True)).backward()
        return -x.grad.numpy()
    if op == "second":
        g, = torch.autograd.grad(sum(_fields(x, net, _near_pairs(net), False)), x, create_graph=True)
        v = np.random.default_rng([seed, 99]).normal(size=net.coord.shape)
        hv, = torch.autograd.grad((g * torch.from_numpy(v)).sum(), x)
        return dict(hv=hv.numpy(), dk=None, dl0=None, iterations=None, converged=None, curvature=None)
    e = _energies(net)
    out = dict(before=np.array([[*e, sum(e)]]), after=None, counts=None, coords=None)
    if op == "step":
        out.update(forces=None, plus=None, minus=None, linker=None, motor=None)
    return out
