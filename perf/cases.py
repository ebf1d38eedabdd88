"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is one of six kinds:

  bd       one Box.propagate step of plain Brownian dynamics with hydrodynamic
           interactions (rpy_smith, Ermak), beads alone or bonded polymer
           chains with Lennard-Jones, bond and angle forces, FP64 or mixed;
  sd       one Box.propagate step of lubricated Stokesian dynamics
           (rpy_smith_lub, midpoint scheme), FP64;
  batch    a ReplicaBatch advanced by a few steps with device noise, then a
           frame of every replica's positions read into pinned host memory;
  tensor   the Smith-Ewald RPY tensor of a device-resident configuration
           (pbg_dev_smith_matrix), as an analysis or another integrator uses it;
  factor   the Cholesky factor of such a tensor in place (pbg_dev_cholesky);
  inverse  its inverse in place (pbg_dev_spd_inverse).

The listed sizes are the workloads that this repository states (64 beads of
plain BD, the 1024-bead headline, the 512-bead lubricated suspension, the 256
replicas, the mixed-size serving stream) and sizes between and below them.
`draw` gives more of the same ranges, odd sizes included.

`exact` computes the same results in FP64 with plain torch and numpy.
"""
import math

import numpy as np
import torch

BOLTZMANN = 1.380649e-23
T, ETA = 293.15, 0.01005
KBT = BOLTZMANN * T
ALPHA, M_MAX, N_MAX = math.sqrt(math.pi), 2, 4


# ----------------------------------------------------------------------------- the cases

def listed():
    return [
        # The smallest ordinary run (64 beads of radius 20 in a box of 750, dt 1): a step is
        # launches, host round trips and the short panel chain, not arithmetic.
        {"name": "bd 64 fp64", "kind": "bd", "beads": 64, "polymer": False, "precision": "fp64", "dt": 1.0},
        # A solution of flexible chains (16 beads each): the force kernels and the
        # deterministic move run every step.
        {"name": "bd polymer 336 fp64", "kind": "bd", "beads": 336, "polymer": True, "precision": "fp64",
         "dt": 0.05},
        # The headline workload, 1024 polydisperse beads, in its mixed precision ...
        {"name": "bd 1024 mixed", "kind": "bd", "beads": 1024, "polymer": False, "precision": "mixed", "dt": 0.5},
        # ... and in FP64, the default precision of the drivers.
        {"name": "bd 1024 fp64", "kind": "bd", "beads": 1024, "polymer": False, "precision": "fp64", "dt": 0.5},
        # The dense lubricated suspension (volume fraction 0.30): two resistance matrices,
        # three factorisations and two triangular solves per midpoint step.
        {"name": "sd 512 fp64", "kind": "sd", "beads": 512, "dt": 0.1},
        # A small lubricated box of odd size, as used for testing a force field or a protocol.
        {"name": "sd 101 fp64", "kind": "sd", "beads": 101, "dt": 0.1},
        # An ensemble of 256 independent replicas of uneven size; a frame every 2 steps.
        {"name": "batch 256 mixed", "kind": "batch", "replicas": 256, "lo": 32, "hi": 512, "log": False,
         "precision": "mixed", "steps": 2, "dt": 0.5},
        # A serving moment: 24 requests in flight, sizes log-uniform up to 2048 beads.
        {"name": "batch 24 serving", "kind": "batch", "replicas": 24, "lo": 16, "hi": 2048, "log": True,
         "precision": "mixed", "steps": 2, "dt": 1.0},
        # Replicas of a job range with the drivers' default precision.
        {"name": "batch 40 fp64", "kind": "batch", "replicas": 40, "lo": 16, "hi": 200, "log": False,
         "precision": "fp64", "steps": 4, "dt": 0.5},
        # Building blocks through the device-pointer calls: the FP32 tensor of a large
        # system, the factor of one of odd order, the inverse of a middle-sized one.
        {"name": "tensor 1999 mixed", "kind": "tensor", "beads": 1999, "precision": "mixed"},
        {"name": "factor 601 fp64", "kind": "factor", "beads": 601, "precision": "fp64"},
        {"name": "inverse 333 fp64", "kind": "inverse", "beads": 333, "precision": "fp64"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bd", "bd", "bd", "sd", "batch", "batch", "tensor", "factor", "inverse"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "bd":
        if rng.random() < 0.3:
            return {"kind": "bd", "beads": 16 * rng.randint(2, 32), "polymer": True, "precision": precision,
                    "dt": 0.05}
        return {"kind": "bd", "beads": _log_uniform(rng, 24, 1300), "polymer": False, "precision": precision,
                "dt": rng.choice([0.5, 1.0])}
    if kind == "sd":
        return {"kind": "sd", "beads": _log_uniform(rng, 30, 540), "dt": 0.1}
    if kind == "batch":
        if rng.random() < 0.3:
            return {"kind": "batch", "replicas": rng.randint(6, 24), "lo": 16, "hi": rng.randint(600, 1600),
                    "log": True, "precision": "mixed", "steps": 2, "dt": 1.0}
        small = precision == "fp64"
        return {"kind": "batch", "replicas": _log_uniform(rng, 8, 48 if small else 200), "lo": 16,
                "hi": rng.randint(60, 200 if small else 500), "log": False, "precision": precision,
                "steps": 4 if small else 2, "dt": 0.5}
    if kind == "tensor":
        return {"kind": "tensor", "beads": _log_uniform(rng, 100, 2200), "precision": precision}
    if kind == "factor":
        return {"kind": "factor", "beads": _log_uniform(rng, 30, 1300), "precision": precision}
    return {"kind": "inverse", "beads": _log_uniform(rng, 30, 600), "precision": "fp64"}


# ----------------------------------------------------------------------------- configurations

def _place(rng, radii, L, gap=0.0):
    """Sequential random placement without overlaps (minimum image): a bead takes the first of a pool of
    uniform candidates that is clear of the beads placed before it."""
    n = len(radii)
    pos = np.empty((n, 3))
    least = gap + float(np.min(radii))
    pool, room = np.empty((3, 0)), np.empty(0)  # candidates, and each one's distance to the nearest surface
    for k in range(n):
        need = radii[k] + gap
        ok = room > need
        at = int(ok.argmax()) if len(room) else 0
        while not len(room) or not ok[at]:
            pool = rng.uniform(-L / 2, L / 2, size=(3, max(64, n)))
            room = np.full(pool.shape[1], np.inf)
            for q in range(0, k, 64):
                d = pool[:, :, None] - pos[q:min(k, q + 64)].T[:, None, :]
                d -= L * np.rint(d / L)
                near = np.sqrt(np.einsum("cij,cij->ij", d, d)) - radii[None, q:min(k, q + 64)]
                room = np.minimum(room, near.min(1))
                keep = room > least
                pool, room = pool[:, keep], room[keep]
            ok = room > need
            at = int(ok.argmax()) if len(room) else 0
        pos[k] = pool[:, at]
        d = pool - pos[k][:, None]
        d -= L * np.rint(d / L)
        room = np.minimum(room, np.sqrt(np.einsum("ci,ci->i", d, d)) - radii[k])
        if k % 8 == 7:
            keep = room > least
            pool, room = pool[:, keep], room[keep]
    return pos


def _single(case, seed):
    """Positions, radii and box of a case with one configuration."""
    rng = np.random.default_rng(seed)
    n = case["beads"]
    if case["kind"] == "sd":
        radii = np.full(n, 20.0)
        L = (n * 4.0 * math.pi * 20.0 ** 3 / 3.0 / 0.30) ** (1.0 / 3.0)
        return _place(rng, radii, L, gap=1.0), radii, L
    if n <= 64:  # identical beads at the density of the 64-bead workload
        radii, L = np.full(n, 20.0), 750.0 * (n / 64.0) ** (1.0 / 3.0)
    else:        # polydisperse, at the density of the 1024-bead workload
        radii, L = rng.uniform(10.0, 40.0, size=n), 1500.0 * (n / 1024.0) ** (1.0 / 3.0)
    return _place(rng, radii, L), radii, L


CHAIN, BOND, RADIUS, HARD, EPS = 16, 4.2, 2.0, 1.9, 0.2


def _polymer(case, seed):
    """Chains of 16 beads (radius 2, bonds of 4.2, angles of 150 degrees) at a volume fraction of 0.02."""
    rng = np.random.default_rng(seed)
    n = case["beads"]
    L = (n * 4.0 / 3.0 * math.pi * RADIUS ** 3 / 0.02) ** (1.0 / 3.0)
    turn = math.radians(30.0)
    placed = np.empty((0, 3))
    while len(placed) < n:
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        pts = [rng.uniform(-L / 2, L / 2, 3)]
        for k in range(CHAIN - 1):
            if k:
                w = rng.normal(size=3)
                w -= (w @ u) * u
                w /= np.linalg.norm(w)
                u = math.cos(turn) * u + math.sin(turn) * w
            pts.append(pts[-1] + BOND * u)
        pts = np.array(pts)
        d = pts[:, None, :] - np.concatenate([placed, pts])[None, :, :]
        d -= L * np.round(d / L)
        near = (d * d).sum(2) <= 4.5 ** 2
        own = np.abs(np.arange(CHAIN)[:, None] - np.arange(CHAIN)[None, :]) <= 1
        near[:, len(placed):] &= ~own
        if not near.any():
            placed = np.concatenate([placed, pts])
    return placed - L * np.round(placed / L), np.full(n, RADIUS), L


def _members(case, seed):
    """(positions, radii, box) of every replica of a batch."""
    rng = np.random.default_rng(seed)
    out = []
    sizes = np.random.default_rng(1)  # the batch's composition belongs to the case, its configurations to the seed
    for _ in range(case["replicas"]):
        if case["log"]:
            n = int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))))
            radii = rng.uniform(10.0, 40.0, size=n)
        else:
            n = int(sizes.integers(case["lo"], case["hi"] + 1))
            radii = rng.uniform(10.0, 30.0, size=n)
        L = float((np.sum(4.0 / 3.0 * np.pi * radii ** 3) / 0.05) ** (1.0 / 3.0))
        out.append((_place(rng, radii, L), radii, L))
    return out


def _input(case, L, seed):
    inp = {"box_length": L, "T": T, "viscosity": ETA, "seed": seed % (2 ** 32), "hydrodynamics": "rpy_smith",
           "ewald_alpha": ALPHA, "ewald_real": M_MAX, "ewald_imag": N_MAX, "propagation_scheme": "ermak",
           "immobile_labels": [], "check_overlaps": True, "overlap_treshold": 0.0, "max_move_attempts": 1000000,
           "external_force": [0.0, 0.0, 0.0], "energy_unit": "joule", "verbose": False, "debug": False,
           "precision": case.get("precision", "fp64"), "lennard_jones_6": False, "lennard_jones_12": False,
           "custom_interactions": False}
    if case["kind"] == "sd":
        inp.update({"hydrodynamics": "rpy_smith_lub", "lubrication_cutoff": 0.5, "cichocki_correction": True,
                    "propagation_scheme": "midpoint", "m_midpoint": 100.0})
    if case.get("polymer"):
        inp.update({"energy_unit": "kcal/mol", "lennard_jones_6": True, "lennard_jones_12": True,
                    "lennard_jones_alpha": 4.0})
    return inp


def _beads(case, pos, radii):
    from pybrown_b200.bead import Bead
    if not case.get("polymer"):
        return [Bead(p, a) for p, a in zip(pos, radii)]
    beads = [Bead(p, a, label="P", hard_core_radius=HARD, epsilon_LJ=EPS, bead_id=i + 1)
             for i, (p, a) in enumerate(zip(pos, radii))]
    for i, b in enumerate(beads):
        if i % CHAIN < CHAIN - 1:
            b.bonded_with.append(i + 2)
            b.bonded_how[i + 2] = [BOND, 5.0]
        if i % CHAIN < CHAIN - 2:
            b.angled_with.append([i + 2, i + 3])
            b.angled_how[(i + 2, i + 3)] = [150.0, 2.0]
    return beads


# ----------------------------------------------------------------------------- what a program has and calls

def _padded(n):
    return (3 * n + 63) // 64 * 64


def prepare(case, seed):
    from pybrown_b200 import _lib
    kind = case["kind"]
    if kind in ("bd", "sd"):
        from pybrown_b200.box import Box
        pos, radii, L = _polymer(case, seed) if case.get("polymer") else _single(case, seed)
        return {"kind": kind, "dt": case["dt"], "box": Box(_beads(case, pos, radii), _input(case, L, seed))}
    if kind == "batch":
        from pybrown_b200.batch import ReplicaBatch
        batch = ReplicaBatch(precision=case["precision"])
        members = _members(case, seed)
        slots = [batch.add(pos, radii, L, seed=seed * 4096 + k, noise="device")
                 for k, (pos, radii, L) in enumerate(members)]
        sizes = [len(radii) for _, radii, _ in members]
        frame = torch.empty((sum(sizes), 3), dtype=torch.float64, pin_memory=True)
        return {"kind": kind, "dt": case["dt"], "steps": case["steps"], "batch": batch, "slots": slots,
                "frame": frame, "parts": list(torch.split(frame, sizes))}
    prec = _lib.PREC[case["precision"]]
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    pos, radii, L = _single(case, seed)
    n, ld = case["beads"], _padded(case["beads"])
    state = {"kind": kind, "n": n, "ld": ld, "L": L, "prec": prec, "pos": torch.from_numpy(pos.reshape(-1)).cuda(),
             "radii": torch.from_numpy(radii).cuda(), "scale": KBT * 1e19 / ETA,
             "M": torch.zeros((ld, ld), dtype=dtype, device="cuda")}
    if kind != "tensor":
        # D from plain torch, so that this input does not depend on the framework's own tensor
        D = _diffusion(pos, radii, L)
        state["D"] = torch.zeros((ld, ld), dtype=dtype, device="cuda")
        state["D"][:3 * n, :3 * n] = D.to(dtype=dtype, device="cuda")
        state["info"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return state


def run(state):
    from pybrown_b200 import _lib
    kind = state["kind"]
    if kind in ("bd", "sd"):
        state["box"].propagate(state["dt"])
        return state["box"].positions()
    if kind == "batch":
        batch = state["batch"]
        for _ in range(state["steps"]):
            batch.propagate(state["dt"])
        for s, part in zip(state["slots"], state["parts"]):
            _lib.call("pbg_batch_get_positions_async", batch._h, s, part.data_ptr(), None)
        torch.cuda.current_stream().synchronize()
        return state["frame"]
    M, n3 = state["M"], 3 * state["n"]
    if kind == "tensor":
        _lib.call("pbg_dev_smith_matrix", state["pos"].data_ptr(), state["radii"].data_ptr(), state["n"], state["L"],
                  ALPHA, M_MAX, N_MAX, state["scale"], state["prec"], M.data_ptr(), state["ld"], None)
        return M[:n3, :n3]
    M.copy_(state["D"])
    if kind == "factor":
        _lib.call("pbg_dev_cholesky", M.data_ptr(), n3, state["ld"], state["prec"], state["info"].data_ptr(), None)
        # the factor is the lower triangle; what lies above it is not defined
        return {"L": torch.tril(M[:n3, :n3]), "info": state["info"]}
    _lib.call("pbg_dev_spd_inverse", M.data_ptr(), n3, state["ld"], state["info"].data_ptr(), None)
    return {"inverse": M[:n3, :n3], "info": state["info"]}


# Operations per pair of beads of the Ewald sums: the images' and the
# half-vectors' additions and products, special functions counted as one.
_PAIR = 25 * 45 + 64 * 12


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = np.random.default_rng(1)
        n = [int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"]))))) if case["log"]
             else int(sizes.integers(case["lo"], case["hi"] + 1)) for _ in range(case["replicas"])]
        # positions and radii in, positions out; D, B and the noise stay inside a step
        return {"bytes": case["steps"] * 56.0 * sum(n),
                "flops": case["steps"] * sum((3.0 * m) ** 3 / 3 + _PAIR * m * m / 2 + 18.0 * m * m for m in n)}
    m = case["beads"]
    order, es = 3.0 * m, 8.0 if case.get("precision", "fp64") == "fp64" else 4.0
    if kind == "bd":
        return {"bytes": 80.0 * m, "flops": order ** 3 / 3 + _PAIR * m * m / 2 + 18.0 * m * m}
    if kind == "sd":
        # twice the far-field inverse and the lubricated one, one factor, one triangular solve
        return {"bytes": 80.0 * m, "flops": 4 * order ** 3 + order ** 3 / 3 + 2 * _PAIR * m * m / 2}
    if kind == "tensor":
        return {"bytes": 32.0 * m + es * order ** 2, "flops": _PAIR * m * m / 2}
    if kind == "factor":
        return {"bytes": 2 * es * order ** 2, "flops": order ** 3 / 3}
    return {"bytes": 2 * es * order ** 2, "flops": order ** 3}


# ----------------------------------------------------------------------------- the same in 64 bits

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _outer6(x, y, z):
    return [x * x, y * y, z * z, x * y, x * z, y * z]


def _lattice(reach):
    r = range(-reach, reach + 1)
    return [(x, y, z) for x in r for y in r for z in r if abs(x) + abs(y) + abs(z) <= reach]


def _mobility(pos, radii, L):
    """Smith's Ewald sum of the RPY mobility (times viscosity), 3N x 3N, FP64."""
    pos = torch.as_tensor(pos, dtype=torch.float64).reshape(-1, 3).to(_dev())
    a = torch.as_tensor(radii, dtype=torch.float64).to(_dev())
    n = len(a)
    r = pos[:, None, :] - pos[None, :, :]
    r = r - L * torch.round(r / L)
    aa = a[:, None] ** 2 + a[None, :] ** 2
    cO, cQ = 1.0 / (8 * math.pi * L), aa / (24 * math.pi * L ** 3)
    s = r / L
    eye = torch.eye(n, dtype=torch.bool, device=pos.device)
    sx, sy, sz = (torch.where(eye, torch.full_like(s[..., c], 0.25), s[..., c]) for c in range(3))
    al, sp = ALPHA, math.sqrt(math.pi)
    comp, diag = [torch.zeros_like(sx) for _ in range(6)], torch.zeros_like(sx)
    for mx, my, mz in _lattice(M_MAX):
        x, y, z = sx + mx, sy + my, sz + mz
        l2 = x * x + y * y + z * z
        l = torch.sqrt(l2)
        ec, e = torch.erfc(al * l), torch.exp(-al * al * l2)
        W = ec + 2 / sp * al * l * e
        diag += cO * ec / l + cQ * W / l ** 3
        oc = (cO * (ec / l + 2 * al / sp * e) - cQ * (3 * W / l ** 3 + 4 * al ** 3 / sp * e)) / l2
        for c, v in enumerate(_outer6(x, y, z)):
            comp[c] += oc * v
    kk = math.pi ** 2 / al ** 2
    for nx, ny, nz in _lattice(N_MAX):
        nl2 = nx * nx + ny * ny + nz * nz
        if not nl2:
            continue
        cs = torch.cos(2 * math.pi * (nx * sx + ny * sy + nz * sz))
        P = 2 / math.pi / nl2 * math.exp(-kk * nl2)
        diag += cO * P * cs
        g = cs * (cQ * (4 * math.pi * math.exp(-kk * nl2) / nl2) - cO * P * (1 + kk * nl2) / nl2)
        for c, v in enumerate(_outer6(nx, ny, nz)):
            if v:
                comp[c] += g * v
    d2 = (r * r).sum(2)
    d = torch.sqrt(d2)
    rs = a[:, None] + a[None, :]
    over = (d < rs) & ~eye
    if bool(over.any()):
        # overlapping pairs: the far form of the pair term is exchanged for the near one
        i, j = torch.nonzero(over, as_tuple=True)
        ai, aj, dd, d2o = a[i], a[j], d[i, j], d2[i, j]
        f1, f2, f3 = 1 / (8 * math.pi * dd), 1 + aa[i, j] / (3 * d2o), (1 - aa[i, j] / d2o) / d2o
        c1 = 1 / (6 * math.pi * ai * aj)
        cd = (16 * dd ** 3 * (ai + aj) - ((ai - aj) ** 2 + 3 * d2o) ** 2) / 32 / dd ** 3
        co = 3 * ((ai - aj) ** 2 - d2o) ** 2 / (32 * dd ** 3) / d2o
        inside = dd <= (ai - aj).abs()
        c1 = torch.where(inside, 1 / (6 * math.pi * torch.maximum(ai, aj)), c1)
        cd, co = torch.where(inside, torch.ones_like(cd), cd), torch.where(inside, torch.zeros_like(co), co)
        for c, v in enumerate(_outer6(*(r[i, j, q] for q in range(3)))):
            comp[c][i, j] += (c1 * co - f1 * f3) * v
        diag[i, j] += c1 * cd - f1 * f2
    # self blocks
    O, Q = np.zeros(6), np.zeros(6)
    for m in _lattice(M_MAX):
        l2 = float(sum(v * v for v in m))
        if l2:
            l = math.sqrt(l2)
            ec, e, mm = math.erfc(al * l), math.exp(-al * al * l2), np.array(_outer6(*m), dtype=float)
            one = np.array([1.0, 1, 1, 0, 0, 0])
            O += ec * (one + mm / l2) / l + 2 * al / sp * e * mm / l2
            Q += (ec + 2 / sp * al * l * e) * (one - 3 * mm / l2) / l ** 3 - 4 * al ** 3 / sp * e * mm / l2
    for m in _lattice(N_MAX):
        l2 = float(sum(v * v for v in m))
        if l2:
            w, mm = math.exp(-kk * l2), np.array(_outer6(*m), dtype=float)
            O += 2 / math.pi / l2 * w * (np.array([1.0, 1, 1, 0, 0, 0]) - (1 / l2 + kk) * mm)
            Q += 4 * math.pi * w / l2 * mm
    c1 = 1 / (6 * math.pi * a)
    for c in range(6):
        o, q = float(O[c]), float(Q[c])
        own = 3 * a / (4 * L) * o + a ** 3 / (2 * L ** 3) * q
        if c < 3:
            own = 1 + own - 3 * a / (4 * L) * 1.5 * al * a / (sp * L) \
                - a ** 3 / (2 * L ** 3) * al ** 3 * a ** 3 / (L ** 3 * 3 * sp)
        comp[c][eye] = c1 * own
    diag[eye] = 0.0
    M = torch.empty((n, 3, n, 3), dtype=torch.float64, device=pos.device)
    for p, q, c in ((0, 0, 0), (1, 1, 1), (2, 2, 2), (0, 1, 3), (0, 2, 4), (1, 2, 5)):
        v = comp[c] + diag if p == q else comp[c]
        M[:, p, :, q] = v
        M[:, q, :, p] = v
    return M.reshape(3 * n, 3 * n)


def _diffusion(pos, radii, L):
    return _mobility(pos, radii, L) * (KBT * 1e19 / ETA)


# Jeffrey & Onishi's f_m polynomials by power of the size ratio (X and Y families).
_XF = [[1], [0, 3], [0, 9], [0, -4, 27, -4], [0, -24, 81, 36], [0, 0, 72, 243, 72], [0, 16, 108, 281, 648, 144],
       [0, 0, 288, 1620, 1515, 1620, 288], [0, 0, 576, 4848, 5409, 4524, 3888, 576],
       [0, 0, 1152, 9072, 14752, 26163, 14752, 9072, 1152],
       [0, 0, 2304, 20736, 42804, 115849, 76176, 39264, 20736, 2304],
       [0, 0, 4608, 46656, 108912, 269100, 319899, 269100, 108912, 46656, 4608]]
_YF = [[1], [0, 1.5], [0, 2.25], [0, 2, 3.375, 2], [0, 6, 5.0625, 18], [0, 0, 31.5, 7.59375, 31.5],
       [0, 4, 54, 19.390625, 81, 72], [0, 0, 144, 131.625, 149.0859375, 131.625, 144],
       [0, 0, 279, 532.625, 493.62890625, -14.625, 648, 288],
       [0, 0, 576, 1134, 1888.84375, 1496.443359375, 1888.84375, 1134, 576],
       [0, 0, 1152, 1964.25, 6155.4375, 10301.1650390625, 8452.125, -175.5, 3888, 1152],
       [0, 0, 2304, 7128, 11035.5, 21441.4453125, 46486.24755859375, 21441.4453125, 11035.5, 7128, 2304]]


def _jo_equal(s, X):
    """A11 and A12 (X or Y family) of two equal spheres at the scaled distance s, per 6 pi a."""
    l = 1.0
    if X:
        g1, g2, g3 = 2 / 8, 0.2 * 9 / 8, (1 + 18 - 29 + 18 + 1) / 42 / 8
    else:
        g1, g2, g3 = 0.0, 4 / 15 * 5 / 8, 2 / 375 * (16 - 45 + 58 - 45 + 16) / 8
    s2 = 1 - 4 / s ** 2
    a11 = g1 / s2 - g2 * np.log(s2) - g3 * s2 * np.log(s2) + 1 - g1
    lg = np.log((s + 2) / (s - 2))
    a12 = 2 / s * g1 / s2 + g2 * lg + g3 * s2 * lg + 4 * g3 / s
    for m in range(1, 12):
        f = float(sum((_XF if X else _YF)[m])) * l / 4.0 ** m
        m1 = -2 if m == 2 else m - 2
        term = (2 / s) ** m * (f - g1 - 2 / m * g2 + 4 / (m * m1) * g3)
        if m % 2:
            a12 = a12 + term
        elif m <= 10:
            a11 = a11 + term
    return a11, -a12


def _lubrication(pos, a, L, cutoff=0.5):
    """The Jeffrey-Onishi correction (with Cichocki's projection) of equal spheres of radius a, 3N x 3N."""
    n = len(pos)
    i, j = np.triu_indices(n, 1)
    r = pos[j] - pos[i]
    r -= L * np.round(r / L)
    d = np.sqrt((r * r).sum(1))
    near = (d - 2 * a) / (2 * a) <= cutoff
    i, j, r, d = i[near], j[near], r[near], d[near]
    C = np.zeros((n, 3, n, 3))
    e = r / d[:, None]
    ee = e[:, :, None] * e[:, None, :]
    one = np.eye(3)[None]
    far = np.where(d > 2 * a, 1.0, 0.0)
    assert far.all()  # the start configurations and their moves keep the beads apart
    c1 = 1 / (8 * math.pi * d)
    cT = c1 * (1 + 2 * a * a / (3 * d * d))
    cL = cT + c1 * (1 - 2 * a * a / (d * d))
    mob = 1 / (6 * math.pi * a)
    block = np.zeros((len(d), 3, 3))
    for X, proj in ((True, ee), (False, one - ee)):
        a11, a12 = _jo_equal(d / a, X)
        c = cL if X else cT
        det = mob * mob - c * c
        self_ = 6 * math.pi * a * a11 - mob / det
        cross = 6 * math.pi * a * a12 + c / det
        block += ((self_ - cross) / 2)[:, None, None] * proj
    np.add.at(C.transpose(0, 2, 1, 3), (i, i), block)
    np.add.at(C.transpose(0, 2, 1, 3), (j, j), block)
    np.add.at(C.transpose(0, 2, 1, 3), (i, j), -block)
    np.add.at(C.transpose(0, 2, 1, 3), (j, i), -block)
    return torch.from_numpy(C.reshape(3 * n, 3 * n)).to(_dev())


def _overlap(pos, radii, L, free=None):
    d = pos[:, None, :] - pos[None, :, :]
    d = d - L * torch.round(d / L)
    hit = torch.sqrt((d * d).sum(2)) <= radii[:, None] + radii[None, :]
    hit.fill_diagonal_(False)
    if free is not None:
        hit &= ~free
    return bool(hit.any())


def _wrapped(pos, L):
    return pos - L * torch.floor(pos / L + 0.5)


def _polymer_forces(pos, L):
    """Lennard-Jones, bond and angle forces of the chains in joules per angstrom."""
    n = len(pos)

    def image(v):
        return v - L * np.round(v / L)

    p = image(pos[None, :, :] - pos[:, None, :])  # p[a, b]: from a to b
    d2 = (p * p).sum(2)
    np.fill_diagonal(d2, 1.0)
    s6 = ((2 * HARD) ** 2 / d2) ** 3
    coef = 4.0 * EPS * (6 * s6 - 12 * s6 * s6) / d2
    np.fill_diagonal(coef, 0.0)
    F = (coef[:, :, None] * p).sum(1)
    for i in range(n):
        if i % CHAIN < CHAIN - 1:
            v = p[i, i + 1]
            d = math.sqrt(v @ v)
            f = v / d * 5.0 * (d - BOND)
            F[i] += f
            F[i + 1] -= f
        if i % CHAIN < CHAIN - 2:
            u, v = p[i, i + 1], p[i + 1, i + 2]
            du, dv = math.sqrt(u @ u), math.sqrt(v @ v)
            angle = math.acos(-(u @ v) / du / dv)
            c = 2.0 * (angle - math.radians(150.0)) / math.sin(angle)
            F[i] += c * (v / dv + math.cos(angle) * u / du) / du
            F[i + 1] += c * ((u - v) / du / dv - math.cos(angle) * (u / du ** 2 - v / dv ** 2))
            F[i + 2] += c * (-u / du / dv - math.cos(angle) * v / dv ** 2)
    return F * 6.9477e-21


def _philox(seed, first, count):
    """`count` normals from draw `first` (even) of the counter-based stream `seed`:
    Philox-4x32-10 by draw pair, two 53-bit uniforms, Box-Muller."""
    pairs = (count + 1) // 2
    ctr = np.arange(first // 2, first // 2 + pairs, dtype=np.uint64)
    lo = np.uint64(0xFFFFFFFF)
    c = [ctr & lo, ctr >> np.uint64(32), np.zeros_like(ctr), np.zeros_like(ctr)]
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & lo,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & lo]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u1, u2 = ((((c[2 * q] << np.uint64(32)) | c[2 * q + 1]) >> np.uint64(11)).astype(np.float64) for q in range(2))
    u1, u2 = (u1 + 0.5) / 2.0 ** 53, (u2 + 0.5) / 2.0 ** 53
    rad = np.sqrt(-2 * np.log(u1))
    return np.stack([rad * np.cos(2 * np.pi * u2), rad * np.sin(2 * np.pi * u2)], 1).reshape(-1)[:count]


def _exact_bd(case, seed):
    pos, radii, L = _polymer(case, seed) if case["polymer"] else _single(case, seed)
    rng = np.random.RandomState(seed % (2 ** 32))
    D = _diffusion(pos, radii, L)
    B = torch.linalg.cholesky(D)
    x, a, free = torch.from_numpy(pos).to(_dev()), torch.from_numpy(radii).to(_dev()), None
    if case["polymer"]:
        k = torch.arange(len(radii), device=_dev())
        free = ((k[:, None] - k[None, :]).abs() == 1) & (k[:, None] // CHAIN == k[None, :] // CHAIN)
        F = torch.from_numpy(_polymer_forces(pos, L).reshape(-1)).to(_dev())
        x = x + (case["dt"] / KBT * (D @ F)).reshape(-1, 3)
    while True:
        xi = torch.from_numpy(rng.normal(0.0, 1.0, 3 * len(radii))).to(_dev())
        y = x + (math.sqrt(2 * case["dt"]) * (B @ xi)).reshape(-1, 3)
        if not _overlap(y, a, L, free):
            return _wrapped(y, L).cpu().numpy()


def _exact_sd(case, seed):
    pos, radii, L = _single(case, seed)
    rng = np.random.RandomState(seed % (2 ** 32))
    m, dt, a = 100.0, case["dt"], torch.from_numpy(radii).to(_dev())

    def build(p):
        R = torch.linalg.inv(_mobility(p, radii, L) * (1e19 / ETA)) \
            + _lubrication(p.cpu().numpy(), 20.0, L) * (ETA / 1e19)
        return KBT * torch.linalg.inv(R)

    x = torch.from_numpy(pos).to(_dev())
    D = build(x)
    B = torch.linalg.cholesky(D)
    while True:
        xi = torch.from_numpy(rng.normal(0.0, 1.0, 3 * len(radii))).to(_dev())
        U = B @ xi
        half = x + (U * math.sqrt(2 * dt) / m).reshape(-1, 3)
        if _overlap(half, a, L):
            continue
        y = torch.linalg.solve_triangular(B.T, xi[:, None], upper=True)[:, 0]
        drift = m / 2 * math.sqrt(2 * dt) * (build(half) @ y - U)
        end = half + (U * math.sqrt(2 * dt) * (1 - 1 / m) + drift).reshape(-1, 3)
        if not _overlap(end, a, L):
            return _wrapped(end, L).cpu().numpy()


def _exact_batch(case, seed):
    out = []
    for k, (pos, radii, L) in enumerate(_members(case, seed)):
        x, a = torch.from_numpy(pos).to(_dev()), torch.from_numpy(radii).to(_dev())
        n3, at = 3 * len(radii), 0
        for _ in range(case["steps"]):
            B = torch.linalg.cholesky(_diffusion(x, radii, L))
            while True:
                xi = torch.from_numpy(_philox(seed * 4096 + k, at, n3)).to(_dev())
                at += n3 + n3 % 2
                y = x + (math.sqrt(2 * case["dt"]) * (B @ xi)).reshape(-1, 3)
                if not _overlap(y, a, L):
                    break
            x = _wrapped(y, L)
        out.append(x.cpu().numpy())
    return np.concatenate(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "bd":
        return _exact_bd(case, seed)
    if kind == "sd":
        return _exact_sd(case, seed)
    if kind == "batch":
        return _exact_batch(case, seed)
    D = _diffusion(*_single(case, seed))
    if kind == "tensor":
        return D
    if case["precision"] == "mixed":
        D = D.float().double()  # the call's input is the FP32 matrix
    if kind == "factor":
        return {"L": torch.linalg.cholesky(D), "info": None}
    return {"inverse": torch.linalg.inv(D), "info": None}
