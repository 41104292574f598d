"""The work this framework is used for, as a list of measurable cases.

A case is a dict of plain values.  ``prepare`` makes what a program holds
before the call (contexts, networks, device or pinned host buffers, inputs
from a seed), ``run`` is one pass through the public entry points, ``work``
counts what the pass cannot do without and ``exact`` computes the same
outputs in 64 bits with plain torch, independently of the library.

Kinds
  solve      dg_set_conserved_device, `steps` x compute_step, state and dts
             back: a simulation from an initial state to its next output
  noalloc    dg_compute_step_noalloc on caller-owned device memory: one step
             of a host program that owns its memory (the latency case)
  batch      many uneven grids in one dg_batch, states set from and read back
             to pinned host memory, `steps` steps between
  forward    inference of the correction network on a batch of feature boxes
  train      one training step of the network: crops, loss, gradients, Adam
  corrector  learned coarse steps (plain step, network, correction)
"""
import ctypes
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path.cwd()
sys.path.insert(0, str(ROOT / "deep-green_b200" / "python"))

from deepgreen import capi, learned, net as dgnet  # noqa: E402

PERIODIC, OUTFLOW, WALL = capi.PERIODIC, capi.OUTFLOW, capi.WALL
BOUNDARIES = {
    "periodic": (PERIODIC,) * 6,
    "outflow": (OUTFLOW,) * 6,
    "walls": (WALL,) * 6,
    "mixed": (WALL, WALL, PERIODIC, PERIODIC, OUTFLOW, OUTFLOW),
    "channel": (OUTFLOW, OUTFLOW, WALL, WALL, PERIODIC, PERIODIC),
}
ROUNDING = {"default": capi.ROUNDING_DEFAULT, "reference": capi.ROUNDING_REFERENCE, "fast": capi.ROUNDING_FAST}
GAMMA, CFL, GRAVITY = 1.4, 0.4, -0.1
FLOPS_PER_CELL = 450          # the step's arithmetic per cell (slopes, predictor, three faces, update, wave speed)
CROP = 64                     # target crop of a training entry
NET_IO, HIDDEN = dgnet.IO_CHANNELS, dgnet.HIDDEN


def listed():
    return [
        # the smallest call: one step of a small grid on a caller's memory, its dt read back (launch latency)
        {"name": "noalloc_48", "kind": "noalloc", "nx": 48, "ny": 48, "nz": 48, "bc": "outflow", "init": "riemann",
         "limiter": 1, "gravity": False, "precision": "f32", "rounding": "default"},
        # the 64^3 periodic shear layer, the size of parity and convergence runs
        {"name": "solve_kh64", "kind": "solve", "nx": 64, "ny": 64, "nz": 64, "bc": "periodic", "init": "kh",
         "limiter": 1, "gravity": False, "precision": "f32", "rounding": "default", "steps": 20},
        # the reference's rising-bubble configuration: walls, gravity, unlimited slopes
        {"name": "solve_bubble", "kind": "solve", "nx": 124, "ny": 124, "nz": 252, "bc": "walls", "init": "bubble",
         "limiter": 0, "gravity": True, "precision": "f32", "rounding": "default", "steps": 20},
        # an ordinary production size that no tile divides, three kinds of faces
        {"name": "solve_ragged", "kind": "solve", "nx": 253, "ny": 239, "nz": 261, "bc": "mixed", "init": "riemann",
         "limiter": 1, "gravity": False, "precision": "f32", "rounding": "default", "steps": 10},
        # the largest ordinary solve: the headline's 512^3 shock tube
        {"name": "solve_shock512", "kind": "solve", "nx": 512, "ny": 512, "nz": 512, "bc": "outflow", "init": "riemann",
         "limiter": 1, "gravity": False, "precision": "f32", "rounding": "default", "steps": 8},
        # DG_F64 as a user gets it by default: the reference's rounding, bit for bit
        {"name": "solve_f64_reference", "kind": "solve", "nx": 128, "ny": 128, "nz": 128, "bc": "periodic", "init": "kh",
         "limiter": 1, "gravity": False, "precision": "f64", "rounding": "default", "steps": 6},
        # FP64 with fused arithmetic, an odd size
        {"name": "solve_f64_fast", "kind": "solve", "nx": 150, "ny": 97, "nz": 131, "bc": "channel", "init": "riemann",
         "limiter": 1, "gravity": False, "precision": "f64", "rounding": "fast", "steps": 8},
        # FP32 in the reference's operation order: the reproducibility option
        {"name": "solve_f32_reference", "kind": "solve", "nx": 100, "ny": 84, "nz": 116, "bc": "walls", "init": "modes",
         "limiter": 0, "gravity": False, "precision": "f32", "rounding": "reference", "steps": 10},
        # many small uneven grids advanced together (ensemble runs)
        {"name": "batch_48", "kind": "batch", "grids": 48, "lo": 32, "hi": 160, "bc": "outflow", "limiter": 1,
         "reorient": True, "steps": 40},
        # inference at the corrector's production size
        {"name": "net_forward_264", "kind": "forward", "batch": 1, "x": 264, "y": 264, "z": 264},
        # one step of the training loop: 8 crops of 64^3
        {"name": "net_train_8", "kind": "train", "batch": 8, "n": 128},
        # the learned coarse solver's own step at its production size
        {"name": "corrector_256", "kind": "corrector", "n": 256, "steps": 2},
    ]


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.45:
        f64 = rng.random() < 0.35
        c = {"kind": "solve", "bc": rng.choice(sorted(BOUNDARIES)), "init": rng.choice(["kh", "riemann", "modes"]),
             "limiter": rng.randint(0, 1), "precision": "f64" if f64 else "f32",
             "rounding": rng.choice(["reference", "fast"]) if f64 else rng.choice(["default"] * 4 + ["reference"])}
        # unlimited slopes are for smooth flow
        if c["limiter"] == 0 and c["init"] == "riemann":
            c["init"] = "modes"
        c["gravity"] = c["bc"] == "walls" and rng.random() < 0.5
        # edges spread log-uniformly around a size drawn log-uniformly
        slow = f64 or c["rounding"] == "reference"
        mid = math.exp(rng.uniform(math.log(24), math.log(160 if slow else 330)))
        top = 220 if slow else 480
        for a in ("nx", "ny", "nz"):
            c[a] = min(top, max(16, _edge(rng, mid / 1.5, mid * 1.5)))
        cells = c["nx"] * c["ny"] * c["nz"]
        # a sharp shear layer amplifies rounding: few steps keep the outputs comparable
        c["steps"] = max(2, min(20 if c["init"] == "kh" else 40, int(3e7 / cells)))
        return c
    if pick < 0.6:
        c = {"kind": "noalloc", "bc": rng.choice(sorted(BOUNDARIES)), "init": rng.choice(["kh", "riemann"]), "limiter": 1,
             "gravity": False, "precision": rng.choice(["f32", "f32", "f64"]), "rounding": "default"}
        mid = math.exp(rng.uniform(math.log(20), math.log(120)))
        for a in ("nx", "ny", "nz"):
            c[a] = max(8, _edge(rng, mid / 1.4, mid * 1.4))
        c["nz"] = (c["nz"] + 3) // 4 * 4      # rows of whole 16-byte units, as the entry point asks
        return c
    if pick < 0.7:
        lo = _edge(rng, 16, 48)
        return {"kind": "batch", "grids": rng.randint(6, 40), "lo": lo, "hi": lo * rng.randint(2, 3),
                "bc": rng.choice(["outflow", "periodic", "mixed"]), "limiter": rng.randint(0, 1),
                "reorient": rng.random() < 0.5, "steps": rng.randint(10, 40)}
    if pick < 0.83:
        mid = math.exp(rng.uniform(math.log(28), math.log(190)))
        c = {"kind": "forward", "batch": rng.randint(1, 4)}
        for a in ("x", "y", "z"):
            c[a] = max(12, _edge(rng, mid / 1.3, mid * 1.3))
        return c
    if pick < 0.92:
        return {"kind": "train", "batch": rng.randint(1, 12), "n": rng.choice([72, 96, 128, 140])}
    return {"kind": "corrector", "n": 4 * rng.randint(12, 60), "steps": rng.randint(1, 4)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _dtype(case):
    return torch.float64 if case.get("precision") == "f64" else torch.float32


def _dev():
    return torch.device("cuda", 0)


def _primitives(init, shape, ds, seed, dev):
    """The five primitive fields on every ghosted cell, FP64."""
    r = random.Random(seed)
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    full = tuple(s + 4 for s in shape)
    ax = [(torch.arange(m, dtype=torch.float64, device=dev) - 1.5) * ds for m in full]
    x, y, z = ax[0].view(-1, 1, 1), ax[1].view(1, -1, 1), ax[2].view(1, 1, -1)
    span = [s * ds for s in shape]
    zero = torch.zeros(full, dtype=torch.float64, device=dev)
    if init == "riemann":
        # two constant states split by a seeded plane, with a little smooth structure
        s = [(math.exp(r.uniform(math.log(0.2), math.log(5))), [r.uniform(-0.8, 0.8) for _ in range(3)],
              math.exp(r.uniform(math.log(0.2), math.log(5)))) for _ in range(2)]
        nrm = [r.gauss(0, 1) for _ in range(3)]
        at = [r.uniform(0.3, 0.7) * w for w in span]
        side = ((x - at[0]) * nrm[0] + (y - at[1]) * nrm[1] + (z - at[2]) * nrm[2]) < 0
        ph = r.uniform(0, 6)
        soft = 1 + 0.05 * torch.sin(6 * x + 7 * y + 5 * z + ph)
        pick = lambda a, b: torch.where(side, a, b).to(torch.float64)  # noqa: E731
        return [pick(s[0][0], s[1][0]) * soft] + [pick(s[0][1][c], s[1][1][c]) + zero for c in range(3)] + [
            pick(s[0][2], s[1][2]) * soft]
    if init == "bubble":
        # near hydrostatic balance with a light bubble
        h = span[2] - z
        p = 2.5 + 0.1 * h + zero
        at = [w * r.uniform(0.4, 0.6) for w in span[:2]] + [span[2] * r.uniform(0.25, 0.4)]
        d2 = (x - at[0]) ** 2 + (y - at[1]) ** 2 + (z - at[2]) ** 2
        rho = 1.0 - 0.5 * torch.exp(-d2 / (0.15 * span[0]) ** 2)
        v = [1e-3 * (2 * torch.rand(full, generator=gen, dtype=torch.float64, device=dev) - 1) for _ in range(3)]
        return [rho] + v + [p]
    if init == "kh":
        ys = y / span[1]
        inner = ((ys - 0.5).abs() < 0.25).to(torch.float64)
        shear, ratio = r.uniform(0.3, 0.7), r.uniform(1.5, 3)
        rho = 1 + (ratio - 1) * inner + zero
        v = [shear * (2 * inner - 1) + zero,
             0.01 * torch.sin(4 * math.pi * x / span[0] + r.uniform(0, 6))
             * (torch.exp(-(ys - 0.25) ** 2 / 0.005) + torch.exp(-(ys - 0.75) ** 2 / 0.005)) + zero, zero.clone()]
        v = [c + 1e-3 * (2 * torch.rand(full, generator=gen, dtype=torch.float64, device=dev) - 1) for c in v]
        return [rho] + v + [2.5 + zero]
    # smooth periodic modes
    q = [1 + zero, zero.clone(), zero.clone(), zero.clone(), 1 + zero]
    for _ in range(4):
        k = [r.randint(-2, 2) for _ in range(3)]
        wave = torch.sin(sum(2 * math.pi * k[a] / span[a] * (x, y, z)[a] for a in range(3)) + r.uniform(0, 6))
        for f in range(5):
            q[f] += r.uniform(-0.06, 0.06) * wave
    return q


def _totals(q, ds):
    vol = ds ** 3
    rho, vx, vy, vz, p = q
    return torch.stack([rho * vol, rho * vx * vol, rho * vy * vol, rho * vz * vol,
                        vol * (0.5 * rho * (vx * vx + vy * vy + vz * vz) + p / (GAMMA - 1))])


def _initial_state(case, seed):
    """(5, nx+4, ny+4, nz+4) conserved totals in the case's precision, and ds."""
    shape = (case["nx"], case["ny"], case["nz"])
    ds = 1.0 / max(shape)
    return _totals(_primitives(case["init"], shape, ds, seed, _dev()), ds).to(_dtype(case)).contiguous(), ds


def _batch_shapes(case):
    r = random.Random(case["grids"] * 1000 + case["lo"])
    return [tuple(_edge(r, case["lo"], case["hi"]) for _ in range(3)) for _ in range(case["grids"])]


def _batch_prims(case, seed, i, shape):
    ds = 1.0 / max(shape)
    return torch.stack(_primitives("riemann" if case["limiter"] else "modes", shape, ds, seed * 131 + i, _dev())).float(), ds


def _net_weights(seed):
    """Seeded weights over real channels: [(w[co][ci][3][3][3], b[co])]."""
    rng = np.random.default_rng(seed)
    out = []
    for l in range(dgnet.LAYERS):
        co, ci = dgnet.layer_shape(l, learned.INPUTS, learned.OUTPUTS)
        bound = math.sqrt(6.0 / (27 * ci)) * (0.5 if l == dgnet.LAYERS - 1 else 1.0)
        out.append((rng.uniform(-bound, bound, (co, ci, 3, 3, 3)).astype(np.float32),
                    rng.uniform(-0.1, 0.1, co).astype(np.float32)))
    return out


def _make_net(seed):
    n = dgnet.Net(learned.INPUTS, learned.OUTPUTS)
    n.set_params(_net_weights(seed))
    return n


def _features_box(case, seed):
    gen = torch.Generator(device=_dev())
    gen.manual_seed(seed)
    f = torch.randn((case["batch"], case["x"], case["y"], case["z"], NET_IO), generator=gen, device=_dev(),
                    dtype=torch.bfloat16)
    f[..., learned.INPUTS:] = 0
    return f


def _norm(out_std):
    n = learned.Norm.identity()
    for c in range(learned.INPUTS, 16):
        n.in_inv_std[c] = 0.0
    for c in range(5):
        n.in_mean[c] = (1.0, 0.0, 0.0, 0.0, 2.5)[c]
        n.in_inv_std[5 + c] = 50.0      # the change over one step is small
        n.out_std[c] = out_std
    n.in_mean[13] = 1.0
    return n


def _train_packs(case, seed):
    """Two coarse states before / after a step and the truth, (2, 5, m, m, m) each."""
    n, ds = case["n"], 1.0 / case["n"]
    out = [[], [], []]
    for k in range(2):
        q = _primitives("modes", (n,) * 3, ds, seed * 7 + k, _dev())
        d = _primitives("modes", (n,) * 3, ds, seed * 7 + k + 3, _dev())
        t = _primitives("modes", (n,) * 3, ds, seed * 7 + k + 5, _dev())
        after = [a + 0.02 * (b - 1 if f in (0, 4) else b) for f, (a, b) in enumerate(zip(q, d))]
        truth = [a + 0.01 * (b - 1 if f in (0, 4) else b) for f, (a, b) in enumerate(zip(after, t))]
        for lst, p in zip(out, (q, after, truth)):
            lst.append(_totals(p, ds).float())
    return [torch.stack(v).contiguous() for v in out]


def _train_picks(case, seed):
    r = random.Random(seed)
    return [(r.randint(0, 1), [r.randrange(case["n"]) for _ in range(3)]) for _ in range(case["batch"])]


def _corrector_state(case, seed):
    n, ds = case["n"], 1.0 / case["n"]
    return _totals(_primitives("modes", (n,) * 3, ds, seed, _dev()), ds).float().contiguous(), ds


def _field_ptrs(t):
    return [t[f].data_ptr() for f in range(5)]


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        u0, ds = _initial_state(case, seed)
        torch.cuda.synchronize()
        ctx = capi.Context((case["nx"], case["ny"], case["nz"]), ds, BOUNDARIES[case["bc"]], gamma=GAMMA, cfl=CFL,
                           g=GRAVITY, gravity=case["gravity"], limiter=case["limiter"],
                           precision=capi.F64 if case["precision"] == "f64" else capi.F32,
                           rounding=ROUNDING[case["rounding"]])
        return {"case": case, "ctx": ctx, "u0": u0, "out": torch.empty_like(u0)}
    if kind == "noalloc":
        u0, ds = _initial_state(case, seed)
        info = capi.SimInfo()
        info.nx, info.ny, info.nz, info.nghosts = case["nx"], case["ny"], case["nz"], 2
        info.ds, info.gamma, info.cfl, info.g = ds, GAMMA, CFL, GRAVITY
        for f, b in enumerate(BOUNDARIES[case["bc"]]):
            info.bcs[f] = b
        info.gravity, info.limiter = int(case["gravity"]), case["limiter"]
        info.precision = capi.F64 if case["precision"] == "f64" else capi.F32
        info.device, info.rounding = 0, ROUNDING[case["rounding"]]
        return {"case": case, "lib": capi.load(), "info": info, "u0": u0, "out": torch.empty_like(u0)}
    if kind == "batch":
        shapes = _batch_shapes(case)
        bcs = BOUNDARIES[case["bc"]]
        specs, host_in, host_out = [], [], []
        for i, sh in enumerate(shapes):
            q, ds = _batch_prims(case, seed, i, sh)
            specs.append({"shape": sh, "ds": ds, "bcs": bcs, "limiter": case["limiter"], "gamma": GAMMA, "cfl": CFL})
            host_in.append(q.cpu().pin_memory())
            host_out.append(torch.empty(q.shape, dtype=torch.float32).pin_memory())
        return {"case": case, "batch": capi.Batch(specs, reorient=case["reorient"]), "in": host_in, "out": host_out,
                "fields": [[f.numpy() for f in t] for t in host_in]}
    if kind == "forward":
        feat = _features_box(case, seed)
        n, x, y, z = feat.shape[:4]
        return {"case": case, "net": _make_net(seed), "feat": feat,
                "out": torch.empty((n, x - 8, y - 8, z - 8, NET_IO), dtype=torch.float32, device=_dev())}
    if kind == "train":
        ext = CROP + 9
        packs = _train_packs(case, seed)
        feat = torch.zeros((case["batch"], ext, ext, ext, NET_IO), dtype=torch.bfloat16, device=_dev())
        tgt = torch.zeros((case["batch"], CROP, CROP, CROP, NET_IO), dtype=torch.float32, device=_dev())
        torch.cuda.synchronize()
        return {"case": case, "net": _make_net(seed), "norm": _norm(0.01), "packs": packs, "feat": feat, "tgt": tgt,
                "picks": _train_picks(case, seed)}
    u0, ds = _corrector_state(case, seed)
    torch.cuda.synchronize()
    ctx = learned.grid(case["n"])
    net = _make_net(seed)
    # a tolerance that no step of these states reaches: every step is corrected
    cor = learned.Corrector(ctx, net, _norm(1e-3), tolerance=1e-5)
    return {"case": case, "ctx": ctx, "net": net, "cor": cor, "u0": u0, "out": torch.empty_like(u0)}


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "solve":
        ctx = state["ctx"]
        ctx.set_conserved_device(_field_ptrs(state["u0"]))
        dts = ctx.compute_step(case["steps"])
        ctx.get_conserved_device(_field_ptrs(state["out"]))
        # dt is computed in the grid's precision
        return {"state": state["out"], "dts": dts.astype(ctx.dtype)}
    if kind == "noalloc":
        dt = ctypes.c_double()
        rc = state["lib"].dg_compute_step_noalloc(ctypes.byref(state["info"]), state["u0"].data_ptr(),
                                                  state["out"].data_ptr(), ctypes.byref(dt), None)
        if rc != capi.DG_OK:
            raise capi.DgError(rc, state["lib"].dg_last_error(None).decode())
        return {"state": state["out"], "dt": torch.tensor(dt.value, dtype=state["out"].dtype)}
    if kind == "batch":
        b = state["batch"]
        for i, q in enumerate(state["fields"]):
            b.set_primitives(i, q)
        b.step(case["steps"])
        for i, t in enumerate(state["out"]):
            b._check(b.lib.dg_batch_get_conserved(b.h, i, capi._PP5(*_field_ptrs(t))))
        return state["out"]
    if kind == "forward":
        return state["net"].forward(state["feat"], state["out"])
    if kind == "train":
        net, (before, after, truth) = state["net"], state["packs"]
        n, ext = case["n"], CROP + 9
        stream = net.stream()
        for i, (k, o) in enumerate(state["picks"]):
            learned.features(state["norm"], before[k].data_ptr(), after[k].data_ptr(), n, [c - 5 for c in o], ext,
                             state["feat"][i].data_ptr(), stream)
            learned.targets(state["norm"], after[k].data_ptr(), truth[k].data_ptr(), n, o, CROP,
                            state["tgt"][i].data_ptr(), stream)
        loss = net.forward_backward_flux(state["feat"], state["tgt"], True)
        net.adam_step(1e-5)
        grads = [t for l in range(dgnet.LAYERS) for t in net.get_grad(l)]
        # the divergence does not see the last bias: its gradient is zero but for rounding
        return {"loss": loss, "grads": grads[:-1]}
    state["ctx"].set_conserved_device(_field_ptrs(state["u0"]))
    state["cor"].step(case["steps"])
    state["ctx"].get_conserved_device(_field_ptrs(state["out"]))
    return state["out"]


def _net_flops(batch, x, y, z):
    total = 0.0
    for l in range(dgnet.LAYERS):
        co, ci = dgnet.layer_shape(l, learned.INPUTS, learned.OUTPUTS)
        k = 2 * (l + 1)
        total += 2.0 * 27 * co * ci * batch * (x - k) * (y - k) * (z - k)
    return total


def work(case):
    kind = case["kind"]
    if kind in ("solve", "noalloc"):
        elem = 8 if case["precision"] == "f64" else 4
        cells = case["nx"] * case["ny"] * case["nz"] * case.get("steps", 1)
        return {"bytes": cells * 10 * elem, "flops": cells * FLOPS_PER_CELL}
    if kind == "batch":
        shapes = _batch_shapes(case)
        cells = sum(a * b * c for a, b, c in shapes) * case["steps"]
        return {"bytes": cells * 40, "flops": cells * FLOPS_PER_CELL}
    if kind == "forward":
        n, x, y, z = case["batch"], case["x"], case["y"], case["z"]
        return {"bytes": n * (x * y * z * 32 + (x - 8) * (y - 8) * (z - 8) * 64), "flops": _net_flops(n, x, y, z)}
    if kind == "train":
        ext = CROP + 9
        # forward, input gradients of three layers, weight gradients of four
        co, ci = dgnet.layer_shape(0, learned.INPUTS, learned.OUTPUTS)
        first = 2.0 * 27 * co * ci * case["batch"] * (ext - 2) ** 3
        return {"bytes": case["batch"] * (ext ** 3 * 40 + CROP ** 3 * 40),
                "flops": 3 * _net_flops(case["batch"], ext, ext, ext) - first}
    n, s = case["n"], case["steps"]
    return {"bytes": s * n ** 3 * 40, "flops": s * (n ** 3 * FLOPS_PER_CELL + _net_flops(1, n + 8, n + 8, n + 8))}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits
# ---------------------------------------------------------------------------
def _at(axis, idx):
    s = [slice(None)] * 4
    s[axis + 1] = idx
    return tuple(s)


def _ghosts(q, bcs, mirror):
    """Ghost layers of a (fields, x, y, z) array, in place: wall mirrors (the
    normal vector component negated) when `mirror`, then copies."""
    if mirror:
        for face, bc in enumerate(bcs):
            ax, up = divmod(face, 2)
            m = q.shape[ax + 1]
            if bc == WALL:
                for dst, src in ((m - 2, m - 3), (m - 1, m - 4)) if up else ((1, 2), (0, 3)):
                    q[_at(ax, dst)] = q[_at(ax, src)]
                    q[1 + ax][_at(ax, dst)[1:]] *= -1
    for face, bc in enumerate(bcs):
        ax, up = divmod(face, 2)
        m = q.shape[ax + 1]
        if bc == OUTFLOW:
            for dst in (m - 2, m - 1) if up else (0, 1):
                q[_at(ax, dst)] = q[_at(ax, m - 3 if up else 2)]
        elif bc == PERIODIC:
            for dst, src in ((m - 2, 2), (m - 1, 3)) if up else ((0, m - 4), (1, m - 3)):
                q[_at(ax, dst)] = q[_at(ax, src)]


def _step64(u, ds, bcs, limiter, gravity):
    """One MUSCL-Hancock / Rusanov step of the conserved totals u (5, x, y, z),
    FP64, with the reference's ghost rules for slopes, predictions and fluxes."""
    vol, gm1 = ds ** 3, GAMMA - 1
    rho = u[0] / vol
    v = u[1:4] / u[0]
    w = torch.cat([rho[None], v, ((u[4] / vol - 0.5 * rho * (v * v).sum(0)) * gm1)[None]])
    del rho, v
    _ghosts(w, bcs, True)
    dt = CFL * float((ds / ((GAMMA * w[4] / w[0]).sqrt() + (w[1:4] ** 2).sum(0).sqrt())).min())
    grads = []
    for ax in range(3):
        m = w.shape[ax + 1]
        lo, mid, hi = (_at(ax, slice(k, m - 2 + k)) for k in range(3))
        g = torch.zeros_like(w)
        if limiter:
            a, b = (w[mid] - w[lo]) / ds, (w[hi] - w[mid]) / ds
            g[mid] = torch.where(a * b > 0, torch.where(a.abs() < b.abs(), a, b), torch.zeros_like(a))
            del a, b
        else:
            g[mid] = (w[hi] - w[lo]) / (2 * ds)
        # the outermost layer of the other axes keeps slope zero
        for other in range(3):
            if other != ax:
                g[_at(other, 0)] = 0
                g[_at(other, -1)] = 0
        _ghosts(g, bcs, False)
        grads.append(g)
    h = 0.5 * dt
    xt = w.clone()
    div = grads[0][1] + grads[1][2] + grads[2][3]
    for ax in range(3):
        xt -= h * w[1 + ax] * grads[ax]
        xt[1 + ax] -= h * grads[ax][4] / w[0]
    xt[0] -= h * w[0] * div
    xt[4] -= h * GAMMA * w[4] * div
    del div, w
    _ghosts(xt, bcs, True)
    new = u.clone()
    for ax in range(3):
        n, t1, t2 = 1 + ax, 1 + (ax + 1) % 3, 1 + (ax + 2) % 3
        m = xt.shape[ax + 1]
        lower, upper = _at(ax, slice(1, m - 2)), _at(ax, slice(2, m - 1))    # faces 1 | 2 .. m-3 | m-2
        left = xt[lower] + grads[ax][lower] * (ds / 2)
        right = xt[upper] - grads[ax][upper] * (ds / 2)

        def cons(s):
            e = 0.5 * s[0] * (s[1] ** 2 + s[2] ** 2 + s[3] ** 2) + s[4] / gm1
            return torch.stack([s[0], s[0] * s[1], s[0] * s[2], s[0] * s[3], e])

        cl, cr = cons(left), cons(right)
        c = torch.maximum((GAMMA * left[4] / left[0]).sqrt() + left[n].abs(),
                          (GAMMA * right[4] / right[0]).sqrt() + right[n].abs())
        star = 0.5 * (cl + cr)
        p = gm1 * (star[4] - 0.5 * (star[1] ** 2 + star[2] ** 2 + star[3] ** 2) / star[0])
        vel = star[n] / star[0]
        f = star * vel
        f[n] += p
        f[4] += p * vel
        if gravity and ax == 2:
            k = torch.arange(1, m - 2, dtype=torch.float64, device=u.device).view(1, 1, -1)
            height = (m - 4) * ds - (k - 2) * ds
            f[3] += star[0] * GRAVITY * height
            f[4] += 0.5 * star[0] * (left[3] + right[3]) * GRAVITY * height
        f -= 0.5 * c * (cr - cl)
        del left, right, cl, cr, c, star, p, vel
        # flux of face k | k+1 stored at k, its ghost rules, then the balance
        flux = torch.zeros_like(xt)
        flux[lower] = f
        del f
        for face in (2 * ax, 2 * ax + 1):
            if bcs[face] == OUTFLOW and face == 2 * ax:
                flux[_at(ax, 1)] = flux[_at(ax, 2)]
            elif bcs[face] == PERIODIC and face == 2 * ax:
                flux[_at(ax, 1)] = flux[_at(ax, m - 3)]
        inner, below = _at(ax, slice(2, m - 2)), _at(ax, slice(1, m - 3))
        new[inner] -= dt * ds * ds * (flux[inner] - flux[below])
        del flux
    _ghosts(new, bcs, True)
    return new, dt


def _solve64(u, ds, bcs, limiter, gravity, steps):
    dts = []
    u = u.double()
    for _ in range(steps):
        u, dt = _step64(u, ds, bcs, limiter, gravity)
        dts.append(dt)
    return u, torch.tensor(dts, dtype=torch.float64)


def _conv64(a, w, b):
    """Valid 3x3x3 convolution of channels-last FP64 a with w[co][ci][3][3][3]."""
    x, y, z = (a.shape[1] - 2, a.shape[2] - 2, a.shape[3] - 2)
    out = b.expand(a.shape[0], x, y, z, b.shape[0]).clone()
    for i in range(3):
        for j in range(3):
            for k in range(3):
                out += a[:, i:i + x, j:j + y, k:k + z] @ w[:, :, i, j, k].t()
    return out


def _gelu64(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _forward64(feat, params):
    a = feat[..., :learned.INPUTS].double()
    for l, (w, b) in enumerate(params):
        a = _conv64(a, w, b)
        if l < dgnet.LAYERS - 1:
            a = _gelu64(a)
    return a


def _params64(seed, grad=False):
    return [tuple(torch.from_numpy(t).to(_dev()).double().requires_grad_(grad) for t in wb) for wb in _net_weights(seed)]


def _features64(norm, before, after, ds):
    """Normalised channels of densities before and after, (x, y, z, INPUTS)."""
    u0, u1 = before.double() / ds ** 3, after.double() / ds ** 3
    v = u1[1:4] / u1[0]
    p = (GAMMA - 1) * (u1[4] - 0.5 * u1[0] * (v * v).sum(0))
    f = torch.cat([u1, u1 - u0, v, p[None]]).permute(1, 2, 3, 0)
    mean = torch.tensor(list(norm.in_mean)[:learned.INPUTS], dtype=torch.float64, device=f.device)
    inv = torch.tensor(list(norm.in_inv_std)[:learned.INPUTS], dtype=torch.float64, device=f.device)
    return (f - mean) * inv


def _exact_train(case, seed):
    n, ds, ext = case["n"], 1.0 / case["n"], CROP + 9
    norm, params = _norm(0.01), _params64(seed, grad=True)
    before, after, truth = _train_packs(case, seed)
    std = torch.tensor(list(norm.out_std)[:5], dtype=torch.float64, device=_dev())
    feats, tgts = [], []
    for k, o in _train_picks(case, seed):
        wrap = lambda off, m: [(torch.arange(m, device=_dev()) + o[a] + off) % n + 2 for a in range(3)]  # noqa: E731
        i, j, l = wrap(-5, ext)
        box = lambda t: t[k][:, i[:, None, None], j[None, :, None], l[None, None, :]]  # noqa: E731
        feats.append(_features64(norm, box(before), box(after), ds))
        i, j, l = wrap(0, CROP)
        tgts.append(((box(truth).double() - box(after).double()) / ds ** 3).permute(1, 2, 3, 0) / std)
    power = torch.stack([(t ** 2).mean() for t in tgts])
    weight = power.mean() / (power + 0.01 * power.mean())
    total, count = 0.0, case["batch"] * CROP ** 3 * 5
    for f, t, wb in zip(feats, tgts, weight):
        o = _forward64(f[None], params)[0]
        up = o[1:, 1:, 1:]
        low = (o[:-1, 1:, 1:], o[1:, :-1, 1:], o[1:, 1:, :-1])
        du = sum(up[..., 5 * d:5 * d + 5] - low[d][..., 5 * d:5 * d + 5] for d in range(3))
        loss = wb * ((du - t) ** 2).sum() / count
        loss.backward()
        total += float(loss.detach())
        del o, du, loss
    return {"loss": total, "grads": [t.grad for wb in params for t in wb][:-1]}


def _exact_corrector(case, seed):
    n = case["n"]
    norm, params = _norm(1e-3), _params64(seed)
    u, ds = _corrector_state(case, seed)
    u = u.double()
    std = torch.tensor(list(norm.out_std)[:5], dtype=torch.float64, device=_dev()).view(5, 1, 1, 1)
    c = (slice(None),) + (slice(2, -2),) * 3
    for _ in range(case["steps"]):
        new, _ = _step64(u, ds, BOUNDARIES["periodic"], 1, False)
        f = _features64(norm, u[c], new[c], ds)
        for a in range(3):
            i = (torch.arange(n + 8, device=_dev()) - 4) % n
            f = f.index_select(a, i)
        o = _forward64(f[None], params)[0].permute(3, 0, 1, 2)
        d = sum(o[5 * a:5 * a + 5] - torch.roll(o[5 * a:5 * a + 5], 1, dims=a + 1) for a in range(3)) * std * ds ** 3
        new[c] += d - d.mean(dim=(1, 2, 3), keepdim=True)
        _ghosts(new, BOUNDARIES["periodic"], True)
        u = new
    return u


@torch.no_grad()
def _exact_plain(case, seed):
    kind = case["kind"]
    if kind in ("solve", "noalloc"):
        u0, ds = _initial_state(case, seed)
        u, dts = _solve64(u0, ds, BOUNDARIES[case["bc"]], case["limiter"], case["gravity"], case.get("steps", 1))
        return {"state": u, "dts": dts} if kind == "solve" else {"state": u, "dt": dts[0]}
    if kind == "batch":
        out = []
        for i, sh in enumerate(_batch_shapes(case)):
            q, ds = _batch_prims(case, seed, i, sh)
            out.append(_solve64(_totals(q.double(), ds), ds, BOUNDARIES[case["bc"]], case["limiter"], False,
                                case["steps"])[0].cpu())
        return out
    if kind == "forward":
        o = _forward64(_features_box(case, seed), _params64(seed))
        return torch.nn.functional.pad(o, (0, NET_IO - learned.OUTPUTS))
    return _exact_corrector(case, seed)


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return _exact_plain(case, seed)
