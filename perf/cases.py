"""Performance cases: the calls a user of gell_b200 makes, at the sizes they are made at.

Each case goes through the public entry points (gell_b200.Simulation, gell_b200.Ensemble and, for
device-resident fields, gell_field_import / gell_field_export of include/gell.h) and returns what the
call computes: cell records, substrate fields, gradients.  The inputs are synthetic tumours with the
statistics of the repository's own workloads (bench.py): jittered-lattice spheroids at volume
fraction 0.6, radii N(5, 0.5) um, 10 um voxels, oxygen and a drug, seeded Ki-67 states.

Families of cases (`kind`):
  step       one mechanics step: FM_update, PreLOD, the LOD substeps (the host loop's inner call)
  run        several mechanics steps in one call (run_mechanics: replayed from a captured graph)
  diffusion  PreLOD and the LOD substeps alone (cells that do not move between two blocks)
  mechanics  FM_update alone (growth without diffusion)
  biology    one biology step on imported records: birth, death, export
  ensemble   run_mechanics of many small tumours side by side (parameter sweeps)
  surrogate  the learned oxygen operator on a new field
  train      one training pair of that operator
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import gell_b200 as gb
from gell_b200 import surrogate as gs

VOXEL = 10.0  # um
RADIUS_COEF = 0.23873241
SPLIT = (1871.0 / 2495.0, 135.0 / 2495.0, 489.0 / 2495.0)  # Vf, Vns, Vcs

_stream = None


def stream():
    """The stream every context of this program works on, one call after the other."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


# ---------------------------------------------------------------------------------------- the cases


def listed():
    return [
        # the smallest grid the repository's own tests step: a call bound by launches
        {"name": "step 32", "kind": "step", "N": 32, "cells": 2000, "subs": 1, "substeps": 10},
        # the small plain workload (100^3, 10^4 cells), driven the way a host loop runs it between biology steps
        {"name": "run 100", "kind": "run", "N": 100, "cells": 10000, "subs": 1, "substeps": 10, "steps": 6},
        # the headline workload: one whole mechanics step, oxygen and drug
        {"name": "step 400 x2", "kind": "step", "N": 400, "cells": 1000000, "subs": 2, "substeps": 10},
        # an odd edge (rows padded, ragged last groups), two substrates
        {"name": "diffusion 131 x2", "kind": "diffusion", "N": 131, "cells": 60000, "subs": 2, "substeps": 10},
        # the block the learned operator stands in for: 50 plain substeps of oxygen
        {"name": "diffusion 256", "kind": "diffusion", "N": 256, "cells": 300000, "subs": 1, "substeps": 50},
        # the largest grid of the repository's workloads (birth and death at 600^3, 5*10^6 cells)
        {"name": "diffusion 600 x2", "kind": "diffusion", "N": 600, "cells": 5000000, "subs": 2, "substeps": 10},
        # cell mechanics of the headline workload
        {"name": "mechanics 1M", "kind": "mechanics", "N": 400, "cells": 1000000},
        # one biology step of a large tumour, counter-based draws
        {"name": "biology 1M", "kind": "biology", "N": 160, "cells": 1000000, "rng": "philox"},
        # one biology step with the default draws (the reference's generator) on the default-sized grid
        {"name": "biology 50k", "kind": "biology", "N": 100, "cells": 50000, "rng": "xorwow"},
        # a parameter sweep: tumours of different sizes, two steps per call
        {"name": "ensemble 24", "kind": "ensemble", "members": 24, "lo": 64, "hi": 160, "substeps": 10, "steps": 2},
        # the packaged operator on the grid it was trained for
        {"name": "surrogate 256", "kind": "surrogate", "N": 256, "cells": 300000},
        # one pair of a fit, gradient returned
        {"name": "train 96", "kind": "train", "N": 96, "cells": 40000, "substeps": 50},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "run", "diffusion", "diffusion", "mechanics", "biology", "ensemble", "surrogate", "train"])
    fill = lambda N, top: max(500, min(top, _log(rng, 0.002 * N ** 3, 0.25 * N ** 3)))  # noqa: E731
    if kind == "step":
        N = _log(rng, 24, 400)
        return {"kind": kind, "N": N, "cells": fill(N, 1000000), "subs": rng.choice([1, 2]), "substeps": 10}
    if kind == "run":
        N = _log(rng, 32, 200)
        return {"kind": kind, "N": N, "cells": fill(N, 300000), "subs": rng.choice([1, 2]), "substeps": 10, "steps": rng.choice([2, 4, 6])}
    if kind == "diffusion":
        N = _log(rng, 32, 600)
        return {"kind": kind, "N": N, "cells": fill(N, 5000000), "subs": rng.choice([1, 2]), "substeps": 10 if N > 256 else rng.choice([1, 10, 50])}
    if kind == "mechanics":
        n = _log(rng, 2000, 2000000)
        return {"kind": kind, "N": max(40, int(1.6 * n ** (1 / 3)) + rng.randrange(1, 60)), "cells": n}
    if kind == "biology":
        n = _log(rng, 2000, 2000000)
        return {"kind": kind, "N": max(32, int(1.6 * n ** (1 / 3)) + rng.randrange(1, 30)), "cells": n, "rng": rng.choice(["philox", "xorwow"])}
    if kind == "ensemble":
        lo = rng.randrange(24, 100)
        return {"kind": kind, "members": rng.randrange(4, 33), "lo": lo, "hi": lo + rng.randrange(1, 60), "substeps": 10, "steps": 2}
    if kind == "surrogate":
        N = _log(rng, 40, 256)
        return {"kind": kind, "N": N, "cells": fill(N, 300000)}
    N = _log(rng, 32, 128)
    return {"kind": kind, "N": N, "cells": fill(N, 40000), "substeps": rng.choice([10, 50])}


# ---------------------------------------------------------------------------------------- the inputs


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def make_cells(n, N, seed):
    """n cells on a jittered cubic lattice around the grid's centre, as [n, 18] float32 words of the
    72-byte record, in a random order (cells of a running model are in no particular order)."""
    g = _gen(2 * seed + 1)
    dev = torch.device("cuda")
    a = (4.0 / 3.0 * math.pi * 125.0 / 0.6) ** (1.0 / 3.0)
    m = int(math.ceil((3.0 * n / (4.0 * math.pi)) ** (1.0 / 3.0))) + 2
    ax = torch.arange(-m, m + 1, device=dev, dtype=torch.float64)
    d2 = (ax[:, None, None] ** 2 + ax[None, :, None] ** 2 + ax[None, None, :] ** 2).reshape(-1)
    site = torch.argsort(d2, stable=True)[:n]
    site = site[torch.randperm(n, generator=g, device=dev)]
    w = 2 * m + 1
    pts = torch.stack([site // (w * w), (site // w) % w, site % w], 1).to(torch.float64) - m
    pts = pts * a + (torch.rand((n, 3), generator=g, device=dev, dtype=torch.float64) - 0.5) * (0.2 * a) + N * VOXEL / 2
    r = (5.0 + 0.5 * torch.randn(n, generator=g, device=dev)).clamp(4.0, 6.0)
    V = (r.double() ** 3 / RADIUS_COEF).float()
    # Ki-67 states of a growing tumour (cells.seed_ki67_states)
    u = torch.rand(n, generator=g, device=dev)
    ph = torch.bucketize(u, torch.tensor([0.60, 0.75, 0.85, 0.90, 0.95], device=dev), right=True).to(torch.int32)
    t = torch.rand(n, generator=g, device=dev)
    clock = torch.where(ph == 1, t * 780.0, torch.where(ph == 2, t * 150.0, torch.zeros_like(t)))
    vcs = V * SPLIT[2]
    vcs = torch.where((ph >= 3) & (t < 1.0 / 3.0), torch.full_like(vcs, 20.0), vcs)
    rec = torch.zeros((n, 18), device=dev, dtype=torch.float32)
    whole = rec.view(torch.int32)
    whole[:, 0] = 1
    rec[:, 2:5] = pts.float()
    ijk = (rec[:, 2:5] / VOXEL).to(torch.int32)
    whole[:, 1] = ijk[:, 0] + ijk[:, 1] * N + ijk[:, 2] * (N * N)
    rec[:, 11], rec[:, 12], rec[:, 13], rec[:, 14], rec[:, 15] = r, V, V * SPLIT[0], vcs, V * SPLIT[1]
    whole[:, 16] = ph
    rec[:, 17] = clock
    return rec


def make_field(n, N, b, seed):
    """A substrate around a tumour of n cells: depleted in the core, the boundary value far out."""
    dev = torch.device("cuda")
    R = 5.93 * n ** (1.0 / 3.0) + VOXEL
    x = (torch.arange(N, device=dev, dtype=torch.float32) + 0.5) * VOXEL - N * VOXEL / 2
    p = (x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2).neg_().div_(R * R).exp_()
    p = p.mul_(-0.9).add_(1.0).mul_(b)
    p.mul_(torch.rand(p.shape, generator=_gen(2 * seed + 2), device=dev).mul_(2e-3).add_(0.999))
    return p.reshape(-1).contiguous()


def _bytes(rec):
    return rec.view(torch.uint8).reshape(-1)


def _substrates(case):
    return [gb.oxygen(), gb.drug()][: case.get("subs", 1)]


def _field_in(sim, s, t):
    sim._check(sim.lib.gell_field_import(sim.h, s, ctypes.c_void_p(t.data_ptr()), 1), "gell_field_import")


def _field_out(sim, s, t):
    sim._check(sim.lib.gell_field_export(sim.h, s, ctypes.c_void_p(t.data_ptr()), 1), "gell_field_export")


def _sim(case, seed, N, n, subs, cap=None, **params):
    """A context with the cells and fields of one tumour, and device buffers for what is read back."""
    sim = gb.Simulation(voxel_num=N, voxel_length=VOXEL, max_cell_num=cap or n, **params)
    sim.set_stream(stream())
    rec = make_cells(n, N, seed)
    fields = []
    for k, s in enumerate(subs):
        sim.add_substrate(s)
        fields.append(make_field(n, N, s.boundary, 16 * seed + k))
    torch.cuda.synchronize()  # the records and fields come from torch's stream
    sim.import_cells(_bytes(rec), on_device=True)
    for k, f in enumerate(fields):
        _field_in(sim, k, f)
    sim.sync()
    return sim, rec, fields


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        sims, cells, fields, N3, n3 = [], [], [], 0, 0
        rng = np.random.Generator(np.random.Philox(seed))
        for k, (N, n) in enumerate(_members(case)):
            s = gb.Substrate(boundary=38.0, diffusion=float(np.float32(rng.uniform(5e4, 2e5))), decay=0.1,
                             uptake=float(np.float32(-rng.uniform(5, 20))), init=38.0)
            sims.append(_sim(case, 64 * seed + k, N, n, [s], rng_mode=gb.GELL_RNG_PHILOX)[0])
            cells.append((n3, n3 + n))
            fields.append((N3, N3 + N ** 3))
            n3 += n
            N3 += N ** 3
        ens = gb.Ensemble(sims)
        ens.set_batched(True)
        return {"case": case, "ens": ens, "sims": sims, "cells": cells, "fields": fields,
                "rec": torch.zeros((n3, 18), device="cuda"), "out": torch.zeros(N3, device="cuda")}
    N, n = case["N"], case["cells"]
    st = {"case": case}
    if kind == "biology":
        mode = gb.GELL_RNG_PHILOX if case["rng"] == "philox" else gb.GELL_RNG_XORWOW
        st["sim"], st["cells"], _ = _sim(case, seed, N, n, [gb.oxygen()], cap=n + n // 4 + 1024, rng_mode=mode)
        st["rec"] = torch.zeros((n + n // 4 + 1024, 18), device="cuda")
    elif kind in ("surrogate", "train"):
        st["sim"], _, f = _sim(case, seed, N, n, [gb.oxygen()], rng_mode=gb.GELL_RNG_PHILOX)
        st["field"] = f[0]
        w = gs.load_weights(gs.DEFAULT_WEIGHTS)
        if kind == "surrogate":
            st["sim"].surrogate_load(0, w.weights, w.substeps, w.rate_scale, w.threshold, w.input_kind)
        else:
            st["sim"].surrogate_train_init(0, w.weights, case["substeps"], w.rate_scale, w.input_kind)
        st["sim"].PreLOD()
        st["out"] = [torch.zeros(N ** 3, device="cuda")]
    else:
        subs = [] if kind == "mechanics" else _substrates(case)
        st["sim"], _, _ = _sim(case, seed, N, n, subs, rng_mode=gb.GELL_RNG_PHILOX)
        st["rec"] = torch.zeros((n, 18), device="cuda")
        st["out"] = [torch.zeros(N ** 3, device="cuda") for _ in subs]
    st["sim"].sync()
    return st


def _members(case):
    """(N, cells) of an ensemble's members: edges and fillings spread evenly over their ranges."""
    k = case["members"]
    out = []
    for i in range(k):
        N = int(round(case["lo"] * (case["hi"] / case["lo"]) ** (i / max(1, k - 1))))
        out.append((N, int(0.25 * N ** 3 * 0.02 ** (((5 * i) % k) / k))))
    return out


# ---------------------------------------------------------------------------------------- one pass


def _records(rec):
    """The 72-byte records by field: whole numbers and floats."""
    whole = rec.view(torch.int32)
    return {"sign_mesh": whole[:, 0:2], "pos": rec[:, 2:5], "force": rec[:, 5:8], "oldforce": rec[:, 8:11],
            "volumes": rec[:, 11:16], "phase": whole[:, 16:17], "clock": rec[:, 17:18]}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "ensemble":
        st["ens"].run_mechanics(case["steps"], case["substeps"])
        for sim, (a, b), (p, q) in zip(st["sims"], st["cells"], st["fields"]):
            sim.export_cells_device(_bytes(st["rec"][a:b]))
            _field_out(sim, 0, st["out"][p:q])
        return {**_records(st["rec"]), "fields": st["out"]}
    sim = st["sim"]
    if kind == "biology":
        sim.import_cells(_bytes(st["cells"]), on_device=True)
        sim.CellBirth_kernel()
        n = sim.CellDeath_kernel()
        sim.export_cells_device(_bytes(st["rec"][:n]))
        return {"count": n, **_records(st["rec"])}  # records past the count stay as they were
    if kind in ("surrogate", "train"):
        _field_in(sim, 0, st["field"])
        if kind == "surrogate":
            sim.surrogate_infer(0)
            _field_out(sim, 0, st["out"][0])
            return {"field": st["out"][0]}
        loss = sim.surrogate_train_pair(0, 1e-5)
        grad = sim.surrogate_train_read(0, 1)
        _field_out(sim, 0, st["out"][0])
        return {"loss": loss, "gradient": grad, "target": st["out"][0]}
    if kind == "step":
        sim.mechanics_step(case["substeps"])
    elif kind == "run":
        sim.run_mechanics(case["steps"], case["substeps"])
    elif kind == "mechanics":
        sim.FM_update()
    else:
        sim.PreLOD()
        sim.LODsolver(case["substeps"])
    out = {}
    if kind != "diffusion":
        sim.export_cells_device(_bytes(st["rec"]))
        out.update(_records(st["rec"]))
    for s, t in enumerate(st["out"]):
        _field_out(sim, s, t)
        out["field%d" % s] = t
    return out


# ---------------------------------------------------------------------------------------- what a pass cannot do without


def work(case):
    kind = case["kind"]
    fm = lambda n: (n * (72 + 72), n * 31 * 12)  # noqa: E731  (records in and out; about 31 candidates a cell)
    lod = lambda v, k: (v * 12, v * 17 * k)  # noqa: E731  (field in and out, uptake map in; 17 operations a voxel and substep)
    parts = []
    if kind == "ensemble":
        for N, n in _members(case):
            parts += [fm(n)] + [(0, n * 31 * 12)] * (case["steps"] - 1) + [lod(N ** 3, case["substeps"] * case["steps"])]
    elif kind == "biology":
        parts = [(case["cells"] * 144, case["cells"] * 100)]
    elif kind in ("surrogate", "train"):
        v = case["N"] ** 3
        macs = 27 * (3 * 32 + 8 * 32 * 32 + 32)
        parts = [(v * 12, 2.0 * macs * v * (3 if kind == "train" else 1))]
        if kind == "train":
            parts.append((0, v * 17 * case["substeps"]))
    else:
        v = case["N"] ** 3 * case.get("subs", 0)
        if kind != "diffusion":
            parts.append(fm(case["cells"]))
            parts += [(0, case["cells"] * 31 * 12)] * (case.get("steps", 1) - 1)
        if v:
            parts.append(lod(v, case["substeps"] * case.get("steps", 1)))
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


# ---------------------------------------------------------------------------------------- the same in 64 bits

_f32 = lambda v: float(np.float32(v))  # noqa: E731
DT_DIFF, DT_MECH = _f32(0.01), _f32(0.1)
CCCA, CCCR, RA, MAX_DIST, DEAD = _f32(0.4), 10.0, 1.25, 25.0, _f32(0.1)


def _voxel(pos, N):
    """Integer bins of float32 positions, as the record's mesh_idx defines them (a float32 division)."""
    ijk = (pos.float() / VOXEL).to(torch.int64)
    ok = ((ijk >= 0) & (ijk < N)).all(1)
    return ijk, ok


def _morton(ijk):
    k = torch.zeros_like(ijk[:, 0])
    for b in range(10):
        for a in range(3):
            k |= ((ijk[:, a] >> b) & 1) << (3 * b + a)
    return k


def _mechanics64(rec, N):
    """FM_update on [n, 18] float32 records, all live and inside the grid: (records in the new order, new
    positions, forces), forces and positions in 64 bits."""
    ijk, _ = _voxel(rec[:, 2:5], N)
    order = torch.argsort(_morton(ijk), stable=True)
    rec, ijk = rec[order], ijk[order]
    lin = ijk[:, 0] + N * (ijk[:, 1] + N * ijk[:, 2])
    n = len(rec)
    first = torch.full((N ** 3,), -1, device=rec.device, dtype=torch.int64)
    count = torch.zeros(N ** 3, device=rec.device, dtype=torch.int64)
    head = torch.ones(n, dtype=torch.bool, device=rec.device)
    head[1:] = lin[1:] != lin[:-1]
    at = torch.nonzero(head)[:, 0]
    first[lin[at]] = at
    count[lin[at]] = torch.diff(at, append=torch.tensor([n], device=rec.device))
    pos, rad = rec[:, 2:5].double(), rec[:, 11].double()
    force = torch.zeros_like(pos)
    thres = torch.full((n,), MAX_DIST, device=rec.device, dtype=torch.float64)
    me = torch.arange(n, device=rec.device)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                q = ijk + torch.tensor([dx, dy, dz], device=rec.device)
                ok = ((q >= 0) & (q < N)).all(1)
                v = torch.where(ok, q[:, 0] + N * (q[:, 1] + N * q[:, 2]), 0)
                c = torch.where(ok, count[v], 0)
                for k in range(int(c.max())):
                    i = me[c > k]
                    j = first[v[i]] + k
                    d3 = pos[i] - pos[j]
                    d = (d3.square().sum(1) + 0.0001).sqrt()
                    near = d < thres[i]
                    i, j, d3, d = i[near], j[near], d3[near], d[near]
                    R = (rad[j] + rad[i]).clamp_min(0.01)
                    t = R * RA
                    thres[i] = t
                    cr = torch.where(d <= R, CCCR * (1 - d / R).square() / d, 0.0)
                    ca = CCCA * (1 - d / t).square() / d
                    cf = torch.where(d < t, cr - ca, 0.0)
                    force[i] += d3 * cf[:, None]
    new = pos + DT_MECH / 2 * (3 * force - rec[:, 8:11].double())
    return rec, new, force


def _records64(rec, new, force):
    return {"sign_mesh": None, "pos": new, "force": torch.zeros_like(force), "oldforce": force,
            "volumes": rec[:, 11:16].double(), "phase": None, "clock": rec[:, 17:18].double()}


def _uptake64(rec, mesh, N, coef):
    rate = torch.zeros(N ** 3, device=rec.device, dtype=torch.float64)
    ph = rec.view(torch.int32)[:, 16]
    r = _f32(coef) * rec[:, 12].double() / VOXEL ** 3
    r = torch.where(ph >= 3, r * DEAD, r)
    rate.index_add_(0, mesh, r)
    return rate


def _diffuse64(p, rate, N, s, substeps):
    """`substeps` LOD substeps of a flat float64 field (x fastest), in place."""
    D, decay, b = _f32(s.diffusion), _f32(s.decay), _f32(s.boundary)
    side = -DT_DIFF * D / VOXEL ** 2
    corner = 1.0 + DT_DIFF * decay / 3.0 - side
    E, F = [0.0], [corner]
    for i in range(1, N - 1):
        E.append(side / F[i - 1])
        F.append(corner - side - E[i] * side)
    v = p.view(N, N, N)
    src = (1.0 - rate * DT_DIFF).view(N, N, N)

    def sweep(w):  # along the first axis
        w[0].fill_(b)
        w[N - 1].fill_(b)
        for i in range(1, N - 1):
            w[i].add_(w[i - 1], alpha=-E[i])
        for i in range(N - 2, 0, -1):
            w[i].add_(w[i + 1], alpha=-side).div_(F[i])
        w[0].fill_(b)

    for _ in range(substeps):
        for a in range(3):
            for k in (0, 1, N - 2, N - 1):
                v.select(a, k).fill_(b)
        v.div_(src)
        t = v.permute(2, 0, 1).contiguous()
        sweep(t)
        v.copy_(t.permute(1, 2, 0))
        sweep(v.permute(1, 0, 2))
        sweep(v)
    return p


def _shell(N, device):
    g = torch.arange(N, device=device)
    s = (g < 2) | (g > N - 3)
    return s[:, None, None] | s[None, :, None] | s[None, None, :]


def _layers64(w):
    out, i = [], 0
    for cin, cout in gs.SHAPES:
        k = cout * cin * 27
        W = torch.from_numpy(np.array(w[i:i + k])).cuda().double().reshape(cout, cin, 3, 3, 3)
        out.append([W, torch.from_numpy(np.array(w[i + k:i + k + cout])).cuda().double()])
        i += k + cout
    return out


def _conv64(x, W, b):
    """3x3x3 convolution of [1, C, N, N, N], a few planes at a time."""
    N = x.shape[2]
    step = max(1, min(N, int(6e9 / (27 * x.shape[1] * N * N * 8))))
    if step >= N:
        return torch.nn.functional.conv3d(x, W, b, padding=1)
    out = torch.empty((1, W.shape[0], N, N, N), device=x.device, dtype=x.dtype)
    for z in range(0, N, step):
        e = min(N, z + step)
        lo, hi = max(0, z - 1), min(N, e + 1)
        slab = torch.nn.functional.pad(x[:, :, lo:hi], (0, 0, 0, 0, lo - (z - 1), (e + 1) - hi))
        out[:, :, z:e] = torch.nn.functional.conv3d(slab, W, b, padding=(0, 1, 1))
    return out


def _operator64(x, L):
    h = torch.relu(_conv64(x, *L[0]))
    for k in range(4):
        h = h + _conv64(torch.relu(_conv64(h, *L[2 * k + 1])), *L[2 * k + 2])
    return _conv64(h, *L[9])[0, 0]


def _delta64(p, rate, N, s, w):
    """The operator's input planes and the scale of its output, from one plain substep."""
    inner = ~_shell(N, p.device)
    d = (_diffuse64(p.clone(), rate, N, s, 1) - p).view(N, N, N)
    m = float(d.abs()[inner].max())
    planes = [torch.where(inner, d, 0.0) / m, rate.view(N, N, N) * _f32(w.rate_scale), (~inner).double()]
    return torch.stack(planes)[None], m, inner


def exact(case, seed):
    kind = case["kind"]
    # several steps in one call: the order of the records after a second step turns on the last bit of
    # the positions, so there is no one value in 64 bits; a biology step turns on its random draws
    if kind in ("run", "ensemble", "biology"):
        return None
    N, n = case["N"], case["cells"]
    rec = make_cells(n, N, seed)
    if kind == "mechanics":
        return _records64(*_mechanics64(rec, N))
    subs = _substrates(case)
    mesh = rec.view(torch.int32)[:, 1].long()
    out = {}
    if kind == "step":
        rec, new, force = _mechanics64(rec, N)
        out.update(_records64(rec, new, force))
        ijk, _ = _voxel(new, N)
        mesh = ijk[:, 0] + N * (ijk[:, 1] + N * ijk[:, 2])
    if kind in ("step", "diffusion"):
        for k, s in enumerate(subs):
            p = make_field(n, N, s.boundary, 16 * seed + k).double()
            out["field%d" % k] = _diffuse64(p, _uptake64(rec, mesh, N, s.uptake), N, s, case["substeps"])
        return out
    s, w = gb.oxygen(), gs.load_weights(gs.DEFAULT_WEIGHTS)
    p = make_field(n, N, s.boundary, 16 * seed).double()
    rate = _uptake64(rec, mesh, N, s.uptake)
    x, m, inner = _delta64(p, rate, N, s, w)
    L = _layers64(w.weights)
    if kind == "surrogate":
        with torch.no_grad():
            q = p.view(N, N, N) + m * _operator64(x, L)
            return {"field": torch.where(inner, q, _f32(s.boundary)).reshape(-1)}
    y = _diffuse64(p.clone(), rate, N, s, case["substeps"])
    for W, b in L:
        W.requires_grad_(True)
        b.requires_grad_(True)
    e = (p.view(N, N, N) - y.view(N, N, N)) / m + _operator64(x, L)
    loss = e[inner].square().mean()
    loss.backward()
    grad = torch.cat([t.grad.reshape(-1) for pair in L for t in pair])
    return {"loss": float(loss), "gradient": grad, "target": y}
