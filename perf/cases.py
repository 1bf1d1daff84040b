"""The work a program gives this framework, as cases that can be timed and compared.

A model with its domains resident on one GPU does four things with it: it exchanges halos every
step (through a communication object, a bulk communication object or an explicit plan), it runs
the adjoint of the exchange in its backward pass, and it trains through the exchange and a
stencil (through torch.autograd, or replayed from one CUDA graph). The cases are those four over
regular grids, the cubed sphere and unstructured columns, from the 64^3 grid of the quick start
to fields of gigabytes.

Fields of one element type are views of one allocation (as a model's state usually is), each
starting on a 512-byte boundary; halos start with stale values.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from ghex_b200 import autograd as AG
from ghex_b200 import unstructured as U
from ghex_b200 import workloads as W
from ghex_b200.structured import cubed_sphere as CS
from ghex_b200.structured import regular as R

DTYPES = {"f64": torch.float64, "f32": torch.float32, "i64": torch.int64, "i32": torch.int32, "u8": torch.uint8}
MIXED = "f64:3,3,3,3,0,0;f64:3,3,3,3,0,0;f64:3,3,3,3,0,0;f32:2,2,2,2,1,1;f32:2,2,2,2,1,1"
ALPHA = 0.1


def listed():
    return [
        # the quick-start grid: a small field exchanged once per step, waited for (launch latency)
        {"name": "regular_small", "kind": "regular", "use": "co", "nx": 64, "ny": 64, "nz": 64, "px": 2, "py": 2, "pz": 2,
         "uneven": False, "periodic": "xyz", "fields": "f64:1,1,1,1,1,1"},
        # every field of a weather model's uneven domains in one exchange, as GHEX's users write it
        {"name": "regular_uneven", "kind": "regular", "use": "co", "nx": 400, "ny": 300, "nz": 96, "px": 3, "py": 3, "pz": 3,
         "uneven": True, "periodic": "y", "fields": MIXED},
        # the same model at twice the resolution: an autotuned plan replayed inside the time loop
        {"name": "regular_large", "kind": "regular", "use": "plan", "nx": 800, "ny": 600, "nz": 192, "px": 3, "py": 3, "pz": 3,
         "uneven": True, "periodic": "y", "fields": MIXED},
        # a scalar and a wind vector on the cubed sphere, registered ahead (bulk communication object)
        {"name": "cubed_sphere", "kind": "cubed", "use": "bulk", "edge": 384, "levels": 90, "split": 2, "halo": 3,
         "fields": "f64:1;f64:2"},
        # columns of a triangulated mesh, levels contiguous: a double and a float field
        {"name": "columns", "kind": "columns", "use": "co", "ni": 1024, "nj": 2048, "parts": 16, "levels": 64,
         "contiguous": True, "fields": "f64,f32"},
        # a small ocean-like mesh with an odd number of levels, single precision (columns of 76 bytes)
        {"name": "columns_odd", "kind": "columns", "use": "co", "ni": 160, "nj": 192, "parts": 8, "levels": 19,
         "contiguous": True, "fields": "f32"},
        # fields stored level by level (vertices contiguous), the layout of edge- and vertex-major codes
        {"name": "columns_by_level", "kind": "columns", "use": "plan", "ni": 512, "nj": 768, "parts": 16, "levels": 30,
         "contiguous": False, "fields": "f64"},
        # the backward pass of an exchange of the weather model's fields
        {"name": "regular_adjoint", "kind": "regular", "use": "adjoint", "nx": 400, "ny": 300, "nz": 96, "px": 3, "py": 3,
         "pz": 3, "uneven": True, "periodic": "y", "fields": MIXED},
        # the backward pass of an exchange of mesh columns
        {"name": "columns_adjoint", "kind": "columns", "use": "adjoint", "ni": 1024, "nj": 2048, "parts": 16, "levels": 64,
         "contiguous": True, "fields": "f64,f32"},
        # training through ten steps of exchange and diffusion with torch.autograd
        {"name": "program_autograd", "kind": "program", "graphed": False, "nx": 256, "ny": 256, "nz": 128, "px": 2, "py": 2,
         "pz": 2, "uneven": False, "dtype": "f64", "steps": 10},
        # the same in single precision, replayed from one CUDA graph
        {"name": "program_graphed_f32", "kind": "program", "graphed": True, "nx": 256, "ny": 256, "nz": 128, "px": 2, "py": 2,
         "pz": 2, "uneven": False, "dtype": "f32", "steps": 10},
        # a grid eight times as large, double precision, uneven odd-sized domains
        {"name": "program_graphed_large", "kind": "program", "graphed": True, "nx": 500, "ny": 510, "nz": 250, "px": 3, "py": 2,
         "pz": 2, "uneven": True, "dtype": "f64", "steps": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["regular", "regular", "regular", "cubed", "columns", "columns", "program", "program"])
    if kind == "regular":
        use = rng.choice(["co", "co", "bulk", "plan", "adjoint"])
        case = {"kind": kind, "use": use, "nx": _log(rng, 40, 640), "ny": _log(rng, 40, 480), "nz": _log(rng, 40, 160),
                "px": rng.randint(2, 4), "py": rng.randint(2, 3), "pz": rng.randint(2, 3), "uneven": rng.random() < 0.6,
                "periodic": rng.choice(["xyz", "xy", "y", "z", ""])}
        types = ["f64", "f64", "f32"] if use == "adjoint" else ["f64", "f64", "f32", "f32", "i32", "i64", "u8"]
        halos = [",".join(str(rng.randint(0, 3)) for _ in range(4)) + ",%d,%d" % (rng.randint(1, 3), rng.randint(0, 3)) for _ in range(2)]
        case["fields"] = ";".join(rng.choice(types) + ":" + halos[i % 2] for i in range(rng.randint(1, 5)))
        return case
    if kind == "cubed":
        split = rng.randint(1, 3)
        return {"kind": kind, "use": rng.choice(["co", "bulk", "plan", "adjoint"]), "edge": split * _log(rng, 16, 360 // split),
                "levels": _log(rng, 3, 90), "split": split, "halo": rng.randint(1, 3),
                "fields": rng.choice(["f64:1", "f64:1;f64:2", "f32:1;f32:2", "f32:2"])}
    if kind == "columns":
        use = rng.choice(["co", "plan", "adjoint"])
        return {"kind": kind, "use": use, "ni": _log(rng, 64, 1000), "nj": _log(rng, 64, 1000), "parts": rng.choice([4, 8, 16]),
                "levels": _log(rng, 1, 90), "contiguous": rng.random() < 0.75, "fields": rng.choice(["f64", "f32", "f64,f32", "f32,f32,f32"])}
    return {"kind": kind, "graphed": rng.random() < 0.6, "nx": _log(rng, 40, 400), "ny": _log(rng, 40, 400), "nz": _log(rng, 40, 200),
            "px": rng.randint(2, 3), "py": rng.randint(2, 3), "pz": rng.randint(1, 2), "uneven": rng.random() < 0.5,
            "dtype": rng.choice(["f64", "f32"]), "steps": rng.randint(4, 10)}


# ---- fields ------------------------------------------------------------------------------------
def _arenas(requests, seed):
    """requests: (dtype name, shape, fastest dimension first?) per field. The allocations by type
    and the fields in them, filled with values of the seed."""
    offsets, size = [], {}
    for dt, shape, _ in requests:
        item = torch.empty((), dtype=DTYPES[dt]).element_size()
        offsets.append(size.get(dt, 0))
        size[dt] = -(-(offsets[-1] + math.prod(shape)) * item // 512) * 512 // item
    gen = torch.Generator(device="cuda").manual_seed(seed)
    arenas = {}
    for dt in sorted(size):
        t = torch.empty(size[dt], dtype=DTYPES[dt], device="cuda")
        arenas[dt] = t.uniform_(-1, 1, generator=gen) if t.is_floating_point() else t.random_(0, 127, generator=gen)
    views = []
    for (dt, shape, first), off in zip(requests, offsets):
        a = arenas[dt][off:off + math.prod(shape)]
        views.append(a.view(tuple(reversed(shape))).permute(tuple(reversed(range(len(shape))))) if first else a.view(shape))
    return arenas, views


def _intervals(n, parts, uneven, seed):
    return W.uneven_splits(n, parts, np.random.default_rng(seed)) if uneven else W.even_splits(n, parts)


def _domains(case):
    """(first, last) of every domain, x fastest."""
    xs, ys, zs = (_intervals(case["n" + a], case["p" + a], case["uneven"], 42 + k) for k, a in enumerate("xyz"))
    return [((x[0], y[0], z[0]), (x[1], y[1], z[1])) for z in zs for y in ys for x in xs]


def _specs(case):
    out = []
    for f in case["fields"].split(";"):
        dt, halos = f.split(":")
        out.append((dt, tuple(int(v) for v in halos.split(","))))
    return out


def _extents(dom, h):
    return tuple(dom[1][k] - dom[0][k] + 1 + h[2 * k] + h[2 * k + 1] for k in range(3))


def _regular_inputs(case, seed):
    doms = _domains(case)
    return (doms,) + _arenas([(dt, _extents(d, h), True) for dt, h in _specs(case) for d in doms], seed)


def _regular_bound(case, doms, views):
    """One pattern per set of halo widths, every field bound to its pattern."""
    ctx = R.make_context()
    glob = ((0, 0, 0), (case["nx"] - 1, case["ny"] - 1, case["nz"] - 1))
    descs = [R.DomainDescriptor(i, d) for i, d in enumerate(doms)]
    patterns, bound, it = {}, [], iter(views)
    for dt, h in _specs(case):
        if h not in patterns:
            hg = R.HaloGenerator(glob, [(h[0], h[1]), (h[2], h[3]), (h[4], h[5])], [a in case["periodic"] for a in "xyz"])
            patterns[h] = R.make_pattern(ctx, hg, descs)
        for d, dd in zip(doms, descs):
            bound.append(patterns[h](R.make_field_descriptor(dd, next(it), (h[0], h[2], h[4]), _extents(d, h))))
    return ctx, bound


def _cubed_inputs(case, seed):
    w = W.config3(edge=case["edge"], levels=case["levels"], split=case["split"], halo=case["halo"])
    comps = [(f.split(":")[0], int(f.split(":")[1])) for f in case["fields"].split(";")]
    return (w, comps) + _arenas([(dt, w.extents(d) + (n,), True) for dt, n in comps for d in w.domains], seed)


def _cubed_bound(w, comps, views):
    ctx = CS.make_context()
    cube = CS.cube(w.edge, w.levels)
    descs = [CS.DomainDescriptor(cube, *d) for d in w.domains]
    pattern = CS.make_pattern(ctx, CS.HaloGenerator(w.halo), descs)
    it = iter(views)
    return ctx, [pattern(CS.make_field_descriptor(dd, next(it), w.offsets(), w.extents(d), n, n > 1))
                 for _, n in comps for d, dd in zip(w.domains, descs)]


@functools.lru_cache(maxsize=4)
def _mesh(ni, nj, parts):
    """The mesh, its domains and their pattern: made once by a program and kept for its fields."""
    w = W.config2(ni=ni, nj=nj, parts=parts)
    ctx = U.make_context()
    descs = [U.DomainDescriptor(i, gids, outer) for i, gids, outer in w.domains]
    return w.domains, ctx, descs, U.make_pattern(ctx, U.HaloGenerator(), descs)


def _column_inputs(case, seed):
    doms = _mesh(case["ni"], case["nj"], case["parts"])[0]
    shape = (lambda n: (n, case["levels"])) if case["levels"] > 1 else (lambda n: (n,))
    return (doms,) + _arenas([(dt, shape(g.size), not case["contiguous"]) for dt in case["fields"].split(",") for _, g, _ in doms], seed)


def _column_bound(case, views):
    _, ctx, descs, pattern = _mesh(case["ni"], case["nj"], case["parts"])
    return ctx, [pattern(U.make_field_descriptor(descs[i % len(descs)], v)) for i, v in enumerate(views)]


PROGRAM_HALO = (1, 1, 1, 1, 1, 1)


def _program_inputs(case, seed):
    doms = _domains(case)
    return (doms,) + _arenas([(case["dtype"], _extents(d, PROGRAM_HALO), True) for d in doms], seed)


# ---- the calls ---------------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "program":
        doms, _, xs = _program_inputs(case, seed)
        ctx, bound = _regular_bound(dict(case, periodic="xyz", fields=case["dtype"] + ":1,1,1,1,1,1"), doms, xs)
        dx = AG.DifferentiableExchange(ctx, bound)
        state = {"use": "graphed" if case["graphed"] else "autograd", "dx": dx, "x": xs, "steps": case["steps"]}
        if case["graphed"]:
            state["graphed"] = AG.GraphedDiffusion(dx, xs, case["steps"], ALPHA)
        return state
    if case["kind"] == "regular":
        doms, arenas, views = _regular_inputs(case, seed)
        ctx, bound = _regular_bound(case, doms, views)
    elif case["kind"] == "cubed":
        w, comps, arenas, views = _cubed_inputs(case, seed)
        ctx, bound = _cubed_bound(w, comps, views)
    else:
        _, arenas, views = _column_inputs(case, seed)
        ctx, bound = _column_bound(case, views)
    state = {"use": case["use"], "fields": arenas, "bound": bound}
    if case["use"] == "co":
        state["co"] = R.make_communication_object(ctx)
    elif case["use"] == "bulk":
        state["co"] = R.make_bulk_communication_object(ctx)
        state["co"].add_fields(*bound)
        state["co"].init()
    else:
        state["plan"] = R.make_exchange_plan(ctx, bound)
        if case["use"] == "plan":
            state["plan"].autotune()
    return state


def run(state):
    use = state["use"]
    if use == "co":
        state["co"].exchange(state["bound"]).wait()
    elif use == "bulk":
        state["co"].exchange().wait()
    elif use == "plan":
        state["plan"].graph_launch()
    elif use == "adjoint":  # the fields hold gradients: each halo's is added to its owner's and zeroed
        state["plan"].adjoint()
    elif use == "graphed":
        loss, grads = state["graphed"].run(state["x"])
        return {"loss": loss, "gradients": grads}
    else:
        leaves = [x.detach().requires_grad_(True) for x in state["x"]]
        ys = AG.diffusion_program(state["dx"], [x.clone() for x in leaves], state["steps"], ALPHA)
        loss = AG.interior_loss(ys)
        grads = torch.autograd.grad(loss, leaves)
        return {"loss": loss.detach(), "fields": [y.detach() for y in ys], "gradients": list(grads)}
    return state["fields"]


# ---- what a pass cannot do without -------------------------------------------------------------
def work(case):
    """An exchange reads every halo cell's source and writes the cell; an adjoint reads and writes
    every image and every distinct owner; the program reads its fields and writes their gradients
    (and, through autograd, the final fields)."""
    size = {d: torch.empty((), dtype=t).element_size() for d, t in DTYPES.items()}
    if case["kind"] == "program":
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": float(cells * size[case["dtype"]] * (2 if case["graphed"] else 3)), "flops": float(2 * 9 * case["steps"] * cells)}
    adjoint, total = case["use"] == "adjoint", 0
    if case["kind"] == "regular":
        for dt, h in _specs(case):
            for first, last in _domains(case):
                whole, inner, alone = 1, 1, 1
                for k, a in enumerate("xyz"):
                    n = last[k] - first[k] + 1
                    lower, upper = (a in case["periodic"] or first[k] > 0), (a in case["periodic"] or last[k] < case["n" + a] - 1)
                    whole *= n + h[2 * k] * lower + h[2 * k + 1] * upper
                    inner *= n
                    alone *= max(0, n - h[2 * k] * upper - h[2 * k + 1] * lower)  # read by no halo along this axis
                total += size[dt] * 2 * (whole - inner + ((inner - alone) if adjoint else 0))
    elif case["kind"] == "cubed":
        e, s, h = case["edge"] // case["split"], case["split"], case["halo"]
        per_level = 6 * s * s * ((e + 2 * h) ** 2 - e * e) - 24 * h * h  # the cube's corners have no owner
        for f in case["fields"].split(";"):
            dt, n = f.split(":")
            total += size[dt] * int(n) * case["levels"] * per_level * (4 if adjoint else 2)
    else:
        doms = _mesh(case["ni"], case["nj"], case["parts"])[0]
        halo = sum(o.size for _, _, o in doms)
        owners = np.unique(np.concatenate([g[o] for _, g, o in doms])).size if adjoint else 0
        total = sum(size[dt] for dt in case["fields"].split(",")) * case["levels"] * 2 * (halo + owners)
    return {"bytes": float(total), "flops": float(total / 8 if adjoint else 0)}


# ---- the results in 64 bits --------------------------------------------------------------------
def _wide(arenas):
    return {k: (v.double() if v.is_floating_point() else v.clone()) for k, v in arenas.items()}


def _as(view, arena, wide):
    return wide.as_strided(view.shape, view.stride(), view.storage_offset() - arena.storage_offset())


def _exact_regular(case, seed):
    doms, arenas, views = _regular_inputs(case, seed)
    wide = _wide(arenas)
    n = (case["nx"], case["ny"], case["nz"])
    it = iter(views)
    for dt, h in _specs(case):
        outs = [_as(v, arenas[dt], wide[dt]) for v in (next(it) for _ in doms)]
        inner = [o[tuple(slice(h[2 * k], h[2 * k] + d[1][k] - d[0][k] + 1) for k in range(3))] for o, d in zip(outs, doms)]
        glob = torch.empty(n, dtype=wide[dt].dtype, device="cuda")
        for v, d in zip(inner, doms):
            glob[tuple(slice(d[0][k], d[1][k] + 1) for k in range(3))] = v
        parts = []
        for o, d in zip(outs, doms):
            at, ix = [], []
            for k, a in enumerate("xyz"):
                g = torch.arange(d[0][k] - h[2 * k], d[1][k] + 1 + h[2 * k + 1], device="cuda")
                ok = (g >= 0) & (g < n[k]) if a not in case["periodic"] else torch.ones_like(g, dtype=torch.bool)
                at.append(slice(int(ok.nonzero()[0]), int(ok.nonzero()[-1]) + 1))
                ix.append(g[ok] % n[k])
            parts.append((o[tuple(at)], (ix[0][:, None, None] * n[1] + ix[1][None, :, None]) * n[2] + ix[2][None, None, :]))
        if case["use"] != "adjoint":
            for v, lin in parts:
                v.copy_(glob.view(-1)[lin])
            continue
        for i, (part, lin) in zip(inner, parts):
            i.zero_()  # what is left of the part is its halo
            glob.view(-1).index_add_(0, lin.reshape(-1), part.reshape(-1))
            part.zero_()
        for i, d in zip(inner, doms):
            i.copy_(glob[tuple(slice(d[0][k], d[1][k] + 1) for k in range(3))])
    return wide


def _exact_columns(case, seed):
    doms, arenas, views = _column_inputs(case, seed)
    wide = _wide(arenas)
    n = case["ni"] * case["nj"]
    it = iter(views)
    for dt in case["fields"].split(","):
        outs = [_as(v, arenas[dt], wide[dt]) for v in (next(it) for _ in doms)]
        table = torch.zeros((n,) + tuple(outs[0].shape[1:]), dtype=torch.float64, device="cuda")
        ids = [(torch.from_numpy(g).cuda(), torch.from_numpy(o).cuda()) for _, g, o in doms]
        for v, (g, o) in zip(outs, ids):
            inner = torch.ones(g.numel(), dtype=torch.bool, device="cuda")
            inner[o] = False
            table[g[inner]] = v[inner]
        if case["use"] != "adjoint":
            for v, (g, o) in zip(outs, ids):
                v[o] = table[g[o]]
            continue
        for v, (g, o) in zip(outs, ids):
            table.index_add_(0, g[o], v[o].contiguous())
        for v, (g, o) in zip(outs, ids):
            v.copy_(table[g])
            v[o] = 0.0
    return wide


def _exact_program(case, seed):
    doms, _, xs = _program_inputs(case, seed)
    x = torch.empty((case["nx"], case["ny"], case["nz"]), dtype=torch.float64, device="cuda")
    at = [tuple(slice(d[0][k], d[1][k] + 1) for k in range(3)) for d in doms]
    for v, s in zip(xs, at):
        x[s] = v[1:-1, 1:-1, 1:-1].double()

    def step(x):
        return x + ALPHA * (sum(torch.roll(x, s, k) for k in range(3) for s in (1, -1)) - 6 * x)

    def split(x):
        out = []
        for s in at:
            out.append(torch.nn.functional.pad(x[s], (1,) * 6))
        return out

    for _ in range(case["steps"]):
        x = step(x)
    loss, fields = (x ** 2).sum(), split(x)
    g = 2 * x
    for _ in range(case["steps"]):
        g = step(g)  # the periodic update is its own transpose
    out = {"loss": loss, "gradients": split(g)}
    return out if case["graphed"] else dict(out, fields=fields)


def exact(case, seed):
    if case["kind"] == "program":
        return _exact_program(case, seed)
    if case["kind"] == "regular":
        return _exact_regular(case, seed)
    if case["kind"] == "columns":
        return _exact_columns(case, seed)
    return None  # copies with changes of sign: compared as they are
