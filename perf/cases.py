"""What this framework is used for, as cases that can be timed.

Every case is one call (or one short sequence of calls) that a program of this framework
makes in its step loop, on GPU-resident inputs:

* ``step``: one planet's implicit heat-transport sub-step (``transport_step``), plain FP64
  or FP32 inside FP64 refinement, uniform or per-edge conductance, returning the new
  temperature and the transport;
* ``batch``: one sub-step of many planets of uneven mesh levels (``LaneBatch``), each planet
  with its own radius and per-edge conductances, with the smoother settings a program keeps
  from an earlier autotune, or the default ones;
* ``lane``: one round of the serving loop: the planets of one mesh level resident in a
  ``Batch``, of which those with a queued request take part;
* ``multi``: many sub-steps of one planet that differ in their sources, as one block
  (``transport_step_multi``);
* ``operators``: gradient, divergence and Laplacian of a set of fields;
* ``columns``: the column radiation of every cell;
* ``newton``: the nonlinear implicit transport on an agglomerated graph with the quartic
  column response evaluated per fine cell on the GPU;
* ``tracer``: the implicit tracer transport on an agglomerated graph.

Sizes are those of the framework's benchmark and tests (mesh levels 3 to 8, 2 to 32
sub-steps in a block, 3 to 16 column layers, 2 to 10 tracer layers).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import planet_game_gb300 as pg
from planet_game_gb300 import workloads as W

CP = 1004.64                      # J/kg/K, the tracer's and the air's heat capacity
QUARTIC_A = 3.0e5 / (30.0 * 86400.0)
QUARTIC_R = 0.75 * 0.97 * 5.670374419e-8


def cells_of(level: int) -> int:
    return 10 * 4 ** level + 2


def listed() -> list[dict]:
    return [
        # a small planet stepped alone: the smallest call, latency and launches
        {"name": "step_L4_fp64", "kind": "step", "level": 4, "precision": "fp64", "per_edge": False, "radius": 6.371e6},
        # the reference's default planet with per-edge diffusivity, FP32 inside FP64 refinement
        {"name": "step_L5_mixed", "kind": "step", "level": 5, "precision": "mixed", "per_edge": True, "radius": 4.2e6},
        # the drop-in solve of a medium planet
        {"name": "step_L6_fp64", "kind": "step", "level": 6, "precision": "fp64", "per_edge": False, "radius": 6.371e6},
        # the largest planet stepped alone
        {"name": "step_L8_fp64", "kind": "step", "level": 8, "precision": "fp64", "per_edge": False, "radius": 6.371e6},
        # the headline workload: 64 uneven planets in one step, settings kept from an autotune
        {"name": "batch64_mixed", "kind": "batch", "l4": 16, "l5": 24, "l6": 16, "l7": 8, "precision": "mixed",
         "tuned": True, "mix": 3},
        # a round of the serving loop: 11 of 16 resident L5 planets have a request
        {"name": "lane_L5_mixed", "kind": "lane", "level": 5, "planets": 16, "active": 11, "precision": "mixed",
         "tuned": True, "mix": 5},
        # an ensemble of one planet's sub-steps with perturbed sources
        {"name": "multi_L7_mixed", "kind": "multi", "level": 7, "count": 32, "precision": "mixed", "radius": 6.371e6},
        # the operator sweep on 8 fields of a medium mesh, and on 4 fields of the largest in FP32
        {"name": "operators_L6_fp64", "kind": "operators", "level": 6, "fields": 8, "dtype": "float64",
         "radius": 6.371e6},
        {"name": "operators_L8_fp32", "kind": "operators", "level": 8, "fields": 4, "dtype": "float32",
         "radius": 6.371e6},
        # radiation of 10 pressure levels in every column of a medium mesh
        {"name": "columns_L6", "kind": "columns", "cells": 40962, "layers": 10},
        # the nonlinear transport one mesh level coarser, as the production step runs it
        {"name": "newton_L6", "kind": "newton", "level": 6, "radius": 6.371e6, "conductance": 1.0},
        # ten layers of a tracer on the same kind of graph
        {"name": "tracer_L6", "kind": "tracer", "level": 6, "layers": 10, "radius": 6.371e6, "flow": 2.0e9},
    ]


def draw(rng) -> dict:
    kind = rng.choice(["step", "step", "batch", "lane", "multi", "operators", "columns", "newton", "tracer"])
    radius = float(round(rng.uniform(3.0e6, 9.0e6)))
    precision = rng.choice(["fp64", "mixed"])
    if kind == "step":
        return {"kind": kind, "level": rng.choice([3, 4, 5, 6, 7, 8]), "precision": precision,
                "per_edge": rng.random() < 0.5, "radius": radius}
    if kind == "batch":
        return {"kind": kind, "l4": rng.randint(1, 16), "l5": rng.randint(0, 24), "l6": rng.randint(1, 16),
                "l7": rng.randint(0, 8), "precision": rng.choice(["mixed", "mixed", "fp64"]),
                "tuned": rng.random() < 0.5, "mix": rng.randint(0, 1000)}
    if kind == "lane":
        level = rng.choice([4, 5, 6, 7])
        planets = rng.randint(2, {4: 32, 5: 24, 6: 12, 7: 6}[level])
        return {"kind": kind, "level": level, "planets": planets, "active": rng.randint(1, planets),
                "precision": precision, "tuned": rng.random() < 0.5, "mix": rng.randint(0, 1000)}
    if kind == "multi":
        return {"kind": kind, "level": rng.choice([4, 5, 6, 7]), "count": rng.randint(2, 32), "precision": precision,
                "radius": radius}
    if kind == "operators":
        level, dtype = rng.choice([4, 5, 6, 7, 8]), rng.choice(["float64", "float32"])
        most = 8 if level < 8 else 3 if dtype == "float32" else 1
        return {"kind": kind, "level": level, "fields": rng.randint(1, most), "dtype": dtype, "radius": radius}
    if kind == "columns":   # any part of a mesh, not whole meshes alone
        return {"kind": kind, "cells": round(math.exp(rng.uniform(math.log(150.0), math.log(200000.0)))),
                "layers": rng.randint(3, 16)}
    if kind == "newton":
        return {"kind": kind, "level": rng.choice([5, 6, 7]), "radius": radius,
                "conductance": round(math.exp(rng.uniform(math.log(0.2), math.log(2.0))), 3)}
    return {"kind": kind, "level": rng.choice([5, 6, 7]), "layers": rng.randint(2, 10), "radius": radius,
            "flow": round(math.exp(rng.uniform(math.log(5e8), math.log(4e9))))}


# ---- what a program has in hand ------------------------------------------------------------

def _gpu(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda").contiguous()


@functools.lru_cache(maxsize=12)
def _unit(level: int):
    """Of one mesh level, the same for every radius: cell centres and insolation."""
    m = pg.make_icosphere(level, W.EARTH_RADIUS)
    return m.arrays()["center"], m.substep_mean_insolation(0)


def _state_of(level: int, rng, spread: float = 0.5):
    """T0 and the source of one sub-step (workloads.step_inputs' fields from one generator)."""
    center, insolation = _unit(level)
    t0 = 288.0 - 40.0 * center[:, 2] ** 2 + rng.normal(0.0, spread, len(center))
    return t0, W.source_term(insolation, t0)


def _edges_of(mesh, rng):
    return W.HEAT_CAPACITY * W.DIFFUSIVITY * np.exp(rng.normal(0.0, 0.5, mesh.edge_count))


def _settings(depth: int) -> dict:
    """Smoother settings as the autotuner picks them on batches of these planets: one fine
    sweep each way, several block-local ones on the first coarse level."""
    return {"pre_sweeps": [1, 2, 1, 1][:depth], "post_sweeps": [1, 2, 1, 1][:depth], "stencil_tiles": [1] * depth,
            "vector_tiles": [1] * depth, "block_sweeps": [1, 6, 1, 1][:depth], "jacobi_omega": 1.0}


def _radii(count: int, mix: int) -> list[float]:
    rng = np.random.default_rng([mix, count])
    return [float(r) for r in rng.uniform(3.0e6, 9.0e6, count)]


@functools.lru_cache(maxsize=96)
def _planet(level: int, radius: float):
    """A planet that batches share (a batch keeps its own matrix, vectors and workspace)."""
    return pg.make_icosphere(level, radius)


def _levels(case) -> list[int]:
    if case["kind"] == "lane":
        return [case["level"]] * case["planets"]
    return [4] * case["l4"] + [5] * case["l5"] + [6] * case["l6"] + [7] * case["l7"]


def _meshes(case):
    levels = _levels(case)
    return [_planet(l, r) for l, r in zip(levels, _radii(len(levels), case["mix"]))]


def _batch_inputs(case, seed):
    meshes = _meshes(case)
    rng = np.random.default_rng([seed, 11])
    t0, src, edges = [], [], []
    for m in meshes:
        t, s = _state_of(m.subdivision, rng)
        t0.append(t)
        src.append(s)
        edges.append(_edges_of(m, rng))
    active = [True] * len(meshes)
    if case["kind"] == "lane":
        on = np.random.default_rng(case["mix"]).permutation(len(meshes))[: case["active"]]
        active = [i in set(on.tolist()) for i in range(len(meshes))]
    return meshes, t0, src, edges, active


def _fields(case, seed):
    """Sums of degree-one to degree-three harmonics and their products: smooth fields of
    order one, and edge fluxes of the same size."""
    center, _ = _unit(case["level"])
    mesh = _planet(case["level"], case["radius"])
    rng = np.random.default_rng([seed, 17])
    fields, fluxes = [], []
    for _ in range(case["fields"]):
        k = rng.normal(0.0, 3.0, (4, 3))
        phase = rng.uniform(0.0, 6.0, 4)
        fields.append(np.cos(center @ k.T + phase).sum(axis=1))
        fluxes.append(rng.normal(0.0, 1.0, mesh.edge_count) * 1e-6)
    return mesh, fields, fluxes


def _columns(case, seed):
    rng = np.random.default_rng([seed, 19])
    surface = 288.0 - 40.0 * rng.uniform(-1.0, 1.0, case["cells"]) ** 2 + rng.normal(0.0, 3.0, case["cells"])
    return W.column_profiles(surface, case["layers"], int(rng.integers(1 << 30)))


@functools.lru_cache(maxsize=6)
def _graph(level: int, radius: float):
    """An agglomerated planet's graph arrays (those of the transport's inputs)."""
    p = pg.agglomerated_transport_graph(level, radius)
    g = pg.mesh_transport_graph(p)
    return {"nodes": p.cell_count, "offset": g.offset.astype(np.int64), "neighbour": g.neighbour.astype(np.int64),
            "weight": np.asarray(g.weight), "area": np.asarray(g.area_m2), "group": p.group_of_cell().astype(np.int64)}


def _newton_inputs(case, seed):
    g = _graph(case["level"], case["radius"])
    b, floor = W.quartic_column(QUARTIC_A, QUARTIC_R, len(g["group"]), int(np.random.default_rng([seed, 23]).integers(1 << 30)))
    node_floor = np.full(g["nodes"], -np.inf)
    np.maximum.at(node_floor, g["group"], floor)
    return g, b, node_floor, case["conductance"] * case["radius"] ** 2


def _tracer_inputs(case, seed):
    g = _graph(case["level"], case["radius"])
    rng = np.random.default_rng([seed, 29])
    flux = W.antisymmetric_layer_fluxes(g["offset"], g["neighbour"], case["layers"], case["flow"],
                                        int(rng.integers(1 << 30)), column_balanced=False)
    mass = g["area"] * 1.0e5 / (9.81 * case["layers"])
    tracer = W.tracer_field(case["layers"] * g["nodes"], int(rng.integers(1 << 30)))
    return g, np.full(len(g["neighbour"]), 2.0e8), flux, mass, tracer


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        mesh = pg.make_icosphere(case["level"], case["radius"])
        rng = np.random.default_rng([seed, 7])
        t0, src = _state_of(case["level"], rng)
        return {"kind": kind, "mesh": mesh, "t0": _gpu(t0), "src": _gpu(src), "precision": case["precision"],
                "edges": _edges_of(mesh, rng) if case["per_edge"] else None}
    if kind in ("batch", "lane"):
        meshes, t0, src, edges, active = _batch_inputs(case, seed)
        batch = pg.LaneBatch(meshes) if kind == "batch" else pg.Batch(meshes)
        batch.set_edge_conductance(edges)
        if case["tuned"]:
            lanes = [b for b in batch.batches] if kind == "batch" else [batch]
            for b in lanes:
                b.set_tuning(_settings(max(len(m.level_rows) for m in b.meshes)))
        return {"kind": kind, "batch": batch, "t0": [_gpu(t) if a else None for t, a in zip(t0, active)],
                "src": [_gpu(s) if a else None for s, a in zip(src, active)],
                "active": None if all(active) else active, "precision": case["precision"]}
    if kind == "multi":
        mesh = pg.make_icosphere(case["level"], case["radius"])
        rng = np.random.default_rng([seed, 13])
        t0, src = _state_of(case["level"], rng)
        sources = [_gpu(src + rng.normal(0.0, 5.0, len(src))) for _ in range(case["count"])]
        return {"kind": kind, "mesh": mesh, "t0": _gpu(t0), "sources": sources, "precision": case["precision"]}
    if kind == "operators":
        mesh, fields, fluxes = _fields(case, seed)
        dtype = getattr(torch, case["dtype"])
        return {"kind": kind, "mesh": mesh, "fields": [_gpu(f, dtype) for f in fields],
                "fluxes": [_gpu(f, dtype) for f in fluxes]}
    if kind == "columns":
        c = _columns(case, seed)
        return {"kind": kind, "constants": pg.column_constants(**W.EARTH_COLUMN),
                "inputs": [_gpu(a) for a in (c.temperature, c.humidity, c.cloud_water, c.surface_temperature,
                                             c.surface_pressure)]}
    if kind == "newton":
        _, b, floor, conductance = _newton_inputs(case, seed)
        planet = pg.agglomerated_transport_graph(case["level"], case["radius"])
        response = pg.QuarticResponse(QUARTIC_A, _gpu(b), QUARTIC_R, hold_stride=0, fine=True)
        return {"kind": kind, "planet": planet, "floor": _gpu(floor), "conductance": conductance, "response": response}
    _, eddies, flux, mass, tracer = _tracer_inputs(case, seed)
    planet = pg.agglomerated_transport_graph(case["level"], case["radius"])
    return {"kind": kind, "planet": planet, "transport": pg.AdvectionDiffusion(case["layers"], _gpu(eddies), _gpu(flux), CP),
            "mass": _gpu(mass), "tracer": _gpu(tracer)}


def run(s):
    kind = s["kind"]
    if kind == "step":
        t, h, report = pg.transport_step(s["mesh"], s["t0"], s["src"], W.HEAT_CAPACITY, W.SUBSTEP_S,
                                         W.HEAT_CAPACITY * W.DIFFUSIVITY, edge_conductance=s["edges"],
                                         precision=s["precision"])
        return {"temperature": t, "transport": h, "status": report.status}
    if kind in ("batch", "lane"):
        out, reports = s["batch"].transport_step(s["t0"], s["src"], W.HEAT_CAPACITY, W.SUBSTEP_S,
                                                 edge_conductance="stored", active=s["active"],
                                                 precision=s["precision"])
        return {"temperature": torch.cat([t for t in out if t is not None]),
                "status": max(r.status for r in reports)}
    if kind == "multi":
        out, _, reports = pg.transport_step_multi(s["mesh"], s["t0"], s["sources"], W.HEAT_CAPACITY, W.SUBSTEP_S,
                                                  W.HEAT_CAPACITY * W.DIFFUSIVITY, precision=s["precision"])
        return {"temperature": out, "status": max(r.status for r in reports)}
    if kind == "operators":
        grads = [pg.gradient(s["mesh"], f) for f in s["fields"]]
        return {"east": [e for e, _ in grads], "north": [n for _, n in grads],
                "divergence": [pg.divergence(s["mesh"], f) for f in s["fluxes"]],
                "laplacian": [pg.laplacian(s["mesh"], f) for f in s["fields"]]}
    if kind == "columns":
        return dict(zip(("emissivity", "absorbed", "fraction", "reflectance", "scalars"),
                        pg.column_radiation(s["constants"], *s["inputs"])))
    if kind == "newton":
        r = pg.solve_implicit_transport(s["planet"], s["conductance"], s["floor"], s["response"])
        return {"source": r.source_W_m2, "mean": r.mean_K}
    r = pg.solve_implicit_tracer(s["planet"], s["transport"], s["mass"], s["tracer"], W.SUBSTEP_S)
    return {"tracer": r.tracer}


# ---- what a call cannot do without -----------------------------------------------------------

def work(case) -> dict:
    """Inputs, mesh arrays and outputs once each; the arithmetic of applying the operator
    once (a solve's preconditioning and iterations are the present method's, not counted)."""
    kind = case["kind"]
    if kind == "step":
        n = cells_of(case["level"])
        # T0, S in; T, H out; columns, weights, area (and the conductances per edge)
        return {"bytes": n * (4 * 8 + 6 * 12 + 8 + (24 if case["per_edge"] else 0)), "flops": n * 30}
    if kind in ("batch", "lane"):
        levels = _levels(case)
        share = case["active"] / case["planets"] if kind == "lane" else 1.0
        n = sum(cells_of(l) for l in levels) * share
        return {"bytes": int(n * (3 * 8 + 6 * 8 + 24 + 8)), "flops": int(n * 30)}
    if kind == "multi":
        n = cells_of(case["level"])
        return {"bytes": n * (case["count"] * 16 + 8 + 6 * 12 + 8), "flops": n * 30 * case["count"]}
    if kind == "operators":
        n, item = cells_of(case["level"]), 8 if case["dtype"] == "float64" else 4
        # per field: value and flux in (3 edges a cell), four results out; the mesh once
        return {"bytes": n * (case["fields"] * item * 8 + 24 + 48 + 48 + 48 + 32 + 24 + 8 + 2 + 24),
                "flops": n * case["fields"] * 80}
    if kind == "columns":
        n, layers = case["cells"], case["layers"]
        return {"bytes": n * (7 * layers + 7) * 8, "flops": n * layers * 60}
    if kind == "newton":
        n, fine = cells_of(case["level"] - 1), cells_of(case["level"])
        return {"bytes": n * (3 * 8 + 6 * 12 + 8) + fine * (8 + 8 + 8), "flops": fine * 100}
    n, layers = cells_of(case["level"] - 1), case["layers"]
    return {"bytes": n * (layers * (16 + 6 * 8) + 8 + 6 * 12), "flops": n * layers * 40}


# ---- the same results from plain torch in 64 bits ---------------------------------------------

def _ell(offset, neighbour):
    """Columns [n, 6] (the row itself where a row has five) and the entry of each, or -1."""
    offset = torch.as_tensor(offset, device="cuda")
    n = len(offset) - 1
    slot = torch.arange(6, device="cuda")[None, :]
    entry = offset[:-1, None] + slot
    valid = entry < offset[1:, None]
    entry = torch.where(valid, entry, torch.zeros_like(entry))
    col = torch.as_tensor(neighbour, device="cuda")[entry]
    col = torch.where(valid, col, torch.arange(n, device="cuda")[:, None])
    return col, entry, valid


def _conjugate_gradients(apply, diagonal, b, x, tolerance, dots):
    """Jacobi-preconditioned conjugate gradients on independent systems side by side;
    `dots(u, v)` gives each row the dot product of its system."""
    r = b - apply(x)
    z = r / diagonal
    p = z.clone()
    rz = dots(r, z)
    goal = tolerance * tolerance * dots(b, b)
    for k in range(20000):
        q = apply(p)
        alpha = rz / torch.clamp(dots(p, q), min=1e-300)
        x = x + alpha * p
        r = r - alpha * q
        if k % 50 == 49:
            r = b - apply(x)
            if bool((dots(r, r) <= goal).all()):
                break
        z = r / diagonal
        new = dots(r, z)
        p = z + new / torch.clamp(rz, min=1e-300) * p
        rz = new
    return x


def _sub_steps(meshes, t0, src, conductances):
    """T and H of independent sub-steps, all planets in one block-diagonal system."""
    arrays = [m.arrays() for m in meshes]
    base = np.cumsum([0] + [m.cell_count for m in meshes])
    entries = np.cumsum([0] + [m.directed_edge_count for m in meshes])
    offset = np.concatenate([a["edge_offset"].astype(np.int64) + e for a, e in zip(arrays, entries)] + [entries[-1:]])
    neighbour = np.concatenate([a["neighbor"].astype(np.int64) + b for a, b in zip(arrays, base)])
    weight = _gpu(np.concatenate([a["graph_weight"] for a in arrays]))
    area = _gpu(np.concatenate([a["area_m2"] for a in arrays]))
    g = _gpu(np.concatenate([np.broadcast_to(k, (a["edge_length_m"].shape[0],))[a["edge"].astype(np.int64)]
                             for a, k in zip(arrays, conductances)]))
    which = torch.as_tensor(np.repeat(np.arange(len(meshes)), np.diff(base)), device="cuda")
    t0, src = _gpu(np.concatenate(t0)), _gpu(np.concatenate(src))
    col, entry, valid = _ell(offset, neighbour)
    gw = torch.where(valid, (g * weight)[entry], torch.zeros((), dtype=torch.float64, device="cuda"))
    capacity = W.HEAT_CAPACITY / W.SUBSTEP_S
    total = gw.sum(1)

    def flux(t):   # sum of G w (T_n - T_c), W
        return (gw * (t[col] - t[:, None])).sum(1)

    def dots(u, v):
        return torch.zeros(len(meshes), dtype=torch.float64, device="cuda").index_add_(0, which, u * v)[which]

    # the departure from T0: a small right-hand side loses no digits
    d = _conjugate_gradients(lambda x: capacity * area * x - flux(x), capacity * area + total,
                             area * src + flux(t0), torch.zeros_like(t0), 1e-13, dots)
    h = flux(t0 + d) / area
    return t0 + (src + h) / capacity, h


def _operators_exact(case, seed):
    mesh, fields, fluxes = _fields(case, seed)
    a = mesh.arrays()
    dtype = getattr(torch, case["dtype"])
    offset = np.append(a["edge_offset"].astype(np.int64), mesh.directed_edge_count)
    col, entry, valid = _ell(offset, a["neighbor"].astype(np.int64))
    zero = torch.zeros((), dtype=torch.float64, device="cuda")
    edge = torch.as_tensor(a["edge"].astype(np.int64), device="cuda")
    distance, length = _gpu(a["edge_distance_m"])[edge], _gpu(a["edge_length_m"])[edge]
    east, north = _gpu(a["normal_east"]), _gpu(a["normal_north"])
    e = torch.where(valid, east[entry], zero)
    n = torch.where(valid, north[entry], zero)
    d = torch.where(valid, distance[entry], zero + 1.0)
    l = torch.where(valid, length[entry], zero)
    first = torch.as_tensor(a["edge_first"].astype(np.int64), device="cuda")[edge]
    rows = torch.arange(mesh.cell_count, device="cuda")[:, None]
    sign = torch.where(first[entry] == rows, zero + 1.0, zero - 1.0)
    area = _gpu(a["area_m2"])
    mee, men, mnn = (e * e).sum(1), (e * n).sum(1), (n * n).sum(1)
    det = mee * mnn - men * men
    out = {"east": [], "north": [], "divergence": [], "laplacian": []}
    for f, x in zip(fields, fluxes):
        f, x = _gpu(f, dtype).double(), _gpu(x, dtype).double()
        rise = torch.where(valid, f[col] - f[:, None], zero)
        slope = rise / d
        re, rn = (slope * e).sum(1), (slope * n).sum(1)
        out["east"].append((mnn * re - men * rn) / det)
        out["north"].append((mee * rn - men * re) / det)
        out["divergence"].append((x[edge][entry] * sign * l).sum(1) / area)
        out["laplacian"].append((rise * l / d).sum(1) / area)
    return out


def _columns_exact(case, seed):
    c = _columns(case, seed)
    k = W.EARTH_COLUMN
    temp, q, cloud, ts, ps = (_gpu(a) for a in (c.temperature, c.humidity, c.cloud_water, c.surface_temperature,
                                                c.surface_pressure))
    layers = case["layers"]
    layer_pa = ps / layers
    depth = k["dry_optical_depth"] * layer_pa / k["reference_pressure_Pa"] + \
        k["vapour_absorption_m2_kg"] * q.clamp(min=0.0) * layer_pa / k["gravity_m_s2"]
    path = cloud.clamp(min=0.0) * ps / (k["gravity_m_s2"] * layers)
    fraction = (path / k["in_cloud_water_path_kg_m2"]).clamp(max=1.0)
    inside = torch.where(fraction > 0.0, path / fraction.clamp(min=1e-300), torch.zeros_like(path))
    tau = 3.0 * inside / (2.0 * 1000.0 * k["effective_radius_m"])
    omg = 1.0 - k["cloud_asymmetry"]
    reflectance = fraction * omg * tau / (2.0 + omg * tau)
    eps = -torch.expm1(-(depth + k["cloud_longwave_absorption_m2_kg"] * path))
    emission = eps * k["stefan_boltzmann"] * temp ** 4
    down = torch.zeros_like(ts)
    above = [None] * layers
    for l in reversed(range(layers)):
        above[l] = down
        down = (1.0 - eps[l]) * down + emission[l]
    up = k["stefan_boltzmann"] * ts ** 4
    absorbed = []
    for l in range(layers):
        absorbed.append(eps[l] * (up + above[l]))
        up = (1.0 - eps[l]) * up + emission[l]
    scalars = torch.stack([down, up, (1.0 - reflectance).prod(0), 1.0 - (1.0 - fraction).prod(0),
                           (fraction * tau).sum(0)])
    return {"emissivity": eps, "absorbed": torch.stack(absorbed), "fraction": fraction, "reflectance": reflectance,
            "scalars": scalars}


def _newton_exact(case, seed):
    g, b, floor, conductance = _newton_inputs(case, seed)
    b, area, group = _gpu(b), _gpu(g["area"]), torch.as_tensor(g["group"], device="cuda")
    col, entry, valid = _ell(g["offset"], g["neighbour"])
    w = torch.where(valid, _gpu(g["weight"])[entry], torch.zeros((), dtype=torch.float64, device="cuda"))
    kw, total = conductance * w, conductance * w.sum(1)
    fine = _gpu(_planet(case["level"], case["radius"]).arrays()["area_m2"])

    def flux(t):
        return (kw * (t[col] - t[:, None])).sum(1)

    def mean_of(x):
        return torch.zeros_like(area).index_add_(0, group, fine * x) / area

    def response(h):
        forcing = b + h[group]
        x = torch.minimum(forcing / QUARTIC_A, (forcing / QUARTIC_R) ** 0.25)
        for _ in range(30):
            x = x - (QUARTIC_A * x + QUARTIC_R * x ** 4 - forcing) / (QUARTIC_A + 4.0 * QUARTIC_R * x ** 3)
        return mean_of(x), mean_of(1.0 / (QUARTIC_A + 4.0 * QUARTIC_R * x ** 3))

    def dots(u, v):
        return (u * v).sum()

    h = torch.maximum(torch.zeros_like(area), _gpu(floor))
    for _ in range(12):
        t, slope = response(h)
        lap = flux(t) / area
        if float((lap - h).abs().max()) < 1e-11:
            break
        # J dh = lap - h with dh = dT / slope: A / slope dT - flux(dT) = A (lap - h)
        dt = _conjugate_gradients(lambda y: area / slope * y - flux(y), area / slope + total, area * (lap - h),
                                  torch.zeros_like(area), 1e-13, dots)
        h = torch.maximum(h + dt / slope, _gpu(floor))
    t, _ = response(h)
    return {"source": flux(t) / area, "mean": t}


def _tracer_exact(case, seed):
    g, eddies, flux, mass, tracer = _tracer_inputs(case, seed)
    layers, n = case["layers"], g["nodes"]
    col, entry, valid = _ell(g["offset"], g["neighbour"])
    out = _gpu(flux).view(layers, -1)[:, entry] * valid          # [layers, n, 6] leaving across each face
    eddy = (_gpu(eddies) / (CP * layers))[entry] * valid
    rate = _gpu(mass) / W.SUBSTEP_S
    c0 = _gpu(tracer).view(layers, n)
    rise = -out.sum(2).cumsum(0)                                 # upward flux over each layer's top
    rise[-1] = 0.0
    gain = (-out).clamp(min=0.0) + eddy                          # from the neighbours
    lose = out.clamp(min=0.0) + eddy
    top = rise.clamp(min=0.0)                                    # leaves upward
    drop = (-rise).clamp(min=0.0)                                # comes down from above
    below_in = torch.cat([torch.zeros_like(rise[:1]), top[:-1]])
    below_out = torch.cat([torch.zeros_like(rise[:1]), drop[:-1]])
    diagonal = rate + lose.sum(2) + top + below_out

    def apply(c):
        y = diagonal * c - (gain * c[:, col]).sum(2)
        y[1:] -= below_in[1:] * c[:-1]
        y[:-1] -= drop[:-1] * c[1:]
        return y

    # BiCGSTAB with the diagonal as preconditioner, on the departure from c0; restarted from
    # the true residual until it stops improving
    x = torch.zeros_like(c0)
    b = rate * c0 - apply(c0)
    best, kept = math.inf, x
    for _ in range(6):
        r = b - apply(x)
        norm = float(r.norm() / b.norm())
        if norm < best:
            best, kept = norm, x
        if norm < 1e-14:
            break
        shadow, p, v = r.clone(), torch.zeros_like(r), torch.zeros_like(r)
        rho = alpha = omega = torch.ones((), dtype=torch.float64, device="cuda")
        for k in range(1200):
            new = (shadow * r).sum()
            p = r + new / rho * (alpha / omega) * (p - omega * v)
            rho = new
            ph = p / diagonal
            v = apply(ph)
            alpha = rho / (shadow * v).sum()
            s = r - alpha * v
            sh = s / diagonal
            t = apply(sh)
            omega = (t * s).sum() / (t * t).sum()
            x = x + alpha * ph + omega * sh
            r = s - omega * t
            if k % 25 == 24 and not float(r.norm()) > 1e-15 * float(b.norm()):
                break
        x = torch.nan_to_num(x)
    return {"tracer": (c0 + kept).clamp(min=0.0).reshape(-1)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        mesh = _planet(case["level"], case["radius"])
        rng = np.random.default_rng([seed, 7])
        t0, src = _state_of(case["level"], rng)
        g = _edges_of(mesh, rng) if case["per_edge"] else W.HEAT_CAPACITY * W.DIFFUSIVITY
        t, h = _sub_steps([mesh], [t0], [src], [g])
        return {"temperature": t, "transport": h, "status": None}
    if kind in ("batch", "lane"):
        meshes, t0, src, edges, active = _batch_inputs(case, seed)
        pick = [i for i, a in enumerate(active) if a]
        t, _ = _sub_steps([meshes[i] for i in pick], [t0[i] for i in pick], [src[i] for i in pick],
                          [edges[i] for i in pick])
        return {"temperature": t, "status": None}
    if kind == "multi":
        mesh = _planet(case["level"], case["radius"])
        rng = np.random.default_rng([seed, 13])
        t0, src = _state_of(case["level"], rng)
        k = W.HEAT_CAPACITY * W.DIFFUSIVITY
        out = [_sub_steps([mesh], [t0], [src + rng.normal(0.0, 5.0, len(src))], [k])[0] for _ in range(case["count"])]
        return {"temperature": out, "status": None}
    if kind == "operators":
        return _operators_exact(case, seed)
    if kind == "columns":
        return _columns_exact(case, seed)
    if kind == "newton":
        return _newton_exact(case, seed)
    return _tracer_exact(case, seed)
