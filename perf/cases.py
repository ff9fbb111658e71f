"""Performance cases of the traversal engine: what a program that uses it asks
for, through the Python API (galoisgpu_b200), over the range of graphs that
the package's workloads, benchmark and tests cover.

A case names an application (``app``), a seeded synthetic graph and the
application's options.  Graphs are the package's own: road-like grids (uniform
low degree, thousands of levels at the large end) and plain grids, which stand
for road networks and meshes, and symmetrised R-MAT graphs (skewed degrees, a
handful of levels), which stand for social and web graphs.  The seed draws the
graph and the sources.

``marked`` False is a graph as it comes from a file or from arrays: its
owner has not said that it is symmetric, so BFS stays top-down and connected
components joins every edge.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import galoisgpu_b200 as gft
from galoisgpu_b200 import workloads

ROAD_DELTA = 20000  # tuned bucket width of the road workloads
RMAT_DELTA = 10000  # tuned bucket width of the R-MAT workloads
BATCH_DELTA = 40000  # bucket width of the mixed batch
MSBFS_LEVELS = 24  # planes kept by a multi-source query on an R-MAT graph


def road(app, name=None, *, side, marked=True, **kw):
    return {**({"name": name} if name else {}), "app": app, "kind": "road", "side": side, "marked": marked, **kw}


def grid(app, name=None, *, rows, cols, marked=True, **kw):
    return {**({"name": name} if name else {}), "app": app, "kind": "grid", "rows": rows, "cols": cols,
            "marked": marked, **kw}


def rmat(app, name=None, *, scale, edge_factor, marked=True, **kw):
    return {**({"name": name} if name else {}), "app": app, "kind": "rmat", "scale": scale,
            "edge_factor": edge_factor, "marked": marked, **kw}


def listed():
    return [
        # The smallest graphs of the batch workload, asked one at a time: latency.
        road("bfs", "bfs-road-33", side=33, parent=False),
        # The benchmark's small high-diameter BFS: hundreds of tiny levels.
        grid("bfs", "bfs-grid-256", rows=256, cols=256, parent=False),
        # The benchmark's large BFS, with bottom-up levels.
        rmat("bfs", "bfs-rmat-24", scale=24, edge_factor=16, parent=False),
        # A graph loaded from a file (not marked symmetric) and a BFS tree wanted: top-down.
        rmat("bfs", "bfs-rmat-21-file", scale=21, edge_factor=16, marked=False, parent=True),
        # End to end: several sources on a road network, levels in host memory.
        road("bfs_host", "bfs-host-road-1021", side=1021, sources=4),
        # The benchmark's headline: shortest paths on a continental road network.
        road("sssp", "sssp-road-4096", side=4096),
        # Shortest paths on a social graph (the tuned R-MAT workload).
        rmat("sssp", "sssp-rmat-20", scale=20, edge_factor=16),
        # Many sources on one graph (distance sketches, closeness estimates).
        rmat("msbfs", "msbfs-rmat-20", scale=20, edge_factor=16, sources=256),
        # A mixed batch of queries over graphs of uneven sizes, one launch.
        {"name": "batch-48", "app": "batch", "queries": 48, "vmax": 2000000},
        # Connected components of a social graph.
        rmat("cc", "cc-rmat-23", scale=23, edge_factor=16),
        # Ranks of a web graph.
        rmat("pr", "pr-rmat-22", scale=22, edge_factor=16),
        # An independent set of a mesh (colouring, coarsening).
        road("mis", "mis-road-2047", side=2047),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: an application, then a graph of its range."""
    app = rng.choice(["bfs", "bfs", "bfs_host", "sssp", "sssp", "msbfs", "batch", "cc", "pr", "mis"])
    marked = rng.random() < 0.7
    if app == "batch":
        return {"app": app, "queries": rng.randint(6, 48), "vmax": _log_int(rng, 20000, 2000000)}
    if app == "msbfs":
        return rmat(app, scale=rng.randint(12, 20), edge_factor=rng.choice([8, 12, 16]), marked=marked,
                    sources=rng.choice([1, 17, 32, 64, 100, 128, 200, 256]))
    if app == "bfs":
        kind = rng.choice(["road", "grid", "rmat"])
        opts = {"parent": rng.random() < 0.4}
    elif app in ("bfs_host", "sssp"):
        kind = rng.choice(["road", "rmat"])
        opts = {"sources": rng.randint(1, 6)} if app == "bfs_host" else {}
    else:
        kind = rng.choice(["road", "rmat"])
        opts = {}
    if kind == "grid":
        return grid(app, rows=_log_int(rng, 24, 1500), cols=_log_int(rng, 24, 1500), marked=marked, **opts)
    if kind == "road":
        top = {"bfs": 3000, "bfs_host": 1100, "sssp": 4000, "cc": 4096, "pr": 2048, "mis": 4096}[app]
        return road(app, side=_log_int(rng, 32, top), marked=marked, **opts)
    top = {"bfs": 23, "bfs_host": 20, "sssp": 21, "cc": 23, "pr": 21, "mis": 23}[app]
    return rmat(app, scale=rng.randint(11, top), edge_factor=rng.choice([8, 12, 16]), marked=marked, **opts)


def _graph(case, seed):
    if case["kind"] == "road":
        g = gft.DeviceGraph.generate("road", seed=seed, side=case["side"], max_weight=10000)
    elif case["kind"] == "grid":
        g = gft.DeviceGraph.generate("grid", seed=seed, rows=case["rows"], cols=case["cols"])
    else:
        g = gft.DeviceGraph.generate("rmat", seed=seed, scale=case["scale"], edge_factor=case["edge_factor"],
                                     max_weight=255 if case["app"] == "sssp" else 0)
    if not case["marked"]:
        g.symmetric = False
    return g


def prepare(case, seed):
    """The resident graph, the engine, the sources and the result buffers."""
    app = case["app"]
    engine = gft.Engine(0)
    if app == "batch":
        queries = []
        for i, spec in enumerate(workloads.batch_specs(case["queries"], vmax=case["vmax"])):
            g = workloads.build({**spec, "seed": spec["seed"] + 10000 * seed})
            src = g.pick_sources(seed, 1)[0]
            q = {"graph": g, "app": "bfs" if i % 4 == 3 else "sssp", "src": src, "delta": BATCH_DELTA,
                 "out": torch.empty(g.nnodes, dtype=torch.int32, device="cuda:0")}
            queries.append(q)
        return {"app": app, "batch": gft.Batch(engine, queries), "outs": [q["out"] for q in queries]}
    g = _graph(case, seed)
    state = {"app": app, "engine": engine, "graph": g}
    if app in ("cc", "mis"):
        state["out"] = torch.empty(g.nnodes, dtype=torch.int32, device="cuda:0")
    elif app == "pr":
        state["out"] = torch.empty(g.nnodes, dtype=torch.float32, device="cuda:0")
    elif app == "msbfs":
        state["sources"] = g.pick_sources(seed, case["sources"])
        state["symmetric"] = case["marked"]
        plane = gft.load().gft_msbfs_plane_bytes(g.nnodes, case["sources"])
        state["wanted"] = [case["sources"] * i // 8 for i in range(min(8, case["sources"]))]
        state["planes"] = torch.empty(MSBFS_LEVELS * plane // 4, dtype=torch.int32, device="cuda:0")
    elif app == "bfs_host":
        state["sources"] = g.pick_sources(seed, case["sources"])
        rows = torch.empty((case["sources"], g.nnodes), dtype=torch.int32, pin_memory=True)
        state["rows"], state["host"] = rows, rows.numpy()
    else:
        state["source"] = g.pick_sources(seed, 1)[0]
        state["out"] = torch.empty(g.nnodes, dtype=torch.int32, device="cuda:0")
        state["parent"] = torch.empty_like(state["out"]) if case.get("parent") else None
        state["delta"] = ROAD_DELTA if case["kind"] != "rmat" else RMAT_DELTA
    return state


def run(state):
    """One query, batch or end-to-end call.  A BFS tree is written but not
    returned: any valid parent may stand in it, so two runs differ.  A
    multi-source query's planes go back as levels of up to eight of its
    sources."""
    app = state["app"]
    if app == "batch":
        state["batch"].run()
        return state["outs"]
    eng, g = state["engine"], state["graph"]
    if app == "bfs":
        return eng.bfs(g, state["source"], out=state["out"], parent=state["parent"])["out"]
    if app == "sssp":
        return eng.sssp(g, state["source"], delta=state["delta"], out=state["out"])["out"]
    if app == "bfs_host":
        eng.bfs_host_many(g, state["sources"], state["host"])
        return state["host"]
    if app == "msbfs":
        r = eng.msbfs(g, state["sources"], max_levels=MSBFS_LEVELS, symmetric=state["symmetric"],
                      planes=state["planes"])
        return [r["levels_of"](i) for i in state["wanted"]]
    if app == "cc":
        r = eng.cc(g, out=state["out"])
        return {"labels": r["out"], "components": r["components"]}
    if app == "pr":
        return eng.pr(g, out=state["out"])["out"]
    r = eng.mis(g, out=state["out"])
    return {"state": r["out"], "size": r["vertices_reached"]}


def _size(case):
    """(vertices, edges): exact for grids, near for roads and R-MAT (whose
    deleted and duplicate edges are drawn)."""
    if case["kind"] == "grid":
        r, c = case["rows"], case["cols"]
        return r * c, 2 * (r * (c - 1) + c * (r - 1))
    if case["kind"] == "road":
        n = case["side"] ** 2
        return n, int(3.8 * n)
    n = 1 << case["scale"]
    return n, int(2 * 0.95 * case["edge_factor"] * n)


def work(case):
    """The graph read once and the results written once."""
    app = case["app"]
    if app == "batch":
        total = 0
        for i, s in enumerate(workloads.batch_specs(case["queries"], vmax=case["vmax"])):
            m = (3.8 if s["kind"] == "road" else 15.2) * s["nodes"]
            total += 8 * s["nodes"] + (4 if i % 4 == 3 else 8) * m
        return {"bytes": total, "flops": 0}
    n, m = _size(case)
    graph = 4 * (n + 1) + 4 * m
    if app == "sssp":
        return {"bytes": graph + 4 * m + 4 * n, "flops": 0}
    if app == "bfs_host":
        return {"bytes": case["sources"] * (graph + 4 * n), "flops": 0}
    if app == "msbfs":
        words = 1 << max(0, math.ceil(math.log2(math.ceil(case["sources"] / 32))))
        return {"bytes": graph + 8 * 4 * n * words + 4 * n * min(8, case["sources"]), "flops": 0}
    return {"bytes": graph + 4 * n * (2 if case.get("parent") else 1), "flops": 2 * m if app == "pr" else 0}


def tolerance(case):
    """Levels, distances, labels and sets are whole numbers that do not depend
    on the schedule.  Ranks are 32-bit sums in schedule order, cut off where a
    residual falls below 1e-6: on the largest graph here they are 7.6e-5
    (2-norm) and 1.7e-4 (largest) from the 64-bit solution, almost all of it
    additions of small updates to a hub's large residual.  Another order of
    the sums may lie anywhere within that error; four times it is allowed."""
    if case["app"] == "pr":
        return {"rel": 3e-4, "max": 7e-4}
    return "exact"


def exact(case, seed):
    """Ranks in 64 bits: the solution of rank = (1 - a) + a * sum over
    in-neighbours of rank / out-degree (the limit of the residual pushes), on
    these symmetric graphs, by the power iteration to its fixed point."""
    if case["app"] != "pr":
        return None
    a = 0.85
    host = _graph(case, seed).download()
    rows = torch.from_numpy(host.row_start.astype(np.int64)).cuda()
    cols = torch.from_numpy(host.edge_dst.astype(np.int64)).cuda()
    n = host.nnodes
    deg = (rows[1:] - rows[:-1]).double()
    adj = torch.sparse_csr_tensor(rows, cols, torch.ones(cols.numel(), dtype=torch.float64, device="cuda"),
                                  size=(n, n))
    inv = torch.where(deg > 0, 1.0 / deg.clamp(min=1), torch.zeros_like(deg))
    x = torch.full((n,), 1 - a, dtype=torch.float64, device="cuda")
    for _ in range(400):
        y = (1 - a) + a * (adj @ (x * inv).unsqueeze(1)).squeeze(1)
        done = float((y - x).abs().max()) < 1e-11 * float(y.abs().max())
        x = y
        if done:
            break
    return x
