"""PageRank (residual push, apps/pr on this engine): the CPU oracle pinned to
the reference's own CUDA build (tests/golden/pr_*), the product's output
writer against the reference format, and gft_pr on the GPU against the
oracle and the golden ranks.

Ranks are float sums accumulated with atomicAdd in whatever order the GPU
runs, in the reference as here, so two runs of the reference itself differ
(by up to 4.2e-5 on the golden graphs, recorded in pr_manifest.json).  The
tolerance used throughout is |a - b| <= RTOL * max(1, |b|), RTOL = 1e-4: the
largest relative difference between the oracle and the reference on the
golden graphs is 5.2e-5, on the 5000-leaf star whose hub holds rank 2298.

A few vertices per run may miss RTOL for a second reason, the reference's:
its crossing test `prev + update > EPSILON && prev < EPSILON`
(apps/pr/kernel.cu:190,222) fails when a residual sum rounds to exactly
EPSILON, and that vertex is never queued again, so the residual it gathers
afterwards never reaches its rank.  Which vertex lands there depends on the
summation order: 0-4 per run on the 32768-vertex R-MAT below in shuffled
sequential schedules of the oracle (which restates that test).  Such a vertex
falls short by what it gathers in the remaining rounds, a few 1e-5 relative.
gft_pr builds each worklist from the residuals above EPSILON instead, so it
has no such vertex, but the oracle and the golden ranks may.  So up to
MAX_STUCK vertices per graph may miss RTOL, and they must still be within
LOOSE_RTOL."""

import json
import re
import subprocess
from pathlib import Path

import numpy as np
import pytest

from test_golden import _graph

RTOL = 1e-4
GOLDEN = Path(__file__).resolve().parent / "golden"
PR_MANIFEST = json.loads((GOLDEN / "pr_manifest.json").read_text())
PR_VALUES = np.load(GOLDEN / "pr_values.npz")
ROOT = Path(__file__).resolve().parent.parent


MAX_STUCK = 8
LOOSE_RTOL = 1e-3


def close(a, b) -> bool:
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    err = np.abs(a - b) / np.maximum(1.0, np.abs(b))
    return bool(np.count_nonzero(err > RTOL) <= MAX_STUCK and np.all(err <= LOOSE_RTOL))


def test_close_allows_only_a_few_stuck_vertices():
    b = np.linspace(1.0, 3.0, 1000)
    a = b.copy()
    a[:MAX_STUCK] -= 3e-4 * b[:MAX_STUCK]
    assert close(a, b)
    a[MAX_STUCK] -= 3e-4 * b[MAX_STUCK]
    assert not close(a, b)  # one too many
    c = b.copy()
    c[0] *= 1 - 2 * LOOSE_RTOL
    assert not close(c, b)  # beyond the loose bound


@pytest.mark.parametrize("key", sorted(PR_MANIFEST))
def test_oracle_pr_matches_reference(gft, orc, key):
    e = PR_MANIFEST[key]
    g = _graph(gft, e["recipe"], e["graph"])
    rank, it = orc.pr(g.row_start, g.edge_dst)
    assert it > 0
    assert close(rank, PR_VALUES[key]), key


def test_pr_golden_noise_is_within_tolerance():
    for key, e in PR_MANIFEST.items():
        assert e["max_abs_diff_between_runs"] <= RTOL * max(1.0, e["rank_max"]), key


def test_product_pr_writer_matches_oracle_text(gft, orc, tmp_path):
    g = _graph(gft, PR_MANIFEST["rmat12w.pr"]["recipe"], "rmat12w")
    rank, _ = orc.pr(g.row_start, g.edge_dst)
    a, b = tmp_path / "a.txt", tmp_path / "b.txt"
    orc.write_pr_output(a, rank)
    gft.write_pr_output(b, rank)
    assert a.read_bytes() == b.read_bytes()


def test_pr_iteration_limit_on_the_oracle(gft, orc):
    g = gft.CSRGraph.road(60, seed=2)
    _, it = orc.pr(g.row_start, g.edge_dst, max_iterations=5)
    assert it == 5


@pytest.mark.gpu
def test_gpu_pr_matches_reference_golden(gft, engine):
    for key, e in sorted(PR_MANIFEST.items()):
        g = _graph(gft, e["recipe"], e["graph"])
        r = engine.pr(g.copy_to_gpu())
        assert close(r["out"].cpu().numpy(), PR_VALUES[key]), key


@pytest.mark.gpu
@pytest.mark.parametrize("tune", [None, {"hub_degree": 32}, {"block_threads": 256, "blocks_per_sm": 4}])
def test_gpu_pr_matches_oracle(gft, orc, engine, tune):
    """Larger graphs, including hubs above the grid-wide split degree (a
    hub's update is stored at its pop and used by the hub phase)."""
    for g in (gft.CSRGraph.rmat(15, 16, seed=12), gft.CSRGraph.road(250, seed=13), gft.CSRGraph.grid(30, 900, 0, 1)):
        want, _ = orc.pr(g.row_start, g.edge_dst)
        r = engine.pr(g.copy_to_gpu(), tune=gft.Tune(**tune) if tune else None)
        assert r["levels"] > 0
        assert close(r["out"].cpu().numpy(), want)


@pytest.mark.gpu
def test_gpu_pr_iteration_limit_and_host_variant(gft, orc, engine):
    g = gft.CSRGraph.road(120, seed=14)
    dg = g.copy_to_gpu()
    r = engine.pr(dg, max_iterations=3)
    assert r["levels"] == 3
    out = np.empty(g.nnodes, dtype=np.float32)
    st = engine.pr_host(dg, out)
    want, _ = orc.pr(g.row_start, g.edge_dst)
    assert st["levels"] > 3 and close(out, want)


def _run_pr_cli(prog: Path, key: str, tmp_path: Path, gft):
    e = PR_MANIFEST[key]
    g = _graph(gft, e["recipe"], e["graph"])
    gr = tmp_path / f"{e['graph']}.gr"
    g.write(gr)
    out = tmp_path / f"{key}.out"
    r = subprocess.run([str(prog), "-o", str(out), str(gr)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert re.search(r"PR took \d+ iterations", r.stdout) and re.search(r"sum: [0-9.]+ \(\d+\)", r.stdout)
    ranks = np.array([float(ln.split()[1]) for ln in out.read_text().splitlines()])
    return ranks


@pytest.mark.gpu
@pytest.mark.parametrize("key", ["rmat14.pr", "road128.pr", "star5000.pr", "disconnected.pr"])
def test_pr_cli_and_dropin_match_reference(gft, tmp_path, key):
    assert close(_run_pr_cli(ROOT / "galoisgpu_b200" / "bin" / "pr", key, tmp_path, gft), PR_VALUES[key])
    dropin = ROOT / "oracle" / "_ref" / "pr_gft"
    if dropin.exists():
        assert close(_run_pr_cli(dropin, key, tmp_path, gft), PR_VALUES[key])


def _pull_cases():
    """Symmetric graphs at the pull path's edges: rows of 0..40 edges (every
    number of lanes per row and its padding), rows around the sizes a warp and
    a whole CTA sum, duplicate edges, self loops."""
    rng = np.random.default_rng(5)
    n = 900
    pairs = [(int(u), int(v)) for u in range(41) for v in rng.choice(np.arange(41, n), size=u, replace=False)]
    yield "rows0to40", n, pairs
    yield "pair", 2, [(0, 1)]
    yield "lonely", 5, []
    yield "dups_loops", 40, [(int(a), int(b)) for a, b in rng.integers(0, 40, size=(300, 2))]
    for leaves in (127, 128, 2047, 2048, 4096, 9000, 70000):
        yield f"star{leaves}", leaves + 3, [(1, i) for i in range(2, leaves + 2)]
    # Graphs on which a sweep moves no rank while all of them are still wrong.
    yield "corona24", *_corona([(i, j) for i in range(24) for j in range(i)], 24, 17)
    yield "corona5000", *_corona([(i, (i + j) % 5000) for i in range(5000) for j in range(1, 24)], 5000, 34)


def _corona(core, n, leaves):
    """The core's edges, and `leaves` vertices on each of its n vertices."""
    return n * (leaves + 1), core + [(v, n + v * leaves + k) for v in range(n) for k in range(leaves)]


def _csr(n, src, dst):
    order = np.argsort(src, kind="stable")
    return np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.uint32), dst[order].astype(np.uint32)


@pytest.mark.gpu
@pytest.mark.parametrize("case", list(_pull_cases()), ids=lambda c: c[0])
def test_gpu_pr_pulled_rows(gft, engine, case):
    """Ranks against the 64-bit solution of the rank equation.  The sweeps end
    at an x(k) whose residual is at most 1e-6 of max(1, rank) at every vertex,
    and at an x(k+1) no further than that from it; a residual's own 32-bit
    rounding (a tree of at most ten additions, the products, the sum) is below
    8e-7 of the rank.  The error, weighted by 1/sqrt(degree), is at most
    1 / (1 - 0.85) times the residual's 2-norm: 1.8e-6 / 0.15 + 1e-6 = 1.3e-5
    of the weighted norm of max(1, rank).  Vertex by vertex the ranks of these
    graphs are within 2.5e-6 (seen, not bounded)."""
    _, n, pairs = case
    a = np.array(pairs, dtype=np.int64).reshape(-1, 2)
    src, dst = np.concatenate([a[:, 0], a[:, 1]]), np.concatenate([a[:, 1], a[:, 0]])
    rs, ed = _csr(n, src, dst)
    deg = np.diff(rs.astype(np.int64)).astype(np.float64)
    want = np.full(n, 0.15)
    for _ in range(250):
        y = want / np.maximum(deg, 1)
        want = 0.15 + 0.85 * np.bincount(dst, weights=y[src], minlength=n) if len(src) else want
    for symmetric in (False, True):
        dg = gft.CSRGraph(rs, ed).copy_to_gpu()
        dg.symmetric = symmetric
        got = engine.pr(dg)["out"].cpu().numpy().astype(np.float64)
        assert np.all(np.abs(got - want) <= 2.5e-6 * np.maximum(1.0, want))
        w = 1 / np.sqrt(np.maximum(deg, 1))
        assert np.linalg.norm(w * (got - want)) <= 1.3e-5 * np.linalg.norm(w * np.maximum(1.0, want))


@pytest.mark.gpu
def test_gpu_pr_pushes_on_graphs_that_are_not_symmetric(gft, orc, engine):
    """A directed graph with hubs, a symmetric one with a single edge
    doubled in one direction (every edge still has a reverse), and a marked
    directed one all take the pushes and match the oracle."""
    rng = np.random.default_rng(6)
    n, m = 20000, 160000
    src = (n * rng.random(m) ** 3).astype(np.int64)
    dst = (n * rng.random(m) ** 2).astype(np.int64)
    g = gft.CSRGraph(*_csr(n, src, dst))
    s2, d2 = np.concatenate([src, dst, src[:1]]), np.concatenate([dst, src, dst[:1]])
    for graph, mark in ((g, False), (gft.CSRGraph(*_csr(n, s2, d2)), False), (g, True)):
        dg = graph.copy_to_gpu()
        dg.symmetric = mark
        r = engine.pr(dg)
        want, _ = orc.pr(graph.row_start, graph.edge_dst)
        assert close(r["out"].cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("claimed", [-6000, -1, 0, 100])
def test_gpu_pr_wrapped_graph_with_a_wrong_edge_count(gft, engine, claimed):
    """A wrapped symmetric graph whose edge count says fewer than its rows
    hold (every row's edges are there): the sweeps, whose buffers are sized by
    the count, leave it to the pushes.  With spare entries behind the edges,
    and with the right count, the ranks are the same."""
    import ctypes as C

    import torch

    g = gft.CSRGraph.grid(80, 80)
    want = engine.pr(g.copy_to_gpu())["out"].cpu().numpy()
    rs = torch.from_numpy(g.row_start.astype(np.int32)).cuda()
    dst = torch.zeros(g.nedges + 128, dtype=torch.int32, device="cuda")
    dst[: g.nedges] = torch.from_numpy(g.edge_dst.astype(np.int32))
    h = C.c_void_p()
    assert gft.load().gft_graph_wrap(0, g.nnodes, g.nedges + claimed, C.c_void_p(rs.data_ptr()),
                                     C.c_void_p(dst.data_ptr()), None, C.byref(h)) == 0
    r = engine.pr(gft.DeviceGraph(h, 0))
    assert close(r["out"].cpu().numpy(), want)
    swept = r["pushes"] == r["levels"] * g.nnodes
    assert claimed > 0 or swept == (claimed == 0)


@pytest.mark.gpu
def test_gpu_pr_on_a_directed_graph_takes_no_sweep_workspace(gft):
    """The pushes need 16 bytes a vertex and the hub list, the sweeps 46 and
    4.5 an edge."""
    rng = np.random.default_rng(7)
    n, m = 30000, 600000
    rs, ed = _csr(n, rng.integers(0, n, m), rng.integers(0, n, m))
    e = gft.Engine(0)
    try:
        before = e.scratch_bytes()
        e.pr(gft.CSRGraph(rs, ed).copy_to_gpu())
        assert e.scratch_bytes() - before <= 16 * n + 8 * (m // 256 + 1) + 4096
    finally:
        e.close()


@pytest.mark.gpu
def test_gpu_pr_without_room_for_the_sweeps(gft, engine):
    """With device memory all but full a symmetric graph takes the pushes, and
    the engine keeps the scratch that it had."""
    import torch

    dg = gft.DeviceGraph.generate("rmat", seed=3, scale=20, edge_factor=16)  # sweeps: about 230 MB, pushes: 17 MB
    want = engine.pr(dg)
    assert want["edges_scanned"] == want["levels"] * dg.nedges  # swept
    e = gft.Engine(0)
    out = torch.empty(dg.nnodes, dtype=torch.float32, device="cuda")
    e.sssp(dg)  # 20 bytes a vertex and more of scratch; the pushes need 16
    e.pr(dg, out=out, max_iterations=2)  # the pushes' kernel is loaded
    had = e.scratch_bytes()
    assert had < 100 << 20
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (128 << 20), dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            r = e.pr(dg, out=out)
            assert r["edges_scanned"] != r["levels"] * dg.nedges
            assert e.scratch_bytes() == had
    finally:
        del fill
        torch.cuda.empty_cache()
    # The pushes' 32-bit sums: 7.6e-5 (2-norm) from the solution on RMAT-22.
    a, b = r["out"].double(), want["out"].double()
    assert float((a - b).norm() / b.norm()) <= 3e-4
    r = e.pr(dg, out=out)
    assert r["edges_scanned"] == r["levels"] * dg.nedges
    e.close()
