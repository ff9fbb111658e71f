"""GPU parity: libgft BFS / SSSP (through the C ABI) against the CPU oracle,
bit for bit, plus parent-tree validity, on hand graphs and seeded synthetic
graphs at sizes the oracle finishes in seconds."""

import numpy as np
import pytest

from graphs import hand_cases

pytestmark = pytest.mark.gpu

TUNES = [
    dict(),  # small graphs run on one CTA, larger ones on the whole grid
    dict(block_threads=256, blocks_per_sm=4, max_blocks=1 << 30),  # always the grid
    dict(block_threads=1024, blocks_per_sm=1, max_blocks=1 << 30),
    dict(hub_degree=32, max_blocks=1 << 30),  # every vertex of degree >= 32 goes through the grid-wide hub phase
    dict(max_blocks=1, hub_degree=32),  # always one CTA
    dict(queue_tile=64, warp_degree=8, max_blocks=1 << 30),  # small push buffers, warps from degree 8
    dict(block_threads=512, queue_tile=256, warp_degree=128, max_blocks=1 << 30),  # edge lists < 128 flattened
]
TUNE_IDS = ["auto", "grid256x4", "grid1024x1", "grid-hub32", "one-cta", "tile64-warp8", "tile256-warp128"]


def _sources(n):
    return sorted({0, n // 2, n - 1})


def _run_bfs(gft, engine, dg, src, tune=None):
    import torch

    par = torch.empty(dg.nnodes, dtype=torch.int32, device="cuda")
    r = engine.bfs(dg, src, parent=par, tune=gft.Tune(**tune) if tune else None)
    return r["out"].cpu().numpy(), r["parent"].cpu().numpy().view(np.uint32), r


def _run_sssp(gft, engine, dg, src, delta, tune=None):
    import torch

    par = torch.empty(dg.nnodes, dtype=torch.int32, device="cuda")
    r = engine.sssp(dg, src, delta=delta, parent=par, tune=gft.Tune(**tune) if tune else None)
    return r["out"].cpu().numpy(), r["parent"].cpu().numpy().view(np.uint32), r


@pytest.mark.parametrize("case", hand_cases(), ids=lambda c: c[0])
def test_hand_graphs_bfs_sssp(gft, orc, engine, case):
    name, rs, dst, w = case
    g = gft.CSRGraph(rs, dst, w)
    dg = g.copy_to_gpu()
    for src in _sources(g.nnodes):
        want = orc.bfs(rs, dst, src)
        got, par, _ = _run_bfs(gft, engine, dg, src)
        np.testing.assert_array_equal(got, want)
        assert orc.check_tree(rs, dst, None, src, got, par) == 0
        for delta in (1, 7, 10000):
            want = orc.sssp(rs, dst, w, src)
            got, par, _ = _run_sssp(gft, engine, dg, src, delta)
            np.testing.assert_array_equal(got, want)
            if w is not None and (w > 0).all():
                assert orc.check_tree(rs, dst, w, src, got, par) == 0


@pytest.mark.parametrize("tune", TUNES, ids=lambda t: ",".join(f"{k}={v}" for k, v in t.items()) or "default")
def test_grid_bfs_closed_form(gft, orc, engine, tune):
    g = gft.CSRGraph.grid(256, 256)
    dg = g.copy_to_gpu()
    got, par, st = _run_bfs(gft, engine, dg, 0, tune)
    r, c = np.divmod(np.arange(g.nnodes), 256)
    np.testing.assert_array_equal(got, (r + c).astype(np.int32))
    assert orc.check_tree(g.row_start, g.edge_dst, None, 0, got, par) == 0
    assert st["levels"] == 511


@pytest.mark.parametrize("tune", TUNES, ids=lambda t: ",".join(f"{k}={v}" for k, v in t.items()) or "default")
def test_rmat_bfs_sssp(gft, orc, engine, tune):
    g = gft.CSRGraph.rmat(16, 16, seed=3, max_weight=255)
    dg = g.copy_to_gpu()
    for src in g.pick_sources(2, 3):
        want = orc.bfs(g.row_start, g.edge_dst, src)
        got, par, _ = _run_bfs(gft, engine, dg, src, tune)
        np.testing.assert_array_equal(got, want)
        assert orc.check_tree(g.row_start, g.edge_dst, None, src, got, par) == 0
        want = orc.sssp(g.row_start, g.edge_dst, g.edge_data, src)
        for delta in (16, 255, 10000):
            got, par, _ = _run_sssp(gft, engine, dg, src, delta, tune)
            np.testing.assert_array_equal(got, want)
            assert orc.check_tree(g.row_start, g.edge_dst, g.edge_data, src, got, par) == 0


@pytest.mark.parametrize("side", [362, 363], ids=["bitmap-in-shared", "bitmap-in-global"])
def test_one_cta_bfs_either_side_of_the_shared_bitmap_limit(gft, orc, engine, side):
    """A one-CTA BFS keeps its visited bitmap in shared memory for graphs of
    at most 2^17 vertices (362^2 = 131,044) and in global memory above
    (363^2 = 131,769); levels and parent trees match the oracle on both
    sides, top-down and with the direction switch."""
    g = gft.CSRGraph.road(side, seed=7)
    dg = g.copy_to_gpu()
    for src in g.pick_sources(8, 2):
        want = orc.bfs(g.row_start, g.edge_dst, src)
        for tune in (dict(max_blocks=1), dict(max_blocks=1, direction=1)):
            got, par, _ = _run_bfs(gft, engine, dg, src, tune)
            np.testing.assert_array_equal(got, want)
            assert orc.check_tree(g.row_start, g.edge_dst, None, src, got, par) == 0


def test_one_cta_bfs_frontier_beyond_the_shared_queue_head(gft, orc, engine):
    """Small uniform-degree graphs run a thread per frontier vertex on one
    CTA, with the first 8,192 entries of each frontier queue in shared
    memory and the rest in global memory.  A random graph of 120,000
    vertices and degree <= 32 has levels of tens of thousands of vertices,
    so both parts of the queue carry vertices; levels and parents stay
    exact."""
    rng = np.random.default_rng(12)
    n, m = 120_000, 240_000
    u = rng.integers(0, n, m, dtype=np.int64)
    v = rng.integers(0, n, m, dtype=np.int64)
    keep = u != v
    a = np.concatenate([u[keep], v[keep]])
    b = np.concatenate([v[keep], u[keep]])
    key = np.unique(a * n + b)
    src_of, dst = (key // n).astype(np.uint32), (key % n).astype(np.uint32)
    rs = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(np.bincount(src_of, minlength=n), out=rs[1:])
    assert int(np.diff(rs.astype(np.int64)).max()) <= 32 and len(dst) <= 1 << 19
    g = gft.CSRGraph(rs, dst, None)
    dg = g.copy_to_gpu()
    for src in g.pick_sources(13, 2):
        want = orc.bfs(rs, dst, src)
        reached = want != np.iinfo(np.int32).max
        assert np.bincount(want[reached]).max() > 16384
        for tune in (None, dict(max_blocks=1)):
            got, par, r = _run_bfs(gft, engine, dg, src, tune)
            np.testing.assert_array_equal(got, want)
            assert orc.check_tree(rs, dst, None, src, got, par) == 0
            assert r["grid_blocks"] == 1
            assert r["vertices_reached"] == int(reached.sum()) - 1  # the source is not counted


def test_one_cta_bfs_on_graphs_with_odd_cycles(gft, orc, engine):
    """Random graphs of degree <= 4 (the one-CTA kernel's per-vertex slot
    path; 131,000 vertices take the 1024-thread CTA) and <= 9 (some
    vertices through the CSR), full of odd cycles, so that a level's
    vertices also claim one another's neighbours: levels, the level count
    and the reached count equal the oracle's, and parent trees are valid,
    with and without the parent output."""
    import torch

    rng = np.random.default_rng(31)
    for n, cap in ((30_000, 4), (50_000, 9), (131_000, 4)):
        u = rng.integers(0, n, 3 * n)
        v = rng.integers(0, n, 3 * n)
        key = np.unique(np.concatenate([u * n + v, v * n + u]))
        key = key[key // n != key % n]
        src_of, dst = key // n, key % n
        deg = np.bincount(src_of, minlength=n)
        first = np.concatenate([[0], np.cumsum(deg)[:-1]])
        rank = np.arange(len(key)) - first[src_of]
        keep = rank < cap
        pairs = set(zip(src_of[keep].tolist(), dst[keep].tolist()))
        sym = np.array(sorted(p for p in pairs if (p[1], p[0]) in pairs), dtype=np.int64)
        rs = np.zeros(n + 1, dtype=np.uint32)
        np.cumsum(np.bincount(sym[:, 0], minlength=n), out=rs[1:])
        g = gft.CSRGraph(rs, sym[:, 1].astype(np.uint32), None)
        dg = g.copy_to_gpu()
        for src in g.pick_sources(5, 3):
            want = orc.bfs(g.row_start, g.edge_dst, src)
            got, par, r = _run_bfs(gft, engine, dg, src)
            np.testing.assert_array_equal(got, want)
            assert orc.check_tree(g.row_start, g.edge_dst, None, src, got, par) == 0
            assert r["grid_blocks"] == 1
            reached = want != np.iinfo(np.int32).max
            assert r["levels"] == int(want[reached].max()) + 1
            assert r["vertices_reached"] == int(reached.sum()) - 1
            out = torch.empty(dg.nnodes, dtype=torch.int32, device="cuda")
            np.testing.assert_array_equal(engine.bfs(dg, src, out=out)["out"].cpu().numpy(), want)


def _wrap(gft, rs, dst):
    """A device graph over caller-owned device arrays (no copy, no BFS slots)."""
    import ctypes as C

    import torch

    d_rs = torch.from_numpy(rs.astype(np.int32)).cuda()
    d_dst = torch.from_numpy(dst.astype(np.int32)).cuda()
    h = C.c_void_p()
    assert gft.load().gft_graph_wrap(0, len(rs) - 1, len(dst), C.c_void_p(d_rs.data_ptr()),
                                     C.c_void_p(d_dst.data_ptr()), None, C.byref(h)) == 0
    return gft.DeviceGraph(h, 0), (d_rs, d_dst)


def test_one_cta_bfs_on_a_wrapped_graph(gft, orc, engine):
    """A wrapped graph has no per-vertex slots, so the one-CTA kernel reads
    every vertex through the CSR: a grid (degree <= 4) and a random graph
    of degree <= 12 give the oracle's levels and valid parent trees."""
    rng = np.random.default_rng(4)
    grid = gft.CSRGraph.grid(90, 110, 0, 1)
    n = 20_000
    u = rng.integers(0, n, 50_000)
    v = rng.integers(0, n, 50_000)
    key = np.unique(np.concatenate([u * n + v, v * n + u]))
    key = key[key // n != key % n]
    src_of, dst = key // n, (key % n).astype(np.uint32)
    deg = np.bincount(src_of, minlength=n)
    first = np.concatenate([[0], np.cumsum(deg)[:-1]])
    keep = np.arange(len(key)) - first[src_of] < 12  # at most 12 edges a vertex
    src_of, dst = src_of[keep], dst[keep]
    rs = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(np.bincount(src_of, minlength=n), out=rs[1:])
    for g_rs, g_dst in ((grid.row_start, grid.edge_dst), (rs, dst)):
        dg, keep_alive = _wrap(gft, g_rs, g_dst)
        for src in (0, len(g_rs) // 2):
            want = orc.bfs(g_rs, g_dst, src)
            got, par, r = _run_bfs(gft, engine, dg, src)
            np.testing.assert_array_equal(got, want)
            assert orc.check_tree(g_rs, g_dst, None, src, got, par) == 0
            assert r["grid_blocks"] == 1
        dg.free()


def test_one_cta_bfs_reports_a_destination_outside_the_graph(gft, engine):
    """An edge leaving the graph (only possible in wrapped, caller-owned
    arrays) ends the one-CTA BFS with GFT_ERR_FORMAT, not a stray write."""
    g = gft.CSRGraph.grid(40, 40, 0, 1)
    dst = g.edge_dst.copy()
    dst[len(dst) // 2] = g.nnodes + 5
    dg, keep_alive = _wrap(gft, g.row_start, dst)
    with pytest.raises(gft.GftError) as ei:
        engine.bfs(dg, 0)
    assert ei.value.status_name == "GFT_ERR_FORMAT"
    dg.free()


def test_road_sssp(gft, orc, engine):
    g = gft.CSRGraph.road(512, seed=1)
    dg = g.copy_to_gpu()
    for src in g.pick_sources(1, 2):
        want = orc.sssp(g.row_start, g.edge_dst, g.edge_data, src)
        for delta in (1000, 10000, 100000):
            got, par, st = _run_sssp(gft, engine, dg, src, delta)
            np.testing.assert_array_equal(got, want)
            assert orc.check_tree(g.row_start, g.edge_dst, g.edge_data, src, got, par) == 0


@pytest.mark.parametrize("cta_small", [2**32 - 1, 64, 2048, 1 << 22], ids=["never", "64", "2048", "all"])
def test_sssp_small_iterations_on_one_cta(gft, orc, engine, cta_small):
    """Grid launches hand runs of small iterations to the first CTA and take
    the loop state back at a grid barrier: distances and the parent tree
    stay exact whether that never happens, happens for tiny piles only, or
    for every iteration (hubs of degree >= 32 included)."""
    for g, hub in ((gft.CSRGraph.road(400, seed=31), 0), (gft.CSRGraph.rmat(16, 16, seed=32, max_weight=255), 32),
                   (gft.CSRGraph.grid(12, 4000, 2, 50), 0)):
        dg = g.copy_to_gpu()
        tune = dict(max_blocks=1 << 30, cta_small=cta_small, hub_degree=hub)
        for src in g.pick_sources(33, 2):
            want = orc.sssp(g.row_start, g.edge_dst, g.edge_data, src)
            for delta in (100, 10000):
                got, par, _ = _run_sssp(gft, engine, dg, src, delta, tune)
                np.testing.assert_array_equal(got, want)
                assert orc.check_tree(g.row_start, g.edge_dst, g.edge_data, src, got, par) == 0


@pytest.mark.parametrize("fuse", [32, 256, 1 << 20], ids=["fuse32", "fuse256", "fuse-unbounded"])
@pytest.mark.parametrize("mode", [dict(max_blocks=1 << 30), dict(max_blocks=1), dict(max_blocks=1 << 30, hub_degree=32)],
                         ids=["grid", "one-cta", "grid-hub32"])
def test_sssp_bucket_fusion(gft, orc, engine, fuse, mode):
    """Warps that expand the near vertices they found in the same iteration
    (claimed by swapping the near tag, so later improvements queue them
    again) give the same distances and a valid parent tree."""
    for g in (gft.CSRGraph.road(400, seed=41), gft.CSRGraph.rmat(16, 16, seed=42, max_weight=255),
              gft.CSRGraph.grid(12, 4000, 3, 50)):
        dg = g.copy_to_gpu()
        for src in g.pick_sources(43, 2):
            want = orc.sssp(g.row_start, g.edge_dst, g.edge_data, src)
            for delta in (100, 10000):
                got, par, _ = _run_sssp(gft, engine, dg, src, delta, dict(mode, fuse_budget=fuse))
                np.testing.assert_array_equal(got, want)
                assert orc.check_tree(g.row_start, g.edge_dst, g.edge_data, src, got, par) == 0


def test_unweighted_sssp_is_zero_weight(gft, orc, engine):
    """An unweighted .gr has weight 0 everywhere (calloc'd edge_data in the
    reference), so every reached vertex has distance 0."""
    g = gft.CSRGraph.rmat(12, 8, seed=5)
    dg = g.copy_to_gpu()
    src = g.pick_sources(1, 1)[0]
    got, _, _ = _run_sssp(gft, engine, dg, src, 10000)
    np.testing.assert_array_equal(got, orc.sssp(g.row_start, g.edge_dst, None, src))


@pytest.mark.parametrize(
    "kind,kw,host",
    [
        ("grid", dict(rows=100, cols=37, max_weight=1), lambda g: g.CSRGraph.grid(100, 37, 1, 1)),
        ("road", dict(side=300), lambda g: g.CSRGraph.road(300, seed=1)),
        ("rmat", dict(scale=14, edge_factor=16, max_weight=255), lambda g: g.CSRGraph.rmat(14, 16, seed=1, max_weight=255)),
        ("rmat", dict(scale=12, edge_factor=8), lambda g: g.CSRGraph.rmat(12, 8, seed=1)),
    ],
)
def test_device_generator_matches_host(gft, kind, kw, host):
    dg = gft.DeviceGraph.generate(kind, seed=1, **kw)
    a = dg.download()
    b = host(gft)
    np.testing.assert_array_equal(a.row_start, b.row_start)
    np.testing.assert_array_equal(a.edge_dst, b.edge_dst)
    if b.edge_data is None:
        assert a.edge_data is None
    else:
        np.testing.assert_array_equal(a.edge_data, b.edge_data)


def test_host_api_matches_device_api(gft, orc, engine):
    g = gft.CSRGraph.road(128, seed=4)
    dg = g.copy_to_gpu()
    out = np.empty(g.nnodes, dtype=np.int32)
    par = np.empty(g.nnodes, dtype=np.uint32)
    engine.sssp_host(dg, 5, out, parent=par)
    np.testing.assert_array_equal(out, orc.sssp(g.row_start, g.edge_dst, g.edge_data, 5))
    assert orc.check_tree(g.row_start, g.edge_dst, g.edge_data, 5, out, par) == 0
    engine.bfs_host(dg, 5, out, parent=par)
    np.testing.assert_array_equal(out, orc.bfs(g.row_start, g.edge_dst, 5))
    assert orc.check_tree(g.row_start, g.edge_dst, None, 5, out, par) == 0


@pytest.mark.parametrize("app", ["bfs", "sssp"])
def test_host_many_rows_equal_single_queries(gft, orc, engine, app):
    """The many-query host calls copy each query's results back while the
    next query runs, through two device buffers: every row equals the oracle
    (and so the single-query host call), in pinned and pageable memory, for
    five sources (both buffers reused), on the grid and on one CTA; no
    sources is a no-op, and a bad source fails before anything runs."""
    import torch

    for g in (gft.CSRGraph.road(700, seed=6), gft.CSRGraph.road(100, seed=6)):
        dg = g.copy_to_gpu()
        srcs = g.pick_sources(21, 5)
        want = [orc.sssp(g.row_start, g.edge_dst, g.edge_data, s) if app == "sssp" else
                orc.bfs(g.row_start, g.edge_dst, s) for s in srcs]
        run = engine.sssp_host_many if app == "sssp" else engine.bfs_host_many
        pinned = torch.empty((len(srcs), g.nnodes), dtype=torch.int32, pin_memory=True).numpy()
        for out in (pinned, np.empty((len(srcs), g.nnodes), dtype=np.int32)):
            out.fill(-7)
            st = run(dg, srcs, out)
            assert len(st) == len(srcs)
            for i in range(len(srcs)):
                np.testing.assert_array_equal(out[i], want[i])
                assert st[i]["levels"] > 0 and st[i]["kernel_ms"] > 0
        assert run(dg, [], pinned[:0]) == []
        pinned.fill(-7)
        with pytest.raises(gft.GftError, match="INVALID_ARG"):
            run(dg, [srcs[0], g.nnodes], pinned)
        assert (pinned == -7).all()


def test_barrier_timeout_is_reported_and_engine_recovers(gft, orc, engine):
    """One CTA never arrives at the first grid barrier (test hook); the other
    CTAs' bounded waits expire, the call returns GFT_ERR_TIMEOUT and the
    context stays usable."""
    g = gft.CSRGraph.grid(64, 64)
    dg = g.copy_to_gpu()
    with pytest.raises(gft.GftError) as ei:
        engine.bfs(dg, 0, tune=gft.Tune(timeout_ms=200, test_skip_block=1))
    assert ei.value.status_name == "GFT_ERR_TIMEOUT"
    with pytest.raises(gft.GftError) as ei:
        engine.sssp(dg, 0, tune=gft.Tune(timeout_ms=200, test_skip_block=0))
    assert ei.value.status_name == "GFT_ERR_TIMEOUT"
    r = engine.bfs(dg, 0)
    np.testing.assert_array_equal(r["out"].cpu().numpy(), orc.bfs(g.row_start, g.edge_dst, 0))


def test_queue_tile_must_be_built(gft, engine):
    """Queue tiles are 64, 128 or 256 entries a warp; SSSP at 1024 threads
    takes at most 128 (its near and far buffers share 48 KB of static
    shared memory).  Anything else is GFT_ERR_INVALID_ARG, not a launch."""
    g = gft.CSRGraph.rmat(12, 8, seed=3, max_weight=255)
    dg = g.copy_to_gpu()
    for app, tune in (("bfs", dict(queue_tile=96)), ("sssp", dict(block_threads=1024, queue_tile=256)),
                      ("sssp", dict(queue_tile=512))):
        t = gft.Tune(max_blocks=1 << 30, **tune)
        with pytest.raises(gft.GftError) as ei:
            engine.sssp(dg, 0, tune=t) if app == "sssp" else engine.bfs(dg, 0, tune=t)
        assert ei.value.status_name == "GFT_ERR_INVALID_ARG"
    ok = engine.sssp(dg, 0, tune=gft.Tune(block_threads=1024, queue_tile=128, max_blocks=1 << 30))
    assert ok["out"].cpu().numpy()[0] == 0


def test_invalid_arguments(gft, engine):
    g = gft.CSRGraph.grid(8, 8)
    dg = g.copy_to_gpu()
    with pytest.raises(gft.GftError, match="INVALID_ARG"):
        engine.bfs(dg, 64)
    with pytest.raises(gft.GftError, match="INVALID_ARG"):
        engine.sssp(dg, 0, delta=0)
    with pytest.raises(gft.GftError, match="INVALID_ARG"):
        engine.bfs(dg, 0, tune=gft.Tune(block_threads=300))


@pytest.mark.parametrize("tune", TUNES, ids=TUNE_IDS)
def test_direction_optimising_bfs(gft, orc, engine, tune):
    """On a graph marked symmetric, BFS runs bottom-up levels when the
    frontier is large: levels equal the oracle's and the top-down-only run's,
    parents form a valid BFS tree, and far fewer edges are examined."""
    g = gft.CSRGraph.rmat(17, 16, seed=11)
    assert g.symmetric
    dg = g.copy_to_gpu()
    assert dg.symmetric
    for src in g.pick_sources(4, 3):
        want = orc.bfs(g.row_start, g.edge_dst, src)
        got, par, r = _run_bfs(gft, engine, dg, src, tune)
        np.testing.assert_array_equal(got, want)
        assert orc.check_tree(g.row_start, g.edge_dst, None, src, got, par) == 0
        td, _, r_td = _run_bfs(gft, engine, dg, src, {**tune, "direction": 1})
        np.testing.assert_array_equal(td, want)
        assert r["edges_scanned"] < r_td["edges_scanned"] / 2


def test_direction_optimising_needs_the_symmetry_mark(gft, orc, engine):
    """A directed graph is never traversed bottom-up: an unmarked upload stays
    top-down, and the mark is the caller's to set."""
    rs = np.array([0, 1, 2, 3, 3], dtype=np.uint32)  # 0 -> 1 -> 2 -> 3, one way
    dst = np.array([1, 2, 3], dtype=np.uint32)
    g = gft.CSRGraph(rs, dst, None)
    assert not g.symmetric
    dg = g.copy_to_gpu()
    assert not dg.symmetric
    for src in range(4):
        got, par, _ = _run_bfs(gft, engine, dg, src)
        np.testing.assert_array_equal(got, orc.bfs(rs, dst, src))
    dg.symmetric = True
    assert dg.symmetric


def test_grid_and_road_bfs_with_static_chunks(gft, orc, engine):
    """Low-degree graphs split large frontiers into one static chunk per
    warp; levels and parents stay exact."""
    for g in (gft.CSRGraph.grid(700, 700, 0, 1), gft.CSRGraph.road(600, seed=4)):
        dg = g.copy_to_gpu()
        for src in g.pick_sources(9, 2):
            got, par, _ = _run_bfs(gft, engine, dg, src)
            np.testing.assert_array_equal(got, orc.bfs(g.row_start, g.edge_dst, src))
            assert orc.check_tree(g.row_start, g.edge_dst, None, src, got, par) == 0


def test_direction_optimising_on_a_uniform_low_diameter_graph(gft, orc, engine):
    """A random graph of small, even degree takes the uniform-degree path of
    the direction switch (no degree loads) and still runs bottom-up."""
    rng = np.random.default_rng(5)
    n, m = 200_000, 800_000
    u = rng.integers(0, n, m, dtype=np.int64)
    v = rng.integers(0, n, m, dtype=np.int64)
    keep = u != v
    a = np.concatenate([u[keep], v[keep]])
    b = np.concatenate([v[keep], u[keep]])
    key = np.unique(a * n + b)
    src_of, dst = (key // n).astype(np.uint32), (key % n).astype(np.uint32)
    rs = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(np.bincount(src_of, minlength=n), out=rs[1:])
    g = gft.CSRGraph(rs, dst, None)
    assert int(np.diff(rs.astype(np.int64)).max()) <= 32
    dg = g.copy_to_gpu()
    dg.symmetric = True
    for src in g.pick_sources(3, 2):
        want = orc.bfs(rs, dst, src)
        got, par, r = _run_bfs(gft, engine, dg, src)
        np.testing.assert_array_equal(got, want)
        assert orc.check_tree(rs, dst, None, src, got, par) == 0
        _, _, r_td = _run_bfs(gft, engine, dg, src, {"direction": 1})
        assert r["edges_scanned"] < r_td["edges_scanned"]


@pytest.mark.parametrize("n", [60_000, 60_001, 60_031, 65_537])
def test_bottom_up_levels_at_bitmap_edges(gft, orc, engine, n):
    """Several bottom-up levels in a row and top-down levels after them, last
    bitmap words of 1, 17 and 31 vertices and a full one: a core of random
    edges (above the one-CTA size), layers of 2000 vertices behind it, a path
    behind those, and vertices without edges at the end."""
    rng = np.random.default_rng(n)
    core, path = n - 25_000, 40
    pairs = [np.stack([rng.integers(0, core, 300_000), rng.integers(0, core, 300_000)], 1)]
    for layer in range(10):
        lo = core + 2000 * layer
        before = rng.integers(0, core, 6000) if layer == 0 else rng.integers(lo - 2000, lo, 6000)
        pairs.append(np.stack([before, rng.integers(lo, lo + 2000, 6000)], 1))
    v = core + 20_000 + np.arange(path)
    pairs.append(np.stack([v - 1, v], 1))
    e = np.concatenate(pairs)
    a, b = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    order = np.argsort(a, kind="stable")
    rs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.uint32)
    dst = b[order].astype(np.uint32)
    dg = gft.CSRGraph(rs, dst).copy_to_gpu()
    dg.symmetric = True
    for src in (0, core - 1, core + 5000, core + 20_000 + path - 1):
        want = orc.bfs(rs, dst, src)
        got, par, r = _run_bfs(gft, engine, dg, src)
        np.testing.assert_array_equal(got, want)
        assert orc.check_tree(rs, dst, None, src, got, par) == 0
        _, _, r_td = _run_bfs(gft, engine, dg, src, {"direction": 1})
        assert r["levels"] == r_td["levels"]
        if src == 0:  # top-down alone scans each reached edge once
            assert r["edges_scanned"] != r_td["edges_scanned"]


def _slot_graph(kind):
    """Graphs of more than 2^17 vertices, at most 4 edges a vertex on average
    and 32 at most: the slot BFS on the grid, except for "random", of whose
    vertices a third have more than 4."""
    n = 150_000
    rng = np.random.default_rng(31)
    if kind == "tree":  # frontiers 1, 3, 9, ...: through every threshold, then the leaves
        v = np.arange(1, n)
        pairs = np.stack([(v - 1) // 3, v], 1)
    elif kind == "bursts":  # a path of hubs with 29 leaves: wide vertices on tiny and on large levels
        v = np.arange(1, n)
        pairs = np.stack([np.where(v % 30 == 0, v - 30, v - v % 30), v], 1)
    else:  # "random", "sparse": a few levels of tens of thousands of vertices
        pairs = rng.integers(0, n, size=(2 * n - n // 8 if kind == "random" else 5 * n // 4, 2))
        pairs = pairs[pairs[:, 0] != pairs[:, 1]]
    a, b = np.concatenate([pairs[:, 0], pairs[:, 1]]), np.concatenate([pairs[:, 1], pairs[:, 0]])
    order = np.argsort(a, kind="stable")
    rs = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.uint32)
    assert int(np.diff(rs.astype(np.int64)).max()) <= 32 and len(a) <= 4 * n
    return rs, b[order].astype(np.uint32)


@pytest.mark.parametrize("kind", ["tree", "bursts", "sparse", "random"])
def test_slot_bfs_on_the_grid(gft, orc, engine, kind):
    import torch

    rs, dst = _slot_graph(kind)
    dg = gft.CSRGraph(rs, dst).copy_to_gpu()
    sms = torch.cuda.get_device_properties(0).multi_processor_count  # one CTA per SM by slots, else two
    assert engine.bfs(dg, 0)["grid_blocks"] == (2 * sms if kind == "random" else sms)
    for src in (0, 1, 149_999, 75_008):
        want = orc.bfs(rs, dst, src)
        got, par, r = _run_bfs(gft, engine, dg, src)
        np.testing.assert_array_equal(got, want)
        assert orc.check_tree(rs, dst, None, src, got, par) == 0
        reached = want != np.iinfo(np.int32).max
        assert r["levels"] == want[reached].max() + 1 and r["vertices_reached"] == reached.sum() - 1
        assert r["edges_scanned"] == int(np.diff(rs.astype(np.int64))[reached].sum())


def test_slot_bfs_reports_an_edge_leaving_the_graph(gft, engine):
    rs, dst = _slot_graph("tree")
    dst[rs[40_000]] = 150_000
    dg = gft.CSRGraph(rs, dst).copy_to_gpu()
    with pytest.raises(gft.GftError) as ei:
        engine.bfs(dg, 0)
    assert ei.value.status_name == "GFT_ERR_FORMAT"


def test_slot_bfs_wait_is_bounded_by_levels_not_by_the_graph(gft, engine):
    """A path's 200,000 levels all run on the first CTA, about 0.2 s in all:
    the other CTAs' waits stay below a 50 ms limit (a run ends after a quarter
    of it)."""
    n = 200_000
    v = np.arange(n)
    deg = np.where((v == 0) | (v == n - 1), 1, 2)
    rs = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint32)
    dst = np.stack([v - 1, v + 1], 1).ravel()
    dst = dst[(dst >= 0) & (dst < n)].astype(np.uint32)
    dg = gft.CSRGraph(rs, dst).copy_to_gpu()
    r = engine.bfs(dg, 0, tune=gft.Tune(timeout_ms=50))
    np.testing.assert_array_equal(r["out"].cpu().numpy(), v)
    assert r["levels"] == n


@pytest.mark.parametrize("side", [1, 2, 90, 91])
def test_one_cta_bfs_either_side_of_the_staged_slots(gft, orc, engine, side):
    """Up to 8192 vertices (90^2 = 8100) the one-CTA kernel builds its slots in
    shared memory, above (91^2 = 8281) it reads the graph's."""
    g = gft.CSRGraph.grid(side, side)
    dg = g.copy_to_gpu()
    for src in {0, g.nnodes // 2, g.nnodes - 1}:
        got, par, r = _run_bfs(gft, engine, dg, src)
        want = orc.bfs(g.row_start, g.edge_dst, src)
        np.testing.assert_array_equal(got, want)
        assert orc.check_tree(g.row_start, g.edge_dst, None, src, got, par) == 0
        assert r["levels"] == want.max() + 1 and r["vertices_reached"] == g.nnodes - 1


@pytest.mark.parametrize("degree", [4, 10, 12, 32])
@pytest.mark.parametrize("marked", [False, True])
def test_grid_bfs_kernels_by_degree(gft, orc, engine, degree, marked):
    """The grid-wide BFS kernels on random graphs of one degree, below, at and
    above 12 edges a vertex, whose large levels run bottom-up when the graph
    is marked, and with a queue tile that has one kernel for all of them."""
    n = 70_001
    rng = np.random.default_rng(degree)
    a = np.tile(np.arange(n), degree // 2)
    b = np.concatenate([rng.permutation(n) for _ in range(degree // 2)])
    src = np.concatenate([a, b])
    order = np.argsort(src, kind="stable")
    rs = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.uint32)
    dst = np.concatenate([b, a])[order].astype(np.uint32)
    assert int(np.diff(rs.astype(np.int64)).max()) == degree
    dg = gft.CSRGraph(rs, dst).copy_to_gpu()
    dg.symmetric = marked
    for src in (0, n - 1):
        want = orc.bfs(rs, dst, src)
        for tune in ({"max_blocks": 1 << 30, "warp_degree": 32}, {"max_blocks": 1 << 30, "queue_tile": 128}):
            got, par, r = _run_bfs(gft, engine, dg, src, tune)
            np.testing.assert_array_equal(got, want)
            assert orc.check_tree(rs, dst, None, src, got, par) == 0
            if not marked:
                reached = want != np.iinfo(np.int32).max
                assert r["edges_scanned"] == int(np.diff(rs.astype(np.int64))[reached].sum())


@pytest.mark.parametrize("claimed", [-5000, -1, 0])
def test_one_cta_bfs_on_a_wrapped_graph_with_a_wrong_edge_count(gft, orc, engine, claimed):
    """The one-CTA kernel stages the slots of every vertex, reached or not: rows
    that end behind the edges the caller claims are left to the CSR, which only
    reads those of reached vertices (here every row's edges are there)."""
    import ctypes as C

    g = gft.CSRGraph.grid(60, 60)
    dg, keep = _wrap(gft, g.row_start, g.edge_dst)
    h = C.c_void_p()
    assert gft.load().gft_graph_wrap(0, g.nnodes, g.nedges + claimed, C.c_void_p(keep[0].data_ptr()),
                                     C.c_void_p(keep[1].data_ptr()), None, C.byref(h)) == 0
    understated = gft.DeviceGraph(h, 0)
    for src in (0, 1799, 3599):
        want = orc.bfs(g.row_start, g.edge_dst, src)
        for graph in (dg, understated):
            got, par, r = _run_bfs(gft, engine, graph, src)
            np.testing.assert_array_equal(got, want)
            assert r["edges_scanned"] == g.nedges


def test_slot_bfs_wait_is_bounded_by_time(gft, orc, engine):
    """A ladder of 5000 levels of 500 vertices, every tenth with 7 edges, read
    through the CSR: a level of the first CTA takes 4 us, all of them 20 ms,
    and the other CTAs wait for at most 5 ms at a time."""
    width, depth = 500, 5000
    n = width * depth
    v = np.arange(n)
    src = [v[:-width], v[width:]]
    dst = [v[width:], v[:-width]]
    wide = v[::10]
    for k in range(1, 6):  # five more edges, to the same level
        a, b = wide, wide // width * width + (wide + k) % width
        src += [a, b]
        dst += [b, a]
    src, dst = np.concatenate(src), np.concatenate(dst)
    order = np.argsort(src, kind="stable")
    rs = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.uint32)
    dst = dst[order].astype(np.uint32)
    assert int(np.diff(rs.astype(np.int64)).max()) <= 32 and len(dst) <= 4 * n
    dg = gft.CSRGraph(rs, dst).copy_to_gpu()
    want = orc.bfs(rs, dst, 0)
    r = engine.bfs(dg, 0, tune=gft.Tune(timeout_ms=5))
    np.testing.assert_array_equal(r["out"].cpu().numpy(), want)


@pytest.mark.parametrize("kind", ["tree", "bursts", "sparse"])
def test_slot_bfs_fills_the_first_query_s_slots_in_scratch(gft, orc, engine, kind):
    """A graph's first query by slots takes no device memory beside the engine's
    scratch, the second builds the graph's own slots, and all agree."""
    import torch

    rs, dst = _slot_graph(kind)
    host = gft.CSRGraph(rs, dst)
    engine.bfs(host.copy_to_gpu(), 0)  # the scratch has its size
    dg = host.copy_to_gpu()
    out = torch.empty(dg.nnodes, dtype=torch.int32, device="cuda")
    par = torch.empty_like(out)
    free = []
    for src in (75_008, 75_008, 149_999):
        out.fill_(-7)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        engine.bfs(dg, src, out=out, parent=par)
        free.append(before - torch.cuda.mem_get_info()[0])
        want = orc.bfs(rs, dst, src)
        np.testing.assert_array_equal(out.cpu().numpy(), want)
        assert orc.check_tree(rs, dst, None, src, want, par.cpu().numpy().view(np.uint32)) == 0
    assert free[0] == 0 and free[1] >= 16 * dg.nnodes and free[2] == 0


@pytest.mark.parametrize("leaves", [1023, 1024, 1025, 4096, 70_001])
@pytest.mark.parametrize("marked", [False, True])
def test_hub_chunks_of_every_kernel(gft, orc, engine, leaves, marked):
    """Two hubs of sizes at the chunks' edges (512, 1024 and 2048), joined by a
    leaf and followed by a path: grid, one CTA, a batch's group and its one CTA,
    BFS and SSSP."""
    n = 2 * leaves + 50
    pairs = [(0, 2 + i) for i in range(leaves)] + [(1, 1 + leaves + i) for i in range(leaves)]
    pairs += [(i, i + 1) for i in range(2 * leaves + 1, n - 1)] + [(2, 2 * leaves + 1)]
    a = np.unique(np.array(pairs), axis=0)
    src, dst = np.concatenate([a[:, 0], a[:, 1]]), np.concatenate([a[:, 1], a[:, 0]])
    order = np.argsort(src, kind="stable")
    rs = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.uint32)
    w = np.random.default_rng(leaves).integers(1, 100, len(src)).astype(np.int32)
    g = gft.CSRGraph(rs, dst[order].astype(np.uint32), w)
    dg = g.copy_to_gpu()
    dg.symmetric = marked
    bfs, sssp = orc.bfs(rs, g.edge_dst, 3), orc.sssp(rs, g.edge_dst, w, 3)
    for tune in (None, {"max_blocks": 1}, {"max_blocks": 1 << 30}):
        t = gft.Tune(**tune) if tune else None
        np.testing.assert_array_equal(engine.bfs(dg, 3, tune=t)["out"].cpu().numpy(), bfs)
        np.testing.assert_array_equal(engine.sssp(dg, 3, delta=50, tune=t)["out"].cpu().numpy(), sssp)
    for group in (1, 4):
        b = gft.Batch(engine, [{"graph": dg, "app": "bfs", "src": 3}, {"graph": dg, "app": "sssp", "src": 3, "delta": 50}],
                      tune=gft.Tune(group_blocks=group, group_min_nodes=1 if group > 1 else 1 << 30))
        b.run()
        np.testing.assert_array_equal(b.queries[0]["out"].cpu().numpy(), bfs)
        np.testing.assert_array_equal(b.queries[1]["out"].cpu().numpy(), sssp)
        b.close()
