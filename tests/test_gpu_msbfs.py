"""Batched multi-source BFS vs the oracle: per-root uint8 levels are the BFS
distances (255 = unreached), bit-exact, for every lane width, with and without
the CUDA graph, under push-only and pull-only level schedules."""
import ctypes as C

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def as_u8(levels16: np.ndarray) -> np.ndarray:
    out = levels16.astype(np.int64)
    out[levels16 == 0xFFFF] = 255
    assert out.max() <= 255
    return out.astype(np.uint8)


@pytest.fixture(scope="module")
def s13(g500, oracle_mod):
    edges = oracle_mod.generate_edges(13)
    og = oracle_mod.Graph(edges, 2)
    g = g500.Graph2DCSR.build(edges, 2)
    roots = og.find_roots(64)
    want = np.stack([as_u8(og.bfs_levels(int(r))) for r in roots])
    yield g, og, roots, want
    g.close()


@pytest.mark.parametrize("lane_width", [32, 64, 128])
@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("alpha", [1e-12, 15.0, 1e12])
def test_msbfs_levels_bit_exact(g500, s13, lane_width, use_graph, alpha):
    g, og, roots, want = s13
    ms = g500.MultiSourceBFS(g, lane_width, alpha, use_graph)
    for n in (len(roots), 7):
        got = ms.levels(roots[:n])
        assert np.array_equal(got, want[:n]), (lane_width, use_graph, alpha, n)
    ms.close()


@pytest.mark.parametrize("lane_width", [32, 64, 128])
@pytest.mark.parametrize("sparse,limit", [(False, 0), (True, 1), (True, 300), (True, 0), (True, 1 << 40)])
def test_msbfs_sparse_levels_keep_levels(g500, s13, lane_width, sparse, limit):
    """Dense levels only, sparse push levels for small frontiers (limits 1 and
    300 put the switch between the two inside the search), and every push
    level sparse: the same levels.  alpha 1e-12 pushes every level; 15 mixes
    push and pull levels."""
    g, og, roots, want = s13
    ms = g500.MultiSourceBFS(g, lane_width, 15.0, True)
    ms.set_sparse(sparse, limit)
    for alpha in (1e-12, 15.0):
        ms.set_params(lane_width, alpha, True)
        for n in (len(roots), 5):
            assert np.array_equal(ms.levels(roots[:n]), want[:n]), (lane_width, sparse, limit, alpha, n)
    with pytest.raises(g500.G500Error) as ei:
        ms.set_sparse(True, -1)
    assert ei.value.code == g500.G500_E_INVAL
    ms.close()


def test_msbfs_repeated_runs_and_device_output(g500, s13):
    import torch
    g, og, roots, want = s13
    ms = g500.MultiSourceBFS(g, 64, 15.0, True)
    out = torch.full((64, g.pred_size()), 7, dtype=torch.uint8, device="cuda")
    for _ in range(3):
        ms.run(roots, out)
        assert np.array_equal(out.cpu().numpy(), want)
    # a different root set reuses the captured graph
    other = roots[::-1].copy()
    assert np.array_equal(ms.levels(other), want[::-1])
    ms.close()


def test_msbfs_root_stats_match_validator(g500, oracle_mod, s13):
    g, og, roots, want = s13
    ms = g500.MultiSourceBFS(g, 64)
    ms.run(roots[:16])
    reached, nedge = ms.root_stats(16)
    edges = oracle_mod.generate_edges(13)
    for i, r in enumerate(roots[:16]):
        assert reached[i] == int((want[i] != 255).sum())
        ok, evc, _ = oracle_mod.validate(edges, og.info["max_used_vertex"] + 1, og.info["pred_size"], int(r),
                                         og.bfs_pred(int(r)))
        assert ok and nedge[i] == evc
    ms.close()


@pytest.mark.parametrize("ran,then", [(32, 64), (32, 128), (64, 32), (128, 64)])
def test_msbfs_root_stats_keep_the_width_that_ran(g500, s13, ran, then):
    """Root statistics and the run's lane width describe the launch that ran, whatever width is set after it:
    after a run, and while a launch is in flight."""
    g, og, roots, _ = s13
    ms = g500.MultiSourceBFS(g, ran)
    ms.run(roots[:20])
    want = [a.tolist() for a in ms.root_stats(20)]
    ms.run(roots[:20])
    ms.set_params(then)
    assert [a.tolist() for a in ms.root_stats(20)] == want
    ms.set_params(ran)
    ms.launch(roots[:20])
    ms.set_params(then)
    assert ms.wait().lane_width == ran
    assert [a.tolist() for a in ms.root_stats(20)] == want
    ms.close()


def test_msbfs_matches_reference_fixture_levels(g500):
    rec, arr = load_golden(18, 2)
    g = g500.Graph2DCSR.generate(18, 16, 2)
    roots = [rec["per_root"][0]["root"], rec["per_root"][1]["root"]]
    ms = g500.MultiSourceBFS(g, 32)
    got = ms.levels(np.array(roots))
    for i in range(2):
        assert np.array_equal(got[i], as_u8(arr[f"levels_{i}"]))
    ms.close()
    g.close()


def test_msbfs_duplicate_and_isolated_roots(g500, oracle_mod):
    pairs = [(1, 2), (2, 3), (3, 4), (10, 11), (40, 40), (5, 6)]
    edges = np.zeros(len(pairs), g500.EDGE_DTYPE)
    for i, (u, v) in enumerate(pairs):
        edges[i] = (u, v, 0)
    og = oracle_mod.Graph(edges, 2)
    g = g500.Graph2DCSR.build(edges, 2)
    roots = np.array([1, 1, 40, 11, 4, 0])  # duplicates, an isolated root with a self loop, a vertex without edges
    ms = g500.MultiSourceBFS(g, 32)
    got = ms.levels(roots)
    for i, r in enumerate(roots):
        assert np.array_equal(got[i], as_u8(og.bfs_levels(int(r)))), r
    ms.close()
    g.close()


def test_msbfs_autotune_keeps_levels(g500, s13):
    g, og, roots, want = s13
    ms = g500.MultiSourceBFS(g, 64)
    tune = ms.autotune(roots, reps=1)
    assert tune["lane_width"] in (32, 64, 128) and tune["configs_tried"] == 15
    assert np.array_equal(ms.levels(roots), want)
    ms.close()


@pytest.fixture(scope="module")
def star(g500, oracle_mod):
    """A star whose centre has more than 2^20 neighbours (a hub row for both
    the pull and the push phase), a 40-vertex path hanging off one leaf, and
    2000 random edges among the leaves."""
    leaves = (1 << 20) + 300
    rng = np.random.default_rng(7)
    pairs = [np.stack([np.zeros(leaves, np.int64), np.arange(1, leaves + 1)], 1)]
    path = np.arange(leaves + 1, leaves + 41)
    pairs.append(np.stack([np.concatenate([[5], path[:-1]]), path], 1))
    pairs.append(rng.integers(1, leaves + 1, (2000, 2)))
    pr = np.concatenate(pairs)
    edges = np.zeros(len(pr), g500.EDGE_DTYPE)
    edges["v0_low"], edges["v1_low"] = pr[:, 0], pr[:, 1]
    og = oracle_mod.Graph(edges, 2)
    g = g500.Graph2DCSR.build(edges, 2)
    roots = np.array([0, 5, int(path[-1]), int(path[20]), 17, 123456, leaves], np.int64)
    want = np.stack([as_u8(og.bfs_levels(int(r))) for r in roots])
    yield g, roots, want
    g.close()


@pytest.mark.parametrize("lane_width", [32, 128])
@pytest.mark.parametrize("alpha", [1e-12, 1e12])
@pytest.mark.parametrize("sparse", [False, True])
def test_msbfs_hub_rows_keep_levels(g500, star, lane_width, alpha, sparse):
    """Rows longer than the hub thresholds are split into chunks that several
    warps take (push: over 256 entries, pull: over 2^20); alpha 1e-12 pushes
    every level and 1e12 pulls every level after the first."""
    g, roots, want = star
    ms = g500.MultiSourceBFS(g, lane_width, alpha, True)
    ms.set_sparse(sparse, 0)
    assert np.array_equal(ms.levels(roots), want), (lane_width, alpha, sparse)
    ms.close()


def test_msbfs_refuses_depth_beyond_uint8(g500):
    n = 300
    edges = np.zeros(n - 1, g500.EDGE_DTYPE)
    for i in range(n - 1):
        edges[i] = (i, i + 1, 0)
    g = g500.Graph2DCSR.build(edges, 0)
    ms = g500.MultiSourceBFS(g, 32)
    with pytest.raises(g500.G500Error) as ei:
        ms.run(np.array([0]))
    assert ei.value.code == g500.G500_E_RANGE
    # the handle stays usable for shallow searches
    assert ms.levels(np.array([150]))[0][150] == 0
    ms.close()
    g.close()


@pytest.mark.parametrize("depth", [13, 14, 15, 16, 17, 33, 253])
@pytest.mark.parametrize("vr", [0, 2])
def test_msbfs_levels_across_bit_planes_and_stats(g500, depth, vr):
    """A path of `depth` edges with leaves, seen from several roots at once: levels on both sides of the first
    four bit planes (14 | 15 | 16) and up to the uint8 limit, in every lane width, with and without sparse
    levels; and each root's statistics against its plain BFS, for a second component and for roots without
    edges (one with a self loop) too."""
    pairs = [(i, i + 1) for i in range(depth)] + [(i, 1000 + i) for i in range(1, depth - 1, 3)]
    pairs += [(2000, 2001), (2001, 2002), (2003, 2003)]
    edges = np.zeros(len(pairs), g500.EDGE_DTYPE)
    edges["v0_low"], edges["v1_low"] = np.array(pairs).T
    bfs = g500.BfsOnGPU(reorder_mode=vr)
    bfs.construct(edges)
    bfs.prepare_bfs()
    n = bfs.graph_.pred_size()
    roots = np.array([0, depth, depth // 2, 1, 1001, 2001, 2003, 1999, 0, 2000] + list(range(2, 12)), np.int64)
    want, stats = [], []
    pred = np.zeros(n, np.int64)
    for r in roots:
        st = bfs.run_bfs(int(r), pred)
        lv = g500.levels_from_pred(pred)
        want.append(np.where(lv == 0xFFFF, 255, lv).astype(np.uint8))
        stats.append((st.reached, st.nedge))
    assert max(int(w[w != 255].max()) for w in want) == depth
    for lanes in (32, 64, 128):
        ms = g500.MultiSourceBFS(bfs.graph_, lanes)
        for sparse in (False, True):
            ms.set_sparse(sparse)
            assert np.array_equal(ms.levels(roots), np.array(want)), (lanes, sparse)
            assert list(zip(*(a.tolist() for a in ms.root_stats(len(roots))))) == stats, (lanes, sparse)
        ms.close()
    bfs.close()


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("lanes,n", [(32, 70), (64, 64), (128, 5)])
def test_msbfs_levels_into_device_memory(g500, s13, offset, lanes, n):
    """Rows in device memory are written by the output pass when they are 4-byte aligned and copied otherwise;
    the handle's own output holds the levels too, and nothing beyond the rows is written."""
    import torch
    g, og, roots, want = s13
    rr = np.resize(roots, n)
    ms = g500.MultiSourceBFS(g, lanes)
    size = n * g.pred_size()
    buf = torch.full((size + 16,), 77, dtype=torch.uint8, device="cuda")
    for _ in range(2):
        ms.run(rr, buf[offset:offset + size])
        got = buf.cpu().numpy()
        assert np.array_equal(got[offset:offset + size].reshape(n, -1), np.resize(want, (n, g.pred_size())))
        assert (got[:offset] == 77).all() and (got[offset + size:] == 77).all()
        assert np.array_equal(ms.device_levels(n).cpu().numpy(), got[offset:offset + size].reshape(n, -1))
    ms.close()


@pytest.mark.parametrize("vr", [0, 1, 2])
def test_msbfs_root_stats_in_small_components(g500, vr):
    """Components of 1 to 40 vertices (some with self loops and double edges) around bitmap words: a word's
    vertices reached by no root, by some lanes, whole or in part, and roots without edges."""
    rng = np.random.default_rng(7)
    pairs, ids, nxt = [], rng.permutation(70000), 0
    for size in list(range(1, 41)) * 4:
        c = ids[nxt:nxt + size]
        nxt += size
        pairs += [(c[rng.integers(0, i)], c[i]) for i in range(1, size)] + [(c[0], c[0])] * int(size % 5 == 0)
        pairs += [(c[0], c[size - 1])] * int(size % 3)
    edges = np.zeros(len(pairs), g500.EDGE_DTYPE)
    edges["v0_low"], edges["v1_low"] = np.array(pairs).T
    bfs = g500.BfsOnGPU(reorder_mode=vr)
    bfs.construct(edges)
    bfs.prepare_bfs()
    roots = np.concatenate([ids[rng.integers(0, nxt, 120)], ids[-8:]])  # the last: no edges
    pred = np.zeros(bfs.graph_.pred_size(), np.int64)
    want = []
    for r in roots:
        st = bfs.run_bfs(int(r), pred)
        want.append((st.reached, st.nedge))
    for lanes in (32, 64, 128):
        ms = g500.MultiSourceBFS(bfs.graph_, lanes)
        for part in (roots[:lanes], roots[-lanes:], roots[:1]):
            ms.run(part)
            got = list(zip(*(a.tolist() for a in ms.root_stats(len(part)))))
            assert got == [want[list(roots).index(r)] for r in part], lanes
        ms.close()
    bfs.close()


@pytest.mark.parametrize("vr,scale,per_sm", [(0, 17, 2), (0, 18, 4), (1, 16, 2), (1, 18, 3), (1, 20, 4), (2, 18, 2),
                                             (2, 20, 3), (2, 21, 4)])
def test_msbfs_default_grid_follows_size_and_order(g500, vr, scale, per_sm):
    """A new handle's blocks per SM, by graph size and vertex order, at most what the device can hold."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = g500.Graph2DCSR.generate(scale, 16, vr)
    ms = g500.MultiSourceBFS(g, 64)
    for lanes in (32, 64, 128):
        blocks, most = ms.grid(lanes)
        assert blocks == min(per_sm * sms, most)
    ms.close()
    g.close()


@pytest.mark.parametrize("spare", [0, 1])
def test_msbfs_refuses_device_memory_shorter_than_its_rows(g500, spare):
    """A device allocation that ends inside the rows is refused by the call (the output pass must not write past
    it); one of exactly their size is written, and the handle works on."""
    import torch
    g = g500.Graph2DCSR.generate(18, 4)
    roots = g500.find_roots(g, 48)  # 48 * 2^18 bytes: 12 MB, a torch allocation of its own
    ms = g500.MultiSourceBFS(g, 64)
    want = ms.levels(roots)
    torch.cuda.empty_cache()
    buf = torch.full((len(roots) * g.pred_size(),), 77, dtype=torch.uint8, device="cuda")
    n = len(roots) + spare * 16
    rr = np.resize(roots, n)
    L, p = g500.lib(), g500.MsStats()
    rc = L.g500_msbfs_run(ms.h, rr.ctypes.data, n, buf.data_ptr(), 1, C.byref(p))
    torch.cuda.synchronize()
    if spare:
        assert rc == g500.G500_E_DEVICE and b"invalid argument" in L.g500_last_error()
        assert (buf == 77).all()
    else:
        assert rc == g500.G500_OK and np.array_equal(buf.cpu().numpy().reshape(want.shape), want)
    assert np.array_equal(ms.levels(roots), want)
    ms.close()
    g.close()


@pytest.mark.parametrize("lane_width", [32, 64, 128])
@pytest.mark.parametrize("alpha", [15.0, 1e6])
@pytest.mark.parametrize("sparse", [True, False])
def test_msbfs_mixed_levels_on_hub_rows(g500, star, lane_width, alpha, sparse):
    """Lanes pulled and pushed at one level, with the hub row (over 2^20 entries) reached by pushed lanes while
    others pull: roots on the star's leaves take the hub at level 1 and everything at level 2, roots on the
    path reach it at levels 2 to 5."""
    g, _, _ = star
    leaves = (1 << 20) + 300
    roots = np.array([17, 123456, leaves, 99] + [leaves + 1 + i for i in (0, 1, 2, 3, 0)] + [5, 0], np.int64)
    bfs = g500.BfsOnGPU()
    bfs.graph_ = g
    bfs.prepare_bfs()
    pred = np.zeros(g.pred_size(), np.int64)
    want, stats = [], []
    for r in roots:
        st = bfs.run_bfs(int(r), pred)
        want.append(as_u8(g500.levels_from_pred(pred)))
        stats.append((st.reached, st.nedge))
    bfs.end_bfs()
    ms = g500.MultiSourceBFS(g, lane_width, alpha)
    ms.set_sparse(sparse)
    for _ in range(2):
        assert np.array_equal(ms.levels(roots), np.array(want))
        assert list(zip(*(a.tolist() for a in ms.root_stats(len(roots))))) == stats
    assert any(lv["pull"] == 2 for lv in ms.level_info()), ms.level_info()
    ms.close()
