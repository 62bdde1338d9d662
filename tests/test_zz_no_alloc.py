"""g500_validate_noalloc: Graph500 validation that allocates no device memory.

It serves callers that cannot call cudaMalloc -- a host framework that owns
all device memory through its own arena or caching allocator, or a serving
loop that forbids allocation once it is running.  Its scratch is a fixed
device array inside libg500.so, so this test checks it against the
allocating entry point (g500_validate) on the same inputs, on calls made back
to back (the shared scratch must not carry state from one call to the next).

The file name makes pytest collect it last.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _noalloc(g5, eptr, m, nglob, nloc, root, pred):
    evc, ok, rep = C.c_int64(), C.c_int(), g5.ValidateReport()
    pptr, on_dev = g5._ptr(pred)
    assert on_dev
    g5.check(g5.lib().g500_validate_noalloc(eptr, m, nglob, nloc, int(root), pptr, None, C.byref(evc), C.byref(ok),
                                           C.byref(rep)))
    return bool(ok.value), evc.value, {f[0]: getattr(rep, f[0]) for f in g5.ValidateReport._fields_}


def test_noalloc_validation_matches_allocating_validation(g500):
    import torch

    bfs = g500.BfsOnGPU(reorder_mode=2)
    bfs.construct(g500.EdgeList(None, 14, 16))
    bfs.prepare_bfs()
    g = bfs.graph_
    eptr, m = g.device_edges()
    assert eptr and m == (1 << 14) * 16
    nglob, nloc = g.info.max_used_vertex + 1, g.pred_size()
    roots = g500.find_roots(g, 3)
    pred = torch.empty(nloc, dtype=torch.int64, device="cuda")

    for r in roots[:2]:
        bfs.run_bfs(int(r), pred)
        want = g500.validate_bfs_result(g, int(r), pred)
        first = _noalloc(g500, eptr, m, nglob, nloc, r, pred)
        second = _noalloc(g500, eptr, m, nglob, nloc, r, pred)
        assert want[0] and first == second == want

    # a wrong level planted in the result (host side), then a valid result again:
    # the second call must not see the first call's counters or flags
    r = int(roots[2])
    bfs.run_bfs(r, pred)
    host = pred.cpu().numpy()
    reached = np.nonzero((host != -1) & (np.arange(len(host)) != r))[0]
    v = int(reached[len(reached) // 2])
    bad = host.copy()
    bad[v] = (bad[v] & 0xFFFFFFFFFFFF) | ((((int(bad[v]) >> 48) & 0xFFFF) + 1) << 48)
    bad_dev = torch.from_numpy(bad).cuda()
    want_bad = g500.validate_bfs_result(g, r, bad_dev)
    got_bad = _noalloc(g500, eptr, m, nglob, nloc, r, bad_dev)
    assert not want_bad[0] and got_bad == want_bad
    want_ok = g500.validate_bfs_result(g, r, pred)
    got_ok = _noalloc(g500, eptr, m, nglob, nloc, r, pred)
    assert want_ok[0] and got_ok == want_ok
    bfs.close()


def test_noalloc_refuses_sizes_beyond_its_scratch(g500):
    import torch

    L = g500.lib()
    limit = 1 << 22  # G500_VALIDATE_STATIC_MAX_VERTS
    pred = torch.full((8,), -1, dtype=torch.int64, device="cuda")
    evc, ok = C.c_int64(), C.c_int()
    rc = L.g500_validate_noalloc(None, 0, 1, limit + 1, 0, pred.data_ptr(), None, C.byref(evc), C.byref(ok), None)
    assert rc == g500.G500_E_RANGE
    assert b"at most" in L.g500_last_error()


def test_noalloc_refuses_buffers_off_the_current_device(g500):
    """pred (or the edge list) that is not memory of the current device is refused
    before any kernel runs; a host array stands in for another device's buffer."""
    L = g500.lib()
    host_pred = np.full(64, -1, dtype=np.int64)
    evc, ok = C.c_int64(), C.c_int()
    rc = L.g500_validate_noalloc(None, 0, 1, 64, 0, host_pred.ctypes.data, None, C.byref(evc), C.byref(ok), None)
    assert rc == g500.G500_E_INVAL
    assert b"device memory" in L.g500_last_error()


@pytest.mark.parametrize("planted", ["none", "level", "deep", "deepest", "self", "range", "negative", "half_reached",
                                     "unreached"])
@pytest.mark.parametrize("skip,drop", [(0, 0), (1, 0), (2, 1), (3, 2), (4, 3)])
def test_packed_and_unpacked_validation_report_alike(g500, planted, skip, drop):
    """g500_validate reads packed entries where they fit, g500_validate_noalloc always pred itself: every count
    must agree, on valid and planted results, for edge lists at every 12-byte alignment and remainder of four."""
    import torch

    bfs = g500.BfsOnGPU(reorder_mode=2)
    bfs.construct(g500.EdgeList(None, 12, 16))
    bfs.prepare_bfs()
    g = bfs.graph_
    root = int(g500.find_roots(g, 1)[0])
    pred = np.zeros(g.pred_size(), np.int64)
    bfs.run_bfs(root, pred)
    reached = np.nonzero((pred != -1) & (np.arange(len(pred)) != root))[0]
    v, w = (int(x) for x in reached[[len(reached) // 3, len(reached) // 2]])
    parent, level = int(pred[v]) & 0xFFFFFFFFFFFF, int(pred[v]) >> 48
    pred[v] = {"none": pred[v], "level": parent | (level + 1) << 48, "deep": parent | 30 << 48,
               "deepest": parent | 31 << 48, "self": v | level << 48, "range": 1 << 30 | level << 48,
               "negative": -2, "half_reached": 0xFFFFFFFFFFFF | level << 48, "unreached": -1}[planted]
    if planted == "deep":
        pred[w] = ((1 << 27) - 1) | 30 << 48  # the largest packed entry
    dev = torch.from_numpy(pred).cuda()
    eptr, m = g.device_edges()
    ptr, n = eptr + 12 * skip, m - skip - drop
    evc, ok, rep = C.c_int64(), C.c_int(), g500.ValidateReport()
    g500.check(g500.lib().g500_validate(g.h, ptr, n, 1, root, dev.data_ptr(), 1, C.byref(evc), C.byref(ok),
                                        C.byref(rep)))
    want = _noalloc(g500, ptr, n, g.info.max_used_vertex + 1, g.pred_size(), root, dev)
    assert (bool(ok.value), evc.value, {f[0]: getattr(rep, f[0]) for f in g500.ValidateReport._fields_}) == want
    if planted not in ("none",):
        assert not ok.value
    bfs.close()


def test_validations_of_one_graph_from_several_threads(g500):
    """Calls on one graph from several threads each report their own result: half validate a right pred, half
    one with two levels planted wrong, and every call's counts are those of the same call alone."""
    import threading

    bfs = g500.BfsOnGPU(reorder_mode=2)
    bfs.construct(g500.EdgeList(None, 14, 16))
    bfs.prepare_bfs()
    g = bfs.graph_
    root = int(g500.find_roots(g, 1)[0])
    good = np.zeros(g.pred_size(), np.int64)
    bfs.run_bfs(root, good)
    bad = good.copy()
    reached = np.nonzero((good != -1) & (np.arange(len(good)) != root))[0]
    for v in reached[[len(reached) // 3, len(reached) // 2]]:
        bad[v] += 2 << 48
    alone = [g500.validate_bfs_result(g, root, p) for p in (good, bad)]
    assert alone[0][0] and not alone[1][0]
    got = [[] for _ in range(8)]

    def work(i):
        for _ in range(40):
            got[i].append(g500.validate_bfs_result(g, root, (good, bad)[i % 2]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(got))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, results in enumerate(got):
        assert results == [alone[i % 2]] * 40, i
    bfs.close()


def test_validation_scratch_is_reported_and_not_needed_whole(g500):
    """With room for the flags but not for the packed entries a validation still runs, and keeps nothing; with
    room it keeps its scratch and the graph's device_bytes say so."""
    import torch

    small = g500.BfsOnGPU()
    small.construct(g500.EdgeList(None, 10, 16))
    g500.validate_bfs_result(small.graph_, 0, np.full(small.graph_.pred_size(), -1, np.int64))  # loads the kernels
    bfs = g500.BfsOnGPU(reorder_mode=2)
    bfs.construct(g500.EdgeList(None, 22, 1))
    bfs.prepare_bfs()
    g = bfs.graph_
    n = g.pred_size()
    root = int(g500.find_roots(g, 1)[0])
    pred = torch.empty(n, dtype=torch.int64, device="cuda")
    bfs.run_bfs(root, pred)
    torch.cuda.synchronize()

    def held():
        info = g500.GraphInfo()
        g500.check(g500.lib().g500_graph_info_get(g.h, C.byref(info)))
        return info.device_bytes

    def fill(size, out):
        try:
            while True:
                out.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            pass

    before, full = held(), []
    small.prepare_bfs()  # a device allocation of 7 MB; the flags take 4.2, with the packed entries 21
    try:
        for size in (1 << 30, 16 << 20, 1 << 20):
            fill(size, full)
        small.end_bfs()
        got = g500.validate_bfs_result(g, root, pred)
    finally:
        full.clear()
        torch.cuda.empty_cache()
    assert held() == before
    assert got == g500.validate_bfs_result(g, root, pred) and got[0]
    assert before + 5 * n <= held() <= before + 5 * n + 4096
    bfs.close()
    small.close()


@pytest.mark.parametrize("validated", [False, True])
def test_device_bytes_is_what_a_graph_holds(g500, validated):
    """device_bytes against the memory that destroying the graph gives back: within the 2 MB granularity of its
    allocations (maps, adjacency, edge list, validator's scratch)."""
    import torch

    g = g500.Graph2DCSR.generate(26, 1)
    if validated:
        root = int(g500.find_roots(g, 1)[0])
        g500.validate_bfs_result(g, root, torch.full((g.pred_size(),), -1, dtype=torch.int64, device="cuda"))
    info = g500.GraphInfo()
    g500.check(g500.lib().g500_graph_info_get(g.h, C.byref(info)))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    g.close()
    held = torch.cuda.mem_get_info()[0] - free
    assert info.device_bytes <= held <= info.device_bytes + (4 << 21)


@pytest.mark.parametrize("planted", ["none", "level", "deep", "deepest", "self", "range", "negative", "half_reached",
                                     "unreached"])
def test_validation_reports_alike_at_every_size(g500, planted):
    """The edge pass reads 64-bit entries, one edge a thread up to 2^19 ids and four up to 2^20, then packed ones,
    two edges a thread up to 2^23 and four above.  The same small graph among 2^16 to 2^24 ids, right and planted,
    for edge lists at every alignment and remainder: every count is the same."""
    import torch

    rng = np.random.default_rng(11)
    ids = rng.integers(0, 3000, (20001, 2))
    reports = {}
    for lg in (16, 19, 20, 21, 23, 24):
        edges = np.zeros(len(ids) + 1, g500.EDGE_DTYPE)
        edges["v0_low"][:-1], edges["v1_low"][:-1] = ids.T
        edges["v0_low"][-1] = edges["v1_low"][-1] = (1 << lg) - 1  # a self loop that sets the number of ids
        bfs = g500.BfsOnGPU(reorder_mode=2)
        bfs.construct(edges)
        bfs.prepare_bfs()
        g = bfs.graph_
        assert g.pred_size() == 1 << lg
        root = int(ids[0, 0])
        pred = np.zeros(g.pred_size(), np.int64)
        bfs.run_bfs(root, pred)
        reached = np.nonzero((pred != -1) & (np.arange(len(pred)) != root))[0]
        v, w = (int(x) for x in reached[[len(reached) // 3, len(reached) // 2]])
        parent, level = min(int(n) for n in np.concatenate([ids[ids[:, 0] == v, 1], ids[ids[:, 1] == v, 0]])
                            if int(pred[n]) >> 48 == (int(pred[v]) >> 48) - 1), int(pred[v]) >> 48
        pred[v] = {"none": parent | level << 48, "level": parent | (level + 1) << 48, "deep": parent | 30 << 48,
                   "deepest": parent | 31 << 48, "self": v | level << 48, "range": 1 << 30 | level << 48,
                   "negative": -2, "half_reached": 0xFFFFFFFFFFFF | level << 48, "unreached": -1}[planted]
        dev, elist = torch.from_numpy(pred).cuda(), torch.from_numpy(edges.view(np.int32)).cuda()
        for skip, drop in ((0, 0), (1, 0), (2, 1), (3, 2)):
            evc, ok, rep = C.c_int64(), C.c_int(), g500.ValidateReport()
            g500.check(g500.lib().g500_validate(g.h, elist.data_ptr() + 12 * skip, len(edges) - skip - drop, 1, root,
                                                dev.data_ptr(), 1, C.byref(evc), C.byref(ok), C.byref(rep)))
            got = (bool(ok.value), evc.value, {f[0]: getattr(rep, f[0]) for f in g500.ValidateReport._fields_})
            assert got == reports.setdefault((skip, drop), got), (lg, skip, drop)
            assert got[0] == (planted == "none") or drop or skip
            if lg <= 21:
                assert got == _noalloc(g500, elist.data_ptr() + 12 * skip, len(edges) - skip - drop,
                                       g.info.max_used_vertex + 1, g.pred_size(), root, dev)
        bfs.close()
