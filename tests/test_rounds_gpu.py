"""GPU tests of the solver's plan and its rounds at the sizes where their
kernels change route."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mix64(z):
    z = z + np.uint64(0x9e3779b97f4a7c15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xbf58476d1ce4e5b9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94d049bb133111eb)
    return z ^ (z >> np.uint64(31))


def _planned_classes(edges, n, seed):
    """The weight classes of the light-first split, from the sorted sample of
    4096 weights (the library's own rule, restated)."""
    m = len(edges)
    with np.errstate(over="ignore"):
        h = _mix64(np.uint64(seed) + np.arange(4096, dtype=np.uint64))
    pos = [(int(x) * m) >> 64 for x in h]
    s = np.sort(edges["w"][pos])
    classes, est, length = 1, m / 2.0, len(s)
    last = None
    while est > 3.0 * n and length >= 16:
        pivot = s[int(length * 0.25)]
        light = int(np.searchsorted(s[:length], pivot, side="right"))
        if abs(0.5 - (1.0 - light / length)) > 0.4 or (last is not None and pivot >= last):
            break
        last, classes, est, length = pivot, classes + 1, est * light / length, light
    return classes


@pytest.mark.parametrize("n,m,wmax", [(64, 100, 254), (1000, 20000, 254), (3000, 200000, 254),
                                      (5000, 100001, 3), (3001, 90000, 1 << 30), (700, 7000, 1)])
def test_class_plan_follows_the_sorted_sample(kamsta, oracle, n, m, wmax):
    import torch
    e = oracle.gen_gnm(n, m, 13, wmax)
    # a separate pair under the heaviest weight: every class is contracted
    pair = np.array([(n, n + 1, wmax + 1), (n + 1, n, wmax + 1)], dtype=kamsta.WEDGE)
    e, n = np.concatenate([e, pair]), n + 2
    d = torch.from_numpy(e.view(np.uint32).reshape(-1, 3).view(np.int32)).cuda()
    o = torch.empty((n, 3), dtype=torch.int32, device="cuda")
    ctx, st = kamsta.Context(0), {}
    cfg = kamsta.AlgorithmConfig(local_preprocessing=1, seed=99)
    k = ctx.boruvka_dev(d.data_ptr(), len(e), n, o.data_ptr(), cfg, stats=st)
    got = o[:k].cpu().numpy().view(np.uint32).reshape(-1).view(kamsta.WEDGE)
    ref, w = oracle.kruskal(e, n)
    assert np.array_equal(oracle.canon_keys(got), oracle.canon_keys(ref))
    assert st["levels"] == _planned_classes(e, n, 99)
    ctx.close()


def _dev_solve(kamsta, ctx, edges, n, cfg, fn="boruvka_dev", shift=0):
    """The forest as it lies in the output buffer, with its weight."""
    import torch
    flat = torch.zeros(3 * (len(edges) + shift), dtype=torch.int32, device="cuda")
    flat[3 * shift:] = torch.from_numpy(edges.view(np.uint32).reshape(-1).view(np.int32)).cuda()
    o = torch.zeros((n, 3), dtype=torch.int32, device="cuda")
    st = {}
    torch.cuda.synchronize()
    k = getattr(ctx, fn)(flat.data_ptr() + 12 * shift, len(edges), n, o.data_ptr(), cfg, stats=st)
    return o.cpu().numpy(), k, st


def _rounds_case(oracle, name):
    """Sizes around the cooperative rounds' limits: one CTA and many, a round
    on either side of the vertices a CTA repeats on its own (4096), segment
    counts, ragged tiles."""
    kind, n, m, wmax = name
    if kind == "gnm":
        return oracle.gen_gnm(n, m, 7, wmax), n
    if kind == "rgg":
        return oracle.gen_rgg2d(n, oracle.rgg_radius(n, m), 9), n
    if kind == "path":  # one hook chain through every vertex
        return oracle.symmetric_from_undirected([(i, i + 1, i + 1) for i in range(n - 1)]), n
    # star and a far, separate pair: a hub and finished components
    und = [(0, i, 1 + i % 7) for i in range(1, n - 2)] + [(n - 2, n - 1, wmax)]
    return oracle.symmetric_from_undirected(und), n


@pytest.mark.parametrize("name", [
    ("gnm", 2, 1, 254), ("gnm", 3, 3, 1), ("star", 5, 0, 9), ("gnm", 1023, 4093, 254),
    ("gnm", 4096, 4097, 254), ("gnm", 4097, 50000, 1), ("gnm", 8193, 8190, 1 << 30),
    ("path", 4099, 0, 0), ("path", 70001, 0, 0), ("star", 30011, 0, 254),
    ("gnm", 30000, 1000003, 254), ("rgg", 20011, 12, 0), ("rgg", 400009, 9, 0),
    ("gnm", 600011, 700001, 254)], ids=lambda c: f"{c[0]}-{c[1]}-{c[2]}")
@pytest.mark.parametrize("lp", [0, 1])
def test_cooperative_rounds_match_host_driven_rounds(kamsta, oracle, name, lp):
    """The cooperative rounds write what the host-driven rounds write, byte
    for byte (a traced solve runs the latter)."""
    e, n = _rounds_case(oracle, name)
    ctx = kamsta.Context(0)
    got, k, st = _dev_solve(kamsta, ctx, e, n, kamsta.AlgorithmConfig(local_preprocessing=lp))
    want, kw, sw = _dev_solve(kamsta, ctx, e, n,
                              kamsta.AlgorithmConfig(local_preprocessing=lp, trace=True))
    assert sw["trace_len"] == sw["rounds"] > 0
    assert k == kw and st["total_weight"] == sw["total_weight"] and st["rounds"] == sw["rounds"]
    assert np.array_equal(got, want)
    if len(e) < 1 << 20:
        ref, w = oracle.kruskal(e, n)
        assert k == len(ref) and st["total_weight"] == w
    # an input that starts off a 16-byte boundary
    off, ko, _ = _dev_solve(kamsta, ctx, e, n, kamsta.AlgorithmConfig(local_preprocessing=lp),
                            shift=1)
    assert ko == kw and np.array_equal(off, want)
    ctx.close()


def test_cooperative_rounds_from_threads(kamsta, oracle):
    """Solves on several threads and streams at once give what they give alone."""
    import threading
    graphs = [oracle.gen_gnm(20000 + 1000 * i, 150000, 50 + i) for i in range(4)]
    cfg = kamsta.AlgorithmConfig(local_preprocessing=1)
    ctxs = [kamsta.Context(0) for _ in graphs]
    want = [_dev_solve(kamsta, c, e, 30000, cfg) for c, e in zip(ctxs, graphs)]
    bad = []

    def work(i):
        for _ in range(10):
            got, k, _ = _dev_solve(kamsta, ctxs[i], graphs[i], 30000, cfg)
            if k != want[i][1] or not np.array_equal(got, want[i][0]):
                bad.append(i)

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(graphs))]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad
    [c.close() for c in ctxs]


def test_scratch_heap_limits_and_trim(kamsta, oracle):
    """A context's scratch block grows to what its largest call needed, is
    counted, gives way to a memory limit and is given back by trim; results
    stay the same throughout."""
    n = 1 << 20
    big, small = oracle.gen_gnm(n, 1 << 23, 3), oracle.gen_gnm(5000, 40000, 4)
    cfg = kamsta.AlgorithmConfig(local_preprocessing=1)
    ctx = kamsta.Context(0)
    first, k0, _ = _dev_solve(kamsta, ctx, big, n, cfg)
    for _ in range(3):
        again, k, _ = _dev_solve(kamsta, ctx, big, n, cfg)
        assert k == k0 and np.array_equal(again, first)
        held = ctx.pool_bytes()
    want, ks, _ = _dev_solve(kamsta, kamsta.Context(0), small, 5000, cfg)
    got, k, _ = _dev_solve(kamsta, ctx, small, 5000, cfg)
    assert k == ks and np.array_equal(got, want)
    # tightest limit (a binary search) under which a fresh context solves it
    lo, hi = 1 << 20, 4 << 30
    while hi - lo > 8 << 20:
        mid = (lo + hi) // 2
        c = kamsta.Context(0)
        c.set_memory_limit(mid)
        try:
            _dev_solve(kamsta, c, big, n, cfg)
            hi = mid
        except kamsta.KamstaError as e:
            assert e.status == kamsta._native.E_OOM
            lo = mid
        c.close()
    ctx.set_memory_limit(hi)  # still enough, whatever the context held before
    for _ in range(3):
        again, k, _ = _dev_solve(kamsta, ctx, big, n, cfg)
        assert k == k0 and np.array_equal(again, first)
    ctx.set_memory_limit(0)
    ctx.trim()
    assert ctx.pool_bytes() < held
    again, k, _ = _dev_solve(kamsta, ctx, big, n, cfg)
    assert k == k0 and np.array_equal(again, first)
    ctx.close()


@pytest.mark.parametrize("family,log_n,degree,wmax", [
    ("gnm", 20, 33, 254), ("gnm", 22, 17, 254), ("rgg2d", 21, 33, 254), ("rmat", 21, 34, 254),
    ("gnm", 21, 17, 254), ("rgg2d", 22, 17, 254), ("rmat", 22, 18, 254),
    ("gnm", 20, 40, 1 << 30), ("gnm", 20, 33, 2), ("gnm", 15, 2000, 254)])
def test_plain_rounds_replayed_on_the_forest(kamsta, family, log_n, degree, wmax):
    """Without preprocessing a large dense input is solved on its forest's
    edges; the output is byte for byte that of rounds over every edge (which
    a traced solve runs), order included, with and without validation."""
    import math

    import torch
    ctx = kamsta.Context(0)
    n, m = (1 << log_n) - 3, int((1 << log_n) * degree / 2)
    if family == "gnm":
        d = torch.empty((2 * m, 3), dtype=torch.int32, device="cuda")
        md = ctx.gen_gnm_dev(n, m, 5, wmax, d.data_ptr())
    elif family == "rgg2d":
        r = math.sqrt(degree / (math.pi * n))
        md = ctx.gen_rgg2d_dev(n, r, 5, wmax)
        d = torch.empty((md, 3), dtype=torch.int32, device="cuda")
        ctx.gen_rgg2d_dev(n, r, 5, wmax, d.data_ptr(), md)
    else:
        n = 1 << log_n
        md = ctx.gen_rmat_dev(log_n, m, 5, max_weight=wmax)
        d = torch.empty((md, 3), dtype=torch.int32, device="cuda")
        ctx.gen_rmat_dev(log_n, m, 5, max_weight=wmax, d_out=d.data_ptr(), capacity=md)
    torch.cuda.synchronize()
    o = torch.zeros((2, n, 3), dtype=torch.int32, device="cuda")
    want, got = {}, {}
    kw = ctx.boruvka_dev(d.data_ptr(), md, n, o[0].data_ptr(),
                         kamsta.AlgorithmConfig(trace=True), stats=want)
    for validate in (False, True):
        o[1].zero_()
        torch.cuda.synchronize()
        k = ctx.boruvka_dev(d.data_ptr(), md, n, o[1].data_ptr(),
                            kamsta.AlgorithmConfig(validate=validate), stats=got)
        assert k == kw and got["total_weight"] == want["total_weight"]
        assert got["rounds"] == want["rounds"] and got["levels"] == want["levels"] == 1
        assert torch.equal(o[0], o[1])
    ctx.close()


def _noalloc(kamsta, edges, n, fill=0):
    import ctypes as C

    import torch
    d = torch.from_numpy(edges.view(np.uint32).reshape(-1, 3).view(np.int32)).cuda()
    o = torch.full((n, 3), fill, dtype=torch.int32, device="cuda")
    cnt, w = C.c_uint64(0), C.c_uint64(0)
    torch.cuda.synchronize()
    kamsta.check(kamsta.lib().kamsta_mst_boruvka_noalloc(
        C.c_void_p(d.data_ptr()), len(edges), n, C.c_void_p(o.data_ptr()), C.byref(cnt),
        C.byref(w), None))
    return o.cpu().numpy(), int(cnt.value), int(w.value)


def _small_graphs(oracle):
    """Around the single-CTA solver's limits: compact CTAs (4096 vertices,
    65536 entries), labels and wide minima in shared memory (16384 vertices),
    32-bit keys (weights against the bits of the entry count), the largest
    graph, hubs, paths, ties, isolated vertices, a full graph."""
    yield oracle.gen_gnm(2, 1, 1), 2
    yield oracle.gen_gnm(300, 900, 2, 1), 300
    for wmax in (254, 3, (1 << 16) - 2, (1 << 16) + 5, 0xffffffff):
        yield oracle.gen_gnm(4096, 32768, 3, wmax), 4096      # 2^16 entries: 16 bits
    yield oracle.gen_gnm(4097, 30000, 4), 4097
    yield oracle.gen_gnm(1000, 40000, 5), 1000                # compact by n, not by entries
    for n in (16383, 16384, 16385, 32767, 32768):
        yield oracle.gen_gnm(n, 60000, 6), n
        yield oracle.gen_gnm(n, 60000, 7, 1 << 30), n
    yield oracle.gen_gnm(32768, 131072, 8, 16381), 32768      # the widest 32-bit weights
    yield oracle.gen_gnm(32768, 131072, 9, 16385), 32768
    yield oracle.gen_gnm(513, 513 * 256 - 257, 10), 513
    yield oracle.gen_gnm(32768, 700, 11), 32768
    yield oracle.symmetric_from_undirected([(i, i + 1, i + 1) for i in range(32767)]), 32768
    yield oracle.symmetric_from_undirected([(i, i + 1, 9) for i in range(4095)]), 4096
    yield oracle.symmetric_from_undirected([(0, i, 1 + i % 5) for i in range(1, 32768)]), 32768
    yield oracle.gen_rgg2d(20000, oracle.rgg_radius(20000, 12), 12), 20000


@pytest.mark.parametrize("threads", [0, 256, 512, 1024])
def test_single_cta_solver_at_its_limits(kamsta, oracle, threads):
    import torch
    graphs = list(_small_graphs(oracle))
    ctx = kamsta.Context(0)
    ctx.set_tuning(threads, 0)
    dev = [torch.from_numpy(e.view(np.uint32).reshape(-1, 3).view(np.int32)).cuda()
           for e, _ in graphs]
    outs = [torch.full((n, 3), -1, dtype=torch.int32, device="cuda") for _, n in graphs]
    descs = (kamsta.GraphDesc * len(graphs))()
    for d, t, o, (e, n) in zip(descs, dev, outs, graphs):
        d.edges, d.m_directed, d.n, d.out = t.data_ptr(), len(e), n, o.data_ptr()
    torch.cuda.synchronize()
    ctx.batch_dev(descs)
    torch.cuda.synchronize()
    for d, o, (e, n) in zip(descs, outs, graphs):
        ref, w = oracle.kruskal(e, n)
        assert d.status == 0 and d.out_count == len(ref) and d.total_weight == w
        got = o[: len(ref)].cpu().numpy().view(np.uint32).reshape(-1).view(kamsta.WEDGE)
        key = (got["src"].astype(np.uint64) << np.uint64(32)) | got["dst"]
        assert np.all(np.diff(key.astype(np.int64)) > 0)  # sorted by (src, dst)
        assert np.array_equal(oracle.canon_keys(got), oracle.canon_keys(ref))
        assert np.array_equal(np.sort(got["w"]), np.sort(ref["w"]))
    ctx.close()


def test_allocation_free_solve_writes_what_the_rounds_write(kamsta, oracle):
    """Same order as the device entry point's plain rounds, byte for byte."""
    ctx = kamsta.Context(0)
    for e, n in _small_graphs(oracle):
        want, kw, st = _dev_solve(kamsta, ctx, e, n, kamsta.AlgorithmConfig(trace=True))
        got, k, w = _noalloc(kamsta, e, n)
        assert k == kw and w == st["total_weight"]
        assert np.array_equal(got, want)
    ctx.close()


@pytest.mark.parametrize("hub,lp", [(3071, 1), (3073, 1), (40000, 1), (200000, 1)])
def test_long_rows_fold_their_minimum(kamsta, oracle, hub, lp):
    """Rows around and far beyond two tiles of the first pass, first and last
    in the input, beside ordinary ones."""
    rng = np.random.default_rng(hub)
    n = hub + 20000
    und = {}
    for h in (0, n - 1):
        for v in rng.choice(np.arange(1, n - 1), hub - 1, replace=False):
            und[(min(h, int(v)), max(h, int(v)))] = int(rng.integers(1, 255))
    for a, b in rng.integers(1, n - 1, (40000, 2)):
        if a != b:
            und[(min(int(a), int(b)), max(int(a), int(b)))] = int(rng.integers(1, 255))
    e = oracle.symmetric_from_undirected([(a, b, w) for (a, b), w in sorted(und.items())])
    ctx = kamsta.Context(0)
    for shift in (0, 1):
        got, k, st = _dev_solve(kamsta, ctx, e, n,
                                kamsta.AlgorithmConfig(local_preprocessing=lp), shift=shift)
        ref, w = oracle.kruskal(e, n)
        f = got[:k].view(np.uint32).reshape(-1).view(kamsta.WEDGE)
        assert st["total_weight"] == w
        assert np.array_equal(oracle.canon_keys(f), oracle.canon_keys(ref))
    ctx.close()


@pytest.mark.parametrize("rows", [(1, 8, 9), (255, 256, 257), (5000, 7, 33)])
def test_row_scans_match_the_streamed_class(kamsta, oracle, rows):
    """Outside rows around the lanes of a row (8) and the row a warp takes
    whole (257 entries), last in the input and between other rows; a traced
    solve contracts the heaviest class by row scans, the other one streams
    it, and both write the same bytes."""
    n0 = 100003
    e0 = oracle.gen_gnm(n0, 1200000, 17)
    rng = np.random.default_rng(5)
    # every third id is left out of the graph; some of those become the rows
    ids = np.arange(n0, dtype=np.uint32) * 3 // 2
    und = [(int(ids[a]), int(ids[b]), int(w)) for a, b, w in e0[e0["src"] < e0["dst"]][::2].tolist()]
    free = np.setdiff1d(np.arange(ids[-1]), ids)[[10, 2000, -10]]
    for v, deg in zip(free, rows):
        for u in rng.choice(ids, deg, replace=False):
            und.append((min(int(v), int(u)), max(int(v), int(u)), 254 - int(rng.integers(0, 3))))
    e, n = oracle.symmetric_from_undirected(und), int(ids[-1]) + 1
    ctx = kamsta.Context(0)
    got, k, st = _dev_solve(kamsta, ctx, e, n, kamsta.AlgorithmConfig(local_preprocessing=1))
    want, kw, sw = _dev_solve(kamsta, ctx, e, n,
                              kamsta.AlgorithmConfig(local_preprocessing=1, trace=True))
    ref, w = oracle.kruskal(e, n)
    assert st["row_scans"] == 0 and st["total_weight"] == sw["total_weight"] == w
    assert k == kw == len(ref) and np.array_equal(got, want)
    ctx.close()
    assert sw["row_scans"] >= 1


@pytest.mark.parametrize("filt,lp", [(False, 1), (False, 0), (True, 0)])
def test_union_read_in_place_matches_the_copied_union(kamsta, filt, lp):
    """A batch of 2^25 entries or more whose graphs start on 16-byte
    boundaries is read in place; one graph off such a boundary makes the same
    batch a copied union.  Entry counts of every remainder mod 4, graphs of
    little more than a tile between larger ones, one with an id out of range:
    the same bytes, counts, weights and status."""
    import torch
    ctx = kamsta.Context(0)
    sizes = [(40001, 1540), (40000, 1536), (50021, 1539)] + \
            [(33000 + 517 * i, 130001 + 1801 * i) for i in range(88)] + [(32769, 1537)]
    assert 2 * sum(m for _, m in sizes) > (1 << 25) + 4 * len(sizes)
    bufs, mds = [], []
    for i, (n, m) in enumerate(sizes):
        d = torch.zeros((2 * m + 1, 3), dtype=torch.int32, device="cuda")
        md = ctx.gen_gnm_dev(n, m, 1000 + i, 254, d.data_ptr())
        # the last entries are the src > dst copies of edges: the solve reads the others
        mds.append(max(3072, md - i % 4))
        bufs.append(d)
    bufs[20][777, 1] = sizes[20][0]  # an id out of range
    n = [s[0] for s in sizes]
    runs = []
    for shift in (0, 1):
        src = bufs[45]
        if shift:
            src = torch.zeros_like(bufs[45])
            src[1:] = bufs[45][:-1]
        outs = [torch.full((x, 3), -1, dtype=torch.int32, device="cuda") for x in n]
        descs = (kamsta.GraphDesc * len(n))()
        for i in range(len(n)):
            b = src if i == 45 else bufs[i]
            descs[i].edges = b.data_ptr() + (12 * shift if i == 45 else 0)
            descs[i].m_directed, descs[i].n, descs[i].out = mds[i], n[i], outs[i].data_ptr()
        st = {}
        torch.cuda.synchronize()
        ctx.batch_dev(descs, kamsta.AlgorithmConfig(filter=filt, local_preprocessing=lp),
                      stats=st)
        torch.cuda.synchronize()
        runs.append(([(d.status, d.out_count, d.total_weight) for d in descs], outs, st))
    (a, ao, sa), (b, bo, sb) = runs
    assert a == b and sa["entries"] == sb["entries"] == sum(mds)
    assert a[20][0] != 0 and all(x[0] == 0 for i, x in enumerate(a) if i != 20)
    for i in range(len(n)):
        if i != 20:
            assert torch.equal(ao[i], bo[i]), i
    # three graphs on their own (whole: a single solve wants both copies of an edge)
    for i in (0, 45, len(n) - 1):
        o = torch.zeros((n[i], 3), dtype=torch.int32, device="cuda")
        s1 = {}
        k = ctx.boruvka_dev(bufs[i].data_ptr(), 2 * sizes[i][1], n[i], o.data_ptr(),
                            kamsta.AlgorithmConfig(local_preprocessing=1), stats=s1)
        assert (k, s1["total_weight"]) == a[i][1:]
    ctx.close()


@pytest.mark.parametrize("n,trace", [(4097, False), (300007, False), (300007, True),
                                     ((1 << 22) + 3, True), ((1 << 24) + 5, False)])
@pytest.mark.parametrize("falling", [False, True])
def test_one_hook_chain_through_all_vertices(kamsta, n, trace, falling):
    """A path whose weights rise or fall along it hooks into one chain: the
    label walks are taken up in turns, and the forest is the whole path."""
    import torch
    i = torch.arange(n - 1, device="cuda", dtype=torch.int32)
    w = (n - i) if falling else (i + 1)
    e = torch.empty((2 * (n - 1), 3), dtype=torch.int32, device="cuda")
    e[0::2] = torch.stack([i, i + 1, w], 1)  # (i, i+1) and (i+1, i), sorted by (src, dst)
    e[1::2] = torch.stack([i + 1, i, w], 1)
    o = torch.zeros((n, 3), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx, st = kamsta.Context(0), {}
    k = ctx.boruvka_dev(e.data_ptr(), len(e), n, o.data_ptr(),
                        kamsta.AlgorithmConfig(trace=trace), stats=st)
    assert k == n - 1 and st["total_weight"] == int(w.to(torch.int64).sum())
    got = o[:k][torch.argsort(o[:k, 0])]
    assert torch.equal(got, e[0::2])
    ctx.close()
