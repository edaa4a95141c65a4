"""Error paths of the context, driven by failures injected on the host: a call
that fails midway leaves nothing running, and a call that can do without what
failed gives the same forest."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL_LAUNCH, POOL_ALLOC, COOP_LAUNCH = 0, 1, 2


def _fail(kamsta, ctx, what, nth):
    left = C.c_uint32(0)
    kamsta.check(kamsta.lib().kamsta_ctx_fail_nth(ctx._h, what, nth, C.byref(left)))
    return int(left.value)


def _dev(edges):
    import torch
    return torch.from_numpy(edges.view(np.uint32).reshape(-1, 3).view(np.int32)).cuda()


def test_failed_small_launch_leaves_nothing_running(kamsta, oracle):
    """Three size classes; the launch of the second or third fails while the
    first is under way.  Its graphs take milliseconds: their forests are
    complete when the call returns, the last one's too, only if it waited."""
    import torch
    big, nb = oracle.gen_gnm(32768, 131072, 3), 32768
    ref = _sorted_forest(oracle, big, nb)
    specs = [(oracle.gen_gnm(500, 3000, 4), 500), (oracle.gen_gnm(3000, 20000, 5), 3000)]
    dev = [_dev(e) for e, _ in specs] + [_dev(big)]
    reps = 1500
    outs = torch.zeros((reps, nb, 3), dtype=torch.int32, device="cuda")
    few = [torch.zeros((n, 3), dtype=torch.int32, device="cuda") for _, n in specs]
    ctx, descs = kamsta.Context(0), (kamsta.GraphDesc * (2 + reps))()
    for k, (e, n) in enumerate(specs):
        descs[k].edges, descs[k].m_directed, descs[k].n = dev[k].data_ptr(), len(e), n
        descs[k].out = few[k].data_ptr()
    for k in range(reps):
        d = descs[2 + k]
        d.edges, d.m_directed, d.n, d.out = dev[2].data_ptr(), len(big), nb, outs[k].data_ptr()
    for nth in (2, 3):
        outs.zero_()
        torch.cuda.synchronize()
        assert _fail(kamsta, ctx, SMALL_LAUNCH, nth) == 0
        with pytest.raises(kamsta.KamstaError) as ei:
            ctx.batch_dev(descs)
        got = outs[reps - 1, :len(ref)].cpu().numpy()
        assert ei.value.status == kamsta._native.E_CUDA
        assert np.array_equal(got.view(np.uint32).reshape(-1).view(kamsta.WEDGE), ref)
    assert _fail(kamsta, ctx, SMALL_LAUNCH, 0) == 0
    ctx.batch_dev(descs)
    assert all(d.status == 0 for d in descs)
    for k, (e, n) in enumerate(specs):
        want = _sorted_forest(oracle, e, n)
        got = few[k][:descs[k].out_count].cpu().numpy()
        assert np.array_equal(got.view(np.uint32).reshape(-1).view(kamsta.WEDGE), want)
    ctx.close()


def _sorted_forest(oracle, edges, n):
    f, _ = oracle.kruskal(edges, n)
    t = f.copy()
    t["src"], t["dst"] = np.minimum(f["src"], f["dst"]), np.maximum(f["src"], f["dst"])
    return t[np.lexsort((t["dst"], t["src"]))]


def _solve(kamsta, ctx, d, md, n, fn, cfg):
    import torch
    o = torch.zeros((n, 3), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    k = getattr(ctx, fn)(d.data_ptr(), md, n, o.data_ptr(), cfg)
    return o[:k].cpu().numpy()


@pytest.mark.parametrize("n,m,fn,lp,without", [
    (1000, 4000, "boruvka_dev", 0, 1),       # one CTA: its scratch
    (20000, 90000, "boruvka_dev", 0, 3),     # cooperative rounds: lists and state
    (20000, 200000, "boruvka_dev", 1, 3),
    (20000, 200000, "filter_boruvka_dev", 0, 3),  # each contraction's tail
    (1 << 20, 17 << 20, "boruvka_dev", 0, 3)])    # the forest first, then its edges
def test_every_scratch_request_may_fail(kamsta, n, m, fn, lp, without):
    """The k-th request to the pool fails, for every k of a new context's
    solve: the call runs out of memory or gives the same forest, and for
    at least `without` of them, which only serve speed, it gives the forest;
    the context then solves as before."""
    import torch
    gen = kamsta.Context(0)
    d = torch.empty((2 * m, 3), dtype=torch.int32, device="cuda")
    md = gen.gen_gnm_dev(n, m, 11, 254, d.data_ptr())
    cfg = kamsta.AlgorithmConfig(local_preprocessing=lp)
    want = _solve(kamsta, gen, d, md, n, fn, cfg)
    done_without = 0
    for k in range(1, 200):
        ctx = kamsta.Context(0)
        _fail(kamsta, ctx, POOL_ALLOC, k)
        got = None
        try:
            got = _solve(kamsta, ctx, d, md, n, fn, cfg)
        except kamsta.KamstaError as e:
            assert e.status == kamsta._native.E_OOM
        unused = _fail(kamsta, ctx, POOL_ALLOC, 0)
        assert got is not None or unused == 0
        if got is not None:
            assert np.array_equal(got, want)
            done_without += unused == 0
        assert np.array_equal(_solve(kamsta, ctx, d, md, n, fn, cfg), want)
        ctx.close()
        if unused:
            break
    assert unused and done_without >= without
    gen.close()


@pytest.mark.parametrize("n,m,fn,lp", [
    (20000, 90000, "boruvka_dev", 0), (20000, 200000, "boruvka_dev", 1),
    (20000, 200000, "filter_boruvka_dev", 0), (1 << 20, 17 << 20, "boruvka_dev", 1)])
def test_refused_cooperative_launch_is_done_without(kamsta, n, m, fn, lp):
    """Whichever cooperative launch of a solve is refused, the rounds run
    host-driven from there (or from the start) and give the same forest."""
    import torch
    ctx = kamsta.Context(0)
    d = torch.empty((2 * m, 3), dtype=torch.int32, device="cuda")
    md = ctx.gen_gnm_dev(n, m, 12, 254, d.data_ptr())
    cfg = kamsta.AlgorithmConfig(local_preprocessing=lp)
    want = _solve(kamsta, ctx, d, md, n, fn, cfg)
    for k in range(1, 60):
        _fail(kamsta, ctx, COOP_LAUNCH, k)
        assert np.array_equal(_solve(kamsta, ctx, d, md, n, fn, cfg), want)
        if _fail(kamsta, ctx, COOP_LAUNCH, 0):
            break
    assert k > 1
    ctx.close()


def _from_the_heap(kamsta, ctx, solve):
    """Whether a solve takes nothing from the pool (a request would fail)."""
    _fail(kamsta, ctx, POOL_ALLOC, 1)
    try:
        solve()
    except kamsta.KamstaError as e:
        assert e.status == kamsta._native.E_OOM
    return _fail(kamsta, ctx, POOL_ALLOC, 0) == 1


def _least_limit(kamsta, op):
    """The tightest memory limit, to 2 MB, under which a new context does op."""
    lo, hi = 1 << 20, 4 << 30
    while hi - lo > 2 << 20:
        mid = (lo + hi) // 2
        c = kamsta.Context(0)
        c.set_memory_limit(mid)
        try:
            op(c)
            hi = mid
        except kamsta.KamstaError as e:
            assert e.status == kamsta._native.E_OOM
            lo = mid
        c.close()
    return hi


@pytest.mark.parametrize("what,m_solve", [("7bit", 1450000), ("gnm", 1 << 20),
                                          ("rgg2d", 1 << 18)])
def test_idle_scratch_block_gives_way(kamsta, oracle, what, m_solve):
    """What a new context does under a memory limit it also does after solves
    that left it a block of scratch: the block is not in use by then."""
    import torch
    n, m = 1 << 16, 1 << 20
    gen = kamsta.Context(0)
    d = torch.empty((2 * m_solve, 3), dtype=torch.int32, device="cuda")
    buf = torch.empty((8 * m, 3), dtype=torch.int32, device="cuda")
    out = torch.empty((n, 3), dtype=torch.int32, device="cuda")
    md = gen.gen_gnm_dev(n, m_solve, 13, 254, d.data_ptr())
    small = gen.gen_gnm_dev(n, m, 14, 254, buf.data_ptr())
    torch.cuda.synchronize()
    edges = buf[:small].cpu().numpy().view(np.uint32).reshape(-1).view(kamsta.WEDGE)
    keep, g = gen._cgraph_dev(kamsta.Compressed(edges, n, 4096))
    op = {"7bit": lambda c: c.boruvka_7bit_dev(g, out.data_ptr()),
          "gnm": lambda c: c.gen_gnm_dev(n, 2 * m, 14, 254, buf.data_ptr()),
          "rgg2d": lambda c: c.gen_rgg2d_dev(1 << 20, 0.0012, 15, 254, buf.data_ptr(), 8 * m),
          }[what]
    ctx = kamsta.Context(0)
    solve = lambda: _solve(kamsta, ctx, d, md, n, "boruvka_dev", kamsta.AlgorithmConfig())
    ctx.set_memory_limit(_least_limit(kamsta, op) + (8 << 20))  # and the solves' vertex arrays
    for _ in range(3):
        solve()
    assert _from_the_heap(kamsta, ctx, solve)
    op(ctx)
    torch.cuda.synchronize()
    if what == "7bit":
        ref, _ = oracle.kruskal(edges, n)
        k = ctx.boruvka_7bit_dev(g, out.data_ptr())
        got = out[:k].cpu().numpy().view(np.uint32).reshape(-1).view(kamsta.WEDGE)
        assert np.array_equal(oracle.canon_keys(got), oracle.canon_keys(ref))
    ctx.close()
    gen.close()


def test_out_of_memory_call_does_not_end_the_heap(kamsta):
    """A call that ran out of memory, and one that fitted only without the
    scratch block, leave later, smaller calls a block of scratch."""
    import torch
    n, cfg = 1 << 16, kamsta.AlgorithmConfig()
    gen = kamsta.Context(0)
    graphs = []
    for m in (1 << 17, 1 << 20, 1 << 21, 1 << 23):
        d = torch.empty((2 * m, 3), dtype=torch.int32, device="cuda")
        graphs.append((d, gen.gen_gnm_dev(n, m, m, 254, d.data_ptr())))
    want = [_solve(kamsta, gen, d, md, n, "boruvka_dev", cfg) for d, md in graphs]
    ctx = kamsta.Context(0)

    def solve(i):
        d, md = graphs[i]
        got = _solve(kamsta, ctx, d, md, n, "boruvka_dev", cfg)
        assert np.array_equal(got, want[i])

    d2, md2 = graphs[2]
    ctx.set_memory_limit(_least_limit(
        kamsta, lambda c: _solve(kamsta, c, d2, md2, n, "boruvka_dev", cfg)))
    for _ in range(3):
        solve(1)
    assert _from_the_heap(kamsta, ctx, lambda: solve(1))
    with pytest.raises(kamsta.KamstaError) as ei:
        solve(3)                       # too large for the limit
    assert ei.value.status == kamsta._native.E_OOM
    solve(1)
    assert _from_the_heap(kamsta, ctx, lambda: solve(1))
    for _ in range(6):                 # fits, but not beside the block
        solve(2)
        solve(0)
        assert _from_the_heap(kamsta, ctx, lambda: solve(0))
    ctx.trim()
    for _ in range(3):
        solve(1)
    assert _from_the_heap(kamsta, ctx, lambda: solve(1))
    ctx.close()
    gen.close()


def test_small_graphs_use_the_idle_scratch_block(kamsta, oracle):
    """A wave of small graphs alone takes its slots from a block that a larger
    wave left, also under a memory limit that the block nearly fills."""
    import torch
    ctx = kamsta.Context(0)
    big = torch.empty((1 << 22, 3), dtype=torch.int32, device="cuda")
    md = ctx.gen_gnm_dev(1 << 16, 1 << 21, 21, 254, big.data_ptr())
    e, n = oracle.gen_gnm(3000, 20000, 22), 3000
    ref = _sorted_forest(oracle, e, n)
    d = _dev(e)
    out = torch.zeros((65, 1 << 16, 3), dtype=torch.int32, device="cuda")
    descs = (kamsta.GraphDesc * 65)()
    for k in range(65):
        descs[k].edges, descs[k].m_directed, descs[k].n = d.data_ptr(), len(e), n
        descs[k].out = out[k].data_ptr()
    descs[64].edges, descs[64].m_directed, descs[64].n = big.data_ptr(), md, 1 << 16
    torch.cuda.synchronize()
    large, small = (kamsta.GraphDesc * 1)(descs[64]), (kamsta.GraphDesc * 64)(*descs[:64])
    for limit in (0, _least_limit(kamsta, lambda c: c.batch_dev(large)) + (1 << 20)):
        ctx.set_memory_limit(limit)
        for _ in range(3):
            ctx.batch_dev(large)
        out.zero_()
        torch.cuda.synchronize()
        assert _from_the_heap(kamsta, ctx, lambda: ctx.batch_dev(small))
        assert all(g.status == 0 and g.out_count == len(ref) for g in small)
        got = out[63, :len(ref)].cpu().numpy().view(np.uint32).reshape(-1).view(kamsta.WEDGE)
        assert np.array_equal(got, ref)
        assert _from_the_heap(kamsta, ctx, lambda: ctx.batch_dev(large))
    ctx.close()


def test_small_graphs_of_all_classes_in_one_slot(kamsta, oracle):
    """A memory limit with room for the largest class's slot (4.7 MB) but not
    for one of each class (6.1 MB)."""
    import torch
    specs = [(500, 3000), (3000, 20000), (20000, 90000)]
    graphs = [(oracle.gen_gnm(n, m, 31 + n), n) for n, m in specs]
    dev = [_dev(e) for e, _ in graphs]
    outs = [torch.zeros((n, 3), dtype=torch.int32, device="cuda") for _, n in graphs]
    descs = (kamsta.GraphDesc * 3)()
    for d, t, o, (e, n) in zip(descs, dev, outs, graphs):
        d.edges, d.m_directed, d.n, d.out = t.data_ptr(), len(e), n, o.data_ptr()
    torch.cuda.synchronize()
    ctx = kamsta.Context(0)
    ctx.set_memory_limit(5500000)
    for _ in range(2):
        ctx.batch_dev(descs)
        for d, o, (e, n) in zip(descs, outs, graphs):
            ref = _sorted_forest(oracle, e, n)
            got = o[:len(ref)].cpu().numpy().view(np.uint32).reshape(-1).view(kamsta.WEDGE)
            assert d.status == 0 and d.out_count == len(ref) and np.array_equal(got, ref)
    ctx.close()


@pytest.mark.parametrize("n,cooperative", [(1 << 24, True), ((1 << 24) + 1, False)])
@pytest.mark.parametrize("lp", [0, 1])
def test_sparse_graphs_at_the_vertex_limit(kamsta, n, cooperative, lp):
    """Few edges on many vertices: cooperative rounds up to 2^24 vertices,
    host-driven ones beyond, the forest byte for byte that of a traced solve."""
    import torch
    ctx = kamsta.Context(0)
    d = torch.empty((1 << 22, 3), dtype=torch.int32, device="cuda")
    md = ctx.gen_gnm_dev(n, 1 << 21, 41, 254, d.data_ptr())
    o = torch.zeros((2, n, 3), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    want, got = {}, {}
    kw = ctx.boruvka_dev(d.data_ptr(), md, n, o[0].data_ptr(),
                         kamsta.AlgorithmConfig(local_preprocessing=lp, trace=True), stats=want)
    _fail(kamsta, ctx, COOP_LAUNCH, 1000)
    k = ctx.boruvka_dev(d.data_ptr(), md, n, o[1].data_ptr(),
                        kamsta.AlgorithmConfig(local_preprocessing=lp), stats=got)
    launches = 1000 - _fail(kamsta, ctx, COOP_LAUNCH, 0)
    assert (got["phases"]["round_verts"]["launches"] == 0) == cooperative
    assert launches == 1 or not cooperative
    assert k == kw and got["total_weight"] == want["total_weight"]
    assert torch.equal(o[0], o[1])
    ctx.close()
