"""Error paths of the context, driven by failures injected on the host: a call
that fails midway leaves nothing running, and a call that can do without what
failed gives the same forest."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL_LAUNCH = 0


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
