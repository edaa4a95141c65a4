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
