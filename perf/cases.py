"""The solver's work, as cases that can be timed.

A case names an entry point, its options and the graph it is called on; the
graphs come from the library's seeded device generators.  Every output is a
forest (whole numbers), so outputs compare for equality.
"""
import ctypes as C
import math

import numpy as np
import torch

import kamsta_gb300 as K
from kamsta_gb300 import _native

ENTRY_BYTES = 12  # one directed entry, and one forest edge: (src, dst, w)
_DESC = np.dtype({"names": ["out_count", "total_weight"], "formats": [np.uint64, np.uint64],
                  "offsets": [K.GraphDesc.out_count.offset, K.GraphDesc.total_weight.offset],
                  "itemsize": C.sizeof(K.GraphDesc)})


def listed():
    return [
        # A plugin without an allocator solves one very small graph: the
        # launch and the single CTA's serial chain are all there is.
        {"name": "noalloc_gnm_n1000", "entry": "noalloc", "family": "gnm", "n": 1000,
         "degree": 8.0, "wmax": 254},
        # One ordinary graph with the default configuration (plain Boruvka
        # rounds); the size of the smallest single-graph benchmark.
        {"name": "plain_gnm_2e16_2e20", "entry": "boruvka", "family": "gnm", "n": 1 << 16,
         "degree": 32.0, "wmax": 254, "lp": 0},
        # The same graph through the drop-in call: pinned host buffers in and out.
        {"name": "host_plain_gnm_2e16_2e20", "entry": "host", "family": "gnm", "n": 1 << 16,
         "degree": 32.0, "wmax": 254, "lp": 0},
        # An odd-sized geometric graph with local preprocessing, the
        # reference benchmark's default level.
        {"name": "local_rgg2d_n1000003", "entry": "boruvka", "family": "rgg2d", "n": 1000003,
         "degree": 16.0, "wmax": 254, "lp": 1, "distance": 0},
        # filter-Boruvka's own recursion (no local preprocessing).
        {"name": "filter_plain_gnm_2e20_2e24", "entry": "filter", "family": "gnm", "n": 1 << 20,
         "degree": 32.0, "wmax": 254, "lp": 0},
        # A large graph with the default configuration: every edge in every round.
        {"name": "plain_gnm_2e23_2e27", "entry": "boruvka", "family": "gnm", "n": 1 << 23,
         "degree": 32.0, "wmax": 254, "lp": 0},
        # The large geometric configuration of the benchmark.
        {"name": "filter_local_rgg2d_2e24", "entry": "filter", "family": "rgg2d", "n": 1 << 24,
         "degree": 16.0, "wmax": 254, "lp": 1, "distance": 0},
        # A skewed graph: hubs of 10^5 neighbours, half the vertices isolated.
        {"name": "filter_local_rmat_2e22", "entry": "filter", "family": "rmat", "n": 1 << 22,
         "degree": 16.0, "wmax": 254, "lp": 1},
        # The headline benchmark graph.
        {"name": "local_gnm_2e26_2e30", "entry": "boruvka", "family": "gnm", "n": 1 << 26,
         "degree": 32.0, "wmax": 254, "lp": 1},
        # A graph kept on the device in the 7-bit difference encoding.
        {"name": "local_7bit_gnm_2e20_2e24", "entry": "7bit", "family": "gnm", "n": 1 << 20,
         "degree": 32.0, "wmax": 254, "lp": 1},
        # Many small requests in one call: the persistent one-CTA-per-graph kernel.
        {"name": "batch_small_1024", "entry": "batch", "family": "mixed", "graphs": 1024,
         "log_n_lo": 8.0, "log_n_hi": 12.0, "wmax": 254, "lp": 0},
        # A slice of the benchmark's uneven batch: 2^8 to 2^20 vertices.
        {"name": "batch_mixed_192", "entry": "batch", "family": "mixed", "graphs": 192,
         "log_n_lo": 8.0, "log_n_hi": 20.0, "wmax": 254, "lp": 1},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another call of the listed kinds: sizes over the logarithm of their
    range, average degree 4 to 32, small and wide weights."""
    kind = rng.choice(["noalloc", "host", "boruvka", "boruvka", "boruvka", "filter", "filter",
                       "7bit", "batch", "batch"])
    if kind == "batch":
        hi = rng.uniform(9.0, 20.0)
        most = 2048 if hi < 13 else 512 if hi < 17 else 192
        return {"entry": kind, "family": "mixed", "graphs": _log(rng, 16, most), "log_n_lo": 8.0,
                "log_n_hi": round(hi, 3), "wmax": 254, "lp": rng.choice([0, 1])}
    family = rng.choice(["gnm", "gnm", "rgg2d", "rmat"])
    degree = round(rng.uniform(4.0, 32.0), 3)
    wmax = rng.choice([254, 254, 65535, 1 << 30])
    if kind == "noalloc":
        return {"entry": kind, "family": rng.choice(["gnm", "rgg2d"]), "n": _log(rng, 256, 1 << 15),
                "degree": min(degree, 7.0), "wmax": wmax, "distance": 0}
    # host and compressed inputs are built on the host: bounded sizes
    top = {"host": 1 << 18, "7bit": 1 << 20}.get(kind, 1 << 26 if family == "gnm" else 1 << 24)
    n = _log(rng, 1 << 10, top)
    if family == "rmat":
        n = 1 << max(10, n.bit_length() - 1)
    case = {"entry": kind, "family": family, "n": n, "degree": degree, "wmax": wmax,
            "lp": rng.choice([0, 1])}
    if family == "rgg2d":
        case["distance"] = rng.choice([0, 0, 1])
    return case


def _graph(gen, case, seed):
    """One graph on the device: (edges tensor (m, 3) int32, directed entries)."""
    n, deg, wmax = case["n"], case["degree"], case["wmax"]
    if case["family"] == "gnm":
        m = min(n * (n - 1) // 2, int(n * deg / 2))
        d = torch.empty((2 * m, 3), dtype=torch.int32, device="cuda")
        return d, gen.gen_gnm_dev(n, m, seed, wmax, d.data_ptr())
    if case["family"] == "rgg2d":
        r = math.sqrt(deg / (math.pi * n))

        def call(ptr, cap):
            return gen.gen_rgg2d_dev(n, r, seed, wmax, ptr, cap, distance=case.get("distance", 0))
    else:
        def call(ptr, cap):
            return gen.gen_rmat_dev(n.bit_length() - 1, int(n * deg / 2), seed, max_weight=wmax,
                                    d_out=ptr, capacity=cap)
    md = call(0, 0)
    d = torch.empty((max(md, 1), 3), dtype=torch.int32, device="cuda")
    return d, call(d.data_ptr(), md)


def _sizes(case):
    """The uneven mix: n log-uniform, average degree in [4, 32], G(n, m) and
    geometric graphs in turn.  The sizes are the case's, the graphs the seed's."""
    rng = np.random.default_rng(case["graphs"])
    return [{"family": "gnm" if i % 2 == 0 else "rgg2d", "wmax": case["wmax"],
             "n": int(round(2.0 ** rng.uniform(case["log_n_lo"], case["log_n_hi"]))),
             "degree": float(rng.uniform(4.0, 32.0))} for i in range(case["graphs"])]


def prepare(case, seed):
    # the generator's scratch is not part of what the solving program keeps
    gen = K.Context(0)
    try:
        if case["entry"] == "batch":
            graphs = [(one["n"], *_graph(gen, one, seed * 1_000_003 + i))
                      for i, one in enumerate(_sizes(case))]
        else:
            edges, md = _graph(gen, case, seed)
        torch.cuda.synchronize()
    finally:
        gen.close()
    s = {"entry": case["entry"]}
    if case["entry"] != "noalloc":
        s["cfg"] = K.AlgorithmConfig(local_preprocessing=K.LocalPreprocessing(case["lp"]))
    if case["entry"] == "host":
        s.update(n=case["n"], md=md, edges=edges[:md].cpu().pin_memory(),
                 out=torch.zeros((case["n"], 3), dtype=torch.int32).pin_memory())
        return s
    s["ctx"] = K.Context(0)
    if case["entry"] == "batch":
        out = torch.zeros((sum(n for n, _, _ in graphs), 3), dtype=torch.int32, device="cuda")
        descs = (K.GraphDesc * len(graphs))()
        at = 0
        for d, (n, e, md) in zip(descs, graphs):
            d.edges, d.m_directed, d.n = e.data_ptr(), md, n
            d.out = out.data_ptr() + ENTRY_BYTES * at
            at += n
        s.update(descs=descs, edges=graphs, out=out)
        return s
    s.update(n=case["n"], md=md, out=torch.zeros((case["n"], 3), dtype=torch.int32, device="cuda"))
    if case["entry"] == "7bit":
        host = edges[:md].cpu().numpy().view(np.uint32).reshape(-1).view(K.WEDGE)
        cg = K.Compressed(host, case["n"], chunk_edges=4096)
        s["keep"] = (torch.from_numpy(cg.offset.view(np.int64)).cuda(),
                     torch.from_numpy(cg.first.view(np.uint32).view(np.int32)).cuda(),
                     torch.from_numpy(cg.data.view(np.int8)).cuda())
        s["graph"] = cg.c_struct(*(t.data_ptr() for t in s["keep"]))
    else:
        s["edges"] = edges
    return s


def run(s):
    entry = s["entry"]
    if entry == "batch":
        s["ctx"].batch_dev(s["descs"], s["cfg"])
        done = np.frombuffer(s["descs"], dtype=_DESC)
        return {"forests": s["out"], "counts": done["out_count"].astype(np.int64),
                "weights": done["total_weight"].astype(np.int64)}
    if entry in ("noalloc", "host"):
        lib, count, weight = _native.lib(), C.c_uint64(0), C.c_uint64(0)
        edges, out = C.c_void_p(s["edges"].data_ptr()), C.c_void_p(s["out"].data_ptr())
        if entry == "noalloc":
            _native.check(lib.kamsta_mst_boruvka_noalloc(
                edges, s["md"], s["n"], out, C.byref(count), C.byref(weight), None))
            return {"forest": s["out"], "count": count.value, "weight": weight.value}
        _native.check(lib.kamsta_mst_boruvka(
            edges, s["md"], s["n"], C.byref(s["cfg"].to_c()), out, C.byref(count), None))
        return {"forest": s["out"], "count": count.value}
    stats = {}
    out = s["out"].data_ptr()
    if entry == "7bit":
        k = s["ctx"].boruvka_7bit_dev(s["graph"], out, s["cfg"], stats=stats)
    else:
        call = s["ctx"].filter_boruvka_dev if entry == "filter" else s["ctx"].boruvka_dev
        k = call(s["edges"].data_ptr(), s["md"], s["n"], out, s["cfg"], stats=stats)
    return {"forest": s["out"], "count": k, "weight": stats["total_weight"]}


def work(case):
    """Each input entry read once, each forest edge written once (expected
    sizes where the graph is drawn); no floating-point work."""
    if case["entry"] == "batch":
        sizes = _sizes(case)
        n, md = sum(g["n"] for g in sizes), sum(g["n"] * g["degree"] for g in sizes)
        entry = ENTRY_BYTES
    else:
        n, md, entry = case["n"], case["n"] * case["degree"], ENTRY_BYTES
        if case["entry"] == "7bit":  # varints of the source step, the target and the weight
            bits = math.log2(max(n, 2)) - 0.5
            entry = 1 + math.ceil(bits / 7) + math.ceil(math.log2(case["wmax"]) / 7 - 0.5)
    return {"bytes": entry * md + ENTRY_BYTES * n, "flops": 0}
