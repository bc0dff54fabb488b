"""The calls by which this framework's speed is judged: every family of entry
points over the range of sizes that its users bring, from a graph of a thousand
vertices to R-MAT scale 24, with odd sizes, both directions (pull and push),
the storage types in use, and the calls that begin from an edge list or a host
graph.

A case is a dict of plain values; `prepare` makes its inputs on the GPU from a
seed, `run` makes one call as a user's program does, `exact` gives the same
result in 64 bits from the edge list alone.
"""
import ctypes as C
import math

import numpy as np
import torch

import accelgraph_express_gb300 as gg

MAP_RANK = gg.MAP_IN                      # what PageRank pull needs
MAP_WEIGHTED = gg.MAP_IN | gg.MAP_IN_W    # SpMV pull
MAP_BOTH = gg.MAP_IN | gg.MAP_OUT         # BFS, connected components


def listed():
    return [
        # a small graph ranked on demand: latency of one call, ranks on the host
        dict(name="rank_1k", kind="rank", V=1000, ef=16, graph="rmat", mode="pull", storage="f32",
             iterations=20, cuda_graph=False, host=True),
        # the 65K-vertex graph ranked again and again in one CUDA graph
        dict(name="rank_64k_graph", kind="rank", V=1 << 16, ef=16, graph="rmat", mode="pull", storage="f32",
             iterations=20, cuda_graph=True, host=False),
        # the reference's quantised pull, odd size
        dict(name="rank_q16_700k", kind="rank", V=700001, ef=16, graph="rmat", mode="pull_q16", storage="f32",
             iterations=20, cuda_graph=False, host=False),
        # 16-bit storage on a graph whose values fit L2
        dict(name="rank_bf16_4m", kind="rank", V=1 << 22, ef=16, graph="rmat", mode="pull", storage="bf16",
             iterations=20, cuda_graph=False, host=False),
        # the headline: R-MAT scale 24
        dict(name="rank_f32_16m", kind="rank", V=1 << 24, ef=16, graph="rmat", mode="pull", storage="f32",
             iterations=20, cuda_graph=False, host=False),
        # the push direction on a graph without hubs, odd size
        dict(name="push_f32_3m", kind="rank", V=3000017, ef=11, graph="uniform", mode="push", storage="f32",
             iterations=10, cuda_graph=False, host=False),
        # repeated weighted products, result on the host
        dict(name="spmv_f32_5m", kind="spmv", V=5000011, ef=16, graph="rmat", mode="pull", storage="f32",
             iterations=20),
        # one search of an undirected social-network-like graph
        dict(name="bfs_4m", kind="bfs", V=1 << 22, ef=16, graph="rmat", mode="do"),
        # components of a directed graph, in-edges mapped
        dict(name="cc_6m", kind="cc", V=6000001, ef=16, graph="rmat", algorithm="afforest"),
        # a full batch of personalised rankings
        dict(name="ppr_64_1m", kind="ppr", V=1 << 20, ef=16, graph="rmat", K=64, storage="bf16", iterations=20),
        # a weighted edge list on the device becomes a graph, and one product
        dict(name="load_4m", kind="load", V=1 << 22, ef=16, graph="rmat", weighted=True),
        # the reference's own call on a host graph: upload, iterations, ranks back
        dict(name="dropin_1m", kind="dropin", V=1 << 20, ef=16, graph="rmat", iterations=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any kind, its size spread over the logarithm of its range."""
    kind = rng.choice(["rank", "rank", "rank", "spmv", "bfs", "cc", "ppr", "load", "dropin"])
    graph = rng.choice(["rmat", "rmat", "uniform"])
    ef = rng.choice([5, 8, 11, 16])
    c = dict(kind=kind, ef=ef, graph=graph)
    if kind == "rank":
        c["mode"] = rng.choice(["pull", "pull", "pull", "push", "pull_q16", "pull_fx32"])
        c["V"] = _log_int(rng, 1000, 8000000 if c["mode"] == "pull" else 3000000)
        c["storage"] = rng.choice(["f32", "f32", "bf16", "f16"]) if c["mode"] == "pull" else "f32"
        c["iterations"] = rng.choice([10, 20])
        c["cuda_graph"] = c["V"] < 200000 and rng.random() < 0.5
        c["host"] = rng.random() < 0.3
    elif kind == "spmv":
        c["V"] = _log_int(rng, 1000, 5000000)
        c["mode"] = rng.choice(["pull", "pull", "push"])
        c["storage"] = rng.choice(["f32", "bf16"])
        c["iterations"] = rng.choice([1, 20]) if c["mode"] == "pull" else 1
    elif kind == "bfs":
        c["V"] = _log_int(rng, 1000, 4000000)
        c["mode"] = rng.choice(["do", "do", "push"])
    elif kind == "cc":
        c["V"] = _log_int(rng, 1000, 6000000)
        c["algorithm"] = rng.choice(["afforest", "sv", "weakly"])
    elif kind == "ppr":
        c["V"] = _log_int(rng, 1000, 1000000)
        c["K"] = rng.choice([1, 10, 16, 24, 32, 64])
        c["storage"] = rng.choice(["f32", "bf16"])
        c["iterations"] = rng.choice([10, 20])
    elif kind == "load":
        c["V"] = _log_int(rng, 1000, 4000000)
        c["weighted"] = rng.random() < 0.5
    else:
        c["V"] = _log_int(rng, 1000, 1000000)
        c["iterations"] = rng.choice([10, 20])
    return c


# ---- inputs ---------------------------------------------------------------

CHUNK = 1 << 26
RMAT = (0.57, 0.19, 0.19)  # the generator's own parameters


def _edges(case, seed):
    """(src, dst) as int32 CUDA tensors.  R-MAT ids are drawn on the next power
    of two and scaled down to V."""
    V, E = case["V"], case["V"] * case["ef"]
    gen = torch.Generator(device="cuda").manual_seed(1000003 * seed + V)
    src = torch.empty(E, dtype=torch.int32, device="cuda")
    dst = torch.empty(E, dtype=torch.int32, device="cuda")
    if case["graph"] == "uniform":
        src.random_(0, V, generator=gen)
        dst.random_(0, V, generator=gen)
    else:
        a, b, c = RMAT
        scale = max(1, (V - 1).bit_length())
        for at in range(0, E, CHUNK):
            n = min(CHUNK, E - at)
            s, d = src[at:at + n], dst[at:at + n]
            s.zero_()
            d.zero_()
            r = torch.empty(n, device="cuda")
            for _ in range(scale):
                r.uniform_(generator=gen)
                down = r >= a + b
                right = ((r >= a) & ~down) | (r >= a + b + c)
                s.mul_(2).add_(down)
                d.mul_(2).add_(right)
            if V != 1 << scale:
                for t in (s, d):
                    t.copy_((t.long() * V) >> scale)
    if case["kind"] == "bfs":  # undirected: every edge both ways
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    return src, dst


def _weights(case, seed, E):
    gen = torch.Generator(device="cuda").manual_seed(7 * seed + 11)
    return torch.rand(E, generator=gen, device="cuda")


def _seed_sets(case, seed):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, case["V"], int(rng.integers(1, 33))).astype(np.uint32) for _ in range(case["K"])]


def prepare(case, seed):
    kind, V = case["kind"], case["V"]
    src, dst = _edges(case, seed)
    s = dict(case=case)
    if kind == "load":
        s["src"], s["dst"] = src, dst
        s["w"] = _weights(case, seed, src.numel()) if case["weighted"] else None
        torch.cuda.synchronize()
        return s
    if kind == "dropin":
        s["graph"] = gg.Graph.from_edges(src.cpu().numpy(), dst.cpu().numpy(), num_vertices=V)
        s["args"] = gg.default_arguments(iterations=case["iterations"], epsilon=0.0)
        return s
    w = _weights(case, seed, src.numel()) if kind == "spmv" else None
    if kind == "spmv":
        what = MAP_WEIGHTED if case["mode"] == "pull" else gg.MAP_OUT | gg.MAP_OUT_W
        s["x"] = np.random.default_rng(seed).random(V, dtype=np.float32)
    elif kind in ("bfs", "cc"):
        what = MAP_BOTH
        s["source"] = int(src[0])
    elif kind == "rank" and case["mode"] == "push":
        what = gg.MAP_OUT
    else:
        what = MAP_RANK
    if kind == "ppr":
        s["sets"] = _seed_sets(case, seed)
    torch.cuda.synchronize()  # the edges are complete before another stream reads them
    s["g"] = gg.DeviceGraph.build(src, dst, w, num_vertices=V, what=what)
    return s


# ---- one call -------------------------------------------------------------

class _Device:
    """A device array of the library as torch sees it."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=2, strides=None)


def _tensor(ptr, shape, typestr):
    return torch.as_tensor(_Device(ptr, shape, typestr), device="cuda")


def run(s):
    case = s["case"]
    kind, V = case["kind"], case["V"]
    if kind == "rank":
        g = s["g"]
        ranks, _ = g.pagerank(case["mode"], storage=case["storage"], iterations=case["iterations"], epsilon=0.0,
                              copy_out=case["host"], cuda_graph=case["cuda_graph"])
        return ranks if case["host"] else _tensor(gg.lib().gg_pagerank_device_ranks(g.h), (V,), "<f4")
    if kind == "spmv":
        x, y, _ = s["g"].spmv(case["mode"], storage=case["storage"], iterations=case["iterations"], x=s["x"])
        return [x, y]
    if kind == "bfs":
        # the distances are the same on every run; which of several possible
        # parents a vertex gets is not, so the parents stay out
        g = s["g"]
        _, _, r = g.bfs(s["source"], case["mode"], copy_out=False)
        dist = C.c_void_p()
        gg.lib().gg_bfs_device_results(g.h, None, C.byref(dist))
        return [_tensor(dist.value, (V,), "<i4"), r["processed_nodes"], r["levels"]]
    if kind == "cc":
        g = s["g"]
        _, r = g.cc(case["algorithm"], copy_out=False)
        lab = C.c_void_p()
        gg.lib().gg_cc_device_labels(g.h, C.byref(lab))
        return [_tensor(lab.value, (V,), "<i4"), r["components"]]
    if kind == "ppr":
        g = s["g"]
        g.ppr(s["sets"], iterations=case["iterations"], storage=case["storage"], copy_out=False)
        stride = C.c_uint32()
        ptr = gg.lib().gg_ppr_device_ranks(g.h, C.byref(stride))
        return _tensor(ptr, (V, stride.value), "<f4")[:, :case["K"]]
    if kind == "load":
        g = gg.DeviceGraph.build(s["src"], s["dst"], s["w"], num_vertices=V, what=gg.MAP_ALL)
        x, y, _ = g.spmv("pull")
        g.free()
        return [x, y]
    ranks, _ = gg.pagerank_csr(s["graph"], s["args"], "pageRankPullGraphCSR")
    return ranks


# ---- what a call cannot do without ----------------------------------------

def work(case):
    """Bytes: ids, offsets and values once per pass over the graph; a graph's
    arrays are read again in each iteration."""
    kind, V = case["kind"], case["V"]
    E = V * case["ef"] * (2 if kind == "bfs" else 1)
    val = {"f32": 4, "bf16": 2, "f16": 2}.get(case.get("storage"), 4)
    if kind in ("rank", "dropin"):
        it = case["iterations"]
        val = {"pull_q16": 2, "pull_fx32": 4}.get(case.get("mode"), val)
        b = it * (4 * E + 4 * (V + 1) + 4 * V + 2 * val * V) + 4 * V
        if kind == "dropin":
            b += 4 * E + 8 * V
        return dict(bytes=b, flops=it * (E + 4 * V))
    if kind == "spmv":
        it = case["iterations"]
        return dict(bytes=it * ((4 + val) * E + 4 * (V + 1) + val * V + 4 * V) + 8 * V, flops=2 * it * E)
    if kind == "bfs":
        # every reached vertex needs one in-edge, the frontier bitmaps and the outputs
        return dict(bytes=4 * V + 8 * V + 8 * V + V // 2, flops=E)
    if kind == "cc":
        return dict(bytes=8 * V + 3 * 4 * V + 4 * V, flops=2 * V)
    if kind == "ppr":
        it, K = case["iterations"], case["K"]
        kp = 16 if K <= 16 else 32 if K <= 32 else 64
        return dict(bytes=it * (4 * E + 4 * (V + 1) + 8 * V + 2 * val * kp * V) + 4 * kp * V, flops=it * K * (E + 3 * V))
    # load: the edge list once, the arrays of both directions once, one product
    w = 4 * E if case["weighted"] else 0
    return dict(bytes=8 * E + w + 2 * (4 * E + 4 * V) + 2 * 4 * E + 4 * V + (8 * E + 4 * V) + 12 * V, flops=2 * E)


# ---- the same results in 64 bits ------------------------------------------

def _gather_sum(x, src, dst, V, w=None):
    """y[v] = sum over edges (u, v) of w * x[u], in float64."""
    y = torch.zeros(V, *x.shape[1:], dtype=torch.float64, device="cuda")
    step = max(1, (1 << 26) // max(1, x[0].numel()))
    for at in range(0, src.numel(), step):
        t = x.index_select(0, src[at:at + step])
        if w is not None:
            t.mul_(w[at:at + step])
        y.index_add_(0, dst[at:at + step], t)
    return y


def exact(case, seed):
    kind, V = case["kind"], case["V"]
    if kind in ("bfs", "cc"):
        return None  # whole numbers: the same on every side
    src, dst = _edges(case, seed)
    deg = torch.bincount(src, minlength=V).double()
    inv = torch.where(deg > 0, 1.0 / deg.clamp(min=1), torch.zeros_like(deg))
    damp = float(np.float32(0.85))
    if kind in ("rank", "dropin"):
        base = float(np.float32(1.0) - np.float32(0.85))
        r = torch.full((V,), base, dtype=torch.float64, device="cuda")
        for _ in range(case["iterations"]):
            r = base + damp * _gather_sum(r * inv, src, dst, V)
        return r / V
    if kind == "ppr":
        init = np.zeros((V, case["K"]))
        for k, st in enumerate(_seed_sets(case, seed)):
            np.add.at(init[:, k], st, 1.0 / len(st))
        init = torch.from_numpy(init).cuda()
        r = init
        for _ in range(case["iterations"]):
            r = (1.0 - damp) * init + damp * _gather_sum(r * inv[:, None], src, dst, V)
        return r
    if kind == "load":
        x = torch.where(deg > 0, 1.0 / deg.clamp(min=1), torch.full_like(deg, 0.001)).float()
        w = _weights(case, seed, src.numel()) if case["weighted"] else torch.full((1,), 0.0001, device="cuda").expand(src.numel())
        return [x.double(), _gather_sum(x.double(), src, dst, V, w.double())]
    x = torch.from_numpy(np.random.default_rng(seed).random(V, dtype=np.float32)).cuda().double()
    w = _weights(case, seed, src.numel()).double()
    return [x, _gather_sum(x, src, dst, V, w)]
