"""What the framework's speed is measured on: the calls its users make, over
their sizes.

Every case goes through the public entry points: ``Index.search`` /
``Index.search_device`` on a loaded index (the query-time path, which is what
the framework is for), ``ground_truth``, the graph constructions of
``parallel_anns_b200.graph`` and the training of the entry network. Sizes are
those of the benchmark workloads (1M x 96 mixture, d = 128 integer set,
100k x 96 small configuration) and of the tests, or lie between them.

A program keeps its index (base, graph, device layout, network) and searches
batch after batch on it, so an index belongs to a case's sizes and is shared by
its states; the queries come from the seed. Constructions and training get new
vectors from the seed.
"""
from __future__ import annotations

import collections
import math

import numpy as np
import torch

from parallel_anns_b200 import datasets as ds
from parallel_anns_b200 import learned as LE
from parallel_anns_b200 import native as N
from parallel_anns_b200.graph import build_nsg, build_nsg_cells
from parallel_anns_b200.searching import Index, ground_truth

STORES = {"fp32": N.STORE_FP32, "bf16": N.STORE_BF16, "fp8": N.STORE_FP8}
MODES = {"top_m": N.MODE_TOP_M, "seq": N.MODE_NSG_SEQ, "pss": N.MODE_PSS_V5, "efanna": N.MODE_EFANNA}
DISTS = {"ip": N.DIST_NORM_IP, "l2": N.DIST_L2}
COMPONENTS = 64
MEANS_SEED = 1001


def _search(name, **kw):
    """A search case: sizes of the index, then of the call."""
    c = {"do": "search", "data": "mixture", "n": 1_000_000, "d": 96, "R": 50, "copy": "fp32", "nq": 10_000, "K": 100,
         "L": 384, "mode": "top_m", "M": 8, "T": 1, "distance": "ip", "storage": "fp32", "learned": False,
         "graph_launch": False, "via": "host"}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # An online service's single query against the 1M index: the whole
        # host call, launch and latency of one search.
        _search("online_1_query", copy="fp8", nq=1),
        # A micro-batch of a server that captures its launch, on a BF16 copy.
        _search("online_64_queries_bf16", n=200_000, copy="bf16", storage="bf16", nq=64, L=256, graph_launch=True),
        # The headline: 10,000 device-resident queries, exact float32 search.
        _search("batch_10k_fp32", copy="fp8", via="device"),
        # The fastest configuration of the benchmark end to end: the FP8 copy
        # with the learned entries, queries and results in pinned host memory.
        _search("batch_10k_fp8_learned", copy="fp8", storage="fp8", learned=True, via="pinned"),
        # Integer-valued descriptors that need a long queue (d = 128, R = 64).
        _search("batch_1k_u8_long_queue", data="uint8", n=100_000, d=128, R=64, nq=1000, L=2048, via="device"),
        # PSS_v5 with its T queues on the small configuration.
        _search("pss_1k_queries", n=100_000, nq=1000, L=200, mode="pss", T=4, M=1),
        # efanna2e's search (full L2, random init lists), a dimension whose
        # reference lane order has a ragged tail, a batch of odd size.
        _search("efanna_999_queries_d200", n=30_000, d=200, nq=999, K=50, L=150, mode="efanna", M=1, distance="l2"),
        # Float64 ground truth of an evaluation set on the 1M base.
        {"name": "ground_truth_10k", "do": "truth", "n": 1_000_000, "d": 96, "nq": 10_000, "k": 100},
        # Graph construction of a medium base (all pairs, tensor-core screen).
        {"name": "build_250k_d96", "do": "build", "n": 250_000, "d": 96, "knn_k": 64, "R": 50},
        # A small base of ragged sizes (all pairs, float32 screen).
        {"name": "build_20011_d104", "do": "build", "n": 20_011, "d": 104, "knn_k": 64, "R": 50},
        # The large configuration's construction, scaled down: k-means cells,
        # k-NN within near cells, reverse edges.
        {"name": "build_cells_200k", "do": "cells", "n": 200_000, "d": 96, "knn_k": 64, "R": 48, "cells": 200,
         "probe": 3, "reverse": True},
        # Training the entry network: forward, backward and Adam.
        {"name": "train_32k", "do": "train", "n": 32_768, "d": 96, "R": 1024, "T": 10, "batch": 1024, "epochs": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _search_bytes(c):
    """Bytes of one query's gathers (see work())."""
    size = {"fp32": 4, "bf16": 2, "fp8": 1}[c["storage"]]
    dist = 15 * c["L"]
    rerank = 0 if c["storage"] == "fp32" else 4 * c["d"] * c["L"]
    return dist * (size * c["d"] + 4) + 4 * 19 * c["L"] + rerank + 4 * c["d"] + 4 * c["K"]


def draw(rng):
    do = rng.choice(["search"] * 5 + ["truth", "build", "cells", "train"])
    if do == "search":
        kind = rng.choice(["top_m"] * 5 + ["seq", "pss", "efanna"])
        n = _log(rng, 4000, 300_000)
        d = 8 * rng.randint(3, 32 if n < 100_000 else 16)
        data = rng.choice(["mixture", "mixture", "mixture", "uint8"])
        storage = rng.choice(["fp32", "fp32", "bf16", "fp8"]) if kind in ("top_m", "seq") else "fp32"
        L = _log(rng, 100, 300 if kind in ("pss", "efanna") else 2500)
        c = _search(None, data=data, n=n, d=d, R=rng.choice([32, 50, 64]), copy=storage, storage=storage,
                    K=rng.choice([10, 50, 100]), L=L, mode=kind,
                    M=rng.choice([2, 4, 8, 16, 33]) if kind == "top_m" else 1,
                    T=rng.choice([2, 4, 8]) if kind == "pss" else 1,
                    distance="ip" if storage != "fp32" else rng.choice(["ip", "l2"]))
        c["learned"] = kind == "top_m" and data == "mixture" and n >= 50_000 and rng.random() < 0.4
        nq = _log(rng, 1, 10_000)
        most = 0.5 * 10_000 * _search_bytes(_search(None)) / _search_bytes(c)
        c["nq"] = max(1, min(nq, int(most), 2000 if kind in ("pss", "efanna") else nq))
        c["via"] = rng.choice(["host", "device", "pinned"])
        c["graph_launch"] = c["nq"] <= 64 and rng.random() < 0.5
        return c
    if do == "truth":
        return {"do": do, "n": _log(rng, 5000, 400_000), "d": 8 * rng.randint(3, 16), "nq": _log(rng, 10, 9000),
                "k": rng.choice([10, 50, 100])}
    if do == "build":
        n = _log(rng, 2000, 200_000)
        d = 8 * rng.randint(3, 32 if n < 60_000 else 16)
        k = rng.choice([32, 50, 64, 100])
        return {"do": do, "n": n, "d": d, "knn_k": k, "R": rng.randint(k // 2, k)}
    if do == "cells":
        n = _log(rng, 20_000, 200_000)
        return {"do": do, "n": n, "d": 8 * rng.randint(3, 16), "knn_k": 64, "R": rng.choice([32, 48, 64]),
                "cells": rng.randint(max(8, n // 2500), n // 800), "probe": rng.randint(1, 3),
                "reverse": rng.random() < 0.5}
    n = _log(rng, 3000, 32_000)
    return {"do": do, "n": n, "d": 8 * rng.randint(3, 16), "R": rng.choice([256, 512, 1024]), "T": rng.randint(1, 10),
            "batch": min(n, _log(rng, 200, 2048)), "epochs": rng.randint(1, 2)}


# -- inputs -------------------------------------------------------------------

def _vectors(data, n, d, seed):
    if data == "uint8":
        return ds.uint8_cube(n, d, seed=seed)
    return ds.gaussian_mixture_gpu(n, d, COMPONENTS, 0.3, seed=seed, means_seed=MEANS_SEED)


_indices = collections.OrderedDict()  # the last few indices, by their sizes


def _index(data, n, d, R, copy, learned):
    """The loaded index of these sizes, as a program keeps it between calls."""
    key = (data, n, d, R, copy)
    have = _indices.pop(key, None)
    if have is None:
        while len(_indices) >= 5:
            _indices.popitem(last=False)[1]["index"].close()
        base = _vectors(data, n, d, 1002 if data == "uint8" else MEANS_SEED)
        ix = Index(0)
        ix.set_base(base, storage=STORES[copy])
        ix.set_graph(build_nsg(base, R=R, knn_k=64))
        have = {"index": ix, "learned": False}
    _indices[key] = have
    if learned and not have["learned"]:
        # The entry network of the benchmark's pipeline on a smaller training set.
        ix = have["index"]
        cells = 1024 if n >= 500_000 else 256
        q = _vectors(data, 20_000, d, 77)
        reps, assign = LE.kmeans(ix, cells, 6, 1)
        lab, y, _ = LE.traces(ix, q, assign, K=min(100, n), L_ref=300, T=10, L_grid=(150,))
        params, _ = LE.train(q, lab, y, cells, epochs=4)
        LE.attach(ix, LE.LearnedModel(d, cells, params, reps), E=8, L_init=8, use_L=False)
        have["learned"] = True
    return have["index"]


def _training_set(case, seed):
    """Queries, the cells of their nearest representatives and ln L targets."""
    x = _vectors("mixture", case["n"], case["d"], seed)
    xt = torch.from_numpy(x).cuda()
    reps = torch.from_numpy(_vectors("mixture", case["R"], case["d"], 5)).cuda()
    near = torch.cdist(xt, reps).topk(case["T"], dim=1, largest=False).indices
    rng = np.random.default_rng(seed)
    y = np.log(rng.choice(np.array(LE.DEFAULT_L_GRID), size=case["n"])).astype(np.float32)
    params = LE.init_params(case["d"], case["R"], seed, float(y.mean()))
    return x, near.cpu().numpy().astype(np.uint16), y, params


def prepare(case, seed):
    do, seed = case["do"], int(seed) % (1 << 30)
    if do == "search":
        ix = _index(case["data"], case["n"], case["d"], case["R"], case["copy"], case["learned"])
        q = _vectors(case["data"], case["nq"], case["d"], 10_000 + seed)
        s = {"index": ix, "case": case}
        flags = (N.FLAG_LEARNED if case["learned"] else 0) | (N.FLAG_CUDA_GRAPH if case["graph_launch"] else 0)
        s["call"] = dict(K=case["K"], L=case["L"], mode=MODES[case["mode"]], distance=DISTS[case["distance"]],
                         M=case["M"], T=case["T"], storage=STORES[case["storage"]], flags=flags)
        if case["via"] == "device":
            s["queries"] = torch.from_numpy(q).cuda()
            s["out"] = torch.empty((case["nq"], case["K"]), dtype=torch.int32, device="cuda")
        elif case["via"] == "pinned":
            s["pinned"] = torch.from_numpy(q).pin_memory(), torch.empty((case["nq"], case["K"]),
                                                                        dtype=torch.int32).pin_memory()
            s["queries"], s["out"] = s["pinned"][0].numpy(), s["pinned"][1].numpy().view(np.uint32)
        else:
            s["queries"], s["out"] = q, None
        return s
    if do == "truth":
        ix = _index("mixture", case["n"], case["d"], 50, "fp8", False)
        return {"index": ix, "case": case, "queries": _vectors("mixture", case["nq"], case["d"], 10_000 + seed)}
    if do == "train":
        x, cells, y, params = _training_set(case, 10_000 + seed)
        return {"case": case, "x": x, "cells": cells, "y": y, "params": params}
    # The adjacency goes to a buffer of fixed size: the edge count depends on the vectors.
    return {"case": case, "base": _vectors("mixture", case["n"], case["d"], 10_000 + seed),
            "nbrs": np.zeros(case["n"] * (case["R"] + 1), dtype=np.int32)}


# -- one pass -----------------------------------------------------------------

def run(state):
    case = state["case"]
    do = case["do"]
    if do == "search":
        if case["via"] == "device":
            state["index"].search_device(state["queries"], state["out"], **state["call"])
            return state["out"]
        ids, stats = state["index"].search(state["queries"], out=state["out"], **state["call"])
        return {"ids": ids.view(np.int32), "n_dist": stats["n_dist"]}
    if do == "truth":
        ids, dist = ground_truth(state["index"], state["queries"], case["k"])
        return {"ids": ids.view(np.int32), "dist": dist}
    if do == "train":
        params, losses = LE.train(state["x"], state["cells"], state["y"], case["R"], epochs=case["epochs"],
                                  batch=case["batch"], params=state["params"])
        return {"params": params, "losses": losses}
    if do == "build":
        g, knn = build_nsg(state["base"], R=case["R"], knn_k=case["knn_k"], with_knn=True)
    else:
        g, knn = build_nsg_cells(state["base"], R=case["R"], knn_k=case["knn_k"], cells=case["cells"],
                                 probe=case["probe"], reverse=case["reverse"], with_knn=True)
    state["nbrs"][:g.nbrs.size] = g.nbrs.view(np.int32)
    return {"entry": g.entry, "offsets": g.offsets, "nbrs": state["nbrs"], "knn": knn.view(np.int32)}


# -- what a pass cannot do without ---------------------------------------------

def work(case):
    do, d = case["do"], case["d"]
    if do == "search":
        # Distances and expansions of a search with queue length L: about 15 L
        # and L on these graphs (mean degree 18), each row read once.
        return {"bytes": case["nq"] * _search_bytes(case), "flops": case["nq"] * 15 * case["L"] * 2 * d}
    if do == "truth":
        return {"bytes": 4 * d * (case["n"] + case["nq"]) + 12 * case["nq"] * case["k"],
                "flops": 2 * d * case["n"] * case["nq"]}
    if do == "train":
        P = d * 256 + 256 * 256 + 256 * (case["R"] + 1)
        steps = case["n"] // case["batch"] * case["epochs"]
        return {"bytes": case["n"] * (4 * d + 2 * case["T"] + 4) + steps * 26 * P,
                "flops": 6 * P * case["batch"] * steps}
    pairs = case["n"] * case["n"]
    if do == "cells":
        pairs = pairs // case["cells"] * (case["probe"] + 1) + 11 * case["n"] * case["cells"]
    return {"bytes": case["n"] * (4 * d + 4 * case["knn_k"] + 4 * 20 + 8), "flops": 2 * d * pairs}


# -- the same in 64 bits --------------------------------------------------------

def _exact_truth(case, seed):
    base = torch.from_numpy(_vectors("mixture", case["n"], case["d"], MEANS_SEED)).cuda().double()
    q = torch.from_numpy(_vectors("mixture", case["nq"], case["d"], 10_000 + seed % (1 << 30))).cuda().double()
    bn, k = (base * base).sum(1), case["k"]
    out = torch.empty((case["nq"], k), dtype=torch.float64)
    for r in range(0, case["nq"], 250):
        x = q[r:r + 250]
        near = torch.topk(bn[None, :] - 2.0 * (x @ base.T), min(k + 16, case["n"]), dim=1, largest=False).indices
        dist = (base[near] - x[:, None, :]).square().sum(2)
        out[r:r + 250] = dist.sort(dim=1).values[:, :k].cpu()
    return {"ids": None, "dist": out}


def _mt19937_64(seed):
    """The 64-bit Mersenne Twister (Nishimura, 2000), as std::mt19937_64 draws it."""
    mask = (1 << 64) - 1
    mt = [seed & mask]
    for i in range(1, 312):
        mt.append((6364136223846793005 * (mt[-1] ^ (mt[-1] >> 62)) + i) & mask)
    while True:
        for i in range(312):
            x = (mt[i] & 0xFFFFFFFF80000000) | (mt[(i + 1) % 312] & 0x7FFFFFFF)
            mt[i] = mt[(i + 156) % 312] ^ (x >> 1) ^ (0xB5026F5AA96619E9 if x & 1 else 0)
        for x in mt:
            x ^= (x >> 29) & 0x5555555555555555
            x ^= (x << 17) & 0x71D67FFFEDA60000
            x ^= (x << 37) & 0xFFF7EEE000000000
            yield (x ^ (x >> 43)) & mask


def _exact_train(case, seed):
    """Adam on the network, sums and state in float64, weights used as BF16."""
    x, cells, y, params = _training_set(case, 10_000 + seed % (1 << 30))
    d, R, T, H, B = case["d"], case["R"], case["T"], 256, case["batch"]
    X, Y = torch.from_numpy(x).cuda().double(), torch.from_numpy(y).cuda().double()
    C = torch.zeros((case["n"], R), dtype=torch.float64, device="cuda")
    idx = torch.from_numpy(cells.astype(np.int64)).cuda()
    C.scatter_add_(1, idx, torch.full(idx.shape, 1.0 / T, dtype=torch.float64, device="cuda"))
    w = torch.from_numpy(params).cuda().double()
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    cut = np.cumsum([0, d * H, H, H * H, H, H * (R + 1), R + 1])
    part = [slice(int(a), int(b)) for a, b in zip(cut[:-1], cut[1:])]
    draws, losses, step = _mt19937_64(0), [], 0
    f32 = lambda t: float(np.float32(t))  # noqa: E731
    lr, b1, b2, eps = f32(2e-3), f32(0.9), f32(0.999), f32(1e-8)
    for _ in range(case["epochs"]):
        order = list(range(case["n"]))
        for i in range(case["n"] - 1, 0, -1):
            j = next(draws) % (i + 1)
            order[i], order[j] = order[j], order[i]
        order = torch.tensor(order, device="cuda")
        total = 0.0
        for s in range(case["n"] // B):
            r = order[s * B:(s + 1) * B]
            xb, cb, yb = X[r], C[r], Y[r]
            wb = w.float().bfloat16().double()
            W1, W2, W3 = wb[part[0]].view(d, H), wb[part[2]].view(H, H), wb[part[4]].view(H, R + 1)
            h1 = (xb @ W1 + w[part[1]]).relu()
            h2 = (h1 @ W2 + w[part[3]]).relu()
            z = h2 @ W3 + w[part[5]]
            lse = torch.logsumexp(z[:, :R], 1)
            e = z[:, R] - yb
            total += float((lse - (cb * z[:, :R]).sum(1) + 0.5 * e * e).mean())
            dz = torch.cat([torch.exp(z[:, :R] - lse[:, None]) - cb, e[:, None]], 1) / B
            g = torch.empty_like(w)
            g[part[4]], g[part[5]] = (h2.T @ dz).reshape(-1), dz.sum(0)
            dh2 = (dz @ W3.T) * (h2 > 0)
            g[part[2]], g[part[3]] = (h1.T @ dh2).reshape(-1), dh2.sum(0)
            dh1 = (dh2 @ W2.T) * (h1 > 0)
            g[part[0]], g[part[1]] = (xb.T @ dh1).reshape(-1), dh1.sum(0)
            step += 1
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            w = w - lr * (m / (1 - b1 ** step)) / ((v / (1 - b2 ** step)).sqrt() + eps)
        losses.append(total / (case["n"] // B))
    return {"params": w, "losses": torch.tensor(losses, dtype=torch.float64)}


def exact(case, seed):
    if case["do"] == "truth":
        return _exact_truth(case, int(seed))
    if case["do"] == "train":
        return _exact_train(case, int(seed))
    return None  # vertex ids and counts: whole numbers
