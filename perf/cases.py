"""The work that users of pydiskann_b200 have it do, as timed cases.

Vectors follow the generators of ``pydiskann_b200/synth.py``: integer-valued
isotropic Gaussian mixtures clipped to [0, 255] (SIFT-like descriptors), not
clipped and Zipf weighted for the posting lists, and unit-norm embeddings with
a power-law spectrum for the cosine cases.  Labels are 1-3 of 100 per vector,
Zipf(1.0).  Everything is drawn on the GPU so that an index of a million rows
is in hand within seconds.

Search graphs come from outside, as ``DiskANN.from_graph`` takes them: a row
holds the nearest rows of its own mixture component (spread over ranks as a
pruned graph spreads them), some random rows of it and some random rows of the
whole set, which is what a Vamana graph of such data consists of.  Building a
graph with the library is a case of its own.

Kinds:
  search    batched beam search: FP32 rows, BF16 / FP8 rows + FP32 rerank, PQ,
            int8, F16 or RaBitQ codes + FP32 rerank; L2 or cosine; queries and
            results in HBM or in host arrays; one beam or a beam per query
  one       one query through ``search_with_dists``
  filtered  label-filtered beam search, a filter per query
  spfresh   posting-list search (routing + scans), raw or quantized postings
  build     Vamana graph construction
  pq_train  PQ codebook training and encoding of the same rows
  knn       exact nearest neighbours (ground truth)
"""
from __future__ import annotations

import math

import numpy as np
import torch

import pydiskann_b200 as dg
from pydiskann_b200 import _lib

_TRAV = {"f32": _lib.TRAVERSE_F32, "bf16": _lib.TRAVERSE_BF16, "fp8": _lib.TRAVERSE_FP8, "codes": _lib.TRAVERSE_CODES}


def listed():
    return [
        # an interactive lookup: one query, the class's default beam, Python lists out
        dict(name="one_query_100k", kind="one", n=100_000, d=128, centres=64, R=64, k=10, L=128),
        # what a serving loop launches at moderate load: a batch far smaller than the GPU
        dict(name="serve_batch64_bf16", kind="search", n=500_000, d=128, centres=256, R=64, nq=64, k=10, L=64,
             trav="bf16", rerank=64, metric="l2", host=False, uneven=False),
        # the benchmark's batch on FP32 rows: 10k queries at the beam that reaches recall 0.95
        dict(name="batch10k_f32", kind="search", n=1_000_000, d=128, centres=256, R=64, nq=10_000, k=10, L=40,
             trav="f32", rerank=0, metric="l2", host=False, uneven=False),
        # the same batch on BF16 rows with the FP32 rerank, the headline variant
        dict(name="batch10k_bf16_rerank", kind="search", n=1_000_000, d=128, centres=256, R=64, nq=10_000, k=10, L=40,
             trav="bf16", rerank=40, metric="l2", host=False, uneven=False),
        # PQ codes (M = 16) at the wide beam that coarse codes need, host arrays in and out
        dict(name="pq_host_L128", kind="search", n=500_000, d=128, centres=64, R=64, nq=5_000, k=10, L=128,
             trav="codes", quant="pq", M=16, rerank=128, metric="l2", host=True, uneven=False),
        # text-embedding search: 768 dimensions, cosine over int8 codes, every query its own beam of 32..256
        dict(name="cosine768_int8_uneven", kind="search", n=150_000, d=768, centres=0, R=64, nq=4_000, k=10, L=256,
             trav="codes", quant="int8", rerank=40, metric="cosine", host=False, uneven=True),
        # label-filtered serving batch: selectivity 0.5-35 %, working lists of 4 L = 256
        dict(name="filtered_k10_bf16", kind="filtered", n=300_000, d=256, centres=512, R=48, nq=2_000, k=10, L=64,
             trav="bf16", rerank=64),
        # filtered retrieval of long result lists: k = 100 expands the working list to 1000
        dict(name="filtered_k100_f32", kind="filtered", n=300_000, d=256, centres=512, R=48, nq=500, k=100, L=64,
             trav="f32", rerank=0),
        # SPFresh search after a bulk load, raw postings of 96-d rows, 64 probes per query
        dict(name="spfresh_raw_p64", kind="spfresh", n=300_000, d=96, centres=1024, quant=None, nq=10_000, k=10,
             nprobe=64, rerank=0, host=False),
        # index construction at the class's defaults (R = 64, build beam 128)
        dict(name="build_25k", kind="build", n=25_000, d=128, centres=64, R=64, Lb=128),
        # PQ codebooks as QuantizedDiskANN.build trains them (50k sample, 20 Lloyd steps) and the codes of 200k rows
        dict(name="pq_train_200k", kind="pq_train", n=200_000, d=128, centres=256, M=16, iters=20),
        # ground truth of 1000 queries, the recall check that goes with every configuration
        dict(name="exact_knn_100k", kind="knn", n=100_000, d=128, centres=64, nq=1_000, k=10, metric="l2"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: kinds by how often they run, sizes over the logarithm of their range."""
    kind = rng.choice(["search"] * 5 + ["one", "filtered", "filtered", "spfresh", "spfresh", "build", "pq_train", "knn"])
    if kind == "one":
        return dict(kind="one", n=_log(rng, 5_000, 200_000), d=rng.choice([32, 64, 96, 100, 128, 200, 256]), centres=64,
                    R=rng.choice([32, 48, 64]), k=rng.choice([1, 10, 50]), L=_log(rng, 50, 256))
    if kind == "search":
        trav = rng.choice(["f32", "f32", "bf16", "bf16", "fp8", "codes", "codes"])
        d = rng.choice([32, 50, 96, 100, 128, 200, 256])
        c = dict(kind="search", n=_log(rng, 20_000, 400_000), d=d, centres=rng.choice([64, 256]),
                 R=rng.choice([32, 48, 64]), nq=_log(rng, 8, 6_000), k=rng.choice([1, 10, 10, 20]),
                 L=_log(rng, 20, 256), trav=trav, rerank=0, metric="l2", host=rng.random() < 0.3,
                 uneven=rng.random() < 0.25)
        if trav != "f32":
            c["rerank"] = rng.choice([0, c["L"], c["L"]])
        if trav == "codes":
            c["quant"] = rng.choice(["pq", "int8", "f16", "rabitq"])
            if c["quant"] == "pq":
                c["M"] = next(m for m in (16, 10, 8) if d % m == 0) if d != 50 else 10
        return c
    if kind == "filtered":
        return dict(kind="filtered", n=_log(rng, 20_000, 300_000), d=rng.choice([64, 100, 128, 256]),
                    centres=rng.choice([64, 512]), R=rng.choice([32, 48, 64]), nq=_log(rng, 50, 1_500),
                    k=rng.choice([10, 10, 25, 100]), L=_log(rng, 40, 200), trav=rng.choice(["f32", "bf16"]), rerank=0)
    if kind == "spfresh":
        return dict(kind="spfresh", n=_log(rng, 20_000, 200_000), d=rng.choice([32, 64, 96, 100, 128]),
                    centres=rng.choice([64, 1024]), quant=rng.choice([None, None, "int8", "f16", "pq"]),
                    nq=_log(rng, 20, 6_000), k=rng.choice([1, 10, 20]), nprobe=_log(rng, 8, 128),
                    rerank=rng.choice([0, 40]), host=rng.random() < 0.3)
    if kind == "build":
        return dict(kind="build", n=_log(rng, 2_000, 20_000), d=rng.choice([32, 64, 100, 128]), centres=64,
                    R=rng.choice([32, 48, 64]), Lb=_log(rng, 48, 128))
    if kind == "pq_train":
        d = rng.choice([32, 64, 96, 128])
        return dict(kind="pq_train", n=_log(rng, 5_000, 150_000), d=d, centres=64, M=rng.choice([8, 16]),
                    iters=rng.choice([5, 10, 20]))
    return dict(kind="knn", n=_log(rng, 10_000, 100_000), d=rng.choice([32, 64, 96, 100, 128]), centres=64,
                nq=_log(rng, 50, 1_000), k=rng.choice([1, 10, 100]), metric=rng.choice(["l2", "l2", "cosine"]))


# ------------------------------------------------------------------ inputs
def _gen(seed, stream):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * (seed + 1) + stream)


def _mixture(n, nq, d, centres, seed, clip=True, zipf=0.0):
    """(rows, component of each row, queries): integer-valued float32 on the GPU."""
    g = _gen(seed, 0)
    C = torch.rand((centres, d), generator=g, device="cuda") * 255.0
    w = torch.arange(1, centres + 1, device="cuda", dtype=torch.float32) ** -zipf

    def rows(m, stream):
        gg = _gen(seed, stream)
        z = torch.multinomial(w, m, replacement=True, generator=gg)
        x = torch.randn((m, d), generator=gg, device="cuda").mul_(20.0).add_(C[z]).round_()
        return (x.clamp_(0.0, 255.0) if clip else x), z

    X, z = rows(n, 1)
    return X, z, rows(max(nq, 1), 2)[0][:nq]


def _embeddings(n, nq, d, seed):
    """Unit-norm rows with variance spectrum (i + 1)^-0.5, stored as BF16 values."""
    sig = torch.arange(1, d + 1, device="cuda", dtype=torch.float32) ** -0.25

    def rows(m, stream):
        x = torch.randn((m, d), generator=_gen(seed, stream), device="cuda").mul_(sig)
        return torch.nn.functional.normalize(x, dim=1).bfloat16().float()

    return rows(n, 1), rows(max(nq, 1), 2)[:nq]


def _near_lists(X, ids, near, spread):
    """For the rows `ids` of X: `near` nearest of them and `spread` more at growing ranks, int64 row numbers."""
    Y = X[ids]
    m = len(ids)
    ranks = torch.arange(1, near + 1)
    if spread:
        far = torch.logspace(math.log10(near + 1), math.log10(max(near + spread + 1, m // 4)), spread).long()
        ranks = torch.cat([ranks, torch.maximum(far, near + 1 + torch.arange(spread))])
    depth = min(int(ranks[-1]) + 1, m)
    ranks = ranks.clamp(max=m - 1).cuda()
    out = []
    y2 = (Y * Y).sum(1)
    for s in range(0, m, 4096):
        D = y2[s:s + 4096, None] + y2[None, :] - 2.0 * (Y[s:s + 4096] @ Y.T)
        # (distance, position) in one sortable whole number: no ties
        key = (D.round().clamp_(min=0).long() << 20) | torch.arange(m, device="cuda")
        out.append(torch.topk(key, depth, dim=1, largest=False, sorted=True).values[:, ranks] & 0xFFFFF)
    return ids[torch.cat(out)]


def _graph(X, z, centres, R, seed):
    """Adjacency u32[n, R] (host) and an entry row."""
    n = len(X)
    g = _gen(seed, 3)
    near, spread, wide = (R * 5) // 8, R // 8, R // 8
    adj = torch.randint(0, n, (n, R), generator=g, device="cuda")  # the last R - near - spread columns: any rows
    if centres:
        order = torch.argsort(z, stable=True)
        bounds = torch.cumsum(torch.bincount(z, minlength=centres), 0).cpu().tolist()
        lo = 0
        for hi in bounds:
            ids = order[lo:hi]
            if hi - lo > 1:
                adj[ids, :near + spread] = _near_lists(X, ids, near, spread)
                pick = torch.randint(0, hi - lo, (hi - lo, wide), generator=g, device="cuda")
                adj[ids, near + spread:near + spread + wide] = ids[pick]  # random rows of the component
            lo = hi
    else:
        for s in range(0, n, 2048):  # one cloud of unit rows: the nearest by inner product
            key = ((1.0 - X[s:s + 2048] @ X.T).clamp_(min=0) * (1 << 30)).long() << 20 | torch.arange(n, device="cuda")
            adj[s:s + 2048, :near] = torch.topk(key, near + 1, dim=1, largest=False).values[:, 1:] & 0xFFFFF
    adj = adj.to(torch.int32)
    # a row lists a neighbour once and never itself: repeats become padding at the end of the row
    srt, pos = torch.sort(adj, dim=1, stable=True)
    rep = torch.zeros_like(srt, dtype=torch.bool)
    rep[:, 1:] = srt[:, 1:] == srt[:, :-1]
    rep |= srt == torch.arange(n, device="cuda", dtype=torch.int32)[:, None]
    mask = torch.zeros_like(rep).scatter_(1, pos, rep)
    keep = torch.argsort(mask.to(torch.int8), dim=1, stable=True)
    adj = torch.where(mask, torch.full_like(adj, -1), adj).gather(1, keep)
    entry = int(((X - X.mean(0)) ** 2).sum(1).round().argmin())
    return adj.cpu().numpy().view(np.uint32), entry


def _labels(n, seed, n_labels=100, per=3):
    """1-3 distinct labels of 1..100 per row, Zipf(1.0), padded with u64::MAX."""
    g = _gen(seed, 4)
    w = torch.arange(1, n_labels + 1, device="cuda", dtype=torch.float32) ** -1.0
    lab = torch.multinomial(w.expand(n, n_labels), per, generator=g) + 1
    cnt = torch.randint(1, per + 1, (n, 1), generator=g, device="cuda")
    lab[torch.arange(per, device="cuda")[None, :] >= cnt] = -1
    return lab.cpu().numpy().view(np.uint64)


def _beams(case, seed):
    rng = np.random.default_rng([seed, 5])
    return rng.integers(max(case["L"] // 8, case["k"]), case["L"] + 1, case["nq"]).astype(np.uint32)


def prepare(case, seed):
    """What a user's program holds before the call: the index (plan) and this seed's inputs."""
    kind, d = case["kind"], case["d"]
    s = {"case": case}
    if kind in ("search", "one"):
        nq = case.get("nq", 1)
        metric = case.get("metric", "l2")
        if metric == "cosine":
            (X, Q), z = _embeddings(case["n"], nq, d, seed), None
        else:
            X, z, Q = _mixture(case["n"], nq, d, case["centres"], seed)
        adj, entry = _graph(X, z, case["centres"], case["R"], seed)
        Xh = X.cpu().numpy()
        trav = case.get("trav", "f32")
        if trav == "codes":
            idx = dg.QuantizedDiskANN(Xh, adj, entry, metric, rerank_size=case["rerank"])
            if case["quant"] == "pq":  # codebooks from a small sample: their training is a case of its own
                idx.attach_pq(dg.pq_train(Xh[:8192], case["M"], 256, 4, 8192, seed=1))
            elif case["quant"] == "int8":
                idx.attach_int8(*dg.int8_params(Xh))
            elif case["quant"] == "f16":
                idx.attach_f16()
            else:
                idx.attach_rabitq(*dg.rabitq_params(Xh, 0))
        else:
            idx = dg.DiskANN.from_graph(Xh, adj, entry, metric)
            if trav == "bf16":
                idx.enable_bf16()
            elif trav == "fp8":
                idx.enable_fp8()
        s["idx"] = idx
        s["Q"] = Q.cpu().numpy() if kind == "one" or case["host"] else Q.contiguous()
        s["beams"] = _beams(case, seed) if case.get("uneven") else None
    elif kind == "filtered":
        X, z, Q = _mixture(case["n"], case["nq"], d, case["centres"], seed)
        adj, entry = _graph(X, z, case["centres"], case["R"], seed)
        idx = dg.FilteredDiskANN(X.cpu().numpy(), adj, entry, _labels(case["n"], seed))
        if case["trav"] == "bf16":
            idx.enable_bf16()
        want = np.random.default_rng([seed, 6]).integers(1, 101, case["nq"])
        s["idx"], s["Q"] = idx, Q.contiguous()
        s["filters"] = dg.pack_filters([dg.Filter.or_([dg.Filter.eq(f, int(w)) for f in range(3)]) for w in want])
    elif kind == "spfresh":
        X, _, Q = _mixture(case["n"], case["nq"], d, case["centres"], seed, clip=False, zipf=1.1)
        s["idx"] = dg.SPFresh.bulk_load(X.cpu().numpy(), "l2", case["quant"], rerank_size=case["rerank"],
                                        max_posting_size=128)
        s["Q"] = Q.cpu().numpy() if case["host"] else Q.contiguous()
    elif kind == "build":
        s["X"] = _mixture(case["n"], 0, d, case["centres"], seed)[0].cpu().numpy()
    elif kind == "pq_train":
        s["X"] = _mixture(case["n"], 0, d, case["centres"], seed)[0].cpu().numpy()
    elif case["metric"] == "cosine":
        X, Q = _embeddings(case["n"], case["nq"], d, seed)
        s["X"], s["Q"] = X.cpu().numpy(), Q.cpu().numpy()
    else:
        X, _, Q = _mixture(case["n"], case["nq"], d, case["centres"], seed)
        s["X"], s["Q"] = X.cpu().numpy(), Q.cpu().numpy()
    return s


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "one":
        return state["idx"].search_with_dists(state["Q"][0], c["k"], c["L"])
    if kind == "search":
        return state["idx"].search_arrays(state["Q"], c["k"], c["L"], traversal=_TRAV[c["trav"]],
                                          rerank_size=c["rerank"], per_query_beam=state["beams"])
    if kind == "filtered":
        return state["idx"].search_arrays(state["Q"], c["k"], c["L"], traversal=_TRAV[c["trav"]],
                                          rerank_size=c["rerank"], filters=state["filters"])
    if kind == "spfresh":
        return state["idx"].search_arrays(state["Q"], c["k"], c["nprobe"])
    if kind == "build":
        return dg.build_graph(state["X"], c["R"], c["Lb"], 1.2)
    if kind == "pq_train":
        cb = dg.pq_train(state["X"], c["M"], 256, c["iters"], 50_000, seed=0)
        return cb, dg.pq_encode(state["X"], cb)
    return dg.exact_knn(state["X"], state["Q"], c["k"], c["metric"])


def work(case):
    """Bytes and operations that a pass cannot do without."""
    kind, d = case["kind"], case["d"]
    if kind in ("search", "one", "filtered"):
        nq, k, R, L = case.get("nq", 1), case["k"], case["R"], case["L"]
        if case.get("uneven"):
            L = (max(case["L"] // 8, k) + L) / 2
        if kind == "filtered":
            L = max(4 * L, 10 * k)
        # every entry of the final list is expanded; about two thirds of the listed neighbours are new
        E = L + 3
        N = min(0.66 * E * R, case["n"])
        row = {"f32": 4 * d, "bf16": 2 * d, "fp8": d + 8}.get(case.get("trav", "f32"))
        if row is None:
            row = {"pq": case.get("M", 0), "int8": d + 4, "f16": 2 * d, "rabitq": d / 8 + 8}[case["quant"]]
        rr = max(case["rerank"], k) * 4 * d if case.get("rerank") else 0
        per = E * 4 * R + N * row + rr + 4 * d + 8 * k + 4
        if kind == "filtered":
            per += N * 24
        # no row, code or neighbour list has to cross HBM twice in one pass
        index = case["n"] * (4 * R + row + (4 * d if rr else 0) + (24 if kind == "filtered" else 0))
        return {"bytes": min(nq * per, index + nq * (4 * d + 8 * k + 4)), "flops": nq * N * 3 * d}
    if kind == "spfresh":
        lists = case["n"] / 40.0  # postings after the splits of a bulk load
        probed = min(case["nprobe"], lists)
        code = {None: 4 * d, "int8": d, "f16": 2 * d, "pq": 8}[case["quant"]]
        scanned = case["nq"] * probed * 40.0
        byts = min(scanned, case["n"]) * (code + 4) + lists * 4 * d + case["nq"] * (4 * d + 12 * case["k"] + 4)
        return {"bytes": byts, "flops": 2 * d * (scanned + case["nq"] * lists)}
    if kind == "build":
        n, R, Lb = case["n"], case["R"], case["Lb"]
        # two passes: three searches per row, the prune's pair distances, the same for the reverse edges
        N = 3 * min(0.66 * (Lb + 3) * R, n)
        return {"bytes": n * (4 * d + 4 * R), "flops": 2 * n * 3 * d * (N + 2 * R * R)}
    if kind == "pq_train":
        n, ns = case["n"], min(case["n"], 50_000)
        return {"bytes": n * (4 * d + case["M"]) + 256 * 4 * d, "flops": 3 * 256 * d * (ns * (case["iters"] + 1) + n)}
    n, nq = case["n"], case["nq"]
    return {"bytes": 4 * d * (n + nq) + 8 * nq * case["k"], "flops": 2 * d * n * nq}


# ------------------------------------------------------ 64-bit results
def _beam64(X, adj, entry, Q, k, L):
    """Best-first beam search in 64 bits, all queries in step: distances f64[nq, k], inf where a list ends early.
    The list holds the L smallest (distance, row) pairs seen; the search ends at its first expanded-out or full list."""
    n, inf = len(X), float("inf")
    out = []
    for s in range(0, len(Q), 2500):
        q = Q[s:s + 2500].double()
        m = len(q)
        dist = torch.full((m, L), inf, dtype=torch.float64, device="cuda")
        ids = torch.full((m, L), n, dtype=torch.int64, device="cuda")
        done = torch.ones((m, L), dtype=torch.bool, device="cuda")
        dist[:, 0] = ((X[entry].double() - q) ** 2).sum(1)
        ids[:, 0], done[:, 0] = entry, False
        alive = torch.arange(m, device="cuda")
        while len(alive):
            first = (~done[alive]).to(torch.int8).argmax(1)
            best = dist[alive, first]
            go = (~done[alive, first]) & (best < dist[alive, L - 1])
            alive, first = alive[go], first[go]
            if not len(alive):
                break
            done[alive, first] = True
            nb = adj[ids[alive, first]]
            dd = ((X[nb.clamp(min=0)].double() - q[alive][:, None, :]) ** 2).sum(2)
            dd = torch.where(nb < 0, inf, dd)
            D = torch.cat([dist[alive], dd], 1)
            I = torch.cat([ids[alive], torch.where(nb < 0, n, nb)], 1)
            E = torch.cat([done[alive], nb < 0], 1)
            for by in "EID":  # in the end by distance, then row, an expanded entry before its repeat
                o = torch.argsort({"E": (~E).to(torch.int8), "I": I, "D": D}[by], dim=1, stable=True)
                D, I, E = D.gather(1, o), I.gather(1, o), E.gather(1, o)
            rep = torch.zeros_like(E)
            rep[:, 1:] = I[:, 1:] == I[:, :-1]
            D, I, E = torch.where(rep, inf, D), torch.where(rep, n, I), E | rep
            o = torch.argsort(D, dim=1, stable=True)[:, :L]
            dist[alive], ids[alive], done[alive] = D.gather(1, o), I.gather(1, o), E.gather(1, o)
        out.append(dist[:, :k])
    return torch.cat(out)


def exact(case, seed):
    """The results in 64 bits, laid out as `run` returns them.

    Searches over FP32 rows, and over BF16 rows of these integer data (which
    BF16 holds exactly), follow the graph search in 64 bits.  The other
    searches answer by what their approximate codes, filters or postings let
    through, and codebooks and graphs by seeded draws: these have no 64-bit
    value of their own, and row numbers, counts and codes are whole numbers.
    """
    kind = case["kind"]
    if kind == "knn":
        if case["metric"] == "cosine":
            X, Q = _embeddings(case["n"], case["nq"], case["d"], seed)
        else:
            X, _, Q = _mixture(case["n"], case["nq"], case["d"], case["centres"], seed)
        X, Q = X.double(), Q.double()
        out = []
        for s in range(0, len(Q), 500):
            q = Q[s:s + 500]
            if case["metric"] == "cosine":
                D = 1.0 - (q @ X.T) / (q.norm(dim=1)[:, None] * X.norm(dim=1)[None, :])
            else:
                D = (q * q).sum(1)[:, None] + (X * X).sum(1)[None, :] - 2.0 * (q @ X.T)
            out.append(torch.topk(D, case["k"], dim=1, largest=False, sorted=True).values)
        return None, torch.cat(out).cpu().numpy()
    plain = kind == "one" or (kind == "search" and case["metric"] == "l2" and not case["uneven"] and (
        case["trav"] == "f32" or (case["trav"] == "bf16" and case["rerank"] in (0, case["L"]))))
    if not plain:
        return None
    X, z, Q = _mixture(case["n"], case.get("nq", 1), case["d"], case["centres"], seed)
    adj, entry = _graph(X, z, case["centres"], case["R"], seed)
    k, L = case["k"], case["L"]
    D = _beam64(X, torch.from_numpy(adj.view(np.int32).astype(np.int64)).cuda(), entry, Q, min(k, L), L).cpu()
    if k > L:
        D = torch.cat([D, torch.full((len(D), k - L), float("inf"), dtype=torch.float64)], 1)
    if kind == "one":
        return [(None, v) for v in D[0].tolist() if v != float("inf")]
    return None, (D.numpy() if case["host"] else D.cuda()), None
