"""Performance cases of the exact k-NN library.

Each case is one call a program makes of the public entry points -- exact
search query by query (`knn`, `knn_device`), the scan of every row (`pscan`,
`pscan_noalloc`), batched search (`knn_batch`, `knn_batch_device`) and index
construction (`HerculesIndex.build_device`) -- at sizes from an interactive
query of a small index to the 25M x 256 batch of bench.py.

Collections are z-normalised random walks or L2-normalised Gaussian vectors
(the two kinds bench.py uses), made with torch on the GPU from the seed.
Queries are rows of the collection plus N(0, sigma2) noise, normalised again,
with sigma2 cycling over the case's levels; where `fresh` is set every tenth
query is a fresh walk instead.

Keys of a case:
  kind    plain | pscan | noalloc | batch | build
  n, L    rows and series length;  leaf: leaf size of the index
  data    walk | unit;  sigma2: noise levels, comma separated
  nq, k   queries of the call and answers per query; k = 0: k cycles over
          1, 10, 100 within the call (batch only)
  lb_sax  plain: per-row LB_SAX filter on
  host    queries and answers in host memory (numpy) instead of on the GPU
"""
import math

import numpy as np
import torch

import hercules_b200 as H

MIXED = (1, 10, 100)
# share of the (query, leaf) pairs that LB_EAPCA keeps for noisy queries of
# random walks (0.36 .. 0.57 at the sizes of bench.py's configurations)
KEPT = 0.38


def _case(name, kind, n, L, **kw):
    c = {"name": name, "kind": kind, "n": n, "L": L, "leaf": 0, "data": "walk", "sigma2": "0.01,0.1,1.0",
         "fresh": False, "nq": 1, "k": 1, "lb_sax": False, "host": False}
    c.update(kw)
    return c


def listed():
    return [
        # one interactive 1-NN query of a small index, host in, host out
        _case("plain 100k x 256 / 1 query", "plain", 100000, 256, leaf=2000, sigma2="0.1", nq=1, k=1, lb_sax=True,
              host=True),
        # a workload file of 100 queries over the 1M x 256 index (leaf
        # 100,000) of the reference's own configuration, with LB_SAX
        _case("plain 1M x 256 / 100 queries", "plain", 1000000, 256, leaf=100000, fresh=True, nq=100, k=10,
              lb_sax=True),
        # a few 100-NN queries of a larger index with the default options
        # (no LB_SAX), through the host entry point
        _case("plain 8M x 256 / 16 queries / k 100", "plain", 8000000, 256, leaf=100000, fresh=True, nq=16, k=100,
              host=True),
        # long series: 64 KB rows, small leaves
        _case("plain 100k x 16384 / 12 queries", "plain", 100000, 16384, leaf=1562, sigma2="0.1", nq=12, k=10,
              lb_sax=True),
        # the index-free scan of every row, a handful of queries
        _case("pscan 2M x 256 / 4 queries", "pscan", 2000000, 256, leaf=100000, nq=4, k=10, host=True),
        # one query over a caller-owned matrix, nothing allocated
        _case("noalloc 1M x 256 / 1 query", "noalloc", 999983, 256, sigma2="0.1", nq=1, k=10),
        # a small service batch over a small index, host in, host out
        _case("batch 100k x 256 / 64 queries", "batch", 100000, 256, leaf=2000, sigma2="0.1", nq=64, k=1, host=True),
        # short embedding-like vectors: nothing prunes, odd counts
        _case("batch 3M x 96 unit / 333 queries", "batch", 3000017, 96, leaf=8000, data="unit", sigma2="0.1", nq=333,
              k=10),
        # series of 1,024 points at bench.py's noise levels
        _case("batch 1M x 1024 / 512 queries", "batch", 1000000, 1024, leaf=25000, sigma2="0.1,1.0", nq=512, k=10),
        # the longest series, batched
        _case("batch 200k x 16384 / 128 queries", "batch", 200000, 16384, leaf=1562, sigma2="0.1", nq=128, k=10),
        # bench.py's headline batch: 4,096 queries of mixed noise and k
        _case("batch 25M x 256 / 4096 queries", "batch", 25000000, 256, leaf=100000, fresh=True, nq=4096, k=0),
        # building an index from rows on the GPU
        _case("build 1M x 256", "build", 1000000, 256, leaf=10000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("plain", "plain", "plain", "pscan", "noalloc", "batch", "batch", "batch", "build"))
    L = rng.choice((64, 96, 128, 256, 256, 256, 16 * rng.randint(2, 64), 1024, 4096, 16384))
    n = _log_uniform(rng, 20000, 4000000)
    n = max(2000, min(n, 1500000000 // L))
    c = _case("", kind, n, L)
    del c["name"]
    if kind != "noalloc":
        c["leaf"] = max(200, min(100000, n // _log_uniform(rng, 6, 200)))
    if kind in ("plain", "pscan", "noalloc", "batch"):
        c["data"] = "unit" if L <= 128 and rng.random() < 0.3 else "walk"
        c["sigma2"] = rng.choice(("0.01", "0.1", "0.01,0.1,1.0", "0.1,1.0"))
    c["fresh"] = c["data"] == "walk" and rng.random() < 0.3
    c["k"] = rng.choice((1, 3, 10, 10, 50, 100, 224))
    c["host"] = kind in ("plain", "pscan", "batch") and rng.random() < 0.5
    if kind == "plain":
        c["nq"] = _log_uniform(rng, 1, 64)
        c["lb_sax"] = rng.random() < 0.6
        if c["data"] == "unit":
            c["nq"] = min(c["nq"], 8)
    elif kind == "pscan":
        c["nq"] = _log_uniform(rng, 1, 8)
    elif kind == "batch":
        c["nq"] = _log_uniform(rng, 8, 2048)
        if rng.random() < 0.3:
            c["k"] = 0
    elif kind == "build":
        c.update(nq=1, k=1, fresh=False)
    return c


# -- inputs -------------------------------------------------------------------

_CHUNK = 1 << 28  # values normalised at a time


def _normalise(x, unit):
    if unit:
        x.div_(x.norm(dim=1, keepdim=True))
    else:
        x.sub_(x.mean(dim=1, keepdim=True))
        x.div_(x.std(dim=1, keepdim=True, unbiased=False))


def _rows(n, L, unit, gen):
    x = torch.empty((n, L), dtype=torch.float32, device="cuda")
    for part in x.split(max(1, _CHUNK // L)):
        part.normal_(generator=gen)
        if not unit:
            part.cumsum_(1)
        _normalise(part, unit)
    return x


def _inputs(case, seed):
    """The collection and the queries of a case (float32, on the GPU)."""
    unit = case["data"] == "unit"
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2 * seed + 1)
    X = _rows(case["n"], case["L"], unit, gen)
    nq = case["nq"]
    gen.manual_seed(2 * seed + 2)
    s2 = [float(v) for v in case["sigma2"].split(",")]
    sd = torch.tensor([math.sqrt(s2[j % len(s2)]) for j in range(nq)], dtype=torch.float32, device="cuda")
    base = torch.randint(case["n"], (nq,), generator=gen, device="cuda")
    Q = X[base] + sd[:, None] * torch.randn((nq, case["L"]), generator=gen, device="cuda")
    if case["fresh"] and nq >= 10:
        at = torch.arange(9, nq, 10, device="cuda")
        Q[at] = torch.randn((len(at), case["L"]), generator=gen, device="cuda").cumsum(1)
    _normalise(Q, unit)
    return X, Q


def _ks(case):
    """k of every query."""
    if case["k"]:
        return np.full(case["nq"], case["k"], dtype=np.uint32)
    levels = len(case["sigma2"].split(","))  # every (noise, k) pair in equal shares
    return np.array([MIXED[(j // levels) % 3] for j in range(case["nq"])], dtype=np.uint32)


def prepare(case, seed):
    X, Q = _inputs(case, seed)
    torch.cuda.synchronize()
    s = {"case": case}
    nq, ks = case["nq"], _ks(case)
    if case["kind"] in ("noalloc", "build"):
        s["X"] = X
    else:
        s["ix"] = H.HerculesIndex.build_device(X.data_ptr(), case["n"], case["L"], case["leaf"])
        del X
    torch.cuda.empty_cache()  # the index allocates outside torch's pool
    s["ks"] = ks
    s["kmax"] = kmax = int(ks.max())
    if case["host"]:
        s["Q"] = Q.cpu().numpy()
    else:
        s["Q"] = Q
        s["dist"] = torch.empty((nq, kmax), dtype=torch.float32, device="cuda")
        s["ids"] = torch.empty((nq, kmax), dtype=torch.int64, device="cuda")
    return s


# -- one pass -----------------------------------------------------------------

def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "build":
        ix = H.HerculesIndex.build_device(s["X"].data_ptr(), c["n"], c["L"], c["leaf"])
        leaves = ix.leaves()
        # row -> dataset id, row -> leaf, and every leaf's envelope; the number
        # of segments depends on the data, so the last comes in a fixed buffer
        env = np.zeros((64 * (c["n"] // c["leaf"] + 16), 4), dtype=np.float32)
        at = 0
        for i in range(len(leaves)):
            _, e = ix.leaf_envelope(i)
            e = e[:len(env) - at]
            env[at:at + len(e)] = e
            at += len(e)
        out = {"ids": ix.row_ids(), "leaf": np.repeat(np.arange(len(leaves)), [size for _, size, _ in leaves]),
               "envelopes": env}
        ix.close()
        return out
    if c["host"]:
        if kind == "plain":
            return s["ix"].knn(s["Q"], c["k"], use_lb_sax=c["lb_sax"])
        if kind == "pscan":
            return s["ix"].pscan(s["Q"], c["k"])
        return s["ix"].knn_batch(s["Q"], s["ks"])
    q, d, i = s["Q"].data_ptr(), s["dist"].data_ptr(), s["ids"].data_ptr()
    if kind == "noalloc":
        H.pscan_noalloc(s["X"].data_ptr(), c["n"], c["L"], q, c["k"], d, i)
    elif kind == "plain":
        s["ix"].knn_device(q, c["nq"], c["k"], d, i, use_lb_sax=c["lb_sax"])
    elif kind == "pscan":
        s["ix"].knn_device(q, c["nq"], c["k"], d, i, mode=H.MODE_PSCAN)
    else:
        s["ix"].knn_batch_device(q, c["nq"], s["ks"], s["kmax"], d, i)
    return s["dist"], s["ids"]


def work(case):
    """What a pass cannot do without.  scan: every row once; plain: the rows
    of each query's approximate leaf (a leaf is about 0.6 full) and, with
    LB_SAX, the iSAX words of the kept leaves; batch: the products of the
    kept (query, row) pairs and the BF16 rows once; build: the rows once in,
    once out, with their ids and iSAX words."""
    n, L, nq = case["n"], case["L"], case["nq"]
    kept = KEPT if case["data"] == "walk" else 1.0
    io = 4 * nq * L + 12 * int(_ks(case).sum())
    if case["kind"] in ("pscan", "noalloc"):
        return {"bytes": 4 * n * L + io, "flops": 3 * n * L}
    if case["kind"] == "build":
        return {"bytes": 8 * n * L + 24 * n, "flops": 2 * n * L}
    if case["kind"] == "plain":
        rows = min(n, 0.6 * case["leaf"] * nq)
        return {"bytes": 4 * rows * L + (16 * kept * n * nq if case["lb_sax"] else 0) + io,
                "flops": 3 * 0.6 * case["leaf"] * L * nq}
    return {"bytes": 2 * n * L + io, "flops": 2 * kept * n * L * nq}


# -- the same in 64 bits -------------------------------------------------------

def exact(case, seed):
    """The k smallest squared distances in 64 bits: candidates by their
    32-bit products (2 k + 32 of them), distances of the candidates from the
    64-bit differences."""
    if case["kind"] == "build":
        return None
    X, Q = _inputs(case, seed)
    ks = _ks(case)
    kmax = int(ks.max())
    m = min(case["n"], 2 * kmax + 32)
    nq, L = Q.shape
    tf32, torch.backends.cuda.matmul.allow_tf32 = torch.backends.cuda.matmul.allow_tf32, False
    best = torch.empty((nq, 0), device="cuda")
    rows = torch.empty((nq, 0), dtype=torch.int64, device="cuda")
    step = max(4 * m, min((1 << 30) // nq, (1 << 31) // L))
    for lo in range(0, case["n"], step):
        part = X[lo:lo + step]
        s = torch.addmm(part.square().sum(1)[None, :], Q, part.T, alpha=-2.0)
        v, i = s.topk(min(m, part.shape[0]), dim=1, largest=False)
        best, rows = torch.cat((best, v), 1), torch.cat((rows, i + lo), 1)
        best, j = best.topk(min(m, best.shape[1]), dim=1, largest=False)
        rows = rows.gather(1, j)
    torch.backends.cuda.matmul.allow_tf32 = tf32
    dist = torch.full((nq, kmax), math.inf, dtype=torch.float64, device="cuda")
    for j in range(nq):
        d = (X[rows[j]].double() - Q[j].double()).square().sum(1).sort().values
        k = min(int(ks[j]), d.shape[0])
        dist[j, :k] = d[:k]
    return dist, None
