"""The joins a program has this library do, as measurable cases.

Every case goes through a public entry point: one join on device-resident
relations (join-project, ordered, COUNT, per-A-tile summaries), the
allocation-free call, the host-array call, a pass of many joins over resident
relations, and a batch of joins in one CUDA graph.  Relations are seeded
synthetic ones of the shapes that bench.py and the tests use, made on the GPU.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "joinproject-dim3_gb300"))
import dim3gpu  # noqa: E402


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a join inside an interactive query or a unit of a larger plan: a
        # thousand tuples, where launches and host round trips are the time
        dict(name="project_tiny", call="project", data="zipf", nR=1237, nS=911, dom_a=400, dom_c=300, dom_b=250, s=0.5),
        # the allocation-free call, near the middle of its limits
        dict(name="noalloc_150k", call="noalloc", data="zipf", nR=150001, nS=90007, dom_a=60000, dom_c=60000,
             dom_b=50000, s=0.3),
        # the reference's own default workload: 10M uniform tuples a side,
        # every row sparse
        dict(name="project_uniform_10m", call="project", data="zipf", nR=10000000, nS=10000000, dom_a=1000000,
             dom_c=1000000, dom_b=1000000, s=0.0),
        # skewed join values over small domains: nearly every pair exists
        # (the tensor-core product's case; the 1M-tuple Zipf workload, smaller)
        dict(name="project_zipf_400k", call="project", data="zipf", nR=400000, nS=400000, dom_a=50000, dom_c=50000,
             dom_b=20000, s=1.0),
        # distinct 2-hop neighbours of a 20M-edge power-law graph: an eighth
        # of the vertices' rows against the whole graph, as a program does
        # whose result does not fit in one buffer
        dict(name="two_hop_20m_part8", call="project", data="graph", vertices=1 << 21, samples=10000000, part=8),
        # the same question on a whole graph of a million edges
        dict(name="two_hop_1m", call="project", data="graph", vertices=1 << 17, samples=600011, part=1),
        # pairs grouped by their first value, for a consumer that walks rows
        dict(name="ordered_200k", call="ordered", data="zipf", nR=200003, nS=150001, dom_a=100000, dom_c=80000,
             dom_b=30000, s=0.8),
        # COUNT(*) GROUP BY (a, c), materialised
        dict(name="count_1m", call="count", data="zipf", nR=1000003, nS=800011, dom_a=300000, dom_c=200000,
             dom_b=100000, s=0.7),
        # COUNT of a result that cannot be materialised (16M tuples a side,
        # 1e12 groups): one of 16 slices of its summary
        dict(name="count_summary_16m", call="summary", data="zipf", nR=16000000, nS=16000000, dom_a=1000000,
             dom_c=1000000, dom_b=200000, s=1.2),
        # a request mix over relations that stay on the GPU
        dict(name="resident_16q", call="resident", relations=12, n_lo=500000, n_hi=4000000, queries=16, layout=3),
        # independent joins of uneven sizes, planned once, one graph launch
        dict(name="batch_48", call="batch", joins=48, n_lo=10000, n_hi=1000000, layout=4),
        # the drop-in call on host arrays, page-locked as a program does that
        # calls it often: copies in, join, result out
        dict(name="host_300k", call="host", data="zipf", nR=300007, nS=290011, dom_a=100000, dom_c=100000, dom_b=30000,
             s=0.0),
    ]


# most tuples a side, pairs out and candidates of a drawn join, by call
_MOST = {"project": (10 ** 7, 1.2e9, 3e9), "ordered": (2 * 10 ** 6, 3e8, 1e9), "count": (2 * 10 ** 6, 2e8, 6e8),
         "noalloc": (1 << 18, 8e5, 4e6), "host": (10 ** 6, 1.2e7, 1e8)}


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    call = rng.choice(["project", "project", "graph", "ordered", "count", "noalloc", "host", "summary", "resident",
                       "batch"])
    if call == "graph":
        v = 1 << rng.randint(12, 19)
        return dict(call="project", data="graph", vertices=v, samples=int(v * rng.uniform(2.0, 5.0)),
                    part=rng.choice([1, 1, 3, 8]))
    if call == "summary":
        while True:
            c = dict(call="summary", data="zipf", nR=_log(rng, 3 * 10 ** 5, 4 * 10 ** 6),
                     nS=_log(rng, 3 * 10 ** 5, 4 * 10 ** 6), dom_a=_log(rng, 3 * 10 ** 5, 10 ** 6),
                     dom_c=_log(rng, 3 * 10 ** 5, 10 ** 6), dom_b=_log(rng, 5 * 10 ** 4, 2 * 10 ** 5),
                     s=round(rng.uniform(0.9, 1.1), 3))
            if _expected(c)[0] <= 1e11:
                return c
    if call == "resident":
        return dict(call="resident", relations=rng.randint(4, 12), n_lo=100000, n_hi=_log(rng, 300000, 4000000),
                    queries=rng.randint(2, 16), layout=rng.randint(100, 10 ** 6))
    if call == "batch":
        return dict(call="batch", joins=rng.randint(8, 48), n_lo=10000, n_hi=_log(rng, 100000, 1000000),
                    layout=rng.randint(100, 10 ** 6))
    n_hi, out_hi, cand_hi = _MOST[call]
    while True:
        c = dict(call=call, data="zipf", nR=_log(rng, 1000, n_hi), nS=_log(rng, 1000, n_hi),
                 dom_a=_log(rng, 300, 10 ** 6), dom_c=_log(rng, 300, 10 ** 6), dom_b=_log(rng, 200, 10 ** 6),
                 s=round(rng.uniform(0.0, 1.2), 3))
        cand, out = _expected(c)
        if cand <= cand_hi and out <= out_hi and out >= 100:
            return c


# ------------------------------------------------------------ expectations
def _zipf_weights(dom, s):
    w = np.arange(1, dom + 1, dtype=np.float64) ** -s
    return w / w.sum()


def _vertex_weights(c):
    """Expected degrees of the Chung-Lu graph (exponent 2.1, weights capped
    at the square root of their sum), over the sum."""
    n = c["vertices"]
    w = np.arange(1, n + 1, dtype=np.float64) ** (-1.0 / 1.1)
    w *= 2.0 * c["samples"] / w.sum()
    w = np.minimum(w, math.sqrt(w.sum()))
    return w / w.sum()


def _expected(c):
    """(candidates, distinct pairs) a join is expected to have."""
    if c["data"] == "graph":
        deg = _vertex_weights(c) * 2.0 * c["samples"]
        cand = float((deg * deg).sum())
        # vertices in classes of nearly equal degree; P(no 2-path) per pair
        at = np.unique(np.geomspace(1, c["vertices"] + 1, 400).astype(np.int64))
        size = np.diff(at).astype(np.float64)
        d = np.add.reduceat(deg, at[:-1] - 1) / size
        paths = np.outer(d, d) * cand / (2.0 * c["samples"]) ** 2
        return cand / c["part"], float((np.outer(size, size) * -np.expm1(-paths)).sum()) / c["part"]
    p = _zipf_weights(c["dom_b"], c["s"])
    cand = float(c["nR"]) * c["nS"] * float((p * p).sum())
    cells = float(c["dom_a"]) * c["dom_c"]
    return cand, cells * -math.expm1(-cand / cells)


def _batch_joins(c):
    """Sizes of a batch's joins: tuples log-uniform, Zipf exponent uniform,
    one domain for all three columns log-uniform; a draw with too large an
    expected result is drawn again."""
    rng, got = random.Random(c["layout"]), []
    while len(got) < c["joins"]:
        dom = _log(rng, 1000, 10 ** 6)
        j = dict(data="zipf", nR=_log(rng, c["n_lo"], c["n_hi"]), nS=_log(rng, c["n_lo"], c["n_hi"]), dom_a=dom,
                 dom_c=dom, dom_b=dom, s=rng.uniform(0.5, 1.5))
        cand, out = _expected(j)
        if cand <= 2 ** 26 and out <= 2 ** 24:
            got.append(j)
    return got


_DOM_B = 1 << 18  # join values that resident relations share


def _resident_plan(c):
    """The resident relations and the pass's (r, s, op, expected rows)
    queries: a relation's join values follow a power law of its own over an
    order of the values of its own, and a quarter of the queries count."""
    rng = random.Random(c["layout"])
    rels = [dict(n=_log(rng, c["n_lo"], c["n_hi"]), s=1.0 / (rng.uniform(1.8, 2.5) - 1.0),
                 mul=rng.randrange(1 << 20) * 2 + 1, add=rng.randrange(1 << 20)) for _ in range(c["relations"])]
    share = []
    for p in rels:
        share.append(np.zeros(_DOM_B))
        share[-1][(np.arange(_DOM_B) * p["mul"] + p["add"]) & (_DOM_B - 1)] = _zipf_weights(_DOM_B, p["s"])
    queries = []
    for k in range(c["queries"]):
        r, s = rng.sample(range(c["relations"]), 2)
        n, m = rels[r]["n"], rels[s]["n"]
        cand, cells = float(n) * m * float(share[r] @ share[s]), float(n // 4) * (m // 4)
        queries.append((r, s, dim3gpu.OP_COUNT if k % 4 == 3 else dim3gpu.OP_PROJECT,
                        cells * -math.expm1(-cand / cells)))
    return rels, queries


def work(case):
    c = case
    if c["call"] == "batch":
        js = _batch_joins(c)
        return {"bytes": sum(8.0 * (j["nR"] + j["nS"]) + 8.0 * _expected(j)[1] for j in js), "flops": 0}
    if c["call"] == "resident":
        # each query reads its two relations and writes its result
        rels, queries = _resident_plan(c)
        return {"bytes": sum(8.0 * (rels[r]["n"] + rels[s]["n"]) + (16.0 if op else 8.0) * rows
                             for r, s, op, rows in queries), "flops": 0}
    cand, out = _expected(c)
    if c["data"] == "graph":
        inputs = 16.0 * c["samples"] * (1.0 + 1.0 / c["part"])
    else:
        inputs = 8.0 * (c["nR"] + c["nS"])
    if c["call"] == "summary":
        return {"bytes": inputs, "flops": 2.0 * cand / 16}
    if c["call"] == "count":
        return {"bytes": inputs + 16.0 * out, "flops": 2.0 * cand}
    return {"bytes": inputs + 8.0 * out, "flops": 0}


# ------------------------------------------------------------------ inputs
def _ranks(weights, n, gen):
    cdf = torch.from_numpy(np.cumsum(weights)).cuda()
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    return torch.searchsorted(cdf, u, right=True).clamp_(max=weights.shape[0] - 1)


def _values(ranks):
    """Ranks scattered over the 32-bit keys (an odd multiplier)."""
    return ((ranks * 2654435761 + 0x3C6EF372) & 0xFFFFFFFF) - (1 << 31)


def _pairs(first, y):
    return torch.stack([first.to(torch.int32), y.to(torch.int32)], 1).contiguous()


def _capacity(expected, cells):
    """Rows of an output buffer: the expected result and room to spare."""
    return int(min(1.3 * expected + 65536, cells))


def _relations(c, gen):
    """(R, S, output capacity) of one join."""
    cells = c["vertices"] ** 2 if c["data"] == "graph" else c["dom_a"] * c["dom_c"]
    cap = _capacity(_expected(c)[1], cells)
    if c["data"] == "graph":
        w = _vertex_weights(c)
        u, v = _ranks(w, c["samples"], gen), _ranks(w, c["samples"], gen)
        keep = u != v
        u, v = u[keep], v[keep]
        first, y = torch.stack([u, v], 1).reshape(-1), torch.stack([v, u], 1).reshape(-1)
        S = _pairs(_values(first), _values(y))
        if c["part"] > 1:
            mine = ((first * 2654435761 & 0xFFFFFFFF) >> 13) % c["part"] == 0
            first, y = first[mine], y[mine]
        R = _pairs(_values(first), _values(y))
        return R, S, cap
    w = _zipf_weights(c["dom_b"], c["s"])
    side = []
    for n, dom in ((c["nR"], c["dom_a"]), (c["nS"], c["dom_c"])):
        first = torch.randint(0, dom, (n,), generator=gen, device="cuda")
        side.append((first, _ranks(w, n, gen)))
    (a, yr), (z, ys) = side
    return _pairs(a, _values(yr)), _pairs(z, _values(ys)), cap


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


_contexts = {}


def _context(**knobs):
    """A program keeps one context for all its joins of a kind."""
    key = tuple(sorted(knobs.items()))
    if key not in _contexts:
        ctx = dim3gpu.Context(0)
        for name, value in key:
            ctx.set_param(name, value)
        _contexts[key] = ctx
    return _contexts[key]


def _noalloc_entry():
    fn, vp, u64 = dim3gpu.load().dim3g_join_project_noalloc, ctypes.c_void_p, ctypes.c_uint64
    fn.argtypes = [vp, u64, vp, u64, vp, u64, ctypes.POINTER(u64), vp]
    return fn


def prepare(case, seed):
    c, gen = case, _generator(seed)
    st = dict(call=c["call"])
    if c["call"] == "batch":
        rels = [_relations(j, gen) for j in _batch_joins(c)]
        st["out"] = [torch.empty((cap, 2), dtype=torch.int32, device="cuda") for _, _, cap in rels]
        specs = [dict(op=dim3gpu.OP_PROJECT, out=o, capacity=o.shape[0]) for o in st["out"]]
        torch.cuda.synchronize()
        st["batch"] = dim3gpu.Batch(_context(), [((R, R.shape[0]), (S, S.shape[0])) for R, S, _ in rels], specs)
        return st
    if c["call"] == "resident":
        plan, queries = _resident_plan(c)
        rels = []
        for p in plan:
            first = torch.randint(0, p["n"] // 4, (p["n"],), generator=gen, device="cuda")
            y = (_ranks(_zipf_weights(_DOM_B, p["s"]), p["n"], gen) * p["mul"] + p["add"]) & (_DOM_B - 1)
            rels.append(_pairs(first, _values(y)))
        st["specs"] = []
        for r, s, op, rows in queries:
            cap = _capacity(rows, (plan[r]["n"] // 4) * (plan[s]["n"] // 4))
            spec = dict(r=r, s=s, op=op, capacity=cap, out=torch.empty((cap, 2), dtype=torch.int32, device="cuda"))
            if op == dim3gpu.OP_COUNT:
                spec["cnt"] = torch.empty(cap, dtype=torch.int64, device="cuda")
            st["specs"].append(spec)
        torch.cuda.synchronize()
        st["set"] = dim3gpu.RelSet(_context(), [(t, t.shape[0]) for t in rels])
        return st
    R, S, cap = _relations(c, gen)
    st.update(R=R, S=S, cap=cap)
    if c["call"] == "host":
        st["ctx"] = _context()
        st["R"], st["S"] = (t.cpu().pin_memory().numpy().view(np.uint32) for t in (R, S))
        st["out"] = torch.empty((cap, 2), dtype=torch.int32, pin_memory=True)
        st["into"] = st["out"].numpy().view(np.uint32)
        return st
    if c["call"] == "noalloc":
        st["join"] = _noalloc_entry()
    else:
        st["ctx"] = _context(ordered_output=1) if c["call"] == "ordered" else \
            _context(keep_roles=1) if c.get("part", 1) > 1 else _context()
    if c["call"] != "summary":
        st["out"] = torch.empty((cap, 2), dtype=torch.int32, device="cuda")
    if c["call"] == "count":
        st["cnt"] = torch.empty(cap, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    return st


# -------------------------------------------------------------------- run
class Rows(dict):
    """The rows of one or several results, as the call left them.

    A result is a set: the library writes its rows in an order that differs
    from call to call.  An entry is put in order when it is read, so that
    equal results compare equal: `rows` holds each result's pairs, packed
    into 64 bits and sorted, `counts` the groups' counts in the same order,
    both -1 past a result's end; `sizes` is the number of rows of each."""

    def __init__(self, parts):
        super().__init__(rows=None, sizes=None)
        self.parts = parts
        if any(cnt is not None for _, cnt, _, _ in parts):
            self["counts"] = None

    def __getitem__(self, key):
        if key == "sizes":
            return torch.tensor([n for _, _, n, _ in self.parts])
        parts = [p for p in self.parts if key == "rows" or p[1] is not None]
        got = torch.full((sum(cap for _, _, _, cap in parts),), -1, dtype=torch.int64, device="cuda")
        at = 0
        for out, cnt, n, cap in parts:
            packed = out[:n].view(torch.int64).reshape(-1)
            got[at:at + n] = torch.sort(packed).values if key == "rows" else cnt[:n][torch.argsort(packed)]
            at += cap
        return got


def run(state):
    st = state
    if st["call"] == "batch":
        return Rows([(o, None, r["n_out"], o.shape[0]) for o, r in zip(st["out"], st["batch"].run())])
    if st["call"] == "resident":
        got = st["set"].join(st["specs"])
        return Rows([(q["out"], q.get("cnt"), r["n_out"], q["capacity"]) for q, r in zip(st["specs"], got)])
    R, S = st["R"], st["S"]
    nR, nS = R.shape[0], S.shape[0]
    if st["call"] == "host":
        return Rows([(st["out"], None, st["ctx"].join_project_into(R, S, st["into"]), st["cap"])])
    if st["call"] == "summary":
        return st["ctx"].join_count_summary(R, nR, S, nS, 16, 0, 1).view(np.int64)
    out = st["out"]
    if st["call"] == "noalloc":
        n = ctypes.c_uint64()
        rc = st["join"](R.data_ptr(), nR, S.data_ptr(), nS, out.data_ptr(), out.shape[0], ctypes.byref(n), None)
        if rc:
            raise dim3gpu.Dim3GError(rc, "dim3g_join_project_noalloc")
        return Rows([(out, None, n.value, st["cap"])])
    if st["call"] == "count":
        n = st["ctx"].join_count_device(R, nR, S, nS, out, st["cnt"], out.shape[0])
        return Rows([(out, st["cnt"], n, st["cap"])])
    n = st["ctx"].join_project_device(R, nR, S, nS, out, out.shape[0])
    return Rows([(out, None, n, st["cap"])])


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """The result's rows from a plain sort-merge expansion.  None where that
    takes too long, and for a summary's hashes."""
    c = case
    if c["call"] in ("batch", "resident", "summary") or _expected(c)[0] > 3e8:
        return None
    R, S, cap = _relations(c, _generator(seed))
    if R.shape[0] < S.shape[0] and c.get("part", 1) == 1:  # the larger relation's values come first
        R, S = S, R
    y, order = torch.sort(S[:, 1])
    z = S[:, 0][order].to(torch.int64)
    lo = torch.searchsorted(y, R[:, 1].contiguous())
    n = torch.searchsorted(y, R[:, 1].contiguous(), right=True) - lo
    at = torch.arange(int(n.sum()), device="cuda") + torch.repeat_interleave(lo - (torch.cumsum(n, 0) - n), n)
    packed = (z[at] << 32) | (torch.repeat_interleave(R[:, 0].to(torch.int64), n) & 0xFFFFFFFF)
    rows, counts = torch.unique(packed, return_counts=True)
    got = dict(rows=torch.full((cap,), -1, dtype=torch.int64, device="cuda"), sizes=torch.tensor([rows.shape[0]]))
    got["rows"][:rows.shape[0]] = rows
    if c["call"] == "count":
        got["counts"] = torch.full_like(got["rows"], -1)
        got["counts"][:rows.shape[0]] = counts
    return got
