"""The engine's work as a user's program has it done, one case per way of use.

Every case goes through the public entry points of pico_gb300 (the Python
classes or the C ABI that they bind) on graphs that this file makes with torch
from the seed alone, so that exact() can restate each result without the
engine.  Graph families and sizes are those of the engine's own configurations
and tests: Erdos-Renyi 65,536 / 1,048,576, R-MAT scales 17 to 25 with edge factor
16, a planted 4,000-vertex dense subgraph at p = 0.6, the batch mix
(n = 10^U(2,5), average degree U(4,64), Erdos-Renyi / R-MAT /
Barabasi-Albert), update batches of 10^3 to 10^6 edges half insertions and half
deletions, and graphs at the limits of the allocation-free entry point.
"""
import ctypes

import numpy as np
import torch

import pico_gb300 as pg

RMAT_A, RMAT_B, RMAT_C = 0.57, 0.19, 0.19
DEV = "cuda"


# ---------------------------------------------------------------- cases ----
def listed():
    return [
        # one small graph per call with the result and the statistics back on
        # the host: launches and latency are all there is
        {"name": "er16_peel_host", "op": "peel", "method": "peelone_dyn", "host": True,
         "family": "er", "n": 65536, "m": 1048576},
        # a mid-size power-law graph, the usual single-graph decomposition;
        # the result stays on the device
        {"name": "rmat22_peel", "op": "peel", "method": "peelone", "host": False,
         "family": "rmat", "scale": 22, "m": 16 << 22},
        # the largest single graph: 33.5 M vertices, 1.06 B entries, a deep core
        {"name": "rmat25_planted_peel", "op": "peel", "method": "peelone_dyn", "host": False,
         "family": "planted", "scale": 25, "m": 16 << 25, "k": 4000, "p": 0.6},
        # the h-index drivers (HistoCore / CntCore / NbrCore) on the power-law graph
        {"name": "rmat22_hindex", "op": "peel", "method": "HistoCore", "host": False,
         "family": "rmat", "scale": 22, "m": 16 << 22},
        # many uneven graphs in one launch, the batched configuration
        {"name": "batch_mix4096", "op": "batch", "graphs": 4096, "log_lo": 2.0, "log_hi": 5.0, "deg_hi": 64.0},
        # a launch's worth of small graphs (a request queue's typical contents)
        {"name": "batch_small256", "op": "batch", "graphs": 256, "log_lo": 2.0, "log_hi": 3.5, "deg_hi": 32.0},
        # the allocation-free call of a framework that owns the device memory
        {"name": "noalloc_rmat", "op": "noalloc", "family": "rmat_n", "n": 20011, "m": 320000},
        # edge list on the device to a sorted, de-duplicated CSR
        {"name": "build_dedup_rmat22", "op": "build", "order": "dedup", "family": "rmat", "scale": 22, "m": 16 << 22},
        # the loader's order-keeping build (rows in edge-list order, parallel edges kept)
        {"name": "build_order_rmat18", "op": "build", "order": "keep", "family": "rmat", "scale": 18, "m": 16 << 18},
        # a resident graph under a mixed edge batch and its undoing
        {"name": "update_mixed_1e4", "op": "update", "kind": "mixed", "scale": 22, "ef": 16, "batch": 10000},
        # deletions only (maintained from the old cores), then their undoing
        {"name": "update_delete_1e3", "op": "update", "kind": "delete", "scale": 20, "ef": 16, "batch": 1000},
        # requests of fresh graphs and an update pair, submitted together to the server
        {"name": "serve_mix32", "op": "serve", "graphs": 32, "log_lo": 2.0, "log_hi": 5.0, "deg_hi": 64.0,
         "batch": 1000},
    ]


def draw(rng):
    def logint(lo, hi):
        return max(2, int(round(lo * (hi / lo) ** rng.random())))

    op = rng.choice(["peel", "peel", "hindex", "batch", "noalloc", "build", "update", "serve"])
    if op in ("peel", "hindex"):
        method = rng.choice(["peelone", "peelone_dyn", "gppeel"]) if op == "peel" else rng.choice(["HistoCore", "NbrCore"])
        host = rng.random() < 0.5
        fam = rng.choice(["er", "rmat_n", "planted"])
        if fam == "er":
            n = logint(1000, 4000000)
            return {"op": "peel", "method": method, "host": host, "family": "er", "n": n, "m": int(n * rng.uniform(2, 24))}
        if fam == "rmat_n":
            n = logint(1000, 6000000)
            return {"op": "peel", "method": method, "host": host, "family": "rmat_n", "n": n,
                    "m": int(n * rng.uniform(4, 20))}
        s = rng.randint(16, 22)
        return {"op": "peel", "method": method, "host": host, "family": "planted", "scale": s, "m": 16 << s,
                "k": logint(200, 3000), "p": rng.uniform(0.3, 0.7)}
    if op == "batch":
        lo = rng.uniform(2.0, 3.0)
        return {"op": "batch", "graphs": logint(16, 2048), "log_lo": lo, "log_hi": lo + rng.uniform(0.5, 5.0 - lo),
                "deg_hi": rng.uniform(8.0, 64.0)}
    if op == "noalloc":
        n = logint(100, 50000)
        return {"op": "noalloc", "family": rng.choice(["er", "rmat_n"]), "n": n,
                "m": min(int(n * rng.uniform(2, 40)), 2000000)}
    if op == "build":
        n = logint(3000, 6000000)
        return {"op": "build", "order": rng.choice(["dedup", "keep", "sort"]), "family": rng.choice(["er", "rmat_n"]),
                "n": n, "m": int(n * rng.uniform(3, 16))}
    if op == "update":
        return {"op": "update", "kind": rng.choice(["mixed", "delete"]), "scale": rng.randint(17, 22), "ef": 16,
                "batch": logint(1000, 300000)}
    lo = rng.uniform(2.0, 3.0)
    return {"op": "serve", "graphs": rng.randint(4, 48), "log_lo": lo, "log_hi": lo + rng.uniform(0.5, 2.0),
            "deg_hi": rng.uniform(8.0, 64.0), "batch": logint(200, 5000)}


# ------------------------------------------------------ graphs from torch ----
def _rand(count, gen):
    return torch.rand(count, generator=gen, device=DEV)


def _rmat_edges(bits, m, gen):
    """m draws of R-MAT over 2^bits ids (bits: a number, or one per edge)."""
    src = torch.empty(m, dtype=torch.int32, device=DEV)
    dst = torch.empty(m, dtype=torch.int32, device=DEV)
    step = 1 << 26
    for i in range(0, m, step):
        c = min(step, m - i)
        b = bits if isinstance(bits, int) else bits[i:i + c]
        s = torch.zeros(c, dtype=torch.int32, device=DEV)
        d = torch.zeros(c, dtype=torch.int32, device=DEV)
        for level in range(b if isinstance(b, int) else int(b.max())):
            r = _rand(c, gen)
            sb = (r >= RMAT_A + RMAT_B).int()
            db = (((r >= RMAT_A) & (r < RMAT_A + RMAT_B)) | (r >= RMAT_A + RMAT_B + RMAT_C)).int()
            if isinstance(b, int):
                s, d = 2 * s + sb, 2 * d + db
            else:
                on = level < b
                s, d = torch.where(on, 2 * s + sb, s), torch.where(on, 2 * d + db, d)
        src[i:i + c] = s
        dst[i:i + c] = d
    return src, dst


def _reject(s, d, n):
    """Draws outside [0, n) become the self-loop (0, 0), which no graph keeps."""
    out = (s >= n) | (d >= n)
    return s.masked_fill(out, 0), d.masked_fill(out, 0)


def _mix_params(case):
    """(n, family, edges, ends per new vertex) of each graph of a batch mix:
    the sizes are the case's own, the edges come from the seed."""
    rng = np.random.default_rng([case["graphs"], int(1e6 * case["log_hi"]), 17])
    G = case["graphs"]
    n = np.floor(10.0 ** rng.uniform(case["log_lo"], case["log_hi"], G)).astype(np.int64)
    kind = rng.integers(0, 3, G)
    d = rng.uniform(4.0, case["deg_hi"], G)
    mba = rng.integers(1, max(2, int(case["deg_hi"] / 2) + 1), G)
    m = np.where(kind == 2, n * mba, np.round(n * d / 2.0).astype(np.int64))
    return n, kind, m, mba


def _mix_edges(case, seed):
    """The mix packed into one id space: (src, dst, vbase), 0 Erdos-Renyi, 1
    R-MAT, 2 Barabasi-Albert (each edge's end copied from a uniformly drawn
    place of the earlier edges' ends)."""
    n, kind, m, mba = _mix_params(case)
    vbase = np.zeros(n.size + 1, dtype=np.int64)
    np.cumsum(n, out=vbase[1:])
    gen = torch.Generator(DEV).manual_seed(int(seed))
    parts = []
    for k in range(3):
        which = np.nonzero(kind == k)[0]
        if not which.size:
            continue
        reps = torch.from_numpy(m[which]).to(DEV)
        total = int(m[which].sum())

        def per_edge(a, dtype=torch.int32):
            return torch.repeat_interleave(torch.from_numpy(a[which]).to(DEV, dtype), reps, output_size=total)

        ne, off = per_edge(n), per_edge(vbase[:-1])
        if k == 0:
            s = (_rand(total, gen).double() * ne).int().clamp_(max=ne - 1)
            d = (_rand(total, gen).double() * ne).int().clamp_(max=ne - 1)
        elif k == 1:
            bits = np.ceil(np.log2(np.maximum(n, 2))).astype(np.int64)
            s, d = _reject(*_rmat_edges(per_edge(bits), total, gen), ne)
        else:
            first = torch.from_numpy((np.cumsum(m[which]) - m[which])).to(DEV)
            base = torch.repeat_interleave(first, reps, output_size=total)
            loc = torch.arange(total, device=DEV) - base
            mb = per_edge(mba, torch.int64)
            place = (_rand(total, gen).double() * (2 * loc + 1)).long().clamp_(max=2 * loc)
            cur = place
            for _ in range(64):
                odd = (cur & 1) == 1
                if not bool(odd.any()):
                    break
                cur = torch.where(odd, place[base + (cur >> 1)], cur)
            s = (loc // mb).int()
            d = ((cur >> 1) // mb).int()
        parts.append((s + off, d + off))
    return (torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts]), vbase)


def _edges(case, seed):
    """(n, src, dst): one graph's undirected edge list on the device."""
    gen = torch.Generator(DEV).manual_seed(int(seed))
    fam, m = case["family"], case["m"]
    if fam == "er":
        n = case["n"]
        return n, torch.randint(0, n, (m,), generator=gen, device=DEV, dtype=torch.int32), \
            torch.randint(0, n, (m,), generator=gen, device=DEV, dtype=torch.int32)
    if fam == "rmat_n" or "scale" not in case:
        n = case["n"]
        s, d = _reject(*_rmat_edges(max(1, (n - 1).bit_length()), m, gen), n)
        return n, s, d
    n = 1 << case["scale"]
    s, d = _rmat_edges(case["scale"], m, gen)
    if fam == "planted":
        k = case["k"]
        who = torch.randperm(n, generator=gen, device=DEV)[:k].int()
        i, j = torch.triu_indices(k, k, 1, device=DEV)
        keep = _rand(i.numel(), gen) < case["p"]
        s, d = torch.cat([s, who[i[keep]]]), torch.cat([d, who[j[keep]]])
    return n, s, d


def _listing(case, seed):
    """(n, src, dst): an edge list of m lines as a builder gets it: 90% distinct
    edges of the family, 1% self-loops, the rest repeated lines, shuffled (the
    shares are fixed, so that every seed's CSR has the same size)."""
    m = case["m"]
    keep, loops = int(0.9 * m), m // 100
    keys = torch.empty(0, dtype=torch.int64, device=DEV)
    turn = 0
    while keys.numel() < keep:
        n, s, d = _edges(case, int(seed) + 1000003 * turn)
        keys = torch.unique(torch.cat([keys, _edge_keys(s, d, n)]))
        turn += 1
    gen = torch.Generator(DEV).manual_seed(int(seed) + 2)
    keys = keys[torch.randperm(keys.numel(), generator=gen, device=DEV)[:keep]]
    again = torch.randint(0, keep, (m - keep - loops,), generator=gen, device=DEV)
    loop = torch.randint(0, n, (loops,), generator=gen, device=DEV)
    keys = torch.cat([keys, keys[again], loop * n + loop])
    keys = keys[torch.randperm(m, generator=gen, device=DEV)]
    a, b = (keys // n).int(), (keys % n).int()
    flip = _rand(m, gen) < 0.5
    return n, torch.where(flip, b, a), torch.where(flip, a, b)


def _expected_edges(case):
    m = case["m"]
    return m + (int(case["k"] * (case["k"] - 1) / 2 * case["p"]) if case.get("family") == "planted" else 0)


def _graph(s, d, n, order="dedup"):
    torch.cuda.synchronize()
    g = pg.Graph.from_edges_device(s.data_ptr(), d.data_ptr(), s.numel(), n, dedup=order == "dedup",
                                   sort_rows=order == "sort")
    return g


class _Resident:
    """Device memory of the engine as torch sees it."""

    def __init__(self, ptr, count, typestr, keep):
        self.keep = keep
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _view(ptr, count, typestr, keep):
    return torch.as_tensor(_Resident(ptr, count, typestr, keep), device=DEV)


def _core(g):
    return _view(g.device_core(), g.n, "<i4", g)


def _csr(g):
    n, nnz, _, _ = g.info()
    rowptr, col = g.device_csr()
    return _view(rowptr, n + 1, "<i8", g), _view(col, nnz, "<i4", g)


# -------------------------------------------------------------- prepare ----
def prepare(case, seed):
    op = case["op"]
    if op == "peel":
        n, s, d = _edges(case, seed)
        return {"case": case, "g": _graph(s, d, n)}
    if op == "batch":
        s, d, vbase = _mix_edges(case, seed)
        g = _graph(s, d, int(vbase[-1]))
        return {"case": case, "g": g, "b": pg.Batch(g, vbase.astype(np.uint32))}
    if op == "noalloc":
        n, s, d = _edges(case, seed)
        rowptr, col = _plain_csr(n, s, d)
        return {"case": case, "n": n, "rowptr": rowptr, "col": col.int(),
                "core": torch.empty(n, dtype=torch.int32, device=DEV)}
    if op == "build":
        n, s, d = _listing(case, seed)
        return {"case": case, "n": n, "s": s, "d": d}
    if op == "update":
        n, s, d, ins, dels = _update(case, seed)
        g = _graph(s, d, n)
        g.decompose_device("peelone_dyn")
        host = [tuple(x.cpu().numpy().astype(np.uint32) for x in e) for e in (ins, dels)]
        return {"case": case, "g": g, "ins": host[0] if ins[0].numel() else None, "dels": host[1]}
    # serve: host CSRs of the requests, and a server around a resident graph
    s, d, vbase = _mix_edges(case, seed)
    rowptr, col = (x.cpu().numpy() for x in _plain_csr(int(vbase[-1]), s, d))
    reqs = []
    for lo, hi in zip(vbase[:-1], vbase[1:]):
        r = rowptr[lo:hi + 1]
        reqs.append(((r - r[0]).copy(), (col[r[0]:r[-1]] - lo).astype(np.uint32)))
    n, s, d, ins, dels = _update(_resident_case(case), seed)
    g = _graph(s, d, n)
    host = [tuple(x.cpu().numpy().astype(np.uint32) for x in e) for e in (ins, dels)]
    return {"case": case, "g": g, "server": pg.Server(g), "reqs": reqs, "ins": host[0], "dels": host[1]}


def _resident_case(case):
    return {"op": "update", "kind": "mixed", "scale": 18, "ef": 16, "batch": case["batch"]}


def _update(case, seed):
    """A base graph, edges to insert that it lacks and edges to delete that it has."""
    n, s, d = _edges({"family": "rmat", "scale": case["scale"], "m": case["ef"] << case["scale"]}, seed)
    keys = _edge_keys(s, d, n)
    gen = torch.Generator(DEV).manual_seed(int(seed) + 1)
    b = case["batch"]
    n_del = b if case["kind"] == "delete" else b - b // 2
    dk = keys[torch.randperm(keys.numel(), generator=gen, device=DEV)[:n_del]]
    dels = ((dk // n).int(), (dk % n).int())
    none = torch.empty(0, dtype=torch.int32, device=DEV)
    ins = (none, none)
    if case["kind"] == "mixed":
        a = torch.randint(0, n, (2, 2 * (b // 2) + 64), generator=gen, device=DEV)
        lo, hi = a.min(0).values, a.max(0).values
        k = torch.unique((lo * n + hi)[lo != hi])
        at = torch.searchsorted(keys, k).clamp_(max=keys.numel() - 1)
        k = k[keys[at] != k]
        k = k[torch.randperm(k.numel(), generator=gen, device=DEV)[:b // 2]]
        ins = ((k // n).int(), (k % n).int())
    return n, s, d, ins, dels


# ------------------------------------------------------------------ run ----
def run(state):
    op = state["case"]["op"]
    g = state.get("g")
    if op == "peel":
        if state["case"]["host"]:
            core, st = g.decompose(state["case"]["method"])
            return core.view(np.int32), st.kmax
        g.decompose_device(state["case"]["method"])
        return _core(g)
    if op == "batch":
        state["b"].decompose_device()
        return _core(g)
    if op == "noalloc":
        core = state["core"]
        pg.check(pg.lib().kc_decompose_noalloc(state["rowptr"].data_ptr(), state["col"].data_ptr(), state["n"],
                                               core.data_ptr(), torch.cuda.current_stream().cuda_stream))
        return core
    if op == "build":
        s, d = state["s"], state["d"]
        order = state["case"]["order"]
        return _csr(pg.Graph.from_edges_device(s.data_ptr(), d.data_ptr(), s.numel(), state["n"],
                                               dedup=order == "dedup", sort_rows=order == "sort"))
    if op == "update":
        ins, dels = state["ins"], state["dels"]
        _, a = g.update(ins, dels, want_core=False)
        changed = _core(g).clone()
        torch.cuda.current_stream().synchronize()  # the core array is the engine's own and is written next
        _, b = g.update(dels, ins, want_core=False)
        return [changed, _core(g), a["inserted"], a["deleted"], b["inserted"], b["deleted"]]
    srv = state["server"]
    tickets = [srv.submit_update(state["ins"], state["dels"], want_core=True)]
    tickets += [srv.submit_decompose(r, c) for r, c in state["reqs"]]
    tickets.append(srv.submit_update(state["dels"], state["ins"], want_core=True))
    sizes = [g.n] + [r.size - 1 for r, _ in state["reqs"]] + [g.n]
    return [srv.wait(t, core_cap=n)["core"].view(np.int32) for t, n in zip(tickets, sizes)]


# ----------------------------------------------------------------- work ----
def work(case):
    """Inputs read once, results written once: 8 B per row offset, 4 B per
    directed entry, 4 B per core number, 8 B per listed edge."""
    op = case["op"]

    def csr(n, m):
        return 8 * (n + 1) + 8 * m

    if op in ("peel", "noalloc", "build"):
        n = 1 << case["scale"] if "scale" in case else case["n"]
        m = _expected_edges(case)
        return {"bytes": csr(n, m) + (8 * m if op == "build" else 4 * n), "flops": 0}
    if op == "update":
        n = 1 << case["scale"]
        # both updates read the graph, write the changed one and the cores
        return {"bytes": 2 * (2 * csr(n, case["ef"] * n) + 4 * n + 8 * case["batch"]), "flops": 0}
    n, _, m, _ = _mix_params(case)
    b = csr(int(n.sum()), int(m.sum())) + 4 * int(n.sum())
    return {"bytes": b + (work(_resident_case(case))["bytes"] if op == "serve" else 0), "flops": 0}


# ---------------------------------------------------------------- exact ----
def _edge_keys(s, d, n):
    """Sorted distinct keys lo * n + hi of an undirected edge list without self-loops."""
    lo, hi = torch.minimum(s, d), torch.maximum(s, d)
    on = lo != hi
    return torch.unique(lo[on].long() * n + hi[on])


def _csr_of_keys(keys, n):
    lo, hi = keys // n, keys % n
    both = torch.cat([keys, hi * n + lo])
    both = torch.sort(both).values
    row = both // n
    rowptr = torch.searchsorted(row, torch.arange(n + 1, device=DEV))
    return rowptr, both % n


def _plain_csr(n, s, d):
    return _csr_of_keys(_edge_keys(s, d, n), n)


def _plain_cores(rowptr, col):
    """Core numbers by peeling: while a vertex has at most k neighbours left it
    leaves with core k, then k grows to the smallest count left."""
    n = rowptr.numel() - 1
    deg = (rowptr[1:] - rowptr[:-1]).clone()
    core = torch.zeros(n, dtype=torch.int64, device=DEV)
    left = torch.ones(n, dtype=torch.bool, device=DEV)
    alive = torch.arange(n, device=DEV)
    k = 0
    while alive.numel():
        da = deg[alive]
        k = max(k, int(da.min()))
        front = alive[da <= k]
        alive = alive[da > k]
        while front.numel():
            left[front] = False
            core[front] = k
            cnt = rowptr[front + 1] - rowptr[front]
            total = int(cnt.sum())
            first = torch.cumsum(cnt, 0) - cnt
            at = torch.arange(total, device=DEV) + torch.repeat_interleave(rowptr[front] - first, cnt, output_size=total)
            u = col[at].long()
            u = u[left[u]]
            deg.index_add_(0, u, torch.full_like(u, -1))
            u = torch.unique(u[deg[u] <= k])
            front = u
        alive = alive[left[alive]]
    return core


def exact(case, seed):
    op = case["op"]
    if op == "serve" or (op == "batch" and case["graphs"] > 1024):
        return _exact_packed(case, seed)
    if op == "build":
        n, s, d = _listing(case, seed)
        if case["order"] == "dedup":
            rowptr, col = _plain_csr(n, s, d)
        else:
            on = s != d
            row = torch.stack([s[on], d[on]], 1).reshape(-1).long()
            other = torch.stack([d[on], s[on]], 1).reshape(-1)
            if case["order"] == "sort":
                key = torch.sort(row * n + other).values
                row, col = key // n, key % n
            else:
                row, at = torch.sort(row, stable=True)
                col = other[at]
            rowptr = torch.searchsorted(row, torch.arange(n + 1, device=DEV))
        return rowptr, col.int()
    if op == "update":
        n, s, d, ins, dels = _update(case, seed)
        keys = _edge_keys(s, d, n)
        dk = _edge_keys(*dels, n)
        changed = torch.sort(torch.cat([keys[~torch.isin(keys, dk)], _edge_keys(*ins, n)])).values
        a, b = (_plain_cores(*_csr_of_keys(k, n)).int() for k in (changed, keys))
        ni, nd = int(ins[0].numel()), int(dels[0].numel())
        return [a, b, ni, nd, nd, ni]
    if op == "batch":
        return _exact_packed(case, seed)
    n, s, d = _edges(case, seed)
    rowptr, col = _plain_csr(n, s, d)
    del s, d
    core = _plain_cores(rowptr, col)
    if case.get("method") == "gppeel":
        core[rowptr[1:] == rowptr[:-1]] = 1
    return (core.int(), int(core.max())) if case.get("host") else core.int()


def _exact_packed(case, seed):
    s, d, vbase = _mix_edges(case, seed)
    cores = _plain_cores(*_plain_csr(int(vbase[-1]), s, d)).int()
    if case["op"] == "batch":
        return cores
    a, b = exact(_resident_case(case), seed)[:2]
    return [a] + [cores[lo:hi] for lo, hi in zip(vbase[:-1], vbase[1:])] + [b]
