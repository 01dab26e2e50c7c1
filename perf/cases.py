"""The work that a user of the solver has it do, as cases that can be timed.

Every case goes through the Python package's public calls (kc_cuda_b200): one
context per process, as a long-lived program keeps it, with its memory pool
grown once.  Graphs are seeded R-MAT (a/b/c/d = .57/.19/.19/.05), Erdos-Renyi
or Chung-Lu draws with a planted dense block (pair probability 0.95), the
families of this repository's configurations, made on the GPU.

Kinds ("do"):
  tsv       solve_tsv on host bytes, the `-f` path in one call
  staged    StagedTsv.solve, the bytes already in device memory
  pairs     load_pairs (unordered records, repeats, self-loops) + kmax_truss
  batch     Batch.add_mix + run + results, many uneven graphs at once
  serve     Server, requests of records one after another (light load)
  support   Graph.tricount, triangles through every edge
  truss     Graph.trussness, every edge's truss number
  cores     Graph.core_numbers
  kcore     Graph.kmax_core, membership of one core
"""
import math

import numpy as np
import torch

from kc_cuda_b200.solver import Context

_CTX = []


def _context():
    if not _CTX:
        _CTX.append(Context(0))
        _CTX[0].set_option("pool_reserve_mb", 16384)
    return _CTX[0]


def _graph(name, do, kind, n, draws, block=0, **more):
    return dict(name=name, do=do, kind=kind, n=n, draws=draws, block=block, **more)


def listed():
    return [
        # The smallest call: a graph of the size of this repository's fixtures
        # (R-MAT scale 10, edge factor 8), host bytes to answer.  Latency.
        _graph("tsv-rmat10", "tsv", "rmat", 1 << 10, 8 << 10, 12),
        # Configuration 1: R-MAT scale 16, edge factor 16, a block of 30.
        _graph("tsv-rmat16", "tsv", "rmat", 1 << 16, 16 << 16, 30),
        # End to end from pinned host memory with the chunked ingest (three
        # chunks or more): configuration 2's family at scale 21.
        _graph("tsv-rmat21", "tsv", "rmat", 1 << 21, 32 << 21, 200, pinned=True),
        # The whole solve from device-resident bytes: configuration 2 (scale
        # 24, edge factor 32) at a quarter of its vertices.
        _graph("staged-rmat22", "staged", "rmat", 1 << 22, 32 << 22, 200),
        # Configuration 3's family (Chung-Lu, exponent 2.1, hubs) at a
        # twentieth of its size; an odd vertex count.
        _graph("staged-chunglu", "staged", "chunglu", 2_500_001, 50_000_000, 150),
        # A program that holds edge records in any order: the sorting route
        # and a sparse graph without a dense core.
        _graph("pairs-er", "pairs", "er", 300_007, 6_000_000, 40),
        # Configuration 4: a batch of the mix (10^3 to 10^6 vertices each).
        dict(name="batch-mix", do="batch", graphs=64),
        # Configuration 5 under light load: small requests that find the
        # server idle, so each is a wave of its own.
        dict(name="serve-light", do="serve", requests=8, n_lo=1_000, n_hi=60_000, ef=16),
        # Triangle counts of a sparse graph (vertex bitmaps / lists).
        _graph("support-er", "support", "er", 250_007, 8_000_000, edges=7_900_000),
        # Truss numbers of configuration 1's graph: every level is climbed.
        _graph("truss-rmat16", "truss", "rmat", 1 << 16, 16 << 16, 30, edges=850_000),
        # Core numbers of a skewed graph with odd sizes.
        _graph("cores-rmat19", "cores", "rmat", 400_009, 8_000_000, 60),
        # Membership of one core and the largest core number.
        _graph("kcore-rmat18", "kcore", "rmat", 1 << 18, 16 << 18, 30, k=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["tsv", "tsv", "staged", "staged", "pairs", "batch", "serve", "support", "truss", "cores", "kcore"])
    if do == "batch":
        return dict(do=do, graphs=_log(rng, 4, 64))
    if do == "serve":
        hi = _log(rng, 2_000, 60_000)
        return dict(do=do, requests=rng.randint(2, 8), n_lo=1_000, n_hi=hi, ef=rng.randint(4, 16))
    top = {"tsv": 1 << 20, "staged": 1 << 22, "pairs": 1 << 20, "support": 250_000, "truss": 1 << 17, "cores": 1 << 20,
           "kcore": 1 << 20}[do]
    kind = rng.choice(["rmat", "rmat", "chunglu", "er"])
    if do == "truss":
        kind = "rmat"
    n = _log(rng, 4000 if do in ("support", "truss") else 500, top) | 1
    ef = rng.randint(4, 32 if n <= 1 << 21 else 24)
    case = dict(do=do, kind=kind, n=n, draws=ef * n + rng.randint(0, 63), block=rng.choice([10, 30, 60, 90]))
    if do in ("support", "truss"):
        case["edges"] = case["draws"] // 2
    if do == "tsv":
        case["pinned"] = rng.random() < 0.5
    if do == "kcore":
        case["k"] = rng.randint(1, 24)
    return case


def _draws(kind, n, draws, block, gen):
    """Raw draws (u, v), repeats and self-loops among them, on the GPU, and
    the pairs of the planted block.  The last draw names the last id, so a
    graph's vertex count does not depend on the seed."""
    dev = "cuda"
    if kind == "rmat":
        scale = max(1, (n - 1).bit_length())
        u = torch.zeros(draws, dtype=torch.int64, device=dev)
        v = torch.zeros(draws, dtype=torch.int64, device=dev)
        for _ in range(scale):
            r = torch.rand(draws, device=dev, generator=gen)
            u = (u << 1) | (r >= 0.76)
            v = (v << 1) | (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        if n < 1 << scale:
            u, v = u % n, v % n
    elif kind == "er":
        u = torch.randint(n, (draws,), device=dev, generator=gen)
        v = torch.randint(n, (draws,), device=dev, generator=gen)
    else:
        w = (5.0 * torch.rand(n, dtype=torch.float64, device=dev, generator=gen).clamp_(min=1e-12) ** (-1.0 / 1.1))
        cdf = torch.cumsum(w.clamp_(max=max(50.0, n / 25.0)), 0)
        r = torch.rand(2, draws, dtype=torch.float64, device=dev, generator=gen) * cdf[-1]
        u, v = torch.searchsorted(cdf, r).clamp_(max=n - 1)
    u[-1] = v[-1] = n - 1
    c = torch.randperm(n, device=dev, generator=gen)[:block]
    i, j = torch.triu_indices(len(c), len(c), 1, device=dev)
    kept = torch.rand(len(i), device=dev, generator=gen) < 0.95
    return u, v, c[i[kept]], c[j[kept]]


def _edges(u, v):
    """Distinct undirected edges u << 32 | v (u < v), ascending."""
    keep = u != v
    u, v = u[keep], v[keep]
    return torch.unique((torch.minimum(u, v) << 32) | torch.maximum(u, v))


def _tsv(keys, pinned):
    """Host bytes of the cleaned edge list: `x<TAB>y` lines, both directions,
    grouped by y ascending (the input form of the command line tool)."""
    a, b = keys >> 32, keys & 0xFFFFFFFF
    arcs = torch.sort(torch.cat([(a << 32) | b, (b << 32) | a]))[0]
    y, x = arcs >> 32, arcs & 0xFFFFFFFF
    del a, b, arcs

    def digits(t):
        d = torch.ones_like(t)
        for p in range(1, 10):
            d += t >= 10 ** p
        return d

    dx, dy = digits(x), digits(y)
    end = torch.cumsum(dx + dy + 2, 0)
    out = torch.empty(int(end[-1]) if len(end) else 0, dtype=torch.uint8, device=keys.device)
    out[end - 1] = 10
    out[end - dy - 2] = 9
    for t, d, last in ((y, dy, end - 2), (x, dx, end - dy - 3)):
        for p in range(int(d.max()) if len(d) else 0):
            m = d > p
            out[(last - p)[m]] = ((t // 10 ** p) % 10 + 48)[m].to(torch.uint8)
    if not pinned:
        return out.cpu().numpy()
    host = torch.empty(out.shape, dtype=torch.uint8, pin_memory=True)
    host.copy_(out)
    return host.numpy()


def _records(u, v):
    return ((u << 32) | v).cpu().numpy().view(np.uint64)


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    return gen


def _case_draws(case, seed):
    gen = _generator(seed)
    u, v, bu, bv = _draws(case["kind"], case["n"], case["draws"], case["block"], gen)
    if "edges" not in case:
        return torch.cat([u, bu]), torch.cat([v, bv])
    # Exactly that many distinct edges (an output has an entry for each): the
    # block's and a random part of the others.
    own, rest = _edges(bu, bv), _edges(u, v)
    rest = rest[~torch.isin(rest, own)]
    rest = rest[torch.randperm(len(rest), device=rest.device, generator=gen)[:case["edges"] - len(own)]]
    keys = torch.cat([own, rest])
    return keys >> 32, keys & 0xFFFFFFFF


def prepare(case, seed):
    do = case["do"]
    s = {"do": do, "case": case}
    if do == "batch":
        b = _context().batch()
        b.add_mix(0, case["graphs"], base_seed=1 + int(seed) % (1 << 40))
        s["batch"] = b
    elif do == "serve":
        gen, k = _generator(seed), case["requests"]
        s["records"] = []
        for i in range(k):
            n = int(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** (i / max(1, k - 1)))
            u, v, bu, bv = _draws("rmat" if i % 2 else "er", n, case["ef"] * n, 20, gen)
            s["records"].append(_records(torch.cat([u, bu]), torch.cat([v, bv])))
        s["server"] = Context(0).server()
    elif do in ("tsv", "staged"):
        data = _tsv(_edges(*_case_draws(case, seed)), bool(case.get("pinned")) or do == "staged")
        s["data"] = data if do == "tsv" else _context().stage_tsv(data)
        _context()
    else:
        s["records"] = _records(*_case_draws(case, seed))
        if do != "pairs":
            s["graph"] = _context().load_pairs(s["records"])
            s["k"] = case.get("k", 0)
    torch.cuda.empty_cache()
    return s


def run(s):
    do = s["do"]
    if do == "tsv":
        return _context().solve_tsv(s["data"])
    if do == "staged":
        return s["data"].solve()
    if do == "pairs":
        g = _context().load_pairs(s["records"])
        answer = g.kmax_truss()
        g.free()
        return answer
    if do == "batch":
        s["batch"].run()
        kmax, edges = s["batch"].results()
        return kmax.astype(np.int64), edges.astype(np.int64)
    if do == "serve":
        answers = []
        for r in s["records"]:
            a = s["server"].wait(s["server"].submit_pairs(r))
            answers.append((int(a["kmax"]), int(a["edges"])))
        return answers
    if do == "support":
        return s["graph"].tricount().view(np.int32)
    if do == "truss":
        return s["graph"].trussness().view(np.int32)
    if do == "cores":
        return s["graph"].core_numbers().view(np.int32)
    member, cmax = s["graph"].kmax_core(s["k"])
    return member, cmax


def work(case):
    """Bytes of one pass: the input as the call is given it, and its result.
    Nothing on the path is floating point."""
    do = case["do"]
    if do == "batch":  # the mix: mean vertices (10^6 - 10^3) / ln 10^3, 34 records each
        return {"bytes": 8.0 * 34 * 144_600 * case["graphs"], "flops": 0}
    if do == "serve":
        k = case["requests"]
        n = sum(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** (i / max(1, k - 1)) for i in range(k))
        return {"bytes": 8.0 * case["ef"] * n, "flops": 0}
    m, n = case.get("edges", case["draws"]), case["n"]
    if do in ("tsv", "staged"):
        return {"bytes": 2.0 * m * (2 * len(str(n)) + 1), "flops": 0}
    if do == "pairs":
        return {"bytes": 8.0 * m, "flops": 0}
    csr = 8.0 * m + 8.0 * n
    return {"bytes": csr + (4.0 * m if do in ("support", "truss") else 4.0 * n if do == "cores" else n), "flops": 0}


def _support(keys, n):
    """Triangles through each edge: every neighbour of the end of smaller
    degree is looked up next to the other end."""
    u, v = keys >> 32, keys & 0xFFFFFFFF
    arcs = torch.sort(torch.cat([u * n + v, v * n + u]))[0]
    deg = torch.bincount(arcs // n, minlength=n)
    first = torch.cumsum(deg, 0) - deg
    swap = deg[u] > deg[v]
    a, b = torch.where(swap, v, u), torch.where(swap, u, v)
    out = torch.zeros_like(u)
    step = 1 << 18
    for i in range(0, len(u), step):
        aa, bb = a[i:i + step], b[i:i + step]
        d = deg[aa]
        own = torch.repeat_interleave(torch.arange(len(aa), device=u.device), d)
        at = torch.arange(len(own), device=u.device) - torch.repeat_interleave(torch.cumsum(d, 0) - d, d)
        want = bb[own] * n + arcs[first[aa][own] + at] % n
        pos = torch.searchsorted(arcs, want).clamp_(max=len(arcs) - 1)
        out[i:i + step].index_add_(0, own, (arcs[pos] == want).to(torch.int64))
    return out


def _cores(keys, n):
    """Core numbers by peeling one level after another."""
    u, v = keys >> 32, keys & 0xFFFFFFFF
    core = torch.zeros(n, dtype=torch.int64, device=keys.device)
    alive = torch.ones(n, dtype=torch.bool, device=keys.device)
    k = 0
    while len(u):
        deg = torch.bincount(u, minlength=n) + torch.bincount(v, minlength=n)
        out = alive & (deg <= k)
        if bool(out.any()):
            core[out] = k
            alive &= ~out
            keep = alive[u] & alive[v]
            u, v = u[keep], v[keep]
        else:
            k = int(deg[alive].min())
    core[alive] = k
    return core


def exact(case, seed):
    """Counts in 64-bit integers; the answers of whole solves have no value
    here (they are whole numbers, compared as such)."""
    do = case["do"]
    if do not in ("support", "cores", "kcore") or case["draws"] > 9_000_000:
        return None
    u, v = _case_draws(case, seed)
    n = int(torch.maximum(u, v).max()) + 1  # ids of self-loops count
    keys = _edges(u, v)
    if do == "support":  # a hub's lookups would take too long
        return _support(keys, n) if case["kind"] == "er" else None
    core = _cores(keys, n)
    return core if do == "cores" else ((core >= case["k"]), int(core.max()))
