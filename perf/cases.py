"""The work that a user of this framework has it do, as measured cases.

One case is one pass through the public entry points (bbtc_b200.core) on a
seeded synthetic graph: a count on a resident graph, a request end to end from
host memory, the device preparation pipeline, a batch, an explicit task list,
the allocation-free count, a burst of served requests.

Graph families, drawn with torch on the GPU from the seed alone:
  rmat     `pairs` R-MAT pairs (.57/.19/.19/.05) over the next power of two;
           ids >= n are dropped, so n may be any number
  chunglu  power-law expected degrees (gamma 2.1, mean 2 pairs / n, weights
           capped at 50,000 at 2^23 vertices)
  rgg      random geometric graph in the unit square, mean degree 12
"""
import ctypes
import math
import os

os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")  # a server's streams want a hardware queue each

import torch  # noqa: E402

from bbtc_b200 import Context, Graph, Server, count_batch, core, options  # noqa: E402

GPU = "cuda"


# ---- the cases -----------------------------------------------------------------
def listed():
    return [
        # A small resident graph counted again and again (a monitor, a service's warm graph): latency.
        dict(name="count-rmat-s12", op="count", family="rmat", n=1 << 12, pairs=16 << 12, parts=8, cuts="pal"),
        # An ordinary resident graph: the reference's CPU-runnable size.
        dict(name="count-rmat-s16", op="count", family="rmat", n=1 << 16, pairs=16 << 16, parts=8, cuts="pal"),
        # The single-graph benchmark workload.
        dict(name="count-rmat-s22", op="count", family="rmat", n=1 << 22, pairs=16 << 22, parts=16, cuts="pal"),
        # The largest vertex count: sparse power-law rows, 32 parts.
        dict(name="count-chunglu-8m", op="count", family="chunglu", n=1 << 23, pairs=10 << 23, parts=32, cuts="n1d"),
        # One request end to end from page-locked host memory: upload, layout, count, free.  The smallest size
        # that the request stream serves, an ordinary one, and the benchmark workload.
        dict(name="request-rmat-s12", op="request", family="rmat", n=1 << 12, pairs=16 << 12, parts=4, cuts="pal"),
        dict(name="request-rmat-s18", op="request", family="rmat", n=1 << 18, pairs=16 << 18, parts=8, cuts="pal"),
        dict(name="request-rmat-s22", op="request", family="rmat", n=1 << 22, pairs=16 << 22, parts=16, cuts="pal"),
        # Raw pairs already in device memory: clean, orient, cut, lay out and count without leaving the GPU;
        # an odd vertex count.
        dict(name="prepare-rmat-1m", op="prepare", family="rmat", n=999_983, pairs=16_000_000, parts=16, cuts="n1d"),
        # Many mixed graphs in one launch (the batched configuration: R-MAT s10-14 and geometric graphs).
        dict(name="batch-96", op="batch", graphs=96, low=10, high=14, parts=8),
        # Part of the task list (a border at half of it): per-task kernels over the forward tiles.
        dict(name="tasks-rmat-s18", op="tasks", family="rmat", n=1 << 18, pairs=16 << 18, parts=16, cuts="pal",
             kernel="auto", mode="persistent"),
        # A caller that owns the device's memory: the CSR is counted where it lies.
        dict(name="noalloc-rmat-s17", op="noalloc", family="rmat", n=1 << 17, pairs=16 << 17),
        # Requests of mixed sizes arriving together at the server.
        dict(name="serve-32", op="serve", requests=32, low=12, high=17, parts=4),
    ]


def _log(rng, low, high):
    """A whole number between low and high, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """A case of the same ranges: every entry point, sizes over their logarithm, any vertex count."""
    op = rng.choice(["count", "count", "request", "request", "prepare", "batch", "tasks", "noalloc", "serve"])
    if op == "batch":
        low = rng.randint(10, 12)
        return dict(op=op, graphs=_log(rng, 4, 96), low=low, high=low + rng.randint(0, 2), parts=rng.randint(4, 16))
    if op == "serve":
        low = rng.randint(12, 15)
        return dict(op=op, requests=_log(rng, 4, 32), low=low, high=low + rng.randint(0, 2), parts=rng.randint(2, 8))
    family = rng.choice(["rmat", "rmat", "chunglu", "rgg"])
    top = {"count": 1 << 21, "request": 1 << 21, "prepare": 400_000, "tasks": 1 << 17, "noalloc": 1 << 17}[op]
    n = _log(rng, 1 << 10, top)
    pairs = n * (6 if family == "rgg" else 10 if family == "chunglu" else rng.randint(8, 16))
    case = dict(op=op, family=family, n=n, pairs=pairs)
    if op != "noalloc":
        case.update(parts=rng.randint(4, 32), cuts=rng.choice(["pal", "n1d", "uni"]))
    if op == "tasks":
        case.update(parts=rng.randint(4, 16), kernel=rng.choice(["auto", "search", "merge"]),
                    mode=rng.choice(["persistent", "persistent", "plain"]))
        if case["mode"] == "plain":  # one launch per task: few parts
            case["parts"] = rng.randint(3, 6)
    return case


# ---- inputs (plain torch on the GPU) -------------------------------------------
def _rmat(n, pairs, gen):
    u = torch.zeros(pairs, dtype=torch.int32, device=GPU)
    v = torch.zeros(pairs, dtype=torch.int32, device=GPU)
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(pairs, device=GPU, generator=gen)
        low = r >= 0.76  # the lower quadrants: c and d
        v = 2 * v + torch.where(low, r >= 0.95, r >= 0.57)
        u = 2 * u + low
    return u, v


def _chunglu(n, pairs, gen):
    rank = torch.arange(n, dtype=torch.float64, device=GPU) + 1
    w = rank.pow(-1 / 1.1)
    w *= 2 * pairs / w.sum()
    w.clamp_(max=50_000 * math.sqrt(n / (1 << 23)))
    total = torch.cumsum((w * (1 << 16)).long() + 1, 0)  # whole numbers: the same sums on every run
    at = torch.randperm(n, dtype=torch.int32, device=GPU, generator=gen)  # ids in no order of degree
    high = int(total[-1])
    return [at[torch.searchsorted(total, torch.randint(high, (pairs,), device=GPU, generator=gen), right=True)]
            for _ in "uv"]


def _rgg(n, _pairs, gen):
    x, y = torch.rand(2, n, dtype=torch.float64, device=GPU, generator=gen)
    radius = math.sqrt(12 / (math.pi * n))
    side = max(1, int(1 / radius))
    cx, cy = (x * side).long().clamp_(max=side - 1), (y * side).long().clamp_(max=side - 1)
    cell = cx * side + cy
    order = torch.argsort(cell)
    starts = torch.searchsorted(cell[order], torch.arange(side * side + 1, device=GPU))
    us, vs = [], []
    for dx, dy in ((0, 0), (1, 0), (0, 1), (1, 1), (1, -1)):
        p = torch.nonzero((cx + dx < side) & (cy + dy < side) & (cy + dy >= 0)).flatten()
        c = (cx[p] + dx) * side + cy[p] + dy
        count = starts[c + 1] - starts[c]
        a = torch.repeat_interleave(p, count)
        first = torch.repeat_interleave(starts[c] - (torch.cumsum(count, 0) - count), count)
        b = order[first + torch.arange(a.numel(), device=GPU)]
        keep = (x[a] - x[b]) ** 2 + (y[a] - y[b]) ** 2 <= radius * radius
        if (dx, dy) == (0, 0):
            keep &= a < b
        us.append(a[keep])
        vs.append(b[keep])
    return torch.cat(us).int(), torch.cat(vs).int()


def _pairs(family, n, pairs, seed):
    gen = torch.Generator(device=GPU)
    gen.manual_seed(seed)
    return {"rmat": _rmat, "chunglu": _chunglu, "rgg": _rgg}[family](n, pairs, gen)


def _orient(n, u, v):
    """Distinct edges without self loops, relabelled by (degree, id), from the lower to the higher new id."""
    keep = (u != v) & (u < n) & (v < n)
    lo, hi = torch.minimum(u, v)[keep].long(), torch.maximum(u, v)[keep].long()
    key = torch.unique(lo * n + hi)
    lo, hi = torch.div(key, n, rounding_mode="floor"), key % n
    degree = torch.bincount(lo, minlength=n) + torch.bincount(hi, minlength=n)
    rank = torch.empty(n, dtype=torch.int64, device=GPU)
    rank[torch.argsort(degree, stable=True)] = torch.arange(n, device=GPU)
    a, b = rank[lo], rank[hi]
    key = torch.sort(torch.minimum(a, b) * n + torch.maximum(a, b)).values
    row = torch.div(key, n, rounding_mode="floor")
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=GPU)
    indptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    return indptr.int(), (key % n).int()


def _csr(case, seed):
    return _orient(case["n"], *_pairs(case["family"], case["n"], case["pairs"], seed))


def _mix(case, seed, how_many):
    """Family, vertices, pairs and seed of the graphs of a batch or a burst; one in eight of a batch geometric.
    Sizes depend on the case alone, so that two seeds cost the same; the smaller ones are the more common."""
    out = []
    for i in range(how_many):
        steps = case["high"] - case["low"] + 1
        scale = case["low"] + min(steps - 1, int(steps * ((i * 0.618) % 1.0) ** 1.5))
        if case["op"] == "batch" and i % 8 == 7:
            n = (1 << scale) * 4 + 37 * i
            out.append(dict(family="rgg", n=n, pairs=6 * n, seed=seed * 1000 + i))
        else:
            n = (1 << scale) - (i % 5)
            out.append(dict(family="rmat", n=n, pairs=(8 + i * 5 % 9) * n, seed=seed * 1000 + i))
    return out


def _room(case):
    """Room for the edges of a preparation: every pair (a geometric graph's number of pairs varies with the seed)."""
    return case["pairs"] + (case["n"] + 1024 if case["family"] == "rgg" else 0)


def _pinned(t):
    h = torch.empty(max(1, t.numel()), dtype=torch.int32, pin_memory=True)
    h[:t.numel()].copy_(t)
    return h


# ---- prepare / run ----------------------------------------------------------------
def prepare(case, seed):
    op = case["op"]
    s = dict(op=op, case=case)
    if op == "serve":
        s["requests"] = []
        for g in _mix(case, seed, case["requests"]):
            ip, ix = _csr(g, g["seed"])
            cuts = [g["n"] * i // case["parts"] for i in range(case["parts"] + 1)]
            hip, hix = _pinned(ip), _pinned(ix)
            s["requests"].append((g["n"], hip.numpy().view("u4"), hix.numpy()[:ix.numel()].view("u4"), cuts, hip, hix))
        s["server"] = Server(0, hbm_budget=4 << 30)
        return s
    s["ctx"] = ctx = Context(0)
    if op == "batch":
        s["graphs"] = []
        for g in _mix(case, seed, case["graphs"]):
            ip, ix = _csr(g, g["seed"])
            cuts = core.cuts_device(ctx, "uni", g["n"], ip.data_ptr(), ix.data_ptr(), ix.numel(), case["parts"])
            torch.cuda.synchronize()
            s["graphs"].append(Graph.upload_device(ctx, g["n"], ip.data_ptr(), ix.data_ptr(), ix.numel(), cuts))
        return s
    if op == "prepare":
        s["src"], s["dst"] = _pairs(case["family"], case["n"], case["pairs"], seed)
        s["indptr"] = torch.empty(case["n"] + 1, dtype=torch.int32, device=GPU)
        s["indices"] = torch.empty(_room(case), dtype=torch.int32, device=GPU)
        torch.cuda.synchronize()
        return s
    ip, ix = _csr(case, seed)
    n, m = case["n"], ix.numel()
    torch.cuda.synchronize()
    if op == "noalloc":
        s.update(indptr=ip, indices=ix, m=m, stream=torch.cuda.current_stream().cuda_stream)
        call = core.lib().bbtc_count_csr_noalloc
        call.restype = ctypes.c_int
        call.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_uint64,
                         ctypes.POINTER(ctypes.c_uint64), ctypes.c_void_p]
        s["call"] = call
        return s
    cuts = core.cuts_device(ctx, case["cuts"], n, ip.data_ptr(), ix.data_ptr(), m, case["parts"])
    if op == "request":
        s.update(indptr=_pinned(ip), indices=_pinned(ix), m=m, cuts=cuts)
        return s
    s["graph"] = graph = Graph.upload_device(ctx, n, ip.data_ptr(), ix.data_ptr(), m, cuts)
    if op == "tasks":
        tasks = graph.task_list(sorted=True)
        s["tasks"] = tasks[: max(1, len(tasks) // 2)]
        s["opts"] = options(kernel=case["kernel"], mode=case["mode"])
    return s


class _DeviceWords:
    """A library-held device array as torch sees it."""

    def __init__(self, ptr, count):
        self.__cuda_array_interface__ = dict(shape=(count,), typestr="<i4", data=(ptr, False), version=2)


def run(s):
    op, case = s["op"], s["case"]
    if op == "count":
        return s["graph"].count()
    if op == "request":
        g = Graph.upload_ptrs(s["ctx"], case["n"], s["indptr"].data_ptr(), s["indices"].data_ptr(), s["m"], s["cuts"])
        count = g.count()
        g.free()
        return count
    if op == "prepare":
        csr = core.DeviceCSR(s["ctx"], case["n"], s["src"].data_ptr(), s["dst"].data_ptr(), s["src"].numel())
        cuts = csr.cuts(case["parts"], case["cuts"])
        g = csr.graph(cuts)
        count = g.count()
        g.free()
        # the program keeps the cleaned graph in a buffer of its own (room for every pair, the rest filled with -1)
        s["indptr"].copy_(torch.as_tensor(_DeviceWords(csr.indptr_ptr, csr.n + 1), device=GPU))
        s["indices"][:csr.m].copy_(torch.as_tensor(_DeviceWords(csr.indices_ptr, csr.m), device=GPU))
        s["indices"][csr.m:].fill_(-1)
        torch.cuda.current_stream().synchronize()  # the copies read the library's arrays
        csr.free()
        return dict(count=count, cuts=torch.from_numpy(cuts.astype("i8")), indptr=s["indptr"], indices=s["indices"])
    if op == "batch":
        return torch.tensor(count_batch(s["ctx"], s["graphs"]))
    if op == "tasks":
        return s["graph"].count(s["tasks"], opts=s["opts"])
    if op == "noalloc":
        out = ctypes.c_uint64()
        core.check(s["call"](s["indptr"].data_ptr(), s["indices"].data_ptr(), case["n"], s["m"], ctypes.byref(out),
                             s["stream"]))
        return out.value
    server = s["server"]
    ids = [server.submit(n, ip, ix, cuts) for n, ip, ix, cuts, _, _ in s["requests"]]
    counts = []
    for rid in ids:
        info = server.wait(rid)
        if info.status != 1:
            raise RuntimeError(f"request failed with status {info.status}")
        counts.append(info.count)
        server.release(rid)
    return torch.tensor(counts)


# ---- what a pass cannot do without, and its answer in plain torch ---------------------
def work(case):
    """Bytes of the arrays that a pass takes and gives, each once (pairs for edges: a few repeat); a count does no
    floating-point work."""
    op = case["op"]
    if op in ("batch", "serve"):
        return dict(bytes=sum(4 * (g["n"] + 1) + 4 * g["pairs"] for g in _mix(case, 0, case.get("graphs") or case["requests"])),
                    flops=0)
    csr = 4 * (case["n"] + 1) + 4 * case["pairs"]
    return dict(bytes=csr + (8 * case["pairs"] if op == "prepare" else 0), flops=0)


MAX_WEDGES = 1_500_000_000  # more than this takes over 20 seconds or does not fit


def _triangles(n, indptr, indices):
    """Triangles of an oriented CSR: every edge (u, v) and w in N+(v), looked up as edge (u, w)."""
    indptr, indices = indptr.long(), indices.long()
    degree = indptr[1:] - indptr[:-1]
    row = torch.repeat_interleave(torch.arange(n, device=GPU), degree)
    key = row * n + indices
    wedges = torch.cumsum(degree[indices], 0)
    if not wedges.numel():
        return 0
    if int(wedges[-1]) > MAX_WEDGES:
        return None
    total, at, step = 0, 0, 1 << 26
    while at < wedges.numel():
        done = int(wedges[at - 1]) if at else 0
        end = max(at + 1, int(torch.searchsorted(wedges, done + step)))
        v = indices[at:end]
        count = degree[v]
        first = torch.repeat_interleave(indptr[v] - (torch.cumsum(count, 0) - count), count)
        w = indices[first + torch.arange(first.numel(), device=GPU)]
        want = torch.repeat_interleave(row[at:end], count) * n + w
        found = torch.searchsorted(key, want).clamp_(max=key.numel() - 1)
        total += int((key[found] == want).sum())
        at = end
    return total


def exact(case, seed):
    """What run() returns, from plain torch in 64-bit whole numbers; None where it would take too long, and for part of
    a task list, whose order is the library's."""
    op = case["op"]
    if op == "tasks":
        return None
    if op in ("batch", "serve"):
        how_many = case.get("graphs") or case["requests"]
        counts = [_triangles(g["n"], *_csr(g, g["seed"])) for g in _mix(case, seed, how_many)]
        return None if None in counts else torch.tensor(counts)
    indptr, indices = _csr(case, seed)
    count = _triangles(case["n"], indptr, indices)
    if op == "prepare":
        rest = torch.full((_room(case) - indices.numel(),), -1, dtype=torch.int32, device=GPU)
        return dict(count=count, cuts=None, indptr=indptr, indices=torch.cat([indices, rest]))
    return count
