"""The work that users of this library have it do, as cases that can be timed:
one pair (on the device and from host buffers), all pairs of a collection
(sparse and dense), and batches of pairs, through set_intersection_b200.api.
Inputs are made on the GPU, or by the library's seeded generators, from the
seed alone."""
import math

import torch

from set_intersection_b200 import api, generate


def listed():
    return [
        # One small pair through the simplest call (default technique, elements out): call latency.
        {"name": "sisi_small_call", "kind": "sisi_call", "na": 1500, "nb": 2300, "gap": 16.0, "tech": "ip"},
        # The plain single-pair configuration: 2^20 elements each of [0, 2^24), intersect path, elements out.
        {"name": "sisi_plain_ip", "kind": "sisi", "na": 1 << 20, "nb": 1 << 20, "gap": 16.0, "tech": "ip", "out": True},
        # The large single-pair configuration: 2^28 elements each of [0, 2^31), the engine's choice, elements out.
        {"name": "sisi_large_auto", "kind": "sisi", "na": 1 << 28, "nb": 1 << 28, "gap": 8.0, "tech": "auto",
         "out": True},
        # The skewed single-pair configuration: 2^16 elements looked up in 2^26, a fifth of them present.
        {"name": "sisi_skewed_auto", "kind": "sisi", "na": 1 << 16, "nb": 1 << 26, "gap": 16.0, "tech": "auto",
         "out": True},
        # One pair that lies in pinned host buffers, of sizes that are no power of two: copies up, count and
        # elements copied back (what the per-technique executables do for a file of two sets).
        {"name": "sisi_host_odd", "kind": "host", "na": 12345679, "nb": 9876543, "gap": 8.0, "tech": "auto"},
        # The power-law all-pairs configuration: 8192 sets of 16..65536 elements over 2^20 values, bitmap probes.
        {"name": "misi_powerlaw_bitmap", "kind": "misi", "k": 8192, "n_max": 65536, "values": 1 << 20,
         "tech": "bitmap", "cross": False},
        # One cross tile of a collection that is worked through tile by tile, hash probes.
        {"name": "misi_cross_tile_hi", "kind": "misi", "k": 3000, "n_max": 65536, "values": 1 << 20, "tech": "hi",
         "cross": True},
        # A smaller collection by intersect path.
        {"name": "misi_ip", "kind": "misi", "k": 1001, "n_max": 16384, "values": 1 << 18, "tech": "ip",
         "cross": False},
        # The dense all-pairs configuration: 16384 sets over 65536 values, 5 % membership, INT8 tensor cores.
        {"name": "dense_int8", "kind": "dense", "k": 16384, "values": 65536, "p": 0.05, "dtype": "int8"},
        # A ragged dense collection with FP8 operands.
        {"name": "dense_fp8_ragged", "kind": "dense", "k": 3001, "values": 40009, "p": 0.1, "dtype": "fp8"},
        # The batched configuration at a fifth of its pool and pairs: tuned table, captured once, replayed.
        {"name": "batch_graph_tuned", "kind": "batch", "k": 20000, "n_min": 32, "n_max": 1 << 18, "dense_part": 0.0,
         "npairs": 200000, "graph": True, "tech": "auto"},
        # A batch sent once, without tuning, over a pool whose sets are partly sparse and partly dense.
        {"name": "batch_call_mixed", "kind": "batch", "k": 1000, "n_min": 32, "n_max": 1 << 15, "dense_part": 0.4,
         "npairs": 20000, "graph": False, "tech": "auto"},
    ]


def _log(rng, lo, hi):
    """A whole number, log-uniform on [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sisi_call", "sisi", "sisi", "sisi", "host", "misi", "misi", "dense", "dense", "batch", "batch"])
    if kind == "sisi_call":
        return {"kind": kind, "na": _log(rng, 16, 1 << 18), "nb": _log(rng, 16, 1 << 18),
                "gap": rng.uniform(2.0, 64.0), "tech": rng.choice(["ip", "ip", "auto", "bitmap", "hi", "obs"])}
    if kind == "sisi":
        nb = _log(rng, 1 << 10, 1 << 27)
        na = max(16, nb // _log(rng, 1, 2048) if rng.random() < 0.3 else int(nb * rng.uniform(0.3, 1.0)))
        # one search per element of the smaller set (obs) is asked for where the sizes differ
        tech = rng.choice(["auto", "auto", "ip", "bitmap", "hi"] + (["obs"] if nb > 16 * na else []))
        return {"kind": kind, "na": na, "nb": nb, "gap": rng.uniform(4.0, 16.0), "tech": tech,
                "out": rng.random() < 0.75}
    if kind == "host":
        return {"kind": kind, "na": _log(rng, 1 << 12, 1 << 24), "nb": _log(rng, 1 << 12, 1 << 24),
                "gap": rng.uniform(4.0, 64.0), "tech": rng.choice(["auto", "ip", "bitmap"])}
    if kind == "misi":
        tech = rng.choice(["bitmap", "bitmap", "auto", "hi", "obs", "ip"])
        slow = tech in ("obs", "ip")
        return {"kind": kind, "k": _log(rng, 64, 1500 if slow else 5000), "n_max": _log(rng, 512, 16384 if slow else 65536),
                "values": _log(rng, 1 << 17, 1 << 21), "tech": tech, "cross": rng.random() < 0.3}
    if kind == "dense":
        return {"kind": kind, "k": _log(rng, 128, 10000), "values": _log(rng, 2000, 65536),
                "p": rng.uniform(0.02, 0.3), "dtype": rng.choice(["int8", "fp8"])}
    k = _log(rng, 200, 10000)
    return {"kind": "batch", "k": k, "n_min": 32, "n_max": _log(rng, 2048, 1 << 17),
            "dense_part": rng.choice([0.0, 0.0, rng.uniform(0.1, 0.8)]), "npairs": _log(rng, 200, 100000),
            "graph": rng.random() < 0.5, "tech": rng.choice(["auto", "auto", "auto", "ip", "obs", "hi", "bitmap"])}


# ------------------------------------------------------------------ inputs --
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _distinct(g, n, hi):
    """n distinct values uniform on [0, hi), ascending: int32 on the GPU."""
    hi = min(max(int(hi), 2 * n), (1 << 31) - 1)
    m = int(-hi * math.log1p(-n / hi) + 6 * math.sqrt(n) + 16)
    x = torch.randint(0, hi, (m,), generator=g, device="cuda", dtype=torch.int32).unique()
    while x.numel() < n:
        x = torch.cat([x, torch.randint(0, hi, (m // 8 + 16,), generator=g, device="cuda", dtype=torch.int32)]).unique()
    while x.numel() > n:  # surplus values leave at random
        keep = torch.ones(x.numel(), dtype=torch.bool, device="cuda")
        keep[torch.randint(0, x.numel(), (x.numel() - n,), generator=g, device="cuda")] = False
        x = x[keep]
    return x


def _pair(case, seed):
    """Two sets whose larger one has a mean gap of case["gap"] between its
    values; where the sizes of device sets differ widely, a fifth of the
    smaller is planted in the larger."""
    g = _generator(seed)
    na, nb = case["na"], case["nb"]
    hi = int(case["gap"] * max(na, nb))
    if case["kind"] != "sisi":  # the calls that return just the common elements: as many for every seed
        common = int(min(na, nb) / case["gap"])
        x = _distinct(g, na + nb - common, hi)
        p = torch.randperm(x.numel(), generator=g, device="cuda")
        return x[p[:na]].sort().values, x[p[na - common:]].sort().values
    a, b = _distinct(g, na, hi), _distinct(g, nb, hi)
    if nb > 64 * na:
        b = torch.cat([b[na // 5:], a[torch.randperm(na, generator=g, device="cuda")[:na // 5]]]).unique()
    return a, b


def _device_collection(elements, offsets, universe):
    return api.Collection(torch.from_numpy(elements.view("int32")).cuda(), torch.from_numpy(offsets).cuda(), universe)


def _pool(case, seed):
    """case["k"] sets of log-uniform sizes with uniform values: of [0, 2^26),
    and dense_part of the sets of [0, 2^16); pairs drawn uniformly."""
    g = _generator(seed)
    k, lo, hi = case["k"], case["n_min"], case["n_max"]
    u = torch.rand(k, generator=g, device="cuda", dtype=torch.float64)
    sizes = (lo * (hi / lo) ** u).long()
    small = torch.rand(k, generator=g, device="cuda") < case["dense_part"]
    sizes = torch.where(small, sizes.clamp(max=1 << 15), sizes)
    values = torch.where(small, 1 << 16, 1 << 26)
    parts, got = [], []
    step = max(1, (1 << 27) // hi)
    for s in range(0, k, step):
        e = min(k, s + step)
        n = sizes[s:e]
        of = torch.repeat_interleave(torch.arange(s, e, device="cuda"), n)
        v = (torch.rand(of.numel(), generator=g, device="cuda", dtype=torch.float64) * values[of]).long()
        key = ((of << 32) | v).sort().values.unique_consecutive()
        got.append(torch.bincount((key >> 32) - s, minlength=e - s))
        parts.append((key & 0xffffffff).int())
    offsets = torch.zeros(k + 1, dtype=torch.int64, device="cuda")
    offsets[1:] = torch.cat(got).cumsum(0)
    col = api.Collection(torch.cat(parts), offsets, (1 << 26) - 1)
    i = torch.randint(0, k, (case["npairs"],), generator=g, device="cuda")
    j = (i + torch.randint(1, k, (case["npairs"],), generator=g, device="cuda")) % k
    return col, torch.stack([i, j], 1).int().contiguous()


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case, "ws": api.Workspace()}
    if kind in ("sisi_call", "sisi", "host"):
        a, b = _pair(case, seed)
        if kind == "host":
            s["a"], s["b"] = a.cpu().pin_memory(), b.cpu().pin_memory()
            s["out"] = torch.empty(min(a.numel(), b.numel()), dtype=torch.int32).pin_memory()
            s["ctx"] = api.HostPair()
        else:
            s["a"], s["b"] = a, b
        if kind == "sisi":  # the result buffers that a program with many pairs keeps
            s["count"] = torch.zeros(1, dtype=torch.int64, device="cuda")
            s["out"] = torch.zeros(min(a.numel(), b.numel()), dtype=torch.int32, device="cuda") if case["out"] else None
            s["ws"].get(api.sisi_workspace_size(a.numel(), b.numel(), case["tech"]))
    elif kind == "misi":
        k = case["k"]
        s["col"] = _device_collection(*generate.powerlaw(seed, k, 16, case["n_max"], 1.1, case["values"], 0.8),
                                      case["values"])
        h = k // 2
        s["a"], s["b"] = ((0, h), (h, k)) if case["cross"] else (None, None)
        n = h * (k - h) if case["cross"] else k * (k - 1) // 2
        s["counts"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    elif kind == "dense":
        k = case["k"]
        s["col"] = _device_collection(*generate.bernoulli(seed, k, case["values"], case["p"]), case["values"] - 1)
        s["counts"] = torch.zeros(k * (k - 1) // 2, dtype=torch.int32, device="cuda")
    else:
        s["col"], s["pairs"] = _pool(case, seed)
        s["counts"] = torch.zeros(case["npairs"], dtype=torch.int32, device="cuda")
        if case["graph"]:
            table = api.batch_tune(s["col"], s["pairs"], 512, s["ws"]) if case["tech"] == "auto" else None
            s["graph"] = api.BatchGraph(s["col"], s["pairs"], s["counts"], case["tech"], table, s["ws"])
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "sisi_call":
        return api.intersect(s["a"], s["b"], case["tech"])
    if kind == "sisi":
        api.sisi_into(s["a"], s["b"], s["count"], s["out"], s["ws"], case["tech"])
        return [s["count"], s["out"]]
    if kind == "host":
        return api.intersect_host(s["a"], s["b"], case["tech"], s["out"], s["ctx"])
    if kind == "misi":
        api.misi_into(s["col"], s["counts"], case["tech"], s["a"], s["b"], workspace=s["ws"])
    elif kind == "dense":
        api.misi_dense_into(s["col"], s["counts"], "mm", case["dtype"], s["ws"])
    elif case["graph"]:
        s["graph"].launch()
    else:
        api.batch_count_into(s["col"], s["pairs"], s["counts"], case["tech"], None, s["ws"])
    return s["counts"]


# -------------------------------------------------------------------- work --
def _mean_sizes(inverse):
    """(mean size, mean of the smaller of two sizes) of a size distribution
    given by its inverse distribution function."""
    q = [inverse((i + 0.5) / 512) for i in range(512)]  # ascending
    return sum(q) / 512, sum(v * (2 * (511 - i) + 1) for i, v in enumerate(q)) / 512 ** 2


def work(case):
    """Each input read once and each output written once; flops: one probe per
    element of the smaller set of every pair, or the two operations per value
    and pair of the incidence product."""
    kind = case["kind"]
    if kind in ("sisi_call", "sisi", "host"):
        na, nb = case["na"], case["nb"]
        common = na / 5 if kind == "sisi" and nb > 64 * na else min(na, nb) / case["gap"]
        searched = kind != "host" and max(na, nb) > 64 * min(na, nb)
        # a search cannot do without one 32-byte sector of the larger set per element
        read = 4 * min(na, nb) + min(4 * max(na, nb), 32 * min(na, nb)) if searched else 4 * (na + nb)
        return {"bytes": read + (4 * common if case.get("out", True) else 0) + 8, "flops": min(na, nb)}
    if kind == "misi":
        k = case["k"]
        lo, hi = 16.0 ** -0.1, float(case["n_max"]) ** -0.1
        mean, smaller = _mean_sizes(lambda u: (lo + u * (hi - lo)) ** -10.0)
        pairs = (k // 2) * (k - k // 2) if case["cross"] else k * (k - 1) // 2
        return {"bytes": 4 * k * mean + 8 * k + 4 * pairs, "flops": pairs * smaller}
    if kind == "dense":
        k, pairs = case["k"], case["k"] * (case["k"] - 1) // 2
        return {"bytes": 4 * k * case["values"] * case["p"] + 8 * k + 4 * pairs, "flops": 2.0 * pairs * case["values"]}
    mean, smaller = _mean_sizes(lambda u: case["n_min"] * (case["n_max"] / case["n_min"]) ** u)
    # every set that is in a pair is read once
    read = min(case["k"], 2 * case["npairs"]) * mean
    return {"bytes": 4 * read + 8 * case["k"] + 12 * case["npairs"], "flops": case["npairs"] * smaller}


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    """Plain torch on the same inputs, where that is quick."""
    kind = case["kind"]
    if kind in ("sisi_call", "sisi", "host"):
        if max(case["na"], case["nb"]) > 1 << 24:
            return None
        a, b = _pair(case, seed)
        c = a[torch.isin(a, b)]
        if kind != "sisi":
            return c.numel(), c
        out = torch.zeros(min(a.numel(), b.numel()), dtype=torch.int32, device="cuda")
        out[:c.numel()] = c
        return [torch.tensor([c.numel()]), out if case["out"] else None]
    if kind == "dense" and case["k"] <= 4096:
        el, off = generate.bernoulli(seed, case["k"], case["values"], case["p"])
        off = torch.from_numpy(off).cuda()
        of = torch.repeat_interleave(torch.arange(case["k"], device="cuda"), off.diff())
        m = torch.zeros(case["k"], case["values"], dtype=torch.float64, device="cuda")
        m[of, torch.from_numpy(el.view("int32")).cuda().long()] = 1.0
        i, j = torch.triu_indices(case["k"], case["k"], 1, device="cuda")
        return (m @ m.T)[i, j].round().int()
    return None
