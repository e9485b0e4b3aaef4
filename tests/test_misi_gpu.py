"""All-pairs counts (MISI) on the GPU, techniques ip / obs / hi / bitmap: every
count equal to the oracle's, for whole collections (triangular order) and for
the reference's tile pairs (triangular self-join tiles, quadratic cross tiles
with the partition as row stride)."""
import numpy as np
import pytest

import oracle
from conftest import golden_path
from set_intersection_b200 import dataset as fmt
from set_intersection_b200 import tiling

pytestmark = pytest.mark.gpu

TECHS = ["ip", "obs", "hi", "bitmap", "auto"]


def collection(elements, offsets, universe):
    import torch
    from set_intersection_b200 import api
    el = torch.from_numpy(np.ascontiguousarray(elements, dtype=np.uint32).view(np.int32)).cuda()
    off = torch.from_numpy(np.ascontiguousarray(offsets, dtype=np.int64)).cuda()
    return api.Collection(el, off, universe)


def run(col, tech, a_range=None, b_range=None, stride=None, ws=None):
    from set_intersection_b200 import api
    return api.misi(col, tech, a_range, b_range, stride, workspace=ws).cpu().numpy().view(np.uint32)


def from_sets(sets, universe=None):
    ds = fmt.from_sets(sets, universe=universe)
    return ds, collection(ds.elements, ds.offsets, ds.universe)


@pytest.mark.parametrize("tech", TECHS)
@pytest.mark.parametrize("name", ["misi_mixed", "misi_onebased"])
def test_golden_datasets(cuda, tech, name):
    """Every pair of the golden datasets equals the reference's result file."""
    ds = fmt.read_dataset(golden_path(f"{name}.bin"))
    got = run(collection(ds.elements, ds.offsets, ds.universe), tech)
    want = fmt.parse_result(golden_path(f"{name}.std.txt"), ds.cardinality)
    np.testing.assert_array_equal(got, want.astype(np.uint32))


@pytest.mark.parametrize("tech", TECHS)
@pytest.mark.parametrize("k,n_max,universe,seed", [
    (2, 100, 1000, 1), (3, 5000, 1 << 16, 2), (40, 3000, 1 << 14, 3), (300, 5000, 1 << 16, 4),
    (257, 40000, 1 << 20, 5), (1000, 2000, 1 << 12, 6),
])
def test_random_powerlaw(cuda, tech, k, n_max, universe, seed):
    from set_intersection_b200 import generate
    el, off = generate.powerlaw(seed, k, 1, n_max, 1.1, universe, 0.8)
    want = oracle.all_pairs(el, off, k, universe, "std")
    np.testing.assert_array_equal(run(collection(el, off, universe), tech), want)


@pytest.mark.parametrize("tech", TECHS)
def test_large_sets_processed_in_chunks(cuda, tech):
    """Sets larger than one shared-memory structure (> 16384 elements, value
    span > 2^20) against each other and against small sets; partners split
    between work items and warp slices."""
    rng = np.random.default_rng(11)
    sets = [np.sort(rng.choice(1 << 26, size=n, replace=False)).astype(np.uint32)
            for n in (100000, 60000, 40000, 20000, 9000, 8193, 8192, 5000, 100, 1)]
    shared = np.sort(rng.choice(1 << 26, size=30000, replace=False)).astype(np.uint32)
    sets += [np.union1d(s, shared).astype(np.uint32) for s in sets[:4]]
    sets.append(np.arange(0, 1 << 26, 7, dtype=np.uint32)[:200000])
    ds, col = from_sets(sets)
    want = oracle.all_pairs(ds.elements, ds.offsets, ds.cardinality, ds.universe, "std")
    np.testing.assert_array_equal(run(col, tech), want)


@pytest.mark.parametrize("tech", TECHS)
def test_edge_sets(cuda, tech):
    """Empty sets, identical sets, subsets, the values 0 and 0xffffffff."""
    top = np.uint32(0xffffffff)
    base = np.arange(0, 3000, 3, dtype=np.uint32)
    sets = [np.zeros(0, np.uint32), base, base.copy(), base[::2].copy(), np.zeros(0, np.uint32),
            np.array([0, top], np.uint32), np.array([top], np.uint32), np.array([0], np.uint32),
            np.concatenate([base, [top]]).astype(np.uint32), np.arange(1, 3000, 3, dtype=np.uint32)]
    ds, col = from_sets(sets)
    want = oracle.all_pairs(ds.elements, ds.offsets, ds.cardinality, ds.universe, "std")
    np.testing.assert_array_equal(run(col, tech), want)
    for k in (0, 1):
        ds, col = from_sets(sets[:k], universe=10)
        assert run(col, tech).size == 0


@pytest.mark.parametrize("tech", TECHS)
@pytest.mark.parametrize("partition", [7, 64, 230])
def test_tile_pairs_match_reference_layout(cuda, tech, partition):
    """The reference's runs (include/util.hpp:40-52): each tile pair's counts,
    triangular (self) or quadratic (cross) with row stride = partition."""
    from set_intersection_b200 import api, generate
    k = 230
    el, off = generate.powerlaw(21, k, 1, 4000, 1.1, 1 << 15, 0.8)
    full = oracle.all_pairs(el, off, k, 1 << 15, "std")
    col = collection(el, off, 1 << 15)
    ws = api.Workspace()
    for A, B in tiling.find_tile_pairs(k, partition):
        got = run(col, tech, (A.start, A.end), (B.start, B.end), partition, ws)
        self_join = A.id == B.id
        for a in range(A.start, A.end):
            bs = range(a + 1, B.end) if self_join else range(B.start, B.end)
            for b in bs:
                idx = (tiling.triangular_index(partition, a - A.start, b - A.start) if self_join
                       else tiling.quadratic_index(partition, a - A.start, b - B.start))
                assert got[idx] == full[tiling.triangular_index(k, a, b)], (A, B, a, b)


@pytest.mark.parametrize("tech", TECHS)
def test_cross_tile_with_uneven_ranges(cuda, tech):
    from set_intersection_b200 import generate
    k = 500
    el, off = generate.powerlaw(31, k, 1, 20000, 1.1, 1 << 18, 0.8)
    full = oracle.all_pairs(el, off, k, 1 << 18, "std")
    col = collection(el, off, 1 << 18)
    for (a0, a1), (b0, b1), stride in [((0, 123), (300, 500), 200), ((450, 500), (0, 77), 77),
                                        ((10, 11), (11, 500), 489)]:
        got = run(col, tech, (a0, a1), (b0, b1), stride)
        for a in range(a0, a1):
            for b in range(b0, b1):
                want = full[tiling.triangular_index(k, min(a, b), max(a, b))]
                assert got[(a - a0) * stride + (b - b0)] == want


@pytest.mark.slow
def test_powerlaw_config_8192_sets(cuda):
    """The full power-law configuration (8192 sets, sizes ~ n^-1.1 on [16, 65536],
    Zipf(0.8) values over [1, 2^20]): the four techniques agree on all 33.5M
    counts, and every count equals the oracle's (its std::set_intersection
    over every pair, OpenMP over all host cores)."""
    import os
    from set_intersection_b200 import api, generate
    el, off = generate.misi_powerlaw()
    k = off.size - 1
    col = collection(el, off, 1 << 20)
    ws = api.Workspace()
    ref = run(col, "bitmap", ws=ws)
    for tech in ("hi", "obs", "ip"):
        assert np.array_equal(run(col, tech, ws=ws), ref), tech
    want = oracle.all_pairs(el, off, k, 1 << 20, "std", threads=os.cpu_count() or 1)
    assert want.size == k * (k - 1) // 2
    np.testing.assert_array_equal(ref, want)

@pytest.mark.parametrize("k", [2, 31, 255, 256, 257, 511, 513])
@pytest.mark.parametrize("sizes", ["equal", "mixed", "tiny"])
def test_plan_orders_ties_and_tiles(cuda, k, sizes):
    """The plan's ranks at the edges of its 256-set tiles: sets of equal sizes,
    empty sets, self-join tiles and cross tiles cut at and off tile edges."""
    rng = np.random.default_rng(k)
    n = {"equal": np.full(k, 20), "mixed": rng.integers(0, 60, k), "tiny": rng.integers(0, 3, k)}[sizes]
    sets = [np.sort(rng.choice(500, size=s, replace=False)).astype(np.uint32) for s in n]
    ds, col = from_sets(sets, universe=500)
    want = oracle.all_pairs(ds.elements, ds.offsets, k, 500, "std")
    full = np.zeros((k, k), np.uint32)
    full[np.triu_indices(k, 1)] = want
    for tech in ("bitmap", "hi"):
        np.testing.assert_array_equal(run(col, tech), want)
        for h in sorted({1, k // 2, min(256, k - 1), k - 1}):
            np.testing.assert_array_equal(run(col, tech, (0, h), (h, k)).reshape(h, k - h), full[:h, h:])


@pytest.mark.parametrize("rows", [16384, 16385])
def test_plan_of_the_most_ranked_sets(cuda, rows):
    """A cross tile of one set against many, at and past the ranked plan's limit."""
    rng = np.random.default_rng(rows)
    sets = [np.arange(0, 300, 2, dtype=np.uint32)]
    sets += [np.unique(rng.integers(0, 300, 1 + i % 7)).astype(np.uint32) for i in range(rows - 1)]
    ds, col = from_sets(sets, universe=300)
    want = np.array([np.count_nonzero(s % 2 == 0) for s in sets[1:]], np.uint32)
    for tech in ("bitmap", "obs"):
        np.testing.assert_array_equal(run(col, tech, (0, 1), (1, rows)), want)


@pytest.mark.parametrize("k,span", [
    (32, 1000), (128, 1), (129, (1 << 21) + 30), (256, 4095), (257, (1 << 20) + 14), (257, (1 << 20) + 15),
    (300, (1 << 21) + 30), (300, (1 << 21) + 31), (512, 40000), (513, 100), (600, (1 << 22) + 62),
    (600, (1 << 22) + 63), (1100, 70000),
])
def test_value_matrix_edges(cuda, k, span):
    """The bitmap technique's value-major matrix: row counts at the edges of
    its entries and groups, value spans at the limits of each entry width (past
    the last the probe kernel counts), values up to 2^32 - 1, partners longer
    than a slice; self-join, cross tiles with few and many rows, a replayed graph."""
    import torch
    from set_intersection_b200 import api
    rng = np.random.default_rng(k * 31 + span % 1000)
    base = (1 << 32) - 1 - span
    sizes = np.minimum(rng.integers(0, 40, k) * rng.integers(1, 12, k), span // 2 + 1)
    sizes[:3] = [min(span // 3 + 1, 9001), 0, min(span // 2 + 1, 4097)]
    sets = [np.unique(rng.integers(0, span + 1, n)) if n else np.zeros(0, np.int64) for n in sizes]
    sets[0] = np.union1d(sets[0], [0, span])  # the span is exact
    sets = [(s + base).astype(np.uint32) for s in sets]
    ds, col = from_sets(sets)
    want = oracle.all_pairs(ds.elements, ds.offsets, k, ds.universe, "std")
    ws = api.Workspace()
    np.testing.assert_array_equal(run(col, "bitmap", ws=ws), want)
    full = np.zeros((k, k), np.uint32)
    full[np.triu_indices(k, 1)] = want
    for h in (1, k // 2):
        np.testing.assert_array_equal(run(col, "auto", (0, h), (h, k), ws=ws).reshape(h, k - h), full[:h, h:])
    counts = torch.zeros(want.size, dtype=torch.int32, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        api.misi_into(col, counts, "bitmap", workspace=ws)
    for _ in range(2):
        counts.fill_(7)
        g.replay()
        np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint32), want)


def test_cross_tile_with_many_groups_on_both_sides(cuda):
    """Rows on both sides (more than eight 512-row groups each)."""
    from set_intersection_b200 import api, generate
    k, h = 9000, 4500
    el, off = generate.powerlaw(41, k, 1, 300, 1.1, 1 << 14, 0.8)
    col = collection(el, off, 1 << 14)
    ws = api.Workspace()
    got, want = run(col, "bitmap", (0, h), (h, k), ws=ws), run(col, "hi", (0, h), (h, k), ws=ws)
    np.testing.assert_array_equal(got, want)
    rows = np.random.default_rng(1).integers(0, h, 50)
    ref = oracle.pairs(el, off, k, np.array([(a, h + b) for a in rows for b in range(0, k - h, 97)], np.uint32))
    np.testing.assert_array_equal(got.reshape(h, k - h)[rows][:, ::97].ravel(), ref)


@pytest.mark.parametrize("k,n_max,span", [
    (32, 300, 1000), (128, 400, 1 << 31), (129, 3000, 5000), (257, 9000, (1 << 20) + 7), (300, 5000, 1 << 22),
    (513, 70, 1 << 24), (1100, 600, 1 << 16),
])
def test_hash_matrix_edges(cuda, k, n_max, span):
    """Technique hi's matrix: row counts at the edges of its entries and
    groups, tables bounded by the elements and by the span, the value that
    marks empty slots, partners longer than a slice; cross tiles; a replayed graph."""
    import torch
    from set_intersection_b200 import api
    rng = np.random.default_rng(k)
    sizes = rng.integers(0, n_max + 1, k)
    sizes[:3] = [n_max, 0, max(1, n_max - 1)]
    common = rng.integers(0, span, 50)
    sets = [np.unique(np.concatenate([rng.integers(0, span, n), common[:n]])) for n in sizes]
    sets = [np.union1d(s, [span]) if i % 3 == 0 else s for i, s in enumerate(sets)]
    sets = [(s + ((1 << 32) - 1 - span)).astype(np.uint32) for s in sets]
    ds, col = from_sets(sets)
    want = oracle.all_pairs(ds.elements, ds.offsets, k, ds.universe, "std")
    ws = api.Workspace()
    np.testing.assert_array_equal(run(col, "hi", ws=ws), want)
    full = np.zeros((k, k), np.uint32)
    full[np.triu_indices(k, 1)] = want
    for h in (1, k // 2):
        np.testing.assert_array_equal(run(col, "hi", (0, h), (h, k), ws=ws).reshape(h, k - h), full[:h, h:])
    counts = torch.zeros(want.size, dtype=torch.int32, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        api.misi_into(col, counts, "hi", workspace=ws)
    for _ in range(2):
        counts.fill_(7)
        g.replay()
        np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("big", [0, 1 << 20, (1 << 20) + 5])
def test_hash_groups_that_fill_the_slots(cuda, big):
    """Sets over the whole 32-bit range, so many elements that a group's rows
    end where half of the slots is full and the table is emptied between
    groups; a set of half the slots, and one larger, which the probe kernel counts."""
    rng = np.random.default_rng(big)
    sets = [np.unique(rng.integers(0, 1 << 32, 60000, dtype=np.uint64)) for _ in range(48)]
    sets = [np.union1d(s, sets[0][i:500 + i]) for i, s in enumerate(sets)]
    sets = [np.union1d(s, [0xffffffff]) if i % 2 else s for i, s in enumerate(sets)]
    if big:
        s = np.unique(rng.integers(0, 1 << 32, big + 5000, dtype=np.uint64))
        sets.append(s[:big])
    ds, col = from_sets([s.astype(np.uint32) for s in sets])
    want = oracle.all_pairs(ds.elements, ds.offsets, ds.cardinality, ds.universe, "std")
    np.testing.assert_array_equal(run(col, "hi"), want)


@pytest.mark.parametrize("tech", ["obs", "ip"])
@pytest.mark.parametrize("span", [0, 1, 16383, 16384, 1 << 20, (1 << 32) - 1])
def test_bucket_search_edges(cuda, tech, span):
    """Buckets of the staged chunk: spans at the bucket limits, sets of one
    bucket and of two far clusters, chunks of exactly 16384 elements and one
    more, values below, between and above the chunk's."""
    rng = np.random.default_rng(span % 1000 + 1)
    base = min(5, (1 << 32) - 1 - span)
    n = [1, 2, 100, 16384, 16385, 40000]
    sets = [np.unique(rng.integers(base, base + span + 1, m, dtype=np.uint64)) for m in n]
    full = np.arange(base, base + min(span + 1, 40000), dtype=np.uint64)
    sets += [full, full[:16384], full[:16385], np.array([base, base + span], np.uint64)]
    sets += [np.union1d(full[:9000], base + span - np.arange(min(span + 1, 9000), dtype=np.uint64)),
             np.array([0], np.uint64), np.array([(1 << 32) - 1], np.uint64), np.zeros(0, np.uint64)]
    ds, col = from_sets([s.astype(np.uint32) for s in sets])
    want = oracle.all_pairs(ds.elements, ds.offsets, ds.cardinality, ds.universe, "std")
    np.testing.assert_array_equal(run(col, tech), want)


@pytest.mark.parametrize("n_a,n_b", [(1, 30), (17, 16), (33, 62), (95, 130), (300, 213)])
def test_plan_totals_of_split_warps(cuda, n_a, n_b):
    """A warp of the plan holds sets of both sides, empty ones, and lanes past
    the last set: the totals and the range of the values still cover every set
    (bitmap and hi leave out values outside the range, obs has work items for the
    totals alone)."""
    rng = np.random.default_rng(n_a)
    k = n_a + n_b
    sets = [np.unique(rng.integers(1 << 19, (1 << 19) + 4000, rng.integers(0, 200))) for _ in range(k)]
    for i in range(0, k, 5):
        sets[i] = sets[i][:0]
    sets[n_a - 1] = np.union1d(sets[n_a - 1], [3, 9, 1 << 20])       # the smallest and the largest value
    sets[k - 1] = np.union1d(sets[k - 1], [5, 9, (1 << 20) + 31])    # lie in single lanes
    ds, col = from_sets([s.astype(np.uint32) for s in sets])
    want = np.array([[len(np.intersect1d(sets[a], sets[n_a + b])) for b in range(n_b)] for a in range(n_a)])
    for tech in ("bitmap", "hi", "obs"):
        np.testing.assert_array_equal(run(col, tech, (0, n_a), (n_a, k)).reshape(n_a, n_b), want)


@pytest.mark.parametrize("tech,k,n_a,span,size", [
    ("bitmap", 128, 0, 1 << 16, 65), ("bitmap", 129, 0, 1 << 16, 6), ("bitmap", 768, 0, 1 << 20, 6),
    ("bitmap", 769, 0, 1 << 12, 2), ("bitmap", 1025, 0, 1 << 13, 1), ("bitmap", 1025, 0, (1 << 21) + 9, 2),
    ("bitmap", 2049, 0, (1 << 22) - 9, 2), ("bitmap", 700, 100, 1 << 14, 4), ("bitmap", 16400, 40, 1 << 15, 1),
    ("hi", 127, 0, 1 << 26, 512), ("hi", 47, 0, 1 << 26, 2048), ("hi", 600, 0, 1 << 14, 36), ("hi", 1024, 0, 1 << 22, 64),
    ("hi", 1025, 0, 1 << 14, 23), ("hi", 2049, 0, 1 << 30, 8), ("hi", 4097, 0, 1 << 12, 5), ("hi", 800, 300, 1 << 12, 8),
    ("hi", 16400, 40, 1 << 12, 5),
])
def test_matrix_or_probes(cuda, tech, k, n_a, span, size):
    """Sets whose pairs take as many probes as the rule between the matrix and the
    probe kernel allows, and one more: one side against itself, and (n_a) two
    sides; rows sorted as well as ranked."""
    rng = np.random.default_rng(k + size)
    for n in (size, size + 1):
        sets = [np.sort(rng.choice(span, n, replace=False)) if span < 1 << 16 else
                np.unique(rng.integers(0, span, 2 * n + 8))[:n] for _ in range(k)]
        ds, col = from_sets([s.astype(np.uint32) for s in sets], span)
        if n_a:
            got = run(col, tech, (0, n_a), (n_a, k))
            pairs = np.stack(np.meshgrid(np.arange(n_a), np.arange(n_a, k), indexing="ij"), -1).reshape(-1, 2)
            want = oracle.pairs(ds.elements, ds.offsets, k, pairs.astype(np.uint32))
        else:
            got = run(col, tech)
            want = oracle.all_pairs(ds.elements, ds.offsets, k, ds.universe, "std")
        np.testing.assert_array_equal(got, want)
