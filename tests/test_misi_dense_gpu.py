"""All-pairs counts of dense collections on the GPU: the tensor-core incidence
product (INT8 and FP8-e4m3) and the plain bitmap AND-popcount kernel, every
count equal to the oracle's (zero error)."""
import numpy as np
import pytest

import oracle
from conftest import golden_path
from set_intersection_b200 import dataset as fmt

pytestmark = pytest.mark.gpu

VARIANTS = [("mm", "int8"), ("mm", "fp8"), ("bitmap_naive", "int8")]


def collection(elements, offsets, universe):
    import torch
    from set_intersection_b200 import api
    el = torch.from_numpy(np.ascontiguousarray(elements, dtype=np.uint32).view(np.int32)).cuda()
    off = torch.from_numpy(np.ascontiguousarray(offsets, dtype=np.int64)).cuda()
    return api.Collection(el, off, universe)


def counts(col, tech, dtype, ws=None):
    from set_intersection_b200 import api
    return api.misi_dense(col, tech, dtype, workspace=ws).cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("tech,dtype", VARIANTS)
@pytest.mark.parametrize("name", ["misi_mixed", "misi_onebased"])
def test_golden_datasets(cuda, tech, dtype, name):
    """Counts of every pair equal the reference's result files (std and
    boost bitset executables)."""
    ds = fmt.read_dataset(golden_path(f"{name}.bin"))
    col = collection(ds.elements, ds.offsets, ds.universe)
    got = counts(col, tech, dtype)
    for ref in ("std", "bitset"):
        want = fmt.parse_result(golden_path(f"{name}.{ref}.txt"), ds.cardinality)
        np.testing.assert_array_equal(got, want.astype(np.uint32))


@pytest.mark.parametrize("tech,dtype", VARIANTS)
@pytest.mark.parametrize("k,n_values,p", [
    (2, 100, 0.5), (3, 1, 1.0), (5, 7, 0.5), (127, 129, 0.3), (128, 128, 0.5), (129, 300, 0.2),
    (255, 1000, 0.1), (256, 4096, 0.05), (257, 5000, 0.1), (300, 4097, 0.3), (513, 200, 0.9),
    (1000, 20000, 0.05), (2100, 3000, 0.02),
])
def test_random_bernoulli(cuda, tech, dtype, k, n_values, p):
    from set_intersection_b200 import generate
    el, off = generate.bernoulli(k * 7 + n_values, k, n_values, p)
    want = oracle.all_pairs(el, off, k, n_values - 1, "bitset")
    got = counts(collection(el, off, n_values - 1), tech, dtype)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("tech,dtype", VARIANTS)
def test_empty_full_and_tiny(cuda, tech, dtype):
    """Empty sets, sets holding the whole universe, one- and zero-pair cases."""
    rng = np.random.default_rng(3)
    U = 777
    sets = [np.arange(U, dtype=np.uint32), np.zeros(0, np.uint32), np.arange(U, dtype=np.uint32),
            np.array([0], np.uint32), np.array([U - 1], np.uint32)]
    sets += [np.sort(rng.choice(U, size=rng.integers(0, U), replace=False)).astype(np.uint32) for _ in range(200)]
    ds = fmt.from_sets(sets, universe=U - 1)
    want = oracle.all_pairs(ds.elements, ds.offsets, ds.cardinality, ds.universe, "std")
    got = counts(collection(ds.elements, ds.offsets, ds.universe), tech, dtype)
    np.testing.assert_array_equal(got, want)
    for k in (0, 1):
        ds = fmt.from_sets(sets[:k], universe=U - 1)
        assert counts(collection(ds.elements, ds.offsets, U - 1), tech, dtype).size == 0


@pytest.mark.parametrize("tech,dtype", VARIANTS)
def test_value_above_universe_is_reported(cuda, tech, dtype):
    from set_intersection_b200._lib import SiError, Status
    el = np.array([1, 5, 9, 2, 40], np.uint32)
    off = np.array([0, 3, 5], np.int64)
    with pytest.raises(SiError) as e:
        counts(collection(el, off, 30), tech, dtype)
    assert e.value.status == Status.INVALID_INPUT


@pytest.mark.parametrize("tech,dtype", VARIANTS)
def test_workspace_reuse(cuda, tech, dtype):
    from set_intersection_b200 import api, generate
    ws = api.Workspace()
    for seed, (k, n, p) in enumerate([(700, 9000, 0.05), (40, 100, 0.5), (1500, 2000, 0.1)]):
        el, off = generate.bernoulli(100 + seed, k, n, p)
        want = oracle.all_pairs(el, off, k, n - 1, "std")
        np.testing.assert_array_equal(counts(collection(el, off, n - 1), tech, dtype, ws), want)


@pytest.mark.slow
def test_dense_config_16384_sets(cuda):
    """The full dense configuration (16384 sets over 65536 values,
    Bernoulli(0.05)): the INT8 and FP8 tensor-core products and the plain
    popcount kernel agree on all 134M counts, and every count equals the
    oracle's (its bitset probe over every pair, the boost_bitset technique,
    OpenMP over all host cores)."""
    import os
    from set_intersection_b200 import generate
    el, off = generate.misi_dense()
    k = off.size - 1
    col = collection(el, off, 65535)
    c_int8 = counts(col, "mm", "int8")
    c_fp8 = counts(col, "mm", "fp8")
    assert np.array_equal(c_int8, c_fp8)
    c_naive = counts(col, "bitmap_naive", "int8")
    assert np.array_equal(c_int8, c_naive)
    want = oracle.all_pairs(el, off, k, 65535, "bitset", threads=os.cpu_count() or 1)
    assert want.size == k * (k - 1) // 2
    np.testing.assert_array_equal(c_int8, want)

@pytest.mark.parametrize("dtype", ["int8", "fp8"])
@pytest.mark.parametrize("k,values", [
    (2, 1), (129, 127), (255, 128), (256, 4096), (257, 4097), (511, 300000), (513, 2049), (769, 5000), (1025, 2048),
    (3000, 3000), (4300, 65536),
])
def test_paired_tiles_edges(cuda, k, values, dtype):
    """Set counts at the edges of the 256-row panels, one to many K stages,
    tiles cut along K and whole, the narrow tile and (4300 sets over 65536
    values) the wide one; some sets empty, some full, against the popcount
    kernel, and the oracle on sampled pairs."""
    from set_intersection_b200 import generate
    el, off = generate.bernoulli(k + values, k, values, min(0.3, 3e6 / (k * values)))
    sets = [el[off[i]:off[i + 1]] for i in range(k)]
    for i in (0, k // 2, k - 1):
        sets[i] = np.arange(values, dtype=np.uint32)
    if k > 2:
        sets[1] = np.zeros(0, np.uint32)
    ds = fmt.from_sets(sets, universe=values - 1)
    col = collection(ds.elements, ds.offsets, values - 1)
    got = counts(col, "mm", dtype)
    np.testing.assert_array_equal(got, counts(col, "bitmap_naive", "int8"))
    rng = np.random.default_rng(k)
    a = rng.integers(0, k - 1, 200)
    b = rng.integers(a + 1, k)
    pairs = np.stack([a, b], 1).astype(np.uint32)
    tri = k * (k - 1) // 2 - (k - a) * (k - a - 1) // 2 + b - a - 1
    np.testing.assert_array_equal(got[tri], oracle.pairs(ds.elements, ds.offsets, k, pairs))


@pytest.mark.parametrize("dtype", ["int8", "fp8"])
def test_dense_call_in_a_graph(cuda, dtype):
    import torch
    from set_intersection_b200 import api, generate
    k, n = 700, 6000
    el, off = generate.bernoulli(7, k, n, 0.1)
    want = oracle.all_pairs(el, off, k, n - 1, "std")
    col, ws = collection(el, off, n - 1), api.Workspace()
    out = torch.zeros(want.size, dtype=torch.int32, device="cuda")
    api.misi_dense_into(col, out, "mm", dtype, ws)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        api.misi_dense_into(col, out, "mm", dtype, ws)
    for _ in range(2):
        out.fill_(3)
        g.replay()
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), want)


def wide_tile(k, values, sms):
    """Whether the tensor-core path takes its 256 x 512 tile: the cheaper of the
    two schedules, in units of a stage's MMAs."""
    pairs, panels, stages = sms // 2, -(-k // 256), -(-values // 128)
    cost = {}
    for n in (1, 2):
        columns = -(-panels // n)
        tiles = sum(columns - i // n for i in range(panels))
        whole = tiles // pairs * pairs
        left = tiles - whole
        cuts = max(1, min(pairs // left, stages // 16)) if left else 1
        stage, out = (1.25 * stages, 18) if n == 1 else (2.1 * stages, 60)
        cost[n] = whole // pairs * (stage + out)
        if left:
            cost[n] += stage / cuts + (1.5 * out if cuts > 1 else out)
    return cost[2] < cost[1]


@pytest.mark.parametrize("dtype", ["int8", "fp8"])
@pytest.mark.parametrize("k,values", [(1400, 200001), (2050, 65536), (3601, 10001), (4609, 40010)])
def test_wide_tile_edges(cuda, k, values, dtype):
    """The 256 x 512 tile where the sets fill neither a row panel nor a column
    panel: an odd number of row panels, whose last column panel lies half past
    the matrix, tiles cut along K in two and six parts, whole tiles, and both; some
    sets empty, some full, against the popcount kernel and the oracle on sampled
    pairs.  (4300 sets over 65536 values take the narrow tile.)"""
    import torch
    assert wide_tile(k, values, torch.cuda.get_device_properties(0).multi_processor_count)
    assert not wide_tile(4300, 65536, 148)
    test_paired_tiles_edges(cuda, k, values, dtype)
