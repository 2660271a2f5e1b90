"""Which count a graph takes: the packed rows, the plain-id tables or one launch.
The packed count is five launches; the plain-id count of more than 4096 rows at
least seven (its scan alone takes three).  Every count is also checked against
the oracle, on either side of each rule."""
import ctypes

import numpy as np
import pytest

import oracle
import trianglecount_gb300 as tc
from trianglecount_gb300 import generators as gen

pytestmark = pytest.mark.gpu

PACKED = 5


def csr(n, u, v):
    key = np.unique(np.asarray(u, np.int64) * n + np.asarray(v, np.int64))
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(key // n, minlength=n), out=rp[1:])
    return rp.astype(np.int32), (key % n).astype(np.int32)


def by_rank(n, src, dst, rank):
    """Every edge from its lower-ranked end to its higher-ranked one."""
    keep = src != dst
    s, d = src[keep], dst[keep]
    swap = rank[s] > rank[d]
    return csr(n, np.where(swap, d, s), np.where(swap, s, d))


def by_degree(n, src, dst):
    deg = np.bincount(np.concatenate((src, dst)), minlength=n).astype(np.int64)
    return by_rank(n, src, dst, deg * n + np.arange(n))


def with_clique(src, dst, size):
    i, j = np.triu_indices(size, 1)
    return np.concatenate((src, i + 5)), np.concatenate((dst, j + 5))


def launches_of(ctx, rp, col, n_roots=None):
    """Launches of one count; the count, the per-root counts and a batch against the oracle."""
    want, pr = oracle.count(rp, col, n_roots=n_roots, per_root=True)
    g = ctx.upload(rp, col, n_roots=n_roots)
    got, st = ctx.count(g, stats=True)
    assert got == want
    assert per_root_and_total(ctx, g, pr) == want
    assert list(ctx.batch([g]).run()) == [want]
    return st["launches"]


def per_root_and_total(ctx, g, want):
    """Checks the per-root counts; the total that the call gives beside them."""
    got, total = np.full(len(want), 7, np.uint64), ctypes.c_uint64()
    st = tc.lib().tc_count_per_root(ctx.handle, g.handle, got.ctypes.data_as(ctypes.c_void_p), ctypes.byref(total))
    assert st == 0 and np.array_equal(got, want)
    return total.value


@pytest.mark.parametrize("self_loops", [False, True])
def test_total_beside_the_per_root_counts(ctx, self_loops):
    """Flat rows of up to 4 and 8, one launch, packed and plain-id tables, all rows and a prefix of them as roots."""
    r = np.random.default_rng(3)
    for n, most in ((5000, 4), (5000, 8), (5000, 40), (60_000, 60), (100_000, 20)):
        u = np.repeat(np.arange(n), r.integers(0, most + 1, n))
        v = r.integers(0, n, len(u)) % max(1, n // 8) if most < 20 else r.integers(0, n, len(u))
        if not self_loops:
            u, v = u[u != v], v[u != v]
        elif most > 4:
            u, v = np.concatenate((u, np.arange(0, n, 7))), np.concatenate((v, np.arange(0, n, 7)))
        rp, col = csr(n, u, v)
        for n_roots in (None, n // 3):
            launches_of(ctx, rp, col, n_roots)


def test_one_clique_does_not_make_a_graph_skewed(ctx):
    """A few long rows in a graph without hubs: the plain-id tables, as without them."""
    n = 100_000
    src, dst = gen.er(n, 16.0, seed=3)
    assert launches_of(ctx, *by_degree(n, src, dst)) > PACKED
    src, dst = with_clique(src, dst, 90)
    rp, col = by_degree(n, src, dst)
    assert np.diff(rp).max() * n > 5 * len(col)
    assert launches_of(ctx, rp, col) > PACKED
    for tie in ("reference", "id_asc"):  # built on the device: whole, and as parts
        g = ctx.graph_from_edges(src, dst, tie=tie)
        assert ctx.count(g, stats=True)[1]["launches"] > PACKED
    src, dst = gen.er(300_000, 16.0, seed=4)
    ug = ctx.ugraph_from_edges(*with_clique(src, dst, 90))
    part = gen.parts_random(ug.info()[0], 2)
    for mode in ("reference", "count"):
        for p in ctx.halo_extract(ug, part, 2, mode=mode):
            assert p.n_rows > 61440 and ctx.count(p, stats=True)[1]["launches"] > PACKED


@pytest.mark.parametrize("maker", ["rmat17", "rmat19", "chung_lu_8", "chung_lu_64"])
def test_skewed_graphs_count_packed(ctx, maker):
    src, dst = {"rmat17": lambda: gen.rmat(17), "rmat19": lambda: gen.rmat(19),
                "chung_lu_8": lambda: gen.chung_lu(80_000, 8.0, seed=1),
                "chung_lu_64": lambda: gen.chung_lu(80_000, 64.0, seed=1)}[maker]()
    g = ctx.graph_from_edges(src, dst)
    rp, col = g.download()
    assert g.n_rows > 61440
    assert ctx.count(g, stats=True)[1]["launches"] == PACKED
    assert launches_of(ctx, rp, col) == PACKED
    ug = ctx.ugraph_from_edges(src, dst)
    parts = ctx.halo_extract(ug, gen.parts_random(ug.info()[0], 3), 3, mode="count")
    assert [ctx.count(p, stats=True)[1]["launches"] for p in parts] == [PACKED] * 3
    assert sum(ctx.count(p) for p in parts) == oracle.count(rp, col)


@pytest.mark.parametrize("maker", ["chung_lu", "rmat18"])
@pytest.mark.parametrize("order", ["ids", "descending"])
def test_edges_that_do_not_go_by_degree_count_on_plain_ids(ctx, maker, order):
    """Rows of thousands of unpopular ids; alone, and in a launch with as many other edges."""
    n, (src, dst) = (100_000, gen.chung_lu(100_000, 16.0, seed=2)) if maker == "chung_lu" else (1 << 18, gen.rmat(18))
    if order == "ids":
        rank = np.random.default_rng(1).permutation(n)
    else:
        rank = -(np.bincount(np.concatenate((src, dst)), minlength=n).astype(np.int64) * n + np.arange(n))
    rp, col = by_rank(n, src, dst, rank)
    assert launches_of(ctx, rp, col) > PACKED
    ordered = by_degree(n, src, dst)
    assert launches_of(ctx, *ordered) == PACKED
    b = ctx.batch([ctx.upload(rp, col), ctx.upload(*ordered), ctx.upload(*ordered)])
    assert list(b.run()) == [oracle.count(rp, col)] + [oracle.count(*ordered)] * 2
    assert b.stats()["launches"] > PACKED


def test_a_small_share_of_such_a_graph_leaves_a_launch_packed(ctx):
    n = 70_000
    far = by_rank(n, *gen.chung_lu(n, 4.0, seed=2), np.random.default_rng(1).permutation(n))
    rp, col = oracle.pipeline(*gen.rmat(18))[:2]
    assert 16 * len(far[1]) < len(col)
    b = ctx.batch([ctx.upload(*far), ctx.upload(rp, col)])
    assert list(b.run()) == [oracle.count(*far), oracle.count(rp, col)]
    assert b.stats()["launches"] == PACKED


@pytest.mark.parametrize("maker", ["rmat20", "chung_lu"])
def test_a_few_roots_of_a_large_graph_count_on_plain_ids(ctx, maker):
    """The packed count packs every row, whether a root holds it or not."""
    src, dst = gen.rmat(20) if maker == "rmat20" else gen.chung_lu(1_000_000, 16.0, seed=1)
    rp, col, _ = oracle.pipeline(src, dst)
    assert launches_of(ctx, rp, col, 300_000) == PACKED
    for n_roots in (1, 2000):
        assert launches_of(ctx, rp, col, n_roots) > PACKED
    g = ctx.upload(rp.astype(np.uint64), col.astype(np.uint64), n_roots=2000)
    assert ctx.count(g, stats=True)[1]["launches"] > PACKED
    ug = ctx.ugraph_from_edges(src, dst)  # a small part and its halo
    part = np.ones(ug.info()[0], np.int32)
    part[::400] = 0
    small, large = ctx.halo_extract(ug, part, 2)
    whole = oracle.count(rp, col)
    b, st = ctx.count(large, stats=True)
    assert ctx.count(small) + b == whole and st["launches"] == PACKED


def test_few_edges_among_many_rows_count_on_plain_ids(ctx):
    rp, col, _ = oracle.pipeline(*gen.rmat(16))

    def among(n_rows):
        return np.concatenate((rp, np.full(n_rows + 1 - len(rp), rp[-1], np.int32)))

    assert launches_of(ctx, among(2_000_000), col) == PACKED
    assert launches_of(ctx, among(8_000_000), col) > PACKED


@pytest.mark.parametrize("m", [(1 << 18) - 1, 1 << 18, (1 << 18) + 1])
def test_one_launch_up_to_2_to_18_edges(ctx, m):
    rp, col = by_degree(20_000, *gen.er(20_000, 27.0, seed=7))
    rp, col = np.minimum(rp, m).astype(np.int32), col[:m]
    assert len(col) == m and np.diff(rp).max() <= 64
    assert launches_of(ctx, rp, col) == (1 if m <= 1 << 18 else PACKED)
    for n_roots in (1, 31, 4097, 19_999):
        assert launches_of(ctx, rp, col, n_roots) == (1 if m <= 1 << 18 else PACKED)


@pytest.mark.parametrize("d", [33, 63, 64, 65, 128, 500, 2000, 8000])
@pytest.mark.parametrize("n_edges", [12_000, 100_000])
def test_one_launch_only_while_every_row_is_short(ctx, d, n_edges):
    """A row is one warp's work in the single launch, however long it is."""
    n = 20_000
    r = np.random.default_rng(d)
    u, v = r.integers(1, n, n_edges - d), r.integers(1, n, n_edges - d)
    hub = 1 + r.choice(n - 1, d, replace=False)
    rp, col = csr(n, np.concatenate((np.zeros(d, np.int64), u)), np.concatenate((hub, v)))
    assert np.diff(rp).max() == d
    for n_roots in (None, 1, 700):
        assert launches_of(ctx, rp, col, n_roots) == (1 if d <= 64 else PACKED)


@pytest.mark.parametrize("n_rows", [64, 65, 4863, 4864, 4865, 19457, 100_000])
def test_one_launch_windows_of_rows(ctx, n_rows):
    """Two to thirty-two rows per warp, as many as it takes to fill the GPU once."""
    r = np.random.default_rng(n_rows)
    m = min(12 * n_rows, 200_000)
    u, v = r.integers(0, n_rows, m), r.integers(0, n_rows, m)
    hub = r.choice(n_rows, 40, replace=False)  # one row past the flat count's eight
    rp, col = csr(n_rows, np.concatenate((u, np.full(40, n_rows // 2))), np.concatenate((v, hub)))
    assert 8 < np.diff(rp).max() <= 64
    assert launches_of(ctx, rp, col) == 1


def wrapped(ctx, rp, col):
    torch = pytest.importorskip("torch")
    a, b = torch.from_numpy(rp).cuda(), torch.from_numpy(col).cuda()
    torch.cuda.synchronize()
    g = ctx.wrap_device(a.data_ptr(), b.data_ptr(), len(rp) - 1, len(col))
    g.arrays = a, b
    return g


def count_async(ctx, g):
    import torch
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    assert tc.lib().tc_count_async(ctx.handle, g.handle, out.data_ptr()) == 0
    ctx.synchronize()
    return int(out.item())


@pytest.mark.parametrize("asynchronous_first", [False, True])
def test_wrapped_graphs_take_the_count_of_their_rows(ctx, asynchronous_first):
    er = by_degree(100_000, *gen.er(100_000, 16.0, seed=3))
    rmat = oracle.pipeline(*gen.rmat(17))[:2]
    few = by_degree(20_000, *gen.er(20_000, 20.0, seed=7))
    for (rp, col), route in ((er, lambda n: n > PACKED), (rmat, lambda n: n == PACKED), (few, lambda n: n == 1)):
        want, pr = oracle.count(rp, col, per_root=True)
        g = wrapped(ctx, rp, col)
        if asynchronous_first:
            assert [count_async(ctx, g) for _ in range(3)] == [want] * 3
        for _ in range(3):
            got, st = ctx.count(g, stats=True)
            assert got == want and route(st["launches"])
        assert np.array_equal(ctx.count_per_root(g), pr)
        assert [count_async(ctx, g) for _ in range(3)] == [want] * 3
        assert list(ctx.batch([wrapped(ctx, rp, col), g]).run()) == [want, want]


def test_wrapped_arrays_may_be_written_anew(ctx):
    """Short rows first (never the flat count: it could not count the longer ones that follow)."""
    torch = pytest.importorskip("torch")
    n, m = 5000, 9000
    r = np.random.default_rng(1)
    short = csr(n, np.repeat(np.arange(n), 2)[:m], (np.repeat(np.arange(n), 2)[:m] + np.tile([1, 2], m)[:m]) % n)
    u, v = np.repeat(np.arange(30), 300), np.concatenate([r.choice(600, 300, replace=False) for _ in range(30)])
    long = csr(n, u, v)
    assert len(short[1]) == len(long[1]) == m
    for first, then in ((short, long), (long, short)):
        g = wrapped(ctx, *first)
        assert [ctx.count(g) for _ in range(3)] == [oracle.count(*first)] * 3
        g.arrays[0].copy_(torch.from_numpy(then[0]))
        g.arrays[1].copy_(torch.from_numpy(then[1]))
        torch.cuda.synchronize()
        want, pr = oracle.count(*then, per_root=True)
        assert [ctx.count(g) for _ in range(3)] == [want] * 3
        assert np.array_equal(ctx.count_per_root(g), pr)
        assert count_async(ctx, g) == want


def test_a_callers_capture_outlives_the_look_at_the_rows():
    """tc_count_async captured by the caller, then a count that takes another form: the capture still counts."""
    torch = pytest.importorskip("torch")
    rp, col, want = oracle.pipeline(*gen.rmat(17))
    c = tc.Context(0)
    s = torch.cuda.Stream()
    c.set_stream(s.cuda_stream)
    g = wrapped(c, rp, col)
    assert count_async(c, g) == want  # sizes the scratch
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    cg = torch.cuda.CUDAGraph()
    with torch.cuda.graph(cg, stream=s):
        assert tc.lib().tc_count_async(c.handle, g.handle, out.data_ptr()) == 0
    assert c.count(g) == want
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        cg.replay()
        torch.cuda.synchronize()
        assert int(out.item()) == want and c.count(g) == want
    g.free()
    c.close()


@pytest.fixture
def tuned(ctx):
    old = ctx.get_tuning()
    yield ctx
    ctx.set_tuning(old["warp_max_deg"], old["light_max_work"], old["unit_work"], old["long_list"],
                   old["probe_kicks"], old["heavy_bitmap"], 0, old["hash_pairs"], old["flat_max_deg"],
                   old["intersect"])


@pytest.mark.parametrize("n", [61_000, 61_440, 61_441, 62_000])
@pytest.mark.parametrize("deg", [40.0, 100.0])
def test_unskewed_graphs_on_either_side_of_61440_rows(tuned, n, deg):
    """Micro, light and heavy tasks of the plain-id cuckoo tables, whole, as a prefix of roots and batched."""
    rp, col = by_degree(n, *gen.er(n, deg, seed=11))
    for tuning in ({}, {"warp_max_deg": 32, "unit_work": 64}, {"light_max_work": 16}, {"warp_max_deg": 32, "unit_work": 4096}):
        tuned.set_tuning(warp_max_deg=256, light_max_work=8192, unit_work=1 << 20)
        tuned.set_tuning(**tuning)
        for n_roots in (None, 1000, n // 2):
            assert (launches_of(tuned, rp, col, n_roots) > PACKED) == (n > 61_440)
        if n > 61_440 and tuning.get("warp_max_deg") == 32:
            assert tuned.count(tuned.upload(rp, col), stats=True)[1]["heavy_units"] > 0


@pytest.mark.parametrize("more", ["plain", "packed"])
def test_mixed_batches_go_with_most_of_their_edges(tuned, more):
    """Unskewed and skewed graphs and halo parts in one launch, on the tables and packed."""
    er = by_degree(100_000, *gen.er(100_000, 16.0, seed=3))
    src, dst = gen.rmat(16)
    skewed = oracle.pipeline(src, dst)[:2]
    ug = tuned.ugraph_from_edges(src, dst)
    parts = tuned.halo_extract(ug, gen.parts_random(ug.info()[0], 3), 3, mode="count")
    plain = [er] * (5 if more == "plain" else 1)
    graphs = [tuned.upload(*c) for c in plain + [skewed]] + parts
    want = [oracle.count(*c) for c in plain + [skewed]] + [tuned.count(p) for p in parts]
    assert sum(want[-3:]) == want[len(plain)]
    gain = sum(g.nnz for g in graphs) - len(plain) * len(er[1])
    assert (2 * gain >= sum(g.nnz for g in graphs)) == (more == "packed")
    for tuning in ({}, {"warp_max_deg": 32, "unit_work": 64}):
        tuned.set_tuning(**tuning)
        for order in (1, -1):
            b = tuned.batch(graphs[::order])
            assert list(b.run()) == want[::order]
            assert (b.stats()["launches"] == PACKED) == (more == "packed")


def test_many_halo_parts_in_one_launch_stay_packed(ctx):
    """A part's roots hold a thirtieth of its entries at k = 64, and the packed launch is the faster one (1.14 against 1.64 ms)."""
    src, dst = gen.rmat(18)
    ug = ctx.ugraph_from_edges(src, dst)
    for k in (16, 64):
        parts = ctx.halo_extract(ug, gen.parts_random(ug.info()[0], k), k, mode="count")
        b = ctx.batch(parts)
        assert int(b.run().sum()) == oracle.count(*oracle.pipeline(src, dst)[:2])
        assert b.stats()["launches"] == PACKED


@pytest.mark.parametrize("n_graphs, n, deg, packed", [(40, 20, 6, True), (500, 20, 6, False), (3000, 8, 3, False),
                                                      (3000, 60, 8, False), (100, 300, 12, True), (2000, 300, 12, True)])
def test_batches_of_tiny_graphs_count_on_plain_ids(ctx, n_graphs, n, deg, packed):
    r = np.random.default_rng(n)
    some = [csr(n, r.integers(0, n, n * deg), r.integers(0, n, n * deg)) for _ in range(20)]
    up, want = [ctx.upload(*c) for c in some], [oracle.count(*c) for c in some]
    b = ctx.batch([up[i % 20] for i in range(n_graphs)])
    assert list(b.run()) == [want[i % 20] for i in range(n_graphs)]
    assert (b.stats()["launches"] == PACKED) == packed
