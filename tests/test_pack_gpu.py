"""The packed-row count (tc_pack.cu) against the oracle and against the plain-id
tables, at the sizes where its layout changes: row lengths around a window (32),
a piece (128), the warp / block border (512) and a block's hash tile; ids around
the low blocks' end (30,720) and around the last full-width mask (63,488 x 16);
graphs around the one-launch and the sampling bound; edges that follow no
order."""
import numpy as np
import pytest

import oracle
from trianglecount_gb300 import generators as gen

pytestmark = pytest.mark.gpu


def csr(n, edges):
    e = np.unique(np.asarray(edges, np.int64).reshape(-1, 2), axis=0)
    rp = np.zeros(n + 1, np.int64)
    np.add.at(rp, e[:, 0] + 1, 1)
    return np.cumsum(rp).astype(np.int32), e[:, 1].astype(np.int32)


def rows_of_lengths(lengths, n, seed):
    """A CSR whose first rows have the given lengths; their members' rows are short or long at random."""
    r = np.random.default_rng(seed)
    out = []
    for u, d in enumerate(lengths):
        out += [(u, v) for v in r.choice(n, d, replace=False)]
    k = len(lengths)
    for u in range(k, min(n, k + 3000)):
        out += [(u, v) for v in r.choice(n, int(r.integers(0, 40)), replace=False)]
    return csr(n, out)


@pytest.fixture
def chain(ctx):
    """Every graph through the launch sequence (flat_max_deg = 0: no one-kernel count)."""
    old = ctx.get_tuning()
    ctx.set_tuning(flat_max_deg=0)
    yield ctx
    ctx.set_tuning(old["warp_max_deg"], old["light_max_work"], old["unit_work"], old["long_list"],
                   old["probe_kicks"], old["heavy_bitmap"], 0, old["hash_pairs"], old["flat_max_deg"],
                   old["intersect"])


def check(ctx, rp, col, n_roots=None):
    want, pr = oracle.count(rp, col, n_roots=n_roots, per_root=True)
    g = ctx.upload(rp, col, n_roots=n_roots)
    assert ctx.count(g) == want
    assert np.array_equal(ctx.count_per_root(g), pr)
    b = ctx.batch([g, g])
    assert list(b.run()) == [want, want]


@pytest.mark.parametrize("n", [4000, 40000])  # with and without high blocks
@pytest.mark.parametrize("d", [1, 2, 3, 8, 9, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513,
                               1023, 1025, 3500])
def test_row_lengths(chain, n, d):
    rp, col = rows_of_lengths([d, d, 32, d, 2, 33, d], n, d)
    check(chain, rp, col)
    check(chain, rp, col, n_roots=4)


@pytest.mark.parametrize("n", [30719, 30720, 30721, 63488 * 16, 63488 * 16 + 1, 3_000_000])
def test_id_ranges(chain, n):
    """Hubs at both ends of the ids, rows longer than a block's hash tile among them."""
    r = np.random.default_rng(n)
    hubs = np.concatenate((np.arange(20), n - 1 - np.arange(20)))
    edges = [(h, v) for h in hubs[:10] for v in r.choice(n, 1500, replace=False)]
    edges += [(u, h) for u in r.choice(n, 3000, replace=False) for h in r.choice(hubs, 12, replace=False)]
    edges += list(zip(r.integers(0, n, 60000), r.integers(0, n, 60000)))
    check(chain, *csr(n, edges))


def test_popular_far_members(chain):
    """Every id equally popular and rows of thousands: several tiles of high entries per root."""
    n = 200_000
    r = np.random.default_rng(3)
    edges = [(u, v) for u in range(40) for v in r.choice(n, 9000, replace=False)]
    edges += [(u, v) for u in range(40) for v in range(40)]
    check(chain, *csr(n, edges))


@pytest.mark.parametrize("m", [(1 << 18) - 1, 1 << 18, (1 << 18) + 1, (1 << 21) - 1, (1 << 21) + 4097])
def test_edge_count_bounds(ctx, m):
    """One launch up to 2^18 edges; a sample of the edges ranks the ids from 2^18 on."""
    src, dst = gen.rmat(17 if m > 1 << 19 else 14, 24)
    rp, col, _ = oracle.pipeline(src, dst)
    col = col[:m]
    rp = np.minimum(rp, m).astype(np.int32)
    assert len(col) == m
    check(ctx, rp, col)


def test_any_direction_of_edges(ctx):
    """No order among the vertices, self-loops: the count is still the sum over u -> v of |N+(u) n N+(v)|."""
    r = np.random.default_rng(8)
    for n, m in ((64, 900), (3000, 90000), (50000, 700000)):
        rp, col = csr(n, np.stack((r.integers(0, n, m), (r.integers(0, n, m) ** 2) // n), 1))
        check(ctx, rp, col)


@pytest.mark.parametrize("n_roots", [0, 1, 31, 32, 33, 5000])
def test_roots_prefix_matches_plain_id_tables(ctx, n_roots):
    rp, col, _ = oracle.pipeline(*gen.rmat(15))
    g = ctx.upload(rp, col, n_roots=n_roots)
    got, pr = ctx.count(g), ctx.count_per_root(g)
    old = ctx.get_tuning()
    ctx.set_tuning(probe_kicks=0)  # the tables of plain ids
    try:
        assert ctx.count(g) == got and np.array_equal(ctx.count_per_root(g), pr)
    finally:
        ctx.set_tuning(probe_kicks=old["probe_kicks"])
    assert ctx.count(g) == got


def test_batch_of_graphs_with_and_without_edges(ctx):
    want, graphs = [], []
    for i, n in enumerate((1, 5, 33, 64, 700, 4097)):
        r = np.random.default_rng(i)
        m = 0 if i % 3 == 1 else 6 * n
        rp, col = csr(n, np.stack((r.integers(0, n, m), r.integers(0, n, m)), 1))
        graphs.append(ctx.upload(rp, col))
        want.append(oracle.count(rp, col))
    for order in (list(range(6)), [1, 4, 0, 1, 3, 5, 2, 4]):
        b = ctx.batch([graphs[i] for i in order])
        assert list(b.run()) == [want[i] for i in order]
