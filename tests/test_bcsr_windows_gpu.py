"""Windows of the device builder at the edges of its two ways (a warp's sort of up to 512 entries, the
column bitmap above), with duplicates and unsorted rows: bit-exact against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _csr(sizes, num_cols, rng, duplicates):
    """One 16-row window per entry of ``sizes``, its entries spread over its rows at random, unsorted."""
    counts = np.concatenate([np.bincount(rng.integers(0, 16, m), minlength=16) for m in sizes])[:-3]
    rp = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    cols = rng.integers(0, num_cols, rp[-1]).astype(np.int32)
    if duplicates:                                    # every fourth entry repeats its neighbour's column
        cols[1::4] = cols[0::4][:cols[1::4].size]
    return len(counts), rp, cols, rng.standard_normal(rp[-1]).astype(np.float32)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("num_cols", [40, 5000, 2_000_000, 2 ** 31 - 1])
def test_windows_of_every_size(oracle, num_cols, dtype):
    from graph_rws_b200 import core
    rng = np.random.default_rng(num_cols)
    sizes = [0, 1, 31, 32, 33, 64, 65, 0, 128, 129, 256, 257, 511, 512, 513, 514, 0, 1500, 9000, 40000, 513, 40]
    n, rp, ci, v = _csr(sizes, num_cols, rng, duplicates=True)
    dev = torch.device("cuda")
    args = (n, torch.from_numpy(rp).to(dev), torch.from_numpy(ci).to(dev), torch.from_numpy(v).to(dev))
    want = oracle.csr_to_bcsr(n, rp, ci, v)
    T = len(want[1]) // 8
    for exact in (True, False):
        wo, cols, vals = core.csr_to_bcsr(*args, values_dtype=dtype, exact=exact)
        assert np.array_equal(wo.cpu().numpy(), want[0])
        assert np.array_equal(cols[:T * 8].cpu().numpy(), want[1])
        assert torch.equal(vals[:T * 128].cpu(), torch.from_numpy(want[2]).to(dtype))
        assert bool((cols[T * 8:] == -1).all()) and bool((vals[T * 128:] == 0).all())


@pytest.mark.parametrize("fanout", [1, 2, 32, 33, 256])
def test_blocks_from_lists(oracle, fanout):
    """A hop's block straight from its fixed-stride lists, on either side of the widest list a warp sorts."""
    from graph_rws_b200 import core
    rng = np.random.default_rng(fanout)
    n = 77
    deg = rng.integers(0, 2 * fanout + 2, n * 8)
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    ci = rng.integers(0, n * 8, rp[-1]).astype(np.int32)
    v = rng.standard_normal(rp[-1]).astype(np.float32)
    dev = torch.device("cuda")
    csr = [torch.from_numpy(a).to(dev) for a in (rp, ci, v)]
    seeds = torch.from_numpy(rng.permutation(n * 8)[:n].astype(np.int32)).to(dev)
    wo, cols, vals, _, src = core.sample_layers_fused(*csr, seeds, [fanout], seed=3)[0]
    nbr, w, _ = core.sample_hop(*csr, seeds, fanout, seed=3)
    local = {int(u): i for i, u in reversed(list(enumerate(src.tolist()))) if u >= 0}
    rows = [[(local[int(u)], x) for u, x in zip(r, xs) if u >= 0] for r, xs in zip(nbr.tolist(), w.tolist())]
    lrp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    lci = np.array([c for r in rows for c, _ in r], dtype=np.int32)
    lv = np.array([x for r in rows for _, x in r], dtype=np.float32)
    want = oracle.csr_to_bcsr(n, lrp, lci, lv)
    T = len(want[1]) // 8
    assert np.array_equal(wo.cpu().numpy(), want[0])
    assert np.array_equal(cols[:T * 8].cpu().numpy(), want[1])
    assert np.array_equal(vals[:T * 128].float().cpu().numpy(), want[2])
    assert bool((cols[T * 8:] == -1).all()) and bool((vals[T * 128:] == 0).all())


@pytest.mark.parametrize("order", ["ascending", "any"])
@pytest.mark.parametrize("num_cols", [3000, 1_200_000])
def test_large_windows_of_distinct_entries(oracle, num_cols, order):
    """Entries that can be written in any order: rows in ascending order (recognised), or the caller's word."""
    from graph_rws_b200 import core
    rng = np.random.default_rng(num_cols)
    rows = [0, 1, 700, 0, 2999, 2998, 5, 0, 0, 600, 13, 0, 0, 0, 0, 2000, 0, 0, 300, 400, 33, 0, 800]
    cols = [rng.choice(num_cols, m, replace=False).astype(np.int32) for m in rows]
    if order == "ascending":
        cols = [np.sort(c) for c in cols]
    rp, ci = np.concatenate([[0], np.cumsum(rows)]).astype(np.int64), np.concatenate(cols)
    v = rng.standard_normal(ci.size).astype(np.float32)
    dev = torch.device("cuda")
    wo, c, x = core.csr_to_bcsr(len(rows), *(torch.from_numpy(a).to(dev) for a in (rp, ci, v)), unique=order == "any")
    for got, want in zip((wo, c, x), oracle.csr_to_bcsr(len(rows), rp, ci, v)):
        assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("rows", [0, 16, 40])
@pytest.mark.parametrize("exact", [True, False])
def test_no_entries(rows, exact):
    """Without entries the row pointers are not read (here there is only one)."""
    from graph_rws_b200 import core
    none = torch.empty(0, device="cuda")
    wo, cols, vals = core.csr_to_bcsr(rows, torch.zeros(1, dtype=torch.int64, device="cuda"), none.int(), none, exact=exact)
    windows = (rows + 15) // 16
    assert wo.tolist() == [0] * (windows + 1)
    assert cols.tolist() == [-1] * (0 if exact else windows * 8) and not vals.any()


def _wide(kind, m, num_cols, rng):
    if kind == "even":
        return rng.integers(0, num_cols, m)
    far = rng.integers(0, num_cols, m // 16)                   # most entries in a narrow band, the others anywhere
    return rng.permutation(np.concatenate([num_cols // 3 + rng.integers(0, min(num_cols // 3, 700_000), m - far.size), far]))


@pytest.mark.parametrize("kind", ["even", "band"])
@pytest.mark.parametrize("num_cols", [524_287, 524_289, 600_000, 3_000_000, 7_000_000, 2 ** 31 - 1])
def test_wide_windows(oracle, num_cols, kind):
    """Large windows about as wide as a column bitmap and wider: a few rounds of bitmaps, one sort of up to 8,192 entries, or
    divided by column ranges that are sorted or marked (of the band's ranges some hold more than a sort takes and
    are wider than a bitmap)."""
    from graph_rws_b200 import core
    rng = np.random.default_rng(num_cols)
    sizes = [513, 1024, 1025, 2048, 2049, 4100, 8191, 8192, 8193, 16_500, 200_000, 700]
    counts = np.concatenate([np.bincount(rng.integers(0, 16, m), minlength=16) for m in sizes])
    rp = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    ci = np.concatenate([_wide(kind, m, num_cols, rng) for m in sizes]).astype(np.int32)
    ci[rp[16 * 3]], ci[rp[16 * 3] + 1] = 0, num_cols - 1       # the whole span
    v = rng.standard_normal(ci.size).astype(np.float32)
    n = len(counts)
    got = core.csr_to_bcsr(n, *(torch.from_numpy(a).cuda() for a in (rp, ci, v)))
    for g, want in zip(got, oracle.csr_to_bcsr(n, rp, ci, v)):
        assert np.array_equal(g.cpu().numpy(), want)


def test_wide_blocks_from_lists(oracle):
    """Lists whose local ids span more than a column bitmap, with empty slots."""
    from graph_rws_b200 import core
    rng = np.random.default_rng(8)
    n, fanout = 2400, 256
    rp = np.concatenate([[0], np.cumsum(rng.integers(200, 400, n))]).astype(np.int64)
    ci = rng.integers(0, 2 ** 30, rp[-1]).astype(np.int32)
    v = rng.standard_normal(rp[-1]).astype(np.float32)
    seeds = rng.permutation(n).astype(np.int32)
    wo, cols, vals, _, src = core.sample_layers_fused(*(torch.from_numpy(a).cuda() for a in (rp, ci, v, seeds)), [fanout], seed=3)[0]
    nbr, w, _ = oracle.sample_hop(rp, ci, v, seeds, fanout, 3, 0)
    src_r, wo_r, cols_r, vals_r = oracle.build_block(seeds, nbr, w)
    assert cols_r.max() >= 524_288
    assert np.array_equal(src[:src_r.size].cpu().numpy(), src_r) and np.array_equal(wo.cpu().numpy(), wo_r)
    assert np.array_equal(cols[:cols_r.size].cpu().numpy(), cols_r) and np.array_equal(vals[:vals_r.size].cpu().numpy(), vals_r)


def test_cost_does_not_grow_with_the_columns():
    """Windows of 640 entries in 400 k and in 100 M columns: within a factor (each 524,288 columns used to cost every
    window two more passes: a factor of 200)."""
    from graph_rws_b200 import core
    times = []
    for num_cols in (400_000, 100_000_000):
        g = torch.Generator(device="cuda").manual_seed(1)
        rp = torch.arange(0, 100_001, device="cuda") * 40
        ci = torch.randint(0, num_cols, (4_000_000,), generator=g, device="cuda", dtype=torch.int32)
        v = torch.ones(4_000_000, device="cuda")
        taken = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            core.csr_to_bcsr(100_000, rp, ci, v, exact=False)
            b.record()
            b.synchronize()
            taken.append(a.elapsed_time(b))
        times.append(min(taken))
    assert times[1] < 8 * times[0]


@pytest.mark.parametrize("twice", [None, "row", "other row"])
@pytest.mark.parametrize("entries,num_cols", [(8193, 30_000), (20_000, 3_000_000), (600_000, 2_000_000), (30_000, 9_000_000)])
def test_unordered_hub_row(oracle, entries, num_cols, twice):
    """A long row in no order next to a short one: distinct entries (found out by more than a bitmap of slots in the
    widest), a column twice in the row (the last one stays), or once in either row."""
    from graph_rws_b200 import core
    rng = np.random.default_rng(entries)
    hub = rng.choice(num_cols, entries, replace=False).astype(np.int32)
    short = rng.choice(num_cols, 300, replace=False).astype(np.int32)
    if twice == "row":
        hub[-1] = hub[entries // 3] = hub.max()                # the last slot, too
    if twice == "other row":
        short[7] = hub[-1]
    rp = np.array([0] * 5 + [entries] * 4 + [entries + 300] * 11, dtype=np.int64)
    ci = np.concatenate([hub, short])
    v = rng.standard_normal(ci.size).astype(np.float32)
    n = rp.size - 1
    got = core.csr_to_bcsr(n, *(torch.from_numpy(a).cuda() for a in (rp, ci, v)))
    for g, want in zip(got, oracle.csr_to_bcsr(n, rp, ci, v)):
        assert np.array_equal(g.cpu().numpy(), want)
