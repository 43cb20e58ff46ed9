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
