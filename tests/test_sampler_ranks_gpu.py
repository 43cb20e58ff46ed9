"""The sampler's lane groups at their edges, and the batch-wide node table: bit-exact against the host replay."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _csr(n, top, num_cols, seed):
    rng = np.random.default_rng(seed)
    deg = rng.integers(0, top, n)
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    return rp, rng.integers(0, num_cols, rp[-1]).astype(np.int32), rng.standard_normal(rp[-1]).astype(np.float32)


@pytest.mark.parametrize("fanout", [1, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33])
def test_hop_groups(oracle, fanout):
    from graph_rws_b200 import core
    rp, ci, vv = _csr(333, 4 * fanout + 2, 333, fanout)
    nodes = np.concatenate([np.arange(333), [-1, 5, -1]]).astype(np.int32)
    got = core.sample_hop(*(torch.from_numpy(a).cuda() for a in (rp, ci, vv, nodes)), fanout, seed=11, hop=2)
    for a, b in zip(got, oracle.sample_hop(rp, ci, vv, nodes, fanout, 11, 2)):
        assert np.array_equal(a.cpu().numpy().reshape(-1), np.asarray(b).reshape(-1))


@pytest.mark.parametrize("n,num_cols,fanouts", [
    (40, 40, [3, 2, 2]),            # one bitmap word and a bit; sources soon cover the graph
    (8192, 8192, [4, 3]),           # exactly one CTA's words
    (20011, 20011, [5, 4]),         # several CTAs, a ragged last word
    (64, 9000, [7]),                # a last hop that names ids past the node count
])
def test_batch_table(oracle, n, num_cols, fanouts):
    from graph_rws_b200 import core
    rp, ci, vv = _csr(n, 12, num_cols, n)
    seeds = np.random.default_rng(1).integers(0, n, 33).astype(np.int32)         # some of them twice
    hops = core.sample_layers_fused(*(torch.from_numpy(a).cuda() for a in (rp, ci, vv, seeds)), fanouts, seed=9)
    dst = seeds
    for h, f in enumerate(fanouts):
        wo, cols, vals, _, src = (t.cpu().numpy() for t in hops[h])
        nbr, w, _ = oracle.sample_hop(rp, ci, vv, dst, f, 9, h)
        src_r, wo_r, cols_r, vals_r = oracle.build_block(dst, nbr, w)
        assert np.array_equal(src[:src_r.size], src_r) and (src[src_r.size:] == -1).all()
        assert np.array_equal(wo, wo_r)
        assert np.array_equal(cols[:cols_r.size], cols_r) and (cols[cols_r.size:] == -1).all()
        assert np.array_equal(vals[:vals_r.size], vals_r) and (vals[vals_r.size:] == 0).all()
        dst = src


@pytest.mark.parametrize("n,num_cols,fanout", [
    (700, 2 ** 31 - 1, 12),         # one short run of ids past the node count
    (3000, 2_000_000, 12),          # three runs, merged in two groups
    (9000, 9_000_000, 30),          # some twenty runs in groups of eight, the last group short
    (40000, 50_000, 32),            # most of the 10 k such ids are met many times
])
@pytest.mark.parametrize("told", [False, True])
def test_many_ids_past_the_node_count(oracle, n, num_cols, fanout, told):
    from graph_rws_b200 import core
    csr = _csr(n, 2 * fanout, num_cols, n)
    seeds = np.random.default_rng(2).permutation(n).astype(np.int32)
    wo, cols, vals, _, src = (t.cpu().numpy() for t in core.sample_layers_fused(
        *(torch.from_numpy(a).cuda() for a in (*csr, seeds)), [fanout], seed=9, num_cols=num_cols if told else None)[0])
    nbr, w, _ = oracle.sample_hop(*csr, seeds, fanout, 9, 0)
    src_r, wo_r, cols_r, vals_r = oracle.build_block(seeds, nbr, w)
    assert np.array_equal(src[:src_r.size], src_r) and (src[src_r.size:] == -1).all()
    assert np.array_equal(wo, wo_r)
    assert np.array_equal(cols[:cols_r.size], cols_r) and np.array_equal(vals[:vals_r.size], vals_r)


def test_ids_past_the_node_count_cost_no_more_than_a_sort():
    """120 k such ids in one hop: near the time of a square graph's hop (a scan of their list for each took forty
    times as long)."""
    from graph_rws_b200 import core
    times = []
    for num_cols in (20000, 5_000_000):
        csr = [torch.from_numpy(a).cuda() for a in _csr(20000, 60, num_cols, 5)]
        seeds = torch.randperm(20000, generator=torch.Generator().manual_seed(1))[:8192].int().cuda()
        taken = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            core.sample_layers_fused(*csr, seeds, [15], seed=9)
            b.record()
            b.synchronize()
            taken.append(a.elapsed_time(b))
        times.append(min(taken))
    assert times[1] < 6 * times[0]


@pytest.mark.parametrize("nodes,bitmap", [(1, True), (14_400_000, True), (17_000_000, False), (2 ** 31 - 2, False)])
def test_small_batches_of_large_graphs_are_sorted(oracle, nodes, bitmap):
    """37 seeds, fan-out 5-5 (1,295 list slots): the bitmap up to 450,000 words and 61 for every slot, sorts above; the
    scratch tells which, the result does not."""
    import ctypes
    from graph_rws_b200 import core
    from graph_rws_b200.core import _native
    fan = (ctypes.c_int * 2)(5, 5)
    lib = _native.lib()
    sized = lib.grws_sample_layers_sized_scratch_bytes(nodes, 37, fan, 2, 0)
    assert (sized != lib.grws_sample_layers_scratch_bytes(37, fan, 2, 0)) == bitmap
    csr = _csr(500, 12, 500, 3)
    seeds = np.arange(0, 74, 2, dtype=np.int32)
    got = core.sample_layers_fused(*(torch.from_numpy(a).cuda() for a in (*csr, seeds)), [5, 5], seed=9, num_cols=nodes)
    dst = seeds
    for h in range(2):
        wo, cols, vals, _, src = (t.cpu().numpy() for t in got[h])
        nbr, w, _ = oracle.sample_hop(*csr, dst, 5, 9, h)
        src_r, wo_r, cols_r, vals_r = oracle.build_block(dst, nbr, w)
        assert np.array_equal(src[:src_r.size], src_r) and (src[src_r.size:] == -1).all() and np.array_equal(wo, wo_r)
        assert np.array_equal(cols[:cols_r.size], cols_r) and np.array_equal(vals[:vals_r.size], vals_r)
        dst = src


@pytest.mark.parametrize("offset", [1, 4, 8, 255])
@pytest.mark.parametrize("nodes", [300, 2 ** 31 - 2])
def test_scratch_may_start_anywhere(monkeypatch, offset, nodes):
    from graph_rws_b200 import core
    from graph_rws_b200.core import sampling
    args = [torch.from_numpy(a).cuda() for a in (*_csr(300, 12, 300, 3), np.arange(0, 74, 2, dtype=np.int32))]
    want = core.sample_layers_fused(*args, [5, 4], seed=9, num_cols=nodes)
    monkeypatch.setattr(sampling, "_scratch", lambda n, dev: torch.empty(n + 256, dtype=torch.uint8, device=dev)[offset:offset + n])
    got = core.sample_layers_fused(*args, [5, 4], seed=9, num_cols=nodes)
    for a, b in zip(got, want):
        assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("pad_to", [0, 64])
def test_entry_without_a_node_count(pad_to):
    """grws_sample_layers, the call that is not told the number of nodes, gives the same hops and counts."""
    import ctypes
    from graph_rws_b200 import core
    from graph_rws_b200.core import _native
    lib = _native.lib()
    rp, ci, vv = (torch.from_numpy(a).cuda() for a in _csr(3000, 12, 3000, 3))
    seeds = torch.arange(0, 3000, 41, dtype=torch.int32, device="cuda")
    fanouts = [5, 4]
    want, counts = core.sample_layers_fused(rp, ci, vv, seeds, fanouts, seed=9, pad_to=pad_to, want_counts=True)
    fan = (ctypes.c_int * 2)(*fanouts)
    outs = [[torch.empty_like(t) for t in (hop[4], hop[0], hop[1], hop[2])] for hop in want]
    got_counts = torch.empty_like(counts)
    scratch = torch.empty(lib.grws_sample_layers_scratch_bytes(seeds.numel(), fan, 2, pad_to), dtype=torch.uint8, device="cuda")
    arrays = [(ctypes.c_void_p * 2)(*[hop[i].data_ptr() for hop in outs]) for i in range(4)]
    _native.check(lib.grws_sample_layers(rp.data_ptr(), ci.data_ptr(), vv.data_ptr(), seeds.data_ptr(), seeds.numel(), fan, 2, 9, 0, pad_to,
                                         _native.F32, *arrays, got_counts.data_ptr(), scratch.data_ptr(), scratch.numel(),
                                         torch.cuda.current_stream().cuda_stream))
    assert torch.equal(got_counts, counts)
    for hop, out in zip(want, outs):
        assert all(torch.equal(a, b) for a, b in zip((hop[4], hop[0], hop[1], hop[2]), out))
