"""The transposed BCSR of matrices in the forms its two passes over the tiles accept: bit-exact against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _matrix(num_rows, num_cols, rng, empty=(), hub=None):
    """Distinct entries, rows ascending; the rows of ``empty`` windows have none, row ``hub`` has one in every column."""
    counts = rng.integers(0, min(num_cols, 12), num_rows)
    for w in empty:
        counts[w * 16:w * 16 + 16] = 0
    if hub is not None:
        counts[hub] = num_cols
    rp = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    ci = np.concatenate([np.sort(rng.choice(num_cols, c, replace=False)) for c in counts]).astype(np.int32)
    return rp, ci, (rng.integers(1, 100, ci.size) / 16).astype(np.float32)         # exact in 16 bits


def _transposed(oracle, rows, rp, ci, v, num_cols):
    """The oracle's BCSR of the transposed matrix, entries of a column in ascending row order."""
    row = np.repeat(np.arange(rows, dtype=np.int32), np.diff(rp))
    order = np.lexsort((row, ci))
    rp_t = np.concatenate([[0], np.cumsum(np.bincount(ci, minlength=num_cols))]).astype(np.int64)
    return oracle.csr_to_bcsr(num_cols, rp_t, row[order], v[order])


def test_range_of_windows(oracle):
    """A range of a matrix's windows over the whole matrix's arrays: its first tile is not tile 0."""
    from graph_rws_b200 import core
    rng = np.random.default_rng(7)
    rows, cols, lo, hi = 160, 90, 3, 8
    rp, ci, v = _matrix(rows, cols, rng)
    wo, c, x = core.csr_to_bcsr(rows, *(torch.from_numpy(a).cuda() for a in (rp, ci, v)))
    got = core.bcsr_transpose(wo[lo:hi + 1], c, x, cols)
    a, b = rp[lo * 16], rp[hi * 16]
    want = _transposed(oracle, (hi - lo) * 16, rp[lo * 16:hi * 16 + 1] - a, ci[a:b], v[a:b], cols)
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w)


FORMS = {"plain": {}, "windows without tiles": dict(empty=(0, 1, 4, 9)), "hub": dict(hub=37), "hub and holes": dict(empty=(0, 5), hub=150)}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("form", FORMS)
def test_forms(oracle, form, dtype):
    """A hub's tiles are shared out over many warps; windows without tiles are passed over; 16-bit values; an entry count
    given by a bound; arrays that go on behind the last tile; and arrays that no 16-byte load may read."""
    from graph_rws_b200 import core
    rng = np.random.default_rng(len(form))
    rows, cols = 160, 9000
    rp, ci, v = _matrix(rows, cols, rng, **FORMS[form])
    csr = [torch.from_numpy(a).cuda() for a in (rp, ci, v)]
    want = _transposed(oracle, rows, rp, ci, v, cols)
    T = len(want[1]) // 8

    def check(got):
        assert np.array_equal(got[0].cpu().numpy(), want[0])
        assert np.array_equal(got[1][:T * 8].cpu().numpy(), want[1])
        assert got[2].dtype == dtype and np.array_equal(got[2][:T * 128].float().cpu().numpy(), want[2])
        assert bool((got[1][T * 8:] == -1).all()) and not got[2][T * 128:].any()

    wo, c, x = core.csr_to_bcsr(rows, *csr, values_dtype=dtype)
    check(core.bcsr_transpose(wo, c, x, cols))
    check(core.bcsr_transpose(wo, c, x, cols, exact=False, nnz_bound=ci.size + 77))
    check(core.bcsr_transpose(*core.csr_to_bcsr(rows, *csr, values_dtype=dtype, exact=False), cols))
    c2, x2 = torch.empty(c.numel() + 1, dtype=c.dtype, device="cuda")[1:], torch.empty(x.numel() + 1, dtype=dtype, device="cuda")[1:]
    check(core.bcsr_transpose(wo, c2.copy_(c), x2.copy_(x), cols))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_unaligned_outputs(oracle, dtype):
    """Column ids and values that do not start on 16-byte boundaries, for small and large windows and the unused tail."""
    from graph_rws_b200.core import _DT, _native
    rng = np.random.default_rng(4)
    rows, cols = 75, 3000
    rp, ci, v = _matrix(rows, cols, rng, empty=(2,), hub=20)
    rp_d, ci_d, v_d = (torch.from_numpy(a).cuda() for a in (rp, ci, v))
    want = oracle.csr_to_bcsr(rows, rp, ci, v)
    T, lib, st = len(want[1]) // 8 + 3, _native.lib(), torch.cuda.current_stream().cuda_stream
    wo = torch.empty(len(want[0]), dtype=torch.int64, device="cuda")
    scratch = torch.empty(lib.grws_csr_to_bcsr_scratch_bytes(rows, ci.size), dtype=torch.uint8, device="cuda")
    _native.check(lib.grws_csr_to_bcsr_count(rows, rp_d.data_ptr(), ci_d.data_ptr(), v_d.data_ptr(), ci.size, wo.data_ptr(),
                                             scratch.data_ptr(), scratch.numel(), st))
    c = torch.full((T * 8 + 2,), 5, dtype=torch.int32, device="cuda")
    x = torch.full((T * 128 + 2,), 5, dtype=dtype, device="cuda")
    _native.check(lib.grws_csr_to_bcsr_fill(rows, ci.size, wo.data_ptr(), T, c[1:].data_ptr(), x[1:].data_ptr(), _DT[dtype],
                                            scratch.data_ptr(), scratch.numel(), st))
    assert np.array_equal(wo.cpu().numpy(), want[0])
    assert c.tolist() == [5] + want[1].tolist() + [-1] * 24 + [5]
    assert np.array_equal(x[1:-1].float().cpu().numpy(), np.concatenate([want[2], np.zeros(3 * 128, np.float32)]))
    assert float(x[0]) == float(x[-1]) == 5


@pytest.mark.parametrize("num_cols", [0, 3000])
def test_entry_count_given_by_a_bound(oracle, num_cols):
    """Only the entries that the row pointers cover exist; duplicates among them keep their order."""
    from graph_rws_b200 import core
    rng = np.random.default_rng(6)
    rows = 100
    rp = np.concatenate([[0], np.cumsum(rng.integers(0, 90, rows))]).astype(np.int64)
    ci, v = rng.integers(0, 3000, rp[-1] + 50).astype(np.int32), rng.standard_normal(rp[-1] + 50).astype(np.float32)
    ci[3:rp[-1]:5] = ci[2:rp[-1] - 1:5]
    want = oracle.csr_to_bcsr(rows, rp, ci[:rp[-1]], v[:rp[-1]])
    got = core.csr_to_bcsr(rows, *(torch.from_numpy(a).cuda() for a in (rp, ci, v)), nnz_is_bound=True, num_cols=num_cols)
    for g, w in zip(got, want):
        assert np.array_equal(g.cpu().numpy(), w)
