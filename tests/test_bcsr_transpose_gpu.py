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
