"""Column ids of a block for the first layer, against the tensor operations they replace, and the layer's
recorded and unrecorded forms against each other."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("tiles", [1, 31, 33, 1000])
def test_relabel_and_sanitize(tiles, dtype):
    from graph_rws_b200 import core
    g = torch.Generator().manual_seed(tiles)
    cols = torch.randint(-2, 50, (tiles * 8,), generator=g).int().cuda()
    ids = torch.randint(0, 900, (50,), generator=g).int().cuda()
    vals = torch.randn(tiles * 128, generator=g).to(dtype).cuda()
    out = core.relabel_columns(cols, ids)
    assert torch.equal(out, torch.where(cols >= 0, ids[cols.clamp(min=0).long()], cols))
    bad = (out == -1) | (out >= 700)
    want_cols, want_vals = out.masked_fill(bad, 0), vals.view(-1, 16, 8).masked_fill(bad.view(-1, 1, 8), 0.0).view(-1)
    versions = out._version, vals._version
    core.sanitize_columns(out, vals, 700)
    assert torch.equal(out, want_cols) and torch.equal(vals, want_vals)
    assert out._version > versions[0] and vals._version > versions[1]


@pytest.mark.parametrize("rows", [37, 48])
@pytest.mark.parametrize("out_feats", [16, 41])
@pytest.mark.parametrize("target", [None, "rows", "fewer", "more"])
def test_layer_without_grad_equals_layer_with_grad(rows, out_feats, target):
    import numpy as np
    from graph_rws_b200 import BCSRGraph
    from graph_rws_b200.layers import BCSRGraphConv
    rng = np.random.default_rng(rows)
    rp = np.concatenate([[0], np.cumsum(rng.integers(0, 9, rows))]).astype(np.int64)
    g = BCSRGraph.from_csr(rows, rp, rng.integers(0, rows, rp[-1]).astype(np.int32), rng.standard_normal(rp[-1]).astype(np.float32))
    torch.manual_seed(3)
    conv = BCSRGraphConv(24, out_feats).cuda()
    x = torch.randn(rows, 24, device="cuda")
    t = {None: None, "rows": x, "fewer": x[:20], "more": torch.randn(80, 24, device="cuda")}[target]
    want = conv(g, x, features_target=t).detach()
    with torch.no_grad():
        got = conv(g, x, features_target=t)
    assert got.shape == want.shape
    # TF32 products of 24 terms, one rounding of the sum more or less
    assert torch.allclose(got, want, rtol=0, atol=24 * 2 ** -11 * float(want.abs().max()))
