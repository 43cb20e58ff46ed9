"""Column ids of a block for the first layer: what the tensor operations refuse is refused, and what they
accept besides whole 16x8 tiles is done."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _arrays(tiles=5, values=None, tile=(16, 8)):
    cols = torch.arange(tiles * tile[1], dtype=torch.int32, device="cuda") - 1
    return cols, torch.ones(tiles * tile[0] * tile[1] if values is None else values, device="cuda")


@pytest.mark.parametrize("cols,values", [(40, 4 * 128), (40, 3 * 128), (40, 128 * 5 + 8), (36, 128 * 5), (36, 128 * 4)])
def test_arrays_that_disagree(cols, values):
    from graph_rws_b200 import core
    c, v = _arrays(values=values)
    with pytest.raises(RuntimeError):
        core.sanitize_columns(c[:cols], v, 20)


def test_leaf_that_requires_grad():
    from graph_rws_b200 import core
    c, v = _arrays()
    v.requires_grad_()
    with pytest.raises(RuntimeError):
        core.sanitize_columns(c, v, 20)
    c, v = _arrays()                                  # the refused call has edited the column ids
    v.requires_grad_()
    with torch.no_grad():
        core.sanitize_columns(c, v, 20)
    assert v._version == 1 and float(v.detach().sum()) == 20 * 16


def test_inference_tensors():
    from graph_rws_b200 import core
    with torch.inference_mode():
        c, v = _arrays()
    with pytest.raises(RuntimeError):
        core.sanitize_columns(c, v, 20)
    with torch.inference_mode():
        c, v = _arrays()
        core.sanitize_columns(c, v, 20)
    assert float(v.sum()) == 20 * 16


def test_other_tiles():
    from graph_rws_b200 import core
    c, v = _arrays(tile=(8, 4))
    core.sanitize_columns(c, v, 7, 8, 4)
    assert torch.equal(v.view(5, 8, 4).sum(1).flatten().cpu(), 8.0 * torch.tensor([0] + [1] * 7 + [0] * 12))


@pytest.mark.parametrize("top,fine", [(49, True), (50, False), (2 ** 31 - 1, False)])
def test_ids_past_the_table(monkeypatch, top, fine):
    """Such an id stops the program; here the condition is taken down instead of being asserted."""
    from graph_rws_b200 import core
    seen = []
    monkeypatch.setattr(torch, "_assert_async", lambda ok, *a: seen.append(bool(ok)))
    cols = torch.tensor([3, -1, top, 0], dtype=torch.int32, device="cuda")
    core.relabel_columns(cols, torch.arange(100, 150, dtype=torch.int32, device="cuda"))
    assert seen == [fine]
