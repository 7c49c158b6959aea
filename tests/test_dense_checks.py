"""Operands of the dense maps that do not fit together are refused before anything reaches the library."""
import pytest
import torch

from cbm4gnn_b200 import dense


@pytest.mark.parametrize("call", [
    lambda: dense.dense_forward(torch.ones(8, 5), torch.ones(3, 6)),
    lambda: dense.dense_forward(torch.ones(8, 6), torch.ones(3, 5)),
    lambda: dense.dense_forward(torch.ones(2, 8, 5), torch.ones(3, 5)),
    lambda: dense.dense_forward(torch.ones(8, 5), torch.ones(5)),
    lambda: dense.dense_grad_input(torch.ones(8, 4), torch.ones(3, 6)),
    lambda: dense.dense_grad_input(torch.ones(8, 3), torch.ones(3, 6), relu_output=torch.ones(7, 6)),
    lambda: dense.dense_grad_input(torch.ones(8, 3), torch.ones(3, 6), relu_output=torch.ones(8, 5)),
    lambda: dense.dense_grad_weight(torch.ones(8, 3), torch.ones(7, 6)),
])
def test_operands_that_do_not_fit_together(call):
    with pytest.raises(RuntimeError, match="shape mismatch"):
        call()


def test_operands_on_two_devices():
    with pytest.raises(RuntimeError, match="operands on cpu and meta"):
        dense.dense_forward(torch.ones(8, 5), torch.ones((3, 5), device="meta"))


@pytest.mark.parametrize("out,fits", [
    (torch.zeros(8, 3), True), (torch.zeros(8, 7)[:, 2:5], True),                      # rows of any width and pitch
    (torch.zeros(8, 3, dtype=torch.float64), False), (torch.zeros(3, 8).t(), False),   # converted, turned
    (torch.zeros(7, 3), None), (torch.zeros(8, 4), None),                              # neither: refused by the copy
])
def test_results_go_straight_only_to_rows_they_fit(out, fits, monkeypatch):
    written = []
    monkeypatch.setattr(dense, "_call", lambda name, dev, *args: written.append(args[4]))
    if fits is None:
        with pytest.raises(RuntimeError, match="size of tensor"):
            dense.dense_forward(torch.ones(8, 5), torch.ones(3, 5), out=out)
    else:
        assert dense.dense_forward(torch.ones(8, 5), torch.ones(3, 5), out=out) is out
    assert (written == [out.data_ptr()]) == (fits is True)
