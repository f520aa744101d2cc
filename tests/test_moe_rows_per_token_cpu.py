"""The router's note that every token has the same number of entries holds only for the map as the router left it."""
import pytest
import torch

from mindspeed_b200.parallel.moe.moe_utils import mark_rows_per_token, rows_per_token


def _map():
    m = torch.zeros(4, 6, dtype=torch.bool).scatter(1, torch.tensor([[0, 1]] * 4), True)
    mark_rows_per_token(m, 2)
    return m


def test_note_of_an_untouched_map():
    assert rows_per_token(_map()) == 2 and rows_per_token(torch.ones(2, 2, dtype=torch.bool)) is None
    assert rows_per_token(_map().clone()) is None


@pytest.mark.parametrize("edit", [lambda m: m.masked_fill_(torch.eye(4, 6, dtype=torch.bool), False), lambda m: m.__iand__(torch.eye(4, 6) > 0),
                                  lambda m: m.__setitem__((0, 5), True), lambda m: m[1].zero_()])
def test_note_ends_with_the_next_write(edit):
    m = _map()
    edit(m)
    assert rows_per_token(m) is None


def test_inference_tensors_count_no_versions():
    with torch.inference_mode():
        assert rows_per_token(_map()) is None
