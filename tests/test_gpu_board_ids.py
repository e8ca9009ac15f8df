"""Board tables and hand ranks of a board read int64 card ids like int16 ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 3, 149])
def test_int64_boards(cuda_device, m):
    from poker2_b200 import rules, showdown

    g = torch.Generator(device=cuda_device).manual_seed(m)
    boards = torch.rand(m, 52, device=cuda_device, generator=g).argsort(dim=1)[:, :5]
    for a, b in zip(rules.rank_hands(boards), rules.rank_hands(boards.to(torch.int16))):
        assert torch.equal(a, b)
    assert torch.equal(showdown.BoardTables(boards).blob, showdown.BoardTables(boards.to(torch.int32)).blob)
