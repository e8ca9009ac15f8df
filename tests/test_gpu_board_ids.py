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


# ids are 13 * suit + rank: no suit can flush; three, four, five of a suit; a steel wheel and a royal flush; trips and quads;
# a paired board and boards with a straight or most of one
@pytest.mark.parametrize("board", [[0, 14, 28, 42, 17], [0, 3, 7, 22, 38], [13, 15, 19, 24, 50], [26, 29, 31, 34, 37],
                                   [0, 1, 2, 3, 12], [8, 9, 10, 11, 12], [5, 18, 31, 44, 12], [4, 5, 6, 17, 20],
                                   [8, 9, 10, 24, 25], [51, 50, 49, 11, 24]])
def test_strengths_and_order(cuda_device, board):
    import numpy as np

    from oracle import rank7
    from poker2_b200 import rules

    boards = torch.tensor([board], dtype=torch.int64)
    want_scores, want_order = rank7.rank_hands(boards.numpy(), rank7.MODE_IDS)
    scores, order = rules.rank_hands(boards.to(cuda_device))
    assert np.array_equal(scores.cpu().numpy(), want_scores)
    assert np.array_equal(order.cpu().numpy(), want_order)
