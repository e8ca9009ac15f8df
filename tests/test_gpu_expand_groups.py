"""The feature expansion takes eight next cards of a root per block, or all of them where the roots fill the chip; and it adds up
what a card leaves of a range by itself where the subtraction cancels.  Both against `chance.expand_next_card`."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("roots", [1, 5, 700])
@pytest.mark.parametrize("kind", ["dense", "one_card", "empty", "odd_stride"])
def test_features_equal_the_expanded_beliefs(cuda_device, roots, kind):
    from poker2_b200 import chance

    g = torch.Generator(device=cuda_device).manual_seed(roots)
    boards = torch.rand(roots, 52, device=cuda_device, generator=g).argsort(dim=1)[:, :5].contiguous()
    boards[:, 4] = -1
    pre = torch.rand(roots, 2, 1326, device=cuda_device, generator=g)
    if kind == "one_card":  # player 0 holds the first free card's hands, all but 1e-9 of the mass
        c1, c2 = torch.triu_indices(52, 52, 1, device=cuda_device)
        card = int((~torch.isin(torch.arange(52, device=cuda_device), boards[0])).nonzero()[0])
        pre[:, 0] *= torch.where((c1 == card) | (c2 == card), 1.0, 1e-9)
    if kind == "empty":
        pre[:, 1] = 0.0
    offsets = chance.sample_offsets_of(boards)
    post, lookup, samples = chance.expand_next_card(pre, boards)
    ctx = torch.rand(roots, 3, device=cuda_device, generator=g)
    stride = 2721 if kind == "odd_stride" else 2720
    x = chance.expand_features_bf16(pre, boards, offsets, int(offsets[-1]), ctx, stride)
    assert torch.equal(x[:, :2652], post.reshape(-1, 2652).to(torch.bfloat16))
    assert torch.equal(x[:, 2704:2707], ctx[lookup].to(torch.bfloat16)) and not x[:, 2707:].any()
    assert torch.equal(x[:, 2652:2704].float().sum(dim=1), torch.full((x.shape[0],), 5.0, device=cuda_device))


@pytest.mark.parametrize("odd", [float("nan"), float("inf")])
def test_features_where_a_card_takes_what_is_no_number(cuda_device, odd):
    """One hand's belief is NaN or infinite: the samples whose card holds that hand are what the unfused expansion, which adds
    up what a card leaves, gives; so are the others."""
    from poker2_b200 import chance

    g = torch.Generator(device=cuda_device).manual_seed(3)
    boards = torch.tensor([[0, 5, 17, 30, -1]], device=cuda_device)
    pre = torch.rand(1, 2, 1326, device=cuda_device, generator=g)
    pre[0, 1, 1325] = odd  # cards 50 and 51
    ctx = torch.rand(1, 3, device=cuda_device, generator=g)
    off = chance.sample_offsets_of(boards)
    got = chance.expand_features_bf16(pre, boards, off, 48, ctx, 2720)[:, :2652].view(48, 2, 1326)
    want, _, samples = chance.expand_next_card(pre, boards)
    takes = (samples == 50).any(1) | (samples == 51).any(1)
    assert int(takes.sum()) == 2 and bool(want[takes].isfinite().all())
    torch.testing.assert_close(got.float(), want.to(torch.bfloat16).float(), rtol=0.0, atol=0.0, equal_nan=True)
