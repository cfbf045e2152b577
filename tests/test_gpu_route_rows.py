"""The experts' router at many tokens (sixteen tokens a block) against the kernel of one token a block: the same choices and weights,
bit for bit."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def parts(h, router, bias, top, scoring):
    """The same in steps of so few tokens that each is a block of its own."""
    from starter_b200 import ops

    got = [ops.moe_route(h[i:i + 300], router, bias, top, scoring, 1.5) for i in range(0, h.shape[0], 300)]
    return torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got])


def same(got, want):
    assert torch.equal(got[0], want[0])
    assert torch.equal(got[1].nan_to_num(7.0), want[1].nan_to_num(7.0))


# experts: one, less than a pass of eight, a pass, several of sixteen, with what is left over; widths that end inside a stage of 512
# and in one; tokens that leave part of a block
@pytest.mark.parametrize("experts,width,tokens", [(1, 8, 592), (5, 72, 601), (8, 512, 608), (9, 520, 593), (16, 2048, 640), (16, 1544, 2400),
                                                  (17, 264, 1186), (33, 136, 1199), (64, 1032, 1185)])
@pytest.mark.parametrize("scoring", ["softmax_top", "sigmoid_normalised", "sigmoid"])
def test_many_tokens_choose_as_few_do(experts, width, tokens, scoring):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(experts + width)
    h = torch.randn(tokens, width, generator=gen).to(BF).cuda()
    router = (torch.randn(experts, width, generator=gen) * width ** -0.5).cuda()
    for bias in (None, torch.randn(experts, generator=gen).cuda()):
        for top in sorted({1, min(experts, 4), min(experts, 16)}):
            same(ops.moe_route(h, router, bias, top, scoring, 1.5), parts(h, router, bias, top, scoring))


def test_equal_infinite_and_missing_logits():
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(3)
    experts, width, tokens = 40, 64, 1200
    h = torch.randn(tokens, width, generator=gen).to(BF).cuda()
    router = torch.randn(experts, width, generator=gen).cuda()
    router[5], router[37] = router[3], router[3]              # equal logits: the lower index first
    h[7] = 0.0                                                # all equal
    h[8, 0] = float("nan")                                    # none
    h[9, 0] = float("inf")
    bias = torch.zeros(experts).cuda()
    bias[2], bias[4], bias[36], bias[6] = float("-inf"), float("inf"), float("inf"), -0.0
    for scoring in ("softmax_top", "sigmoid_normalised"):
        same(ops.moe_route(h, router, bias, 6, scoring, 1.5), parts(h, router, bias, 6, scoring))
        same(ops.moe_route(h, router, None, 16, scoring, 1.5), parts(h, router, None, 16, scoring))
    none = torch.full((experts,), float("-inf")).cuda()
    same(ops.moe_route(h, router, none, 3, "sigmoid", 1.5), parts(h, router, none, 3, "sigmoid"))


@pytest.mark.parametrize("which", ["h", "router", "width"])
def test_rows_that_are_not_in_whole_pieces(which):
    """Rows off 16 bytes, or of 4 entries more than whole pieces: served as before."""
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(5)
    experts, width, tokens = 12, 68 if which == "width" else 72, 700
    h = torch.randn(tokens * width + 4, generator=gen).to(BF).cuda()[4 if which == "h" else 0:][:tokens * width].view(tokens, width)
    router = torch.randn(experts * width + 2, generator=gen).cuda()[2 if which == "router" else 0:][:experts * width].view(experts, width)
    same(ops.moe_route(h, router, None, 3, "sigmoid", 1.5), parts(h, router, None, 3, "sigmoid"))
