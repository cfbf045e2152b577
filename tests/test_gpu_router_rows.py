"""The routers' kernels that take four tokens a block (steps of many tokens) against those that take one."""

import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = 595                       # the last block has three tokens


def portions(call, h):
    """The same rows, few at a time: a token a block."""
    parts = [call(rows) for rows in h.split(119)]
    return [torch.cat(p) for p in zip(*parts)]


def rows_of(width, dtype):
    gen = torch.Generator().manual_seed(width)
    h = torch.randn(ROWS, width, generator=gen)
    h[7] = 0.0                   # every logit equal
    return h.to(dtype).cuda(), gen


# widths: rows brought into shared memory in one loop and in several; too wide for it; no whole pieces of 16 bytes
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [264, 1028, 4104, 50])
@pytest.mark.parametrize("experts, top, scoring, bias", [(5, 2, "softmax_top", True), (64, 8, "sigmoid_normalised", False), (512, 4, "sigmoid", True)])
def test_router_of_many_tokens(experts, top, scoring, bias, width, dtype):
    from starter_b200 import ops

    h, gen = rows_of(width, dtype)
    router = (torch.randn(experts, width, generator=gen) * width ** -0.5).cuda()
    b = torch.randn(experts, generator=gen).cuda() if bias else None

    def call(x):
        return ops.moe_route(x.contiguous(), router, b, top, scoring, 1.5)

    ids, weights = call(h)
    want_ids, want = portions(call, h)
    # (a logit is the same sum in the same order)
    assert torch.equal(ids, want_ids) and torch.equal(weights, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [264, 4104, 50])
@pytest.mark.parametrize("outputs, top, groups, keep, gate", [(12, 3, 2, 1, True), (256, 8, 8, 4, True), (256, 16, 256, 16, False),
                                                              (255, 5, 255, 9, True), (330, 4, 3, 2, False)])
def test_router_over_all_of_many_tokens(outputs, top, groups, keep, gate, width, dtype):
    """Up to the most outputs and groups whose numbers four tokens have room for, and beyond."""
    from starter_b200 import ops

    h, gen = rows_of(width, dtype)
    router = (torch.randn(outputs + gate, width, generator=gen) * width ** -0.5).cuda()
    correction = (torch.randn(outputs, generator=gen) * 0.1).cuda()

    def call(x):
        return [t for t in ops.moe_route_all(x.contiguous(), router, correction, top, groups, keep, shared_gate=gate) if t is not None]

    for got, want in zip(call(h), portions(call, h)):
        assert torch.equal(got, want)
