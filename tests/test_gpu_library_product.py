"""Products of 129 to 511 rows, which the library does: the short way to it gives torch.mm's bits, and leaves to torch.mm whatever is no
plain product."""

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("rows", [129, 300, 511])
@pytest.mark.parametrize("width, k", [(3072, 2048), (264, 72), (33, 17), (8, 8)])
def test_the_library_products_bits(rows, width, k):
    from starter_b200 import ops

    gen = torch.Generator().manual_seed(rows + k)
    x, w = torch.randn(rows, k, generator=gen).to(BF).cuda(), torch.randn(width, k, generator=gen).to(BF).cuda()
    want = torch.mm(x, w.t())
    assert torch.equal(ops.linear(x, w), want)
    assert torch.equal(ops._product(x, w, 128, 512), want)
    graph = torch.cuda.CUDAGraph()
    with torch.inference_mode(), torch.cuda.graph(graph):
        y = ops.linear(x, w)
    graph.replay()
    assert torch.equal(y, want)


def test_what_is_no_plain_product_goes_the_general_way():
    from starter_b200 import ops

    x, w = torch.randn(200, 64).to(BF).cuda(), torch.randn(48, 64).to(BF).cuda()
    ops.linear(x, w)
    go = lambda a, b: ops._product(a, b, 128, 512)
    assert go(x[:128], w) is None and go(torch.cat([x, x, x]), w) is None          # other kernels' rows
    assert go(x.float(), w.float()) is None and go(x.cpu(), w.cpu()) is None and go(x[:, :32], w[:, :32]) is None
    assert go(x, torch.randn(48, 32).to(BF).cuda()) is None and go(x[None], w) is None and go(x, None) is None
    assert go(x[:, :0].contiguous(), w[:, :0].contiguous()) is None
    grown = w.clone().requires_grad_()
    assert go(x, grown) is None
    y = ops.linear(x, grown)
    assert y.requires_grad
    with torch.no_grad():
        assert torch.equal(go(x, grown), y)
    with torch.autocast("cuda", dtype=torch.float16):
        assert go(x, w) is None and ops.linear(x, w).dtype == torch.float16
    with pytest.raises(ops.KernelError):
        ops.linear(x, torch.randn(47, 64).to(BF).cuda(), gated=True)
    with pytest.raises(ops.KernelError):
        ops.linear(x, w, gated="no such activation")
    with pytest.raises(ops.KernelError):
        ops.linear(x, torch.randn(48, 32).to(BF).cuda())


@pytest.mark.parametrize("which", ["x", "w", "both"])
def test_tangents_are_carried(which):
    from torch.autograd import forward_ad

    from starter_b200 import ops

    x, w, dx, dw = (torch.randn(*shape).to(BF).cuda() for shape in ((200, 64), (48, 64), (200, 64), (48, 64)))
    with forward_ad.dual_level():
        a = forward_ad.make_dual(x, dx) if which != "w" else x
        b = forward_ad.make_dual(w, dw) if which != "x" else w
        assert ops._product(a, b, 128, 512) is None
        got, want = (forward_ad.unpack_dual(y) for y in (ops.linear(a, b), torch.mm(a, b.t())))
        assert torch.equal(got.primal, want.primal) and torch.equal(got.tangent, want.tangent)
    assert torch.equal(ops._product(x, w, 128, 512), torch.mm(x, w.t()))


def test_a_profiler_sees_the_product():
    from starter_b200 import ops

    x, w = torch.randn(200, 64).to(BF).cuda(), torch.randn(48, 64).to(BF).cuda()
    ops.linear(x, w)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as seen:
        ops.linear(x, w)
    assert "aten::mm" in {e.key for e in seen.key_averages()}
