"""The routed experts' grouped products on tcgen05, against float64; which other tokens are in the step, and the other form."""
import pytest
import torch

from leone_b200.parts.base import Runtime
from tests.test_kernels_gpu import DEV, _randn, ops16  # noqa: F401

pytestmark = pytest.mark.gpu


# rows of an expert around a tile of 128 (by how unevenly the tokens choose), experts without any; inner sizes around a k-block
# of 64; columns around a tile of 128 + 128 or 256; the weight at the input or the output; gated and ungated
@pytest.mark.parametrize("form,scale_input", [("gated", True), ("gated", False), ("relu", False)])
@pytest.mark.parametrize("n,experts,top,width,ff,spread", [(300, 4, 2, 64, 128, 0.0), (513, 5, 3, 200, 136, 2.0), (1000, 32, 4, 256, 520, 1.0),
                                                           (129, 1, 1, 72, 8, 0.0), (640, 64, 8, 512, 256, 3.0)])
def test_grouped_products(ops16, form, scale_input, n, experts, top, width, ff, spread):  # noqa: F811
    x = _randn((n, width + 8), 1, torch.bfloat16)[:, :width]
    gate, up = (_randn((experts, ff, width), s, torch.bfloat16, 1.5 * width ** -0.5) for s in (2, 3))
    down = _randn((experts, width, ff), 4, torch.bfloat16, ff ** -0.5)
    lean = spread * torch.arange(experts, device=DEV) / experts
    weight, chosen = torch.topk(torch.rand((n, experts), device=DEV, generator=torch.Generator(DEV).manual_seed(5)) - lean, top, -1)
    weight = torch.rand((n, top), device=DEV, generator=torch.Generator(DEV).manual_seed(6)) + 0.2
    hidden = _randn((n, width), 7)
    want, size = hidden.double(), hidden.double().abs()
    b16 = lambda t: t.float().to(torch.bfloat16).double()                     # noqa: E731
    for e in range(experts):
        row, at = torch.nonzero(chosen == e, as_tuple=True)
        w = weight[row, at].double()[:, None]
        u = x[row].double() @ up[e].double().t()
        if form == "gated":
            f = w if scale_input else 1.0
            act = torch.nn.functional.silu(b16(x[row].double() @ gate[e].double().t() * f)) * b16(u * f)
        else:
            act = torch.clamp(b16(u), min=0) ** 2
        y = b16(act) @ down[e].double().t() * (1.0 if scale_input else w)
        want = want.index_add(0, row, y)
        size = size.index_add(0, row, (act.abs() @ down[e].double().abs().t()) * (1.0 if scale_input else w))
    rt = Runtime(torch.device(DEV), torch.bfloat16, ops16, n)
    got, before = hidden.clone(), ops16.launches
    ops16.experts_forward(x, gate if form == "gated" else None, up, down, chosen.int().flatten(), weight.flatten(), top, scale_input,
                          got, rt)
    assert ops16.launches - before == 5                 # grouping, the rows in order, two products, the sum over a token's experts
    # a projection near a rounding boundary may fall on its other side: 2^-8 of it, through silu and a product of two, twice;
    # the activation's own rounding likewise
    assert ((got.double() - want).abs() <= 3 * 2.0 ** -8 * size + 1e-6).all()
    assert (got.double() - want).norm() <= 1e-3 * (want - hidden.double()).norm()
    # which other tokens are in the step does not change a token's bits while the form is the same
    part = hidden.clone()[: n // 2 + 1]
    m = part.shape[0]
    ops16.experts_forward(x[:m], gate if form == "gated" else None, up, down, chosen[:m].int().flatten().contiguous(),
                          weight[:m].flatten().contiguous(), top, scale_input, part, rt)
    assert m * top >= experts and torch.equal(part, got[:m])
    # fewer pairs than experts: the mma.sync form, whose sums over k are grouped differently; a projection near a rounding
    # boundary may fall on its other side
    if top < experts:
        alone = hidden[:1].clone()
        ops16.experts_forward(x[:1], gate if form == "gated" else None, up, down, chosen[:1].int().flatten().contiguous(),
                              weight[:1].flatten().contiguous(), top, scale_input, alone, rt)
        assert (alone - got[:1]).norm() <= 2e-3 * (got[:1] - hidden[:1]).norm()
