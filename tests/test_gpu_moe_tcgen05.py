"""The experts' products of prompts on tcgen05 tiles of 128 rows: lists with empty experts, full and nearly full tiles and identity
pairs, inner sizes that fill no tile, every gated unit, rows placed by list and by pair, each against 64-bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def units(gate, up, act, limit, alpha):
    if act == "clamped_swish":
        g, u = gate.clamp(max=limit), up.clamp(-limit, limit)
        return g * torch.sigmoid(alpha * g) * (u + 1.0)
    return torch.nn.functional.gelu(gate, approximate="tanh") * up if act.startswith("gelu") else gate * torch.sigmoid(gate) * up


@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "clamped_swish"])
@pytest.mark.parametrize("counts,identity", [([0, 128, 129, 1], 40), ([300], 0), ([7, 0, 0, 255, 256, 3], 9)])
@pytest.mark.parametrize("width,inner", [(72, 40), (128, 264), (520, 128)])
def test_against_64_bit(act, counts, identity, width, inner):
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(width + len(counts))
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    n = len(counts)
    chosen = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)] + [torch.full((identity,), n + 1)])
    top = 1 if len(chosen) % 2 else 2
    chosen = chosen[torch.randperm(len(chosen), generator=torch.Generator().manual_seed(2))].to(torch.int32).view(-1, top).cuda()
    tokens = chosen.shape[0]
    h = make(tokens, width).bfloat16()
    w_up, w_down = (make(n, 2 * inner, width) * width ** -0.5 * 2).bfloat16(), (make(n, width, inner) * inner ** -0.5).bfloat16()
    lists = K.moe_sort(chosen, n, torch.bfloat16, 128)
    got = K.moe_tcgen05(K.moe_gather(h, lists), w_up, lists, act, False, torch.bfloat16, 1.5, 1.702)
    y = K.moe_tcgen05(got, w_down, lists, None, True, torch.float32)
    listed = int(lists.offsets[-1])
    assert listed == sum(counts)
    order = lists.order[:listed].long()
    expert = chosen.view(-1)[order].long()
    both = torch.einsum("pk,pnk->pn", h[order // top].double(), w_up[expert].double())
    want = units(both[:, :inner], both[:, inner:], act, 1.5, 1.702)
    # rounded to bfloat16 (2^-8 of the value at most) from 32-bit sums
    assert ((got[:listed].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()
    back = torch.einsum("pk,pnk->pn", got[:listed].double(), w_down[expert].double())
    assert (y[order].double() - back).abs().max() <= 1e-5 * back.abs().max()
    K.check_async_errors()


@pytest.mark.parametrize("counts,identity", [([0, 32, 1, 7], 5), ([33], 0), ([3, 0, 65], 1)])
@pytest.mark.parametrize("width,n", [(72, 40), (256, 136), (520, 128)])
def test_few_rows_against_64_bit(counts, identity, width, n):
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(width + n)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    experts = len(counts)
    chosen = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)] + [torch.full((identity,), experts)])
    chosen = chosen[torch.randperm(len(chosen), generator=torch.Generator().manual_seed(2))].to(torch.int32).view(-1, 1).cuda()
    h, w = make(chosen.shape[0], width).bfloat16(), make(experts, n, width).bfloat16()
    lists = K.moe_sort(chosen, experts, torch.bfloat16, 32)
    rows = K.moe_gather(h, lists)
    listed = int(lists.offsets[-1])
    order = lists.order[:listed].long()
    want = torch.einsum("pk,pnk->pn", h[order].double(), w[chosen.view(-1)[order].long()].double())
    for by_pair in (False, True):
        got = K.moe_skinny(rows, w, lists, by_pair)
        assert ((got[order] if by_pair else got[:listed]).double() - want).abs().max() <= 1e-5 * want.abs().max()      # 32-bit sums
    K.check_async_errors()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("scoring", ["sigmoid", "softmax", "softmax_chosen"])
def test_the_router_by_rows_and_a_row_a_block(dtype, scoring):
    """The router of a long prompt (512 rows and more) takes eight rows a block: the same choices and weights as the rows one decoding step at a time."""
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(5)
    h, router = torch.randn(531, 516, device="cuda", generator=gen).to(dtype), torch.randn(19, 516, device="cuda", generator=gen) * 0.1
    correction = torch.randn(19, device="cuda", generator=gen) * 0.1
    experts, weights = K.moe_route(h, router, correction, 5, 1, 1, 1, scoring, True, 1.5)
    for at in range(0, 531, 40):
        e, w = K.moe_route(h[at : at + 40].contiguous(), router, correction, 5, 1, 1, 1, scoring, True, 1.5)
        assert torch.equal(e, experts[at : at + 40]) and torch.equal(w, weights[at : at + 40])


def test_the_bounded_unit_keeps_the_librarys_exponential():
    """Rows that pick one weight each, so that the products are exact and the unit's own error shows."""
    from kapel_b200 import kernels as K

    width, inner = 160, 8
    gate = -0.25 * torch.arange(width, device="cuda", dtype=torch.float32)[None, :] - torch.arange(inner, device="cuda")[:, None] * 0.25
    w = torch.cat([gate, torch.full((inner, width), 0.5, device="cuda")])[None].bfloat16()
    h = torch.eye(width, device="cuda").bfloat16()
    lists = K.moe_sort(torch.zeros((width, 1), dtype=torch.int32, device="cuda"), 1, torch.bfloat16, 128)
    got = K.moe_tcgen05(K.moe_gather(h, lists), w, lists, "clamped_swish", False, torch.float32, 50.0, 1.0)
    g = gate.T[lists.order[:width].long()].double()
    want = g * torch.sigmoid(g) * 1.5
    # an exponential within an ulp, a sum, a quotient and a product: 4 roundings of 2^-24 and that ulp
    assert ((got.double() - want).abs() <= 6.0 * 2.0 ** -24 * want.abs()).all()
