"""Residual += norm(branch), then the next norm, with rows in registers (bfloat16 weights and output): either norm centered or not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def norm(x, w, eps, center):
    c = x - x.mean(-1, keepdim=True) if center else x
    return c / torch.sqrt((c * c).mean(-1, keepdim=True) + eps) * w


@pytest.mark.parametrize("rows", [3, 70])
@pytest.mark.parametrize("width", [4, 8, 44, 2048, 8200, 16368])
@pytest.mark.parametrize("slices", [0, 1, 3, 20])
def test_against_64_bit(rows, width, slices):
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(width + slices)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    x, w1, w2 = make(rows, width) * 3 + 1.5, make(width).bfloat16(), make(width).bfloat16()
    if slices:                                               # split-K partial sums whose mean is far from zero
        parts = make(slices, rows, width) - 4.0
        b, branch = parts.double().sum(0), K.SplitSum(parts)
    else:
        branch = (make(rows, width) - 4.0).bfloat16()
        b = branch.double()
    for post, nxt in ((True, True), (True, False), (False, True)):
        res = x.clone()
        h = K.add_rmsnorm(res, branch, (w1, 1e-5, 0.0, post), (w2, 1e-6, 0.0, nxt), torch.bfloat16)
        want = x.double() + norm(b, w1.double(), 1e-5, post)
        want_h = norm(want, w2.double(), 1e-6, nxt)
        assert (res.double() - want).abs().max() <= 1e-5 * want.abs().max()           # 32-bit sums of up to 16,368 values
        assert (h.double() - want_h).abs().max() <= (2.0 ** -8 + 2e-5) * want_h.abs().max()
    K.check_async_errors()
