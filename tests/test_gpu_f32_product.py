"""The 32-bit product: every kernel that can compute an element gives the same bits (one accumulator, ascending k), and is as near to
64-bit as such a sum can be."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def product(a, w, variant, cap):
    from kapel_b200 import kernels as K

    c = torch.full((a.shape[0], w.shape[0]), 7.0, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    lib = K.library()
    assert lib.kb_gemm_f32_variant(p(c), p(a), p(w), a.shape[0], w.shape[0], a.shape[1], 1 if cap else 0, ctypes.c_float(cap), variant,
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0, lib.kb_last_error()
    return c


@pytest.mark.parametrize("m", [1, 2, 3, 5, 9, 16, 17, 33, 65, 129])
@pytest.mark.parametrize("n,k", [(1, 1), (15, 4), (16, 16), (17, 127), (65, 128), (129, 129), (200, 516)])
def test_every_kernel_gives_the_same_bits(m, n, k):
    gen = torch.Generator(device="cuda").manual_seed(m * 1000 + n + k)
    whole_a, whole_w = (torch.randn(rows * k + 1, device="cuda", generator=gen) for rows in (m, n))
    for off in (0, 1):                                       # rows at 16-byte boundaries or not
        a, w = whole_a[off : off + m * k].view(m, k), whole_w[off : off + n * k].view(n, k)
        got = [product(a, w, v, 0.0) for v in range(0 if m <= 16 else 1, 6)]
        assert all(torch.equal(g, got[0]) for g in got[1:])
        assert torch.equal(product(a, w, -1, 0.0), got[0])
        # a sum of k products, each rounded once as it is added: k * 2^-24 of the sum of their sizes
        assert ((got[0].double() - a.double() @ w.double().T).abs() <= k * 2.0 ** -24 * (a.abs().double() @ w.abs().double().T) + 1e-30).all()
        capped = product(a, w, -1, 5.0)
        assert (capped.double() - 5.0 * torch.tanh(got[0].double() / 5.0)).abs().max() <= 5.0 * 2.0 ** -21
        if m > 1:                                            # a row does not depend on the others
            assert torch.equal(product(a[: m // 2].contiguous(), w, -1, 0.0), got[0][: m // 2])


def test_the_launchers_rules_ask_the_device():
    from kapel_b200 import kernels as K

    assert K.library().kb_multiprocessors() == torch.cuda.get_device_properties(0).multi_processor_count
