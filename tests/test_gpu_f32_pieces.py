"""The 32-bit product by bfloat16 pieces on the tensor cores: against 64-bit and against the multiply-adds it stands in for, at the edges of its tiles,
chunks and segments; values that have no pieces; which products go that way."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def pieces(a, w, segments, cap=0.0):
    from kapel_b200 import kernels as K

    m, (n, k) = a.shape[0], w.shape
    lib, ptr = K.library(), lambda t: ctypes.c_void_p(t.data_ptr())
    guarded = torch.full((m + 2, n), 7.0, device="cuda")
    scratch = torch.full((m * (3 * ((k + 7) // 8 * 4) + 1),), float("nan"), device="cuda")
    assert lib.kb_gemm_f32_pieces(ptr(guarded[1:]), ptr(a), ptr(w), m, n, k, 1 if cap else 0, ctypes.c_float(cap), segments, ptr(scratch),
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0, lib.kb_last_error()
    assert (guarded[0] == 7.0).all() and (guarded[-1] == 7.0).all()
    return guarded[1:-1]


def chains(a, w):
    from kapel_b200 import kernels as K

    c, lib, ptr = torch.empty(a.shape[0], w.shape[0], device="cuda"), K.library(), lambda t: ctypes.c_void_p(t.data_ptr())
    assert lib.kb_gemm_f32(ptr(c), ptr(a), ptr(w), a.shape[0], w.shape[0], a.shape[1], 0, ctypes.c_float(0.0),
                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0, lib.kb_last_error()
    return c


@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 64, 65, 129, 300])
@pytest.mark.parametrize("n,k", [(1, 4), (127, 64), (128, 68), (513, 1028), (700, 2304)])
def test_against_64_bit_and_the_chains(m, n, k):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda", generator=gen) * torch.exp2(torch.randint(-8, 9, (m, k), device="cuda", generator=gen).float())
    w = torch.randn(n, k, device="cuda", generator=gen)
    want, sizes, by_chains = a.double() @ w.double().T, a.abs().double() @ w.abs().double().T, chains(a, w)
    off = float((by_chains - want).norm())
    for segments in (1, 2, 4, 8):                            # 17 chunks of 64 k by eight: the last two segments are empty
        got = pieces(a, w, segments)
        # a chunk's four large additions round towards zero, 2^-23 each at most, the chunks' additions to nearest
        assert ((got - want).abs() <= (4 * 2.0 ** -23 + (k // 64 + 2) * 2.0 ** -24) * sizes + 1e-30).all()
        if k >= 1024:
            assert float((got - want).norm()) <= 0.5 * off
        capped = pieces(a, w, segments, 5.0)
        assert (capped.double() - 5.0 * torch.tanh(got.double() / 5.0)).abs().max() <= 5.0 * 2.0 ** -21
        few = min(m, 5)                                      # a row does not depend on the others, nor on the kernel's width
        assert torch.equal(pieces(a[:few].contiguous(), w, segments), got[:few])


def test_values_without_pieces():
    gen = torch.Generator(device="cuda").manual_seed(2)
    for m in (20, 200):
        a, w = torch.randn(m, 1100, device="cuda", generator=gen), torch.randn(600, 1100, device="cuda", generator=gen)
        a[3, 5], a[7, 1099], a[9, 0], a[m - 1, 700] = float("inf"), float("nan"), 3.4e38, -float("inf")
        # 3.4e38 rounds to infinity in bfloat16. One such value a dot product: whether the sum of two that nearly cancel overflows on its way is a
        # matter of the order, 0.9 X - 1.2 X is finite in one chain, and -1.2 X alone in its segment is not
        w[11, 0], w[599, 1000] = -float("inf"), float("nan")
        want = chains(a, w)
        for segments in (1, 4):
            got = pieces(a, w, segments)
            assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
            known = torch.isfinite(want)
            assert torch.equal(got[want.isinf()], want[want.isinf()])
            assert ((got - want)[known].abs() <= 1100 * 2.0 ** -23 * (a.abs().double() @ w.abs().double().T)[known]).all()


def test_which_products_go_that_way():
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(3)
    flat, w = torch.randn(40 * 1024 + 1, device="cuda", generator=gen), torch.randn(2048, 1024, device="cuda", generator=gen)
    a, shifted = flat[:-1].view(40, 1024), flat[1:].view(40, 1024)
    by_pieces = [m for m in (1, 2, 3, 8, 33, 40) if not torch.equal(K.gemm(a[:m], w), chains(a[:m], w))]
    assert by_pieces == [3, 8, 33, 40]
    assert torch.equal(K.gemm(shifted, w), chains(shifted, w))                 # rows that do not begin at 16-byte boundaries
    shorter = lambda t, k: t[:, :k].contiguous()
    by_pieces = [(m, k) for m in (16, 17) for k in (252, 256, 1020, 1024) if not torch.equal(K.gemm(shorter(a[:m], k), shorter(w, k)), chains(shorter(a[:m], k), shorter(w, k)))]
    assert by_pieces == [(16, 1024), (17, 256), (17, 1020), (17, 1024)]
    got, want = K.gemm(a, w, softcap=30.0).double(), 30.0 * torch.tanh(a.double() @ w.double().T / 30.0)
    assert (got - want).abs().max() <= 1e-4
    K.check_async_errors()
