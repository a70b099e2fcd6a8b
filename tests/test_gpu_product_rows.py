"""The tcgen05 products of many rows store their tiles a row's neighbouring columns at a time: whole numbers small enough that every sum is
exact, at rows and columns around the edges of tiles and of the 32 columns stored together; nothing outside the result is written."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("m,n,k", [(1, 32, 8), (129, 31, 72), (128, 36, 64), (257, 256, 200), (300, 296, 64), (70, 544, 136), (513, 290, 64)])
def test_edges(dtype, kernel, m, n, k):
    from kapel_b200 import kernels as K

    g = torch.Generator(device="cuda").manual_seed(m + n)
    a, w = (torch.randint(-2, 3, s, device="cuda", generator=g).to(torch.bfloat16) for s in ((m, k), (n, k)))
    buf = torch.full((m + 2, n), float("nan"), dtype=dtype, device="cuda")
    point = lambda t: ctypes.c_void_p(t.data_ptr())
    lib = K.library()
    if n * buf.element_size() % 16 == 0:
        c = buf[1 : m + 1]
    else:                                                    # the result starts on 16 bytes
        c = buf[:m]
    assert lib.kb_gemm_tcgen05(point(c), K._CODES[dtype], point(a), point(w), m, n, k, 0, ctypes.c_float(0.0), kernel,
                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want = (a.float() @ w.float().T).to(dtype)               # |sum| <= 4 k = 800: exact in 32-bit
    assert torch.equal(c, want)
    assert int(torch.isnan(buf).sum()) == 2 * n and lib.kb_tcgen05_error() == 0
