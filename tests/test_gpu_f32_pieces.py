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


BESIDE, WHOLE, APART = 0, 1, 2


def by_way(a, w, groups, way, cap=0.0):
    from kapel_b200 import kernels as K

    m, (n, k) = a.shape[0], w.shape
    lib, ptr = K.library(), lambda t: ctypes.c_void_p(t.data_ptr())
    guarded = torch.full((m + 2, n), 7.0, device="cuda")
    floats = m * 3 * ((k + 7) // 8 * 4) + groups * m * n
    scratch = torch.full((floats + n,), float("nan"), device="cuda")
    assert lib.kb_gemm_f32_pieces_by(ptr(guarded[1:]), ptr(a), ptr(w), m, n, k, 1 if cap else 0, ctypes.c_float(cap), groups, way, ptr(scratch),
                                     ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0, lib.kb_last_error()
    assert (guarded[0] == 7.0).all() and (guarded[-1] == 7.0).all() and torch.isnan(scratch[floats:]).all()
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
    assert not any(torch.equal(K.gemm(a[:m], w), chains(a[:m], w)) for m in (1, 2, 3, 8, 33, 40))
    assert torch.equal(K.gemm(shifted, w), chains(shifted, w))                 # rows that do not begin at 16-byte boundaries
    shorter = lambda t, k: t[:, :k].contiguous()
    by_pieces = [(m, k) for m in (1, 16, 17) for k in (252, 256, 257, 1024) if not torch.equal(K.gemm(shorter(a[:m], k), shorter(w, k)), chains(shorter(a[:m], k), shorter(w, k)))]
    assert by_pieces == [(m, k) for m in (1, 16, 17) for k in (256, 1024)]     # by the inner size alone: a row's bits do not depend on the batch
    got, want = K.gemm(a, w, softcap=30.0).double(), 30.0 * torch.tanh(a.double() @ w.double().T / 30.0)
    assert (got - want).abs().max() <= 1e-4
    K.check_async_errors()


@pytest.mark.parametrize("tokens,top,experts,n,k", [(1, 1, 3, 130, 256), (9, 4, 5, 128, 1028), (150, 2, 4, 300, 512), (70, 3, 20, 64, 260)])
def test_experts_products(tokens, top, experts, n, k):
    """By lists of rows with gaps (experts without rows, pairs of no expert) against 64-bit and against the multiply-adds, rows by token and by place."""
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(tokens)
    chosen = torch.randint(0, experts + 2, (tokens, top), device="cuda", generator=gen, dtype=torch.int32)     # the last two have no weights
    if experts > 3:
        chosen[chosen == 1] = 2
    a, w = torch.randn(tokens, k, device="cuda", generator=gen), torch.randn(experts, n, k, device="cuda", generator=gen)
    a[tokens // 2, 3] = float("inf")
    lists = K.moe_sort(chosen, experts, torch.float32)
    pairs = (chosen.reshape(-1) < experts).nonzero()[:, 0]
    rows, which = pairs // top, chosen.reshape(-1)[pairs].long()
    want = torch.einsum("pk,pnk->pn", a[rows].double(), w[which].double())
    sizes = torch.einsum("pk,pnk->pn", a[rows].abs().double(), w[which].abs().double())
    got = K.moe_grouped(a, w, lists, "none", True, True, torch.float32)[pairs]
    known = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), known)
    assert ((got - want)[known].abs() <= ((4 * 2.0 ** -23 + (k // 64 + 2) * 2.0 ** -24) * sizes)[known]).all()
    by_place = K.moe_grouped(a, w, lists, "none", True, False, torch.float32)
    listed = int(lists.offsets[-1])
    order = lists.order[:listed].long()
    where = torch.empty(tokens * top, dtype=torch.long, device="cuda")
    where[order] = torch.arange(listed, device="cuda")
    assert torch.equal(torch.nan_to_num(by_place[where[pairs]]), torch.nan_to_num(got))
    # the second product: rows by place in, rows by pair out
    back = torch.randn(experts, 36, n // 4 * 4, device="cuda", generator=gen)
    inner = torch.nan_to_num(by_place[:, : n // 4 * 4], 0.0, 0.0, 0.0).contiguous()
    out = K.moe_grouped(inner, back, lists, "none", False, True, torch.float32)[pairs]
    want = torch.einsum("pk,pnk->pn", inner[where[pairs]].double(), back[which].double())
    assert float((out - want).norm()) <= 1e-6 * float(want.norm())
    K.check_async_errors()


@pytest.mark.parametrize("tokens,width,top", [(1, 4, 1), (33, 2048, 4), (513, 12, 5), (7, 7, 3)])
def test_experts_sum_by_fours_and_one_by_one(tokens, width, top):
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(width)
    y, weights = torch.randn(tokens * top, width, device="cuda", generator=gen), torch.rand(tokens, top, device="cuda", generator=gen)
    own, also = torch.randn(tokens, width, device="cuda", generator=gen), torch.randn(tokens, width, device="cuda", generator=gen)
    experts = torch.randint(0, 6, (tokens, top), device="cuda", generator=gen, dtype=torch.int32)
    pad = lambda t: torch.cat([torch.zeros(1, device="cuda"), t.reshape(-1)])[1:].view(t.shape)                # one element further: not by fours
    for kw in ({}, {"experts": experts, "real": 4, "own": own}):
        for extra in (None, also):
            a = K.moe_combine(y, weights, torch.float32, also=extra, **kw)
            b = K.moe_combine(pad(y), weights, torch.float32, also=extra, **kw)
            assert torch.equal(a, b)


@pytest.mark.parametrize("m,more,k", [(33, 0, 260), (64, 1, 256), (65, 5, 256), (300, 300, 324), (500, 1, 1028)])
def test_blocks_that_walk_over_tiles(m, more, k):
    """More tiles of 128 weight rows than multiprocessors: every block takes several, and the results are a tile's own, rows without pieces included."""
    gen = torch.Generator(device="cuda").manual_seed(m)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = -(-sms // -(-m // (64 if m <= 64 else 128))) * 128 + more + 128
    a, w = torch.randn(m, k, device="cuda", generator=gen), torch.randn(n, k, device="cuda", generator=gen)
    for odd in (False, True):
        if odd:
            a[m - 1, k - 1], a[2, 0] = float("inf"), float("nan")
            w[n - 1, 3], w[130, 7], w[n // 2, k - 2] = -float("inf"), float("nan"), 3.4e38
        got = pieces(a, w, 1, 5.0 if m == 65 else 0.0)
        for n0 in range(0, n, 4096):                         # few tiles: a block has one
            assert torch.equal(torch.nan_to_num(got[:, n0 : n0 + 4096], nan=1e30),
                               torch.nan_to_num(pieces(a, w[n0 : n0 + 4096].contiguous(), 1, 5.0 if m == 65 else 0.0), nan=1e30))
        if not odd and m != 65:
            want, sizes = a.double() @ w.double().T, a.abs().double() @ w.abs().double().T
            assert ((got - want).abs() <= (4 * 2.0 ** -23 + (k // 64 + 2) * 2.0 ** -24) * sizes + 1e-30).all()      # as above


def overflowing(m, n, k, gen):
    """Finite values some of whose products are beyond the largest float, or so near it that the product of their first pieces is."""
    a, w = torch.randn(m, k, device="cuda", generator=gen), torch.randn(n, k, device="cuda", generator=gen)
    a[3] = 2.0 ** 70 * (1 + torch.rand(k, device="cuda", generator=gen))
    a[7] = -a[3]
    w[11] = 2.0 ** 75 * (1 + torch.rand(k, device="cuda", generator=gen))
    w[n - 1] = -w[11]
    a[9], w[20] = 0.0, 0.0                                   # one product each that is the largest float less 2^-9 of it
    a[9, 4], w[20, 4] = 2.0 ** 64 * (1 - 2.0 ** -10), 2.0 ** 64 * (1 - 2.0 ** -10)
    a[m - 1], w[21] = a[9], w[20]
    return a, w


@pytest.mark.parametrize("m,n", [(20, 600), (50, 600), (200, 600), (200, 9700)])
@pytest.mark.parametrize("cap", [0.0, 5.0])
def test_finite_values_whose_products_overflow(m, n, cap):
    """What is no finite number by pieces is what the multiply-adds make of it: infinities with their signs, under a soft cap the cap, and the
    finite products next to the largest float."""
    k = 260
    a, w = overflowing(m, n, k, torch.Generator(device="cuda").manual_seed(m + n))
    want = chains(a, w)
    assert want[3, 11] == float("inf") and want[7, 11] == -float("inf") and torch.isfinite(want[9, 20]) and want[9, 20] > 3.3e38
    known = torch.isfinite(want)
    sizes = a.abs().double() @ w.abs().double().T
    for segments in (1, 4):
        got = pieces(a, w, segments, cap)
        if cap:
            far = want.abs() > 100 * cap                     # tanh is one there
            assert torch.equal(got[far], cap * torch.sign(want[far])) and not torch.isnan(got).any()
            continue
        assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[want.isinf()], want[want.isinf()])
        assert got[9, 20] == want[9, 20]
        assert ((got.double() - want.double()).abs() <= k * 2.0 ** -23 * sizes)[known].all()


def test_experts_products_that_overflow():
    from kapel_b200 import kernels as K

    a, flat = overflowing(40, 256, 260, torch.Generator(device="cuda").manual_seed(5))
    w = flat.view(2, 128, 260)
    lists = K.moe_sort(torch.arange(2, device="cuda", dtype=torch.int32).repeat(40, 1), 2, torch.float32)       # both experts for every token
    got = K.moe_grouped(a, w, lists, "none", True, True, torch.float32).view(40, 256)
    want = chains(a, flat)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[want.isinf()], want[want.isinf()])
    assert got[9, 20] == want[9, 20] and torch.isfinite(got[9, 20])


@pytest.mark.parametrize("n,k", [(1, 256), (130, 260), (512, 1024), (2048, 2304), (2304, 2048), (2304, 9216), (4096, 2304), (19072, 324)])
def test_a_row_does_not_depend_on_the_batch(n, k):
    """Bit for bit, through the entry point that models call, for every number of rows."""
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(n + k)
    a, w = torch.randn(1200, k, device="cuda", generator=gen), torch.randn(n, k, device="cuda", generator=gen)
    want = K.gemm(a[:500].contiguous(), w)
    for m in (1, 2, 3, 16, 17, 32, 33, 64, 65, 128, 129, 200, 300, 700, 1200):
        rows = min(m, 500)
        assert torch.equal(K.gemm(a[:m].contiguous(), w)[:rows], want[:rows]), m
    assert torch.equal(K.gemm(a[499:500].clone(), w), want[499:])
    K.check_async_errors()


@pytest.mark.parametrize("m,n,k", [(33, 1, 256), (64, 257, 1028), (65, 700, 324), (300, 513, 2304), (129, 9700, 260), (40, 19100, 1100)])
def test_the_groups_of_k_by_either_way(m, n, k):
    """Blocks beside each other, one block after another group, and sums that lie apart: the same bits, with what is no finite number, too."""
    for finite in (True, False):
        a, w = overflowing(m, max(n, 22), k, torch.Generator(device="cuda").manual_seed(m))
        w = w[:n].contiguous()
        if finite:
            a, w = a.clamp(-4.0, 4.0), w.clamp(-4.0, 4.0)
        else:
            a[m - 1, k - 1], w[n // 2, 3] = float("nan"), -float("inf")
        for groups in (1, 2, 4, 8):
            for cap in (0.0, 5.0):
                want = torch.nan_to_num(by_way(a, w, groups, BESIDE, cap), nan=1e30)
                for way in (WHOLE, APART):
                    assert torch.equal(torch.nan_to_num(by_way(a, w, groups, way, cap), nan=1e30), want), (groups, way, cap)


@pytest.mark.parametrize("m,n", [(5, 130), (50, 130), (200, 700), (200, 9700)])
def test_the_smallest_values(m, n):
    """Values down to the subnormal ones: rows of nothing else, against weights of every size, with the error that ordinary values have."""
    k = 260
    gen = torch.Generator(device="cuda").manual_seed(m)
    a, w = torch.randn(m, k, device="cuda", generator=gen), torch.randn(n, k, device="cuda", generator=gen)
    a[1], a[2], a[3], a[4] = a[1] * 2.0 ** -115, a[2] * 2.0 ** -126, a[3] * 2.0 ** -60 * 2.0 ** -74, a[4] * 2.0 ** -60 * 2.0 ** -88
    w[:50] *= 2.0 ** 100
    w[60:120] *= 2.0 ** -60
    want, sizes = a.double() @ w.double().T, a.abs().double() @ w.abs().double().T
    for groups in (1, 4):
        for way in (BESIDE, WHOLE, APART) if m > 32 else (BESIDE,):
            got = by_way(a, w, groups, way)
            # as in the first test; 2^-150: half of the smallest subnormal
            assert ((got - want).abs() <= (4 * 2.0 ** -23 + (k // 64 + 2) * 2.0 ** -24) * sizes + 2.0 ** -150).all(), (groups, way)


def test_scratch_is_bounded():
    """More rows than a launch's scratch has room for go by several; the last of one row."""
    from kapel_b200 import kernels as K

    k, n = 18432, 130
    at_once = (256 << 20) // (6 * k) // 128 * 128
    gen = torch.Generator(device="cuda").manual_seed(4)
    a, w = torch.randn(at_once + 1, k, device="cuda", generator=gen), torch.randn(n, k, device="cuda", generator=gen)
    lib, ptr = K.library(), lambda t: ctypes.c_void_p(t.data_ptr())
    for m in (at_once + 1, 1 << 20):
        assert lib.kb_gemm_f32_scratch_floats(ptr(a), ptr(w), m, n, k) * 4 <= 512 << 20
    got = K.gemm(a, w)
    for rows in (slice(0, 40), slice(at_once - 40, at_once), slice(at_once, at_once + 1)):
        assert torch.equal(got[rows], K.gemm(a[rows].clone(), w))


@pytest.mark.parametrize("k", [256, 260, 512, 1024])
@pytest.mark.parametrize("kind", ["random", "one sign", "left out", "left out, either sign"])
def test_no_larger_an_error_than_the_chains(kind, k):
    """From the shortest inner size on, where chains are short too; sums of one sign; values whose second and third pieces are as large as they can be, so that the
    three products that are left out are 2^-24 of every product, all of one sign."""
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(k)

    def values(rows):
        if kind == "random":
            return torch.randn(rows, k, device="cuda", generator=gen)
        if kind == "one sign":
            return torch.rand(rows, k, device="cuda", generator=gen) + 0.5
        x = (1.0 + 2.0 ** -8 - 2.0 ** -17) * torch.exp2(torch.randint(-3, 4, (rows, k), device="cuda", generator=gen).float())
        return x if kind == "left out" else x * (2.0 * torch.randint(0, 2, (rows, k), device="cuda", generator=gen) - 1.0)

    a, w = values(200), values(600)
    want = a.double() @ w.double().T
    off = [float((c.double() - want).norm() / want.norm()) for c in (K.gemm(a, w), chains(a, w))]
    assert off[0] <= 1.01 * off[1], off                      # 120,000 results: the norms of two errors of one size agree to 1 %
