"""Kernels of a decoding step's few rows and of a pass's first: latent layers' per-head products, the delta rule's inputs at other head sizes, the embedding."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 8, 16])
@pytest.mark.parametrize("heads,n_in,n_out,tail", [(3, 128, 65, 4), (2, 33, 8, 0), (1, 20, 3, 2), (2, 520, 70, 0), (2, 1028, 16, 0)])
def test_per_head_products(rows, heads, n_in, n_out, tail):
    """Columns and inputs that fill no tile, more inputs than a lane holds at once; 32-bit inputs (whole and in slices) and bfloat16 ones."""
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(n_in + rows)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)
    m = rand(heads, n_out, n_in).bfloat16()
    slices = rand(3, rows, heads * (n_in + tail))
    gate, cs = rand(rows, heads * n_out + 5), rand(rows, tail // 2, 2)
    for x in (K.SplitSum(slices), slices[0].contiguous(), slices[1].bfloat16()):
        whole = x.partials.double().sum(0) if isinstance(x, K.SplitSum) else x.double()
        whole = whole.view(rows, heads, n_in + tail)
        want = torch.einsum("rhi,hoi->rho", whole[..., :n_in], m.double())
        sizes = torch.einsum("rhi,hoi->rho", whole[..., :n_in].abs(), m.double().abs())
        for gated in (False, True):
            kw = {"gate": gate, "g_off": 5} if gated else {"tail_off": n_in, "tail": tail, "cos_sin": cs} if tail else {}
            y = K.head_linear(x, heads, n_in + tail, 0, m, pad_to=heads * (n_out + (tail if not gated else 0)) + 3, transposed=True, **kw)
            assert (y[:, -3:] == 0).all()
            got = y[:, :-3].reshape(rows, heads, -1)[..., :n_out].double()
            factor = torch.sigmoid(gate[:, 5:].double()).view(rows, heads, n_out) if gated else 1.0
            # bfloat16's rounding of the result, and 32-bit sums (round towards zero, n_in / 16 additions a piece)
            assert ((got - want * factor).abs() <= 2.0 ** -8 * (want * factor).abs() + n_in / 16 * 2.0 ** -22 * sizes + 1e-30).all()
    if n_in >= 32:                                           # infinity is infinity, not the difference of two
        x = slices[0].clone()
        x[0, 5] = float("inf")
        y = K.head_linear(x, heads, n_in + tail, 0, m, transposed=True)[0].reshape(heads, -1)[:, :n_out].float()
        assert torch.equal(y[0], torch.where(m[0, :, 5] > 0, float("inf"), -float("inf")).float()) and torch.isfinite(y[1:]).all()


@pytest.mark.parametrize("H,G,d,e", [(2, 1, 128, 20), (3, 3, 160, 4), (2, 2, 256, 12), (4, 2, 64, 132)])
def test_delta_inputs_by_a_warp_a_head(H, G, d, e):
    """Head sizes of one to eight components a lane, values that fill no warp, requests that begin within a warp's rows: the same bits as the kernel of a row a
    block, which reads the columns one place further."""
    from kapel_b200 import kernels as K

    sizes, taps = (3, 70, 1, 2, 90), 4
    rows, n, nv = sum(sizes), G * d, H * e
    gen = torch.Generator(device="cuda").manual_seed(d)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)
    conv, a_log, dt_bias = rand(2 * n + nv, taps), rand(H), rand(H)
    entry = torch.tensor(np.repeat(np.arange(len(sizes)), sizes), dtype=torch.int32, device="cuda")
    slots = torch.tensor([1, 2, 0, 3, 4], dtype=torch.int32, device="cuda")
    ranges, start = K.entry_ranges(entry, len(sizes)), rand(5, K.delta_state_floats(H, G, d, e, taps)) * 0.1
    width = 2 * n + nv + 2 * H + (-(2 * n + nv + 2 * H)) % 4
    states = [start.clone(), start.clone()]
    x = rand(rows, width)
    shifted = torch.zeros(rows, width + 4, device="cuda")
    shifted[:, 1:-3] = x
    a, b = (K.delta_scan(src, off, off + n, off + 2 * n, off + 2 * n + nv, off + 2 * n + nv + H, conv, a_log, dt_bias, state, entry, ranges, slots,
                         len(sizes), H, G, d, e, taps, d ** -0.5, 1e-6) for src, off, state in ((x, 0, states[0]), (shifted, 1, states[1])))
    assert torch.equal(a, b) and torch.equal(states[0], states[1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [4, 2048, 2308, 2049])
def test_embedding(width, dtype):
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(width)
    table, places = (torch.randn(n, width, device="cuda", generator=gen).to(dtype) for n in (11, 5))
    ids = torch.tensor([0, 10, -1, 11, 7], dtype=torch.int32, device="cuda")
    positions = torch.tensor([0, 4, 1, 2, 5], dtype=torch.int32, device="cuda")
    for copies in (1, 4):
        got = K.embed(table, ids, 3.0, pos_table=places, positions=positions, copies=copies).view(5, copies, width)
        want = torch.stack([table[0].double() * 3 + places[0].double(), table[10].double() * 3 + places[4].double(), table[7].double() * 3])
        assert torch.isnan(got[2:4]).all()
        assert ((got[[0, 1, 4]].double() - want[:, None]).abs() <= 2.0 ** -23 * (want[:, None].abs() + 4.0)).all()


@pytest.mark.parametrize("rows,n", [(1, 4), (3, 1020), (65, 1024), (70, 1028), (500, 9216)])
@pytest.mark.parametrize("act", ["gelu_tanh", "silu"])
@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16])
def test_gated_unit_by_fours_and_one_by_one(rows, n, act, out):
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(rows, 2 * n, device="cuda", generator=gen) * 4
    beside = torch.empty(rows * 2 * n + 1, device="cuda")[1:].view(rows, 2 * n)      # begins off a 16-byte boundary: a value a thread
    beside.copy_(x)
    assert torch.equal(K.glu(x, act, out_dtype=out), K.glu(beside, act, out_dtype=out))


@pytest.mark.parametrize("rows", [1, 5, 16])
@pytest.mark.parametrize("n_in", [32, 128, 512, 2040, 2048, 2052, 2100, 4097, 13000])
def test_per_head_products_keep_32_bits(rows, n_in):
    """Pairs of inputs that differ by 2^-12 of their size, against each other: whatever the inner size nothing of an input is lost, on both sides of what lies in
    shared memory at once and of what a lane holds."""
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(n_in)
    m = torch.ones(2, 9, n_in, device="cuda").bfloat16()
    m[:, :, 1::2] = -1.0
    m[1, 3] *= 2.0
    big = torch.rand(rows, 2, n_in, device="cuda", generator=gen) + 1.0
    big[..., 1::2] = big[..., : n_in // 2 * 2 : 2] * (1.0 - 2.0 ** -12)
    if n_in % 2:
        big[..., -1] = 0.0
    want = torch.einsum("rhi,hoi->rho", big.double(), m.double())
    sizes = torch.einsum("rhi,hoi->rho", big.double(), m.double().abs())
    got = K.head_linear(big.reshape(rows, -1), 2, n_in, 0, m, transposed=True).view(rows, 2, 9).double()
    # bfloat16's rounding; of 32 inputs the last two additions are of full size and round towards zero (2^-23 of that sum each), those of the groups to nearest
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + (2.0 ** -22 / max(1, n_in // 32) + 2.0 ** -23 * 3) * sizes).all()


@pytest.mark.parametrize("rows", [1, 16])
@pytest.mark.parametrize("n_in", [33, 520, 2600])
def test_per_head_products_beyond_what_pieces_hold(rows, n_in):
    """Finite inputs that round to infinity in bfloat16, products beyond the largest float, infinities."""
    from kapel_b200 import kernels as K

    x, m = torch.zeros(rows, 3, n_in, device="cuda"), torch.zeros(3, 8, n_in, device="cuda").bfloat16()
    x[:, 0, 4], m[0, :, 4] = 3.4e38, 0.5
    x[-1, 1], m[1] = 2.0 ** 70 * 1.01, 2.0 ** 70
    m[1, 5] = -(2.0 ** 70)
    x[0, 2, 7], m[2, :, 7], m[2, 2, 7] = float("inf"), 1.0, -1.0
    y = K.head_linear(x.view(rows, -1), 3, n_in, 0, m, transposed=True).view(rows, 3, 8).float()
    assert torch.equal(y[:, 0], torch.full_like(y[:, 0], 1.7e38).bfloat16().float())
    signs = torch.ones(8, device="cuda")
    signs[5] = -1.0
    assert torch.equal(y[-1, 1], signs * float("inf"))
    signs = torch.ones(8, device="cuda")
    signs[2] = -1.0
    assert torch.equal(y[0, 2], signs * float("inf"))
    assert rows == 1 or bool((y[1:, 2] == 0).all() and (y[:-1, 1] == 0).all())


def test_per_head_products_of_the_smallest_inputs():
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(3, 2, 100, device="cuda", generator=gen) * 2.0 ** -60 * torch.tensor([2.0 ** -56, 2.0 ** -68, 2.0 ** -84], device="cuda")[:, None, None]
    m = (torch.randn(2, 16, 100, device="cuda", generator=gen) * 2.0 ** 100).bfloat16()
    want = torch.einsum("rhi,hoi->rho", x.double(), m.double())
    got = K.head_linear(x.view(3, -1), 2, 100, 0, m, transposed=True).view(3, 2, 16).double()
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -21 * torch.einsum("rhi,hoi->rho", x.double().abs(), m.double().abs())).all()
