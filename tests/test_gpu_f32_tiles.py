"""The 32-bit attention by tiles of rows against 64-bit and against the row-wise kernel: windows, soft caps, sinks, several requests, keys at
the borders of tiles and pages."""
import pytest
import torch

from test_gpu_flash import cut

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("portions", [[(0, 16), (0, 65)], [(0, 63), (64, 17)], [(129, 40), (0, 130), (500, 16)]])
@pytest.mark.parametrize("hq,hkv,d,window,cap", [(2, 2, 128, None, None), (8, 4, 256, None, 50.0), (8, 2, 128, 70, None), (3, 1, 256, 64, 5.0)])
@pytest.mark.parametrize("sink", [False, True])
def test_against_64_bit_and_by_rows(portions, hq, hkv, d, window, cap, sink):
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(6)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    longest = max(b + n for b, n in portions)
    width = -(-longest // 16)
    order = torch.randperm(width * len(portions) + 2, generator=torch.Generator().manual_seed(1))
    k_table, v_table = (torch.full((len(order), hkv, 16, d), float("nan"), device="cuda") for _ in range(2))
    table = torch.full((len(portions), width + 1), -1, dtype=torch.int32)
    rows = sum(n for _, n in portions)
    q, sinks = make(rows, hq, d) * 2, (make(hq) * 2 if sink else None)
    counts, want, entries, at = [], [], [], 0
    for e, (before, n) in enumerate(portions):
        T = before + n
        k, v = make(T, hkv, d), make(T, hkv, d)
        k[T // 2] *= 4.0
        for pg in range(-(-T // 16)):
            where = int(order[e * width + pg])
            table[e, pg] = where
            m = min(16, T - pg * 16)
            k_table[where, :, :m] = k[pg * 16 : pg * 16 + m].transpose(0, 1)
            v_table[where, :, :m] = v[pg * 16 : pg * 16 + m].transpose(0, 1)
        s = torch.einsum("nhd,thd->hnt", q[at : at + n].double(), k.double().repeat_interleave(hq // hkv, 1)) * d ** -0.5
        s = cap * torch.tanh(s / cap) if cap else s
        count, t = torch.arange(before + 1, T + 1, device="cuda")[:, None], torch.arange(T, device="cuda")[None, :]
        s = s.masked_fill(~((t < count) & (t >= (count - window if window else 0)))[None], -torch.inf)
        if sink:
            s = torch.cat([s, sinks.double()[:, None, None].expand(hq, n, 1)], 2)
        want.append(torch.einsum("hnt,thd->nhd", torch.softmax(s, -1)[..., :T], v.double().repeat_interleave(hq // hkv, 1)))
        counts += list(range(before + 1, T + 1))
        entries += [e] * n
        at += n
    args = (q, k_table, v_table, table.cuda(), torch.tensor(entries, dtype=torch.int32, device="cuda"), torch.tensor(counts, dtype=torch.int32, device="cuda"),
            16, window, d ** -0.5, cap, longest // K.attention_chunk() + 2)
    want = torch.cat(want)
    by_rows, by_tiles = K.paged_attention_rows(*args, sinks=sinks), K.paged_attention_rows(*args, sinks=sinks, tiles=cut(portions, 32 // (hq // hkv)))
    off = lambda x: float((x.double() - want).abs().max() / want.abs().max())
    # products of d terms and sums of up to 630 weights in 32-bit; a score of 30 moves by 2^-19 when it is rounded
    assert off(by_tiles) <= 1e-5 and off(by_tiles) <= 3.0 * off(by_rows) + 1e-6, (off(by_tiles), off(by_rows))


@pytest.mark.parametrize("window", [None, 40])
@pytest.mark.parametrize("hq,hkv,d", [(4, 2, 256), (8, 2, 128)])
def test_what_a_row_does_not_see_does_not_reach_it(hq, hkv, d, window):
    """Values that are no finite numbers reach the rows that see them and no other, and a key without a page is seen by nobody: as row by row."""
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(8)
    before, n = 70, 60
    T = before + n
    width = -(-T // 16)
    k_table, v_table = (torch.randn(width, hkv, 16, d, device="cuda", generator=gen) for _ in range(2))
    at = lambda t: (t // 16, slice(None), t % 16)
    v_table[at(100)] = float("nan")
    v_table[at(111)] = float("inf")
    v_table[at(5)] = float("nan")                            # below the window; without one every row sees it
    k_table[at(120)] = float("nan")
    if window is None:
        v_table[at(5)] = 1.0
    table = torch.arange(width, dtype=torch.int32, device="cuda")[None].contiguous()
    table[0, 3] = -1                                         # positions 48 to 63
    q = torch.randn(n, hq, d, device="cuda", generator=gen)
    counts = torch.arange(before + 1, T + 1, dtype=torch.int32, device="cuda")
    args = (q, k_table, v_table, table, torch.zeros(n, dtype=torch.int32, device="cuda"), counts, 16, window, d ** -0.5, None, T // K.attention_chunk() + 2)
    by_rows, by_tiles = K.paged_attention_rows(*args), K.paged_attention_rows(*args, tiles=cut([(before, n)], 32 // (hq // hkv)))
    seen = counts > 100                                      # these rows see position 100
    assert torch.isfinite(by_rows[~seen]).all() and not torch.isfinite(by_rows[seen]).any()
    assert torch.equal(torch.isfinite(by_rows), torch.isfinite(by_tiles))
    # sums of at most 100 weights in 32-bit, in another order
    assert (by_rows - by_tiles)[~seen].abs().max() <= 1e-5 * by_rows[~seen].abs().max()


@pytest.mark.parametrize("hq,hkv,d,cap", [(8, 4, 256, 50.0), (16, 4, 128, None)])
@pytest.mark.parametrize("before,n,peak", [(0, 500, 1.0), (2500, 96, 1.0), (2500, 96, 4.0)])
def test_as_near_to_64_bit_as_row_by_row(hq, hkv, d, cap, before, n, peak):
    """The 2-norm of the error: short chains of products and of keys, as the row-wise kernel's lanes and chunks have them."""
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(9)
    T = before + n
    width = -(-T // 16)
    k_table, v_table = (torch.randn(width, hkv, 16, d, device="cuda", generator=gen) for _ in range(2))
    k, v = (t.transpose(1, 2).reshape(width * 16, hkv, d)[:T].double().repeat_interleave(hq // hkv, 1) for t in (k_table, v_table))
    q = torch.randn(n, hq, d, device="cuda", generator=gen) * peak
    counts = torch.arange(before + 1, T + 1, dtype=torch.int32, device="cuda")
    s = torch.einsum("nhd,thd->hnt", q.double(), k) * d ** -0.5
    s = cap * torch.tanh(s / cap) if cap else s
    s = s.masked_fill((torch.arange(T, device="cuda")[None, :] >= counts[:, None])[None], -torch.inf)
    want = torch.einsum("hnt,thd->nhd", torch.softmax(s, -1), v)
    args = (q, k_table, v_table, torch.arange(width, dtype=torch.int32, device="cuda")[None].contiguous(), torch.zeros(n, dtype=torch.int32, device="cuda"),
            counts, 16, None, d ** -0.5, cap, -(-T // K.attention_chunk()))
    off = [float((K.paged_attention_rows(*args, tiles=t).double() - want).norm() / want.norm()) for t in (None, cut([(before, n)], 32 // (hq // hkv)))]
    assert off[1] <= 1.03 * off[0], off                      # 190,000 results and more: the norms of two random errors of one size agree to 1 %


@pytest.mark.parametrize("hq,hkv,d,at_once", [(8, 4, 256, 1), (16, 4, 128, 2)])
@pytest.mark.parametrize("more,window", [(0, None), (1, None), (0, 600), (0, 100), (1, 100)])
def test_on_both_sides_of_two_blocks_a_tile(hq, hkv, d, at_once, more, window):
    """Up to a wave of tiles two blocks take one, every second step of 64 keys each; the first tiles have one step, so that the second has none."""
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(10)
    per = 32 // (hq // hkv)
    n = at_once * torch.cuda.get_device_properties(0).multi_processor_count // hkv * per + more
    width = -(-n // 16)
    k_table, v_table = (torch.randn(width, hkv, 16, d, device="cuda", generator=gen) for _ in range(2))
    q = torch.randn(n, hq, d, device="cuda", generator=gen)
    counts = torch.arange(1, n + 1, dtype=torch.int32, device="cuda")
    args = (q, k_table, v_table, torch.arange(width, dtype=torch.int32, device="cuda")[None].contiguous(), torch.zeros(n, dtype=torch.int32, device="cuda"),
            counts, 16, window, d ** -0.5, 50.0, -(-n // K.attention_chunk()) + 1)
    by_rows, by_tiles = K.paged_attention_rows(*args), K.paged_attention_rows(*args, tiles=cut([(0, n)], per))
    # sums of up to 600 weights in 32-bit in another order; each side is within 1e-5 of 64 bits (above)
    assert (by_rows - by_tiles).abs().max() <= 2e-5 * by_rows.abs().max()


def test_the_merge_of_many_slots_does_not_depend_on_the_batch():
    """More slots of keys than a merging block of 128 threads has threads: a row alone and among many others, whose blocks have another size."""
    from kapel_b200 import kernels as K

    T, d = 256 * 140, 256
    gen = torch.Generator(device="cuda").manual_seed(11)
    k_table, v_table = (torch.randn(T // 16, 1, 16, d, device="cuda", generator=gen) for _ in range(2))
    q, rows = torch.randn(1, 1, d, device="cuda", generator=gen), 700
    table, ints = torch.arange(T // 16, dtype=torch.int32, device="cuda")[None].contiguous(), lambda v, n: torch.full((n,), v, dtype=torch.int32, device="cuda")
    alone, beside = (K.paged_attention_rows(q.expand(n, 1, d).contiguous(), k_table, v_table, table, ints(0, n), ints(T, n), 16, None, d ** -0.5, None,
                                            T // K.attention_chunk()) for n in (1, rows))
    assert torch.equal(beside, alone.expand(rows, 1, d))
