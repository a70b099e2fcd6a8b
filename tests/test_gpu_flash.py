"""The tcgen05 attention for scores without a bound: over the paged cache (windows, sinks, key slots) and over the dense keys and
values that latent attention makes of its lines, each against 64-bit; and latent attention's two paths against each other."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(q, k, v, first_count, scale, window, sinks):
    """q [n, H, d] of the rows that have seen first_count, first_count + 1, .. positions; k [T, G, d], v [T, G, e]: 64-bit."""
    n, H, _ = q.shape
    q, k, v = q.double(), k.double().repeat_interleave(H // k.shape[1], 1), v.double().repeat_interleave(H // v.shape[1], 1)
    s = torch.einsum("nhd,thd->hnt", q, k) * scale
    count = torch.arange(first_count, first_count + n, device=q.device)[:, None]
    t = torch.arange(k.shape[0], device=q.device)[None, :]
    seen = (t < count) & (t >= (count - window if window else 0))
    s = s.masked_fill(~seen[None], -torch.inf)
    top = s.max(-1, keepdim=True).values
    if sinks is not None:
        top = torch.maximum(top, sinks.double()[:, None, None])
    p = torch.exp(s - top)
    total = p.sum(-1, keepdim=True) + (torch.exp(sinks.double()[:, None, None] - top) if sinks is not None else 0.0)
    return torch.einsum("hnt,thd->nhd", p / total, v)


# A weight is rounded to bfloat16 (2^-9 of itself) and so is the result: 2^-8 of the largest value, and half as much again for the
# scores' own arithmetic (products of bfloat16 numbers, sums and exponentials in 32-bit).
def bound(v):
    return 1.5 * 2.0 ** -8 * float(v.abs().max())


def cut(portions, rows_a_tile):
    entry, row0, nq, at = [], [], [], 0
    for e, (_, n) in enumerate(portions):
        for a in range(0, n, rows_a_tile):
            entry.append(e), row0.append(at + a), nq.append(min(rows_a_tile, n - a))
        at += n
    return tuple(torch.tensor(x, dtype=torch.int32, device="cuda") for x in (entry, row0, nq))


@pytest.mark.parametrize("portions", [[(0, 1), (0, 127), (300, 5)], [(0, 128), (127, 2)], [(0, 129), (0, 385)], [(1000, 40), (0, 33)]])
@pytest.mark.parametrize("hq,hkv,d,window,split", [(4, 4, 64, None, 0), (8, 2, 128, None, 0), (8, 2, 128, 70, 0), (16, 1, 64, 200, 128), (8, 4, 128, None, 256)])
@pytest.mark.parametrize("sink", [False, True])
def test_paged(portions, hq, hkv, d, window, split, sink):
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(3)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    longest = max(b + n for b, n in portions)
    width = -(-longest // 16)
    pages = width * len(portions) + 3
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(1))
    k_table, v_table = (torch.full((pages, hkv, 16, d), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    table = torch.full((len(portions), width + 2), -1, dtype=torch.int32)
    q = make(sum(n for _, n in portions), hq, d).bfloat16()
    sinks = make(hq) * 2 if sink else None
    counts, want, at = [], [], 0
    for e, (before, n) in enumerate(portions):
        T = before + n
        k, v = make(T, hkv, d).bfloat16(), make(T, hkv, d).bfloat16()
        k[T // 2] *= 6.0                                     # a key that stands out, whichever slot or tile it falls into
        if before == 0 and n > 128:
            k[: T // 3] *= 0.01                              # the largest score rises late: the reference has to move
            k[-1] *= 8.0
        for pg in range(-(-T // 16)):
            where = int(order[e * width + pg])
            table[e, pg] = where
            m = min(16, T - pg * 16)
            k_table[where, :, :m] = k[pg * 16 : pg * 16 + m].transpose(0, 1)
            v_table[where, :, :m] = v[pg * 16 : pg * 16 + m].transpose(0, 1)
        want.append((reference(q[at : at + n], k, v, before + 1, d ** -0.5, window, sinks), bound(v)))
        counts += list(range(before + 1, T + 1))
        at += n
    slots = -(-longest // split) if split else 1
    got = K.paged_attention_mma(q, k_table, v_table, table.cuda(), torch.tensor(counts, dtype=torch.int32, device="cuda"), cut(portions, 128 // (hq // hkv)),
                                16, window, d ** -0.5, None, 0, split, slots, sinks=sinks, prompt_kernel="flash")
    at = 0
    for (_, n), (w, limit) in zip(portions, want):
        assert (got[at : at + n].double() - w).abs().max() <= limit
        at += n
    K.check_async_errors()


@pytest.mark.parametrize("portions", [[(0, 64)], [(0, 127), (5, 130)], [(513, 100), (0, 256), (127, 129)]])
@pytest.mark.parametrize("heads", [1, 3, 16])
def test_dense_heads(portions, heads):
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(4)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()
    lengths = [b + n for b, n in portions]
    base = np.cumsum(lengths) - lengths
    kv, rot_keys = make(sum(lengths), heads * 256), make(sum(lengths), 64)
    q = make(sum(n for _, n in portions), heads, 192)
    sinks = torch.randn(heads, device="cuda", generator=gen)
    counts = [c for b, n in portions for c in range(b + 1, b + n + 1)]
    got = K.latent_prompt(q, kv, rot_keys, torch.tensor(base, dtype=torch.int32, device="cuda"), torch.tensor(counts, dtype=torch.int32, device="cuda"),
                          cut(portions, 128), 192 ** -0.5, sinks, 128, 128)
    at = 0
    for (b, n), start, T in zip(portions, base, lengths):
        mine = kv[start : start + T]
        k = torch.cat([mine[:, : heads * 128].view(T, heads, 128), rot_keys[start : start + T, None].expand(T, heads, 64)], 2)
        v = mine[:, heads * 128 :].view(T, heads, 128)
        assert (got[at : at + n].double() - reference(q[at : at + n], k, v, b + 1, 192 ** -0.5, None, sinks)).abs().max() <= bound(v)
        at += n
    K.check_async_errors()


LATENT = {"architecture": "Kofutar", "vocab": 97, "width": 64, "norm": {"eps": 1e-5}, "layers": [
    {"type": "latent_attention", "mlp": None, "mixer": {"heads": 3, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 32, "kv_rank": 64,
                                                        "scale": 192 ** -0.5, "rot": {"base": 100.0, "dims": 64}}},
    {"type": "attention", "mlp": {"kind": "dense", "ff": 48}, "mixer": {"heads": 4, "kv_heads": 2, "dim": 64, "vdim": 64, "scale": 0.125,
                                                                       "rot": {"base": 100.0, "dims": 64}}}]}


def test_latent_attention_by_heads_and_over_lines():
    """The same steps with the prompt path from 64 rows on and without it, each against the 32-bit path: whole prompts, portions behind
    a history beside single tokens, single tokens behind a portion (no prompt path then), several portions."""
    from kapel_b200.engine import Engine, batch

    steps = [[("a", 200)], [("c", 63), ("b", 64)], [("a", 1), ("b", 90), ("d", 128)], [("d", 65), ("a", 1)], [("a", 1), ("b", 3), ("c", 70)], [("c", 1), ("d", 1)]]
    rng = np.random.default_rng(5)
    tokens = [[(r, rng.integers(0, 97, n).tolist()) for r, n in s] for s in steps]
    taken = []

    def run(dtype, from_rows):
        kept, batch.LATENT_PROMPT_ROWS = batch.LATENT_PROMPT_ROWS, from_rows
        whole = batch.StepBatch.latent_tiles
        def tiles(self):
            got = whole(self)
            taken.append(got is not None)
            return got
        batch.StepBatch.latent_tiles = tiles
        try:
            eng = Engine.random(LATENT, seed=2, dtype=dtype, max_tokens=2048, max_sequences=5)
            return [eng.step([(r, t, list(range(len(t)))) for r, t in s]).double().cpu() for s in tokens]
        finally:
            batch.LATENT_PROMPT_ROWS, batch.StepBatch.latent_tiles = kept, whole

    exact, lines = run("float32", 64), run("bfloat16", 1 << 30)
    assert not any(taken)
    taken.clear()
    heads = run("bfloat16", 64)
    assert taken == [True, True, True, False, True]          # a short portion behind a long one: over the lines; the last step: recorded
    for e, l, h in zip(exact, lines, heads):
        off = lambda x: float((x - e).norm() / e.norm())
        assert off(h) <= 2e-2 and off(h) <= 1.5 * off(l) + 1e-3, (off(h), off(l))


@pytest.mark.parametrize("kv_rank", [512, 576, 640])
def test_single_tokens_beside_a_prompt_at_wide_ranks(kv_rank):
    """Lines wider than the tensor-core kernel over lines takes: the single tokens of a mixed pass go row by row, the prompt by heads."""
    import copy

    from kapel_b200.engine import Engine

    model = copy.deepcopy(LATENT)
    model["layers"][0]["mixer"]["kv_rank"] = kv_rank
    rng = np.random.default_rng(6)
    draw = lambda n: rng.integers(0, 97, n).tolist()
    steps = [[("a", draw(40), []), ("b", draw(25), [])], [("a", draw(1), [0]), ("b", draw(1), [0]), ("c", draw(90), list(range(90)))]]

    def run(dtype):
        eng = Engine.random(model, seed=2, dtype=dtype, max_tokens=512, max_sequences=3)
        return [eng.step(s).double().cpu() for s in steps][1]

    exact, got = run("float32"), run("bfloat16")
    assert got.shape == (92, 97) and float((got - exact).norm() / exact.norm()) <= 2e-2


def test_a_request_reads_nothing_of_its_neighbour():
    """Two prompts of lengths that fill no tile in one pass, laid out densely one behind the other, the second's lines no finite numbers: the
    first's logits are what they are alone."""
    from kapel_b200.engine import Engine

    eng = Engine.random(LATENT, seed=2, dtype="bfloat16", max_tokens=1024, max_sequences=4, graphs=False)
    eng.model.embedding.table[96] = float("nan")             # a token that the second prompt alone has
    tokens = np.random.default_rng(7).integers(0, 96, 100).tolist()
    want = list(range(100))
    alone = eng.step([("a", tokens, want), ("b", [3] * 70, [])])[:, :96]
    beside = eng.step([("c", tokens, want), ("d", [96] * 70, [69])])[:, :96]
    assert torch.isfinite(alone).all() and torch.equal(alone, beside[:100]) and not torch.isfinite(beside[100]).any()


@pytest.mark.parametrize("hq,hkv,d,n", [(8, 2, 128, 300), (4, 4, 64, 513)])
@pytest.mark.parametrize("peak", [1.0, 4.0])
def test_as_near_to_64_bit_as_the_kernel_before(hq, hkv, d, n, peak):
    """Flat and peaked rows, whose largest weight is nearly all: the error's 2-norm is no larger than that of the mma.sync kernel, whose weights are
    taken against the row's true maximum."""
    from kapel_b200 import kernels as K

    gen = torch.Generator(device="cuda").manual_seed(12)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    width = -(-n // 16)
    k_table, v_table = (make(width, hkv, 16, d).bfloat16() for _ in range(2))
    k, v = (t.transpose(1, 2).reshape(width * 16, hkv, d)[:n] for t in (k_table, v_table))
    q = (make(n, hq, d) * peak).bfloat16()
    table, counts = (torch.arange(a, a + m, dtype=torch.int32, device="cuda") for a, m in ((0, width), (1, n)))
    want = reference(q, k, v, 1, d ** -0.5, None, None)
    off = [float((K.paged_attention_mma(q, k_table, v_table, table[None].contiguous(), counts, cut([(0, n)], rows // (hq // hkv)), 16, None, d ** -0.5, None,
                                        0, 0, 1, prompt_kernel=kernel).double() - want).norm() / want.norm())
           for kernel, rows in (("mma", K.attention_mma_rows(False)), ("flash", 128))]
    assert off[1] <= 1.03 * off[0], off                      # 40,000 results and more: the norms of two random errors of one size agree to 1 %
