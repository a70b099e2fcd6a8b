"""The gated delta rule by chunks of rows against 64-bit and against the scan: portions of every remainder, behind a memory and a history,
beside short portions, with decays of 0; rows of no request."""
import numpy as np
import pytest
import torch

import plain_kofutar as PK

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,d,e,taps", [(4, 2, 32, 16, 4), (2, 1, 128, 48, 4), (3, 3, 64, 16, 3), (4, 1, 96, 32, 4)])
def test_against_64_bit_and_the_scan(H, G, d, e, taps, monkeypatch):
    from kapel_b200 import kernels as K

    monkeypatch.setattr(K, "DELTA_CHUNK_LONGEST", 64)       # shorter portions than where chunks pay

    dev = lambda x, dtype=torch.float32: torch.tensor(np.asarray(x), dtype=dtype, device="cuda")
    rng = np.random.default_rng(d + e)
    n, nv = G * d, H * e
    width = 2 * n + nv + 2 * H
    conv, a_log, dt_bias = rng.standard_normal((2 * n + nv, taps)) * 0.6, rng.standard_normal(H) * 0.5, rng.standard_normal(H)
    data, want = {}, {}
    for name, T in {"a": 300, "b": 161, "c": 33}.items():
        x = rng.standard_normal((T, width))
        x[:, -2 * H :] *= 3.0                                # decays and step sizes that swing
        x[T // 2, -H:] = 400.0                               # a decay that is 0 in 32-bit: everything is forgotten
        x = x.astype(np.float32).astype(np.float64)
        data[name] = x
        q, k, v, g, beta = PK.delta_inputs(x, conv.astype(np.float32).astype(np.float64), a_log.astype(np.float32).astype(np.float64),
                                           dt_bias.astype(np.float32).astype(np.float64), H, G, d, e)
        want[name] = np.stack([PK.delta_recurrence(q[:, h // (H // G)], k[:, h // (H // G)], v[:, h], g[:, h], beta[:, h]) for h in range(H)], axis=1)
    steps = [[("a", 1, 0, 64), ("b", 2, 0, 3)], [("b", 2, 3, 100), ("a", 1, 64, 65)], [("c", 3, 0, 33), ("a", 1, 65, 194)], [("a", 1, 194, 300), ("b", 2, 100, 161)]]
    per = K.delta_state_floats(H, G, d, e, taps)

    def run(chunked):
        state, worst = torch.zeros((4, per), dtype=torch.float32, device="cuda"), 0.0
        for step in steps:
            sizes = [b - a for _, _, a, b in step]
            entry = dev(np.repeat(np.arange(len(step)), sizes), torch.int32)
            out = K.delta_scan(dev(np.concatenate([data[m][a:b] for m, _, a, b in step])), 0, n, 2 * n, 2 * n + nv, 2 * n + nv + H, dev(conv), dev(a_log),
                               dev(dt_bias), state, entry, K.entry_ranges(entry, len(step)), dev([s for _, s, _, _ in step], torch.int32), len(step),
                               H, G, d, e, taps, d ** -0.5, 1e-6, max(sizes) if chunked else 0, min(sizes)).cpu().numpy()
            at = 0
            for (m, _, a, b), size in zip(step, sizes):
                worst = max(worst, float(np.abs(out[at : at + size] - want[m][a:b]).max() / np.abs(want[m]).max()))
                at += size
        return worst, state

    (scan, by_scan), (chunks, by_chunks) = run(False), run(True)
    print(f"scan {scan:.2e}, chunks {chunks:.2e}")
    assert chunks < 5e-5 and chunks < 2.0 * scan + 1e-6      # the same recurrence in 32-bit, summed in another order
    assert (by_scan - by_chunks).abs().max() <= 5e-5 * by_scan.abs().max()
    before = by_chunks.clone()
    entry = dev(np.zeros(70), torch.int32)
    out = K.delta_scan(dev(data["a"][:70]), 0, n, 2 * n, 2 * n + nv, 2 * n + nv + H, dev(conv), dev(a_log), dev(dt_bias), by_chunks, entry,
                       K.entry_ranges(entry, 1), dev([0], torch.int32), 1, H, G, d, e, taps, d ** -0.5, 1e-6, 70, 70)
    assert float(out.abs().max()) == 0.0 and torch.equal(before, by_chunks)


@pytest.mark.parametrize("taps,rows", [(1, 3), (2, 1), (4, 64), (4, 65), (8, 5)])
def test_single_tokens_move_their_own_history(taps, rows):
    """Told that every request brings one row, the first kernel moves the history on; the bits are those of the kernel made for any portion."""
    from kapel_b200 import kernels as K

    H, G, d, e = 4, 2, 32, 16
    rng = torch.Generator(device="cuda").manual_seed(taps * rows)
    n, nv = G * d, H * e
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=rng)
    conv, a_log, dt_bias = rand(2 * n + nv, taps), rand(H), rand(H)
    entry = torch.arange(rows, dtype=torch.int32, device="cuda")
    slots = torch.arange(1, rows + 1, dtype=torch.int32, device="cuda")
    slots[rows // 2] = 0                                     # a row of no request
    ranges, start = K.entry_ranges(entry, rows), rand(rows + 1, K.delta_state_floats(H, G, d, e, taps))
    states = [start.clone(), start.clone()]
    for _ in range(3):
        x = rand(rows, 2 * n + nv + 2 * H)
        a, b = (K.delta_scan(x, 0, n, 2 * n, 2 * n + nv, 2 * n + nv + H, conv, a_log, dt_bias, state, entry, ranges, slots, rows, H, G, d, e, taps,
                             d ** -0.5, 1e-6, longest, longest) for state, longest in zip(states, (0, 1)))
        assert torch.equal(a, b)
    assert torch.equal(states[0], states[1]) and torch.equal(states[1][0], start[0])


@pytest.mark.parametrize("sizes", [(512,), (515,), (300, 1, 2, 260), (63, 510, 3)])
def test_inputs_by_four_rows_and_by_rows(sizes):
    """Prompts' convolutions and unit vectors four rows a block, against the same columns one place further, which the kernel of a row a
    block reads: the same bits, behind a history and beside a row of no request."""
    from kapel_b200 import kernels as K

    H, G, d, e, taps = 4, 2, 32, 16, 4
    rows, n, nv = sum(sizes), G * d, H * e
    rng = torch.Generator(device="cuda").manual_seed(rows)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=rng)
    conv, a_log, dt_bias = rand(2 * n + nv, taps), rand(H), rand(H)
    entry = torch.tensor(np.repeat(np.arange(len(sizes)), sizes), dtype=torch.int32, device="cuda")
    slots = torch.arange(1, len(sizes) + 1, dtype=torch.int32, device="cuda")
    if len(sizes) > 3:
        slots[2] = 0
    ranges, start = K.entry_ranges(entry, len(sizes)), rand(len(sizes) + 1, K.delta_state_floats(H, G, d, e, taps))
    states = [start.clone(), start.clone()]
    for _ in range(2):
        x = rand(rows, 2 * n + nv + 2 * H)
        shifted = torch.zeros(rows, 2 * n + nv + 2 * H + 4, device="cuda")
        shifted[:, 1:-3] = x
        a, b = (K.delta_scan(src, off, off + n, off + 2 * n, off + 2 * n + nv, off + 2 * n + nv + H, conv, a_log, dt_bias, state, entry, ranges, slots,
                             len(sizes), H, G, d, e, taps, d ** -0.5, 1e-6) for src, off, state in ((x, 0, states[0]), (shifted, 1, states[1])))
        assert torch.equal(a, b)
    assert torch.equal(states[0], states[1])


def test_a_row_takes_nothing_from_later_rows():
    """A value that is no finite number reaches its own row and the rows behind it, by chunks as row by row."""
    from kapel_b200 import kernels as K

    H, G, d, e, taps, rows = 2, 1, 32, 16, 4, 200
    rng = torch.Generator(device="cuda").manual_seed(3)
    n, nv = G * d, H * e
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=rng)
    conv, a_log, dt_bias, x = rand(2 * n + nv, taps), rand(H), rand(H), rand(rows, 2 * n + nv + 2 * H)
    x[75, 2 * n + 3] = float("nan")                          # a value's component of the first head, in the middle of a chunk
    entry = torch.zeros(rows, dtype=torch.int32, device="cuda")
    one, ranges = torch.ones(1, dtype=torch.int32, device="cuda"), K.entry_ranges(entry, 1)
    out = [K.delta_scan(x, 0, n, 2 * n, 2 * n + nv, 2 * n + nv + H, conv, a_log, dt_bias, torch.zeros(2, K.delta_state_floats(H, G, d, e, taps), device="cuda"),
                        entry, ranges, one, 1, H, G, d, e, taps, d ** -0.5, 1e-6, longest, longest) for longest in (0, rows)]
    assert torch.isfinite(out[0][:75]).all() and not torch.isfinite(out[0][75:, 0, 3]).any()
    assert torch.equal(torch.isfinite(out[0]), torch.isfinite(out[1]))


@pytest.mark.parametrize("decay", [0.0, -3.0, -6.0])
def test_as_near_to_64_bit_as_the_scan(decay):
    """The 2-norm of the error over memories that forget within a row, within a chunk and hardly at all (64-bit sums row by row)."""
    from kapel_b200 import kernels as K

    H, G, d, e, taps, rows = 8, 2, 128, 128, 4, 400
    gen = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)
    n, nv = G * d, H * e
    conv, a_log, dt_bias, x = rand(2 * n + nv, taps) * 0.5, rand(H) * 0.5 + decay, rand(H) * 0.5, rand(rows, 2 * n + nv + 2 * H)
    entry = torch.zeros(rows, dtype=torch.int32, device="cuda")
    one, ranges = torch.ones(1, dtype=torch.int32, device="cuda"), K.entry_ranges(entry, 1)
    scan, chunks = (K.delta_scan(x, 0, n, 2 * n, 2 * n + nv, 2 * n + nv + H, conv, a_log, dt_bias, torch.zeros(2, K.delta_state_floats(H, G, d, e, taps), device="cuda"),
                                 entry, ranges, one, 1, H, G, d, e, taps, d ** -0.5, 1e-6, longest, longest).double() for longest in (0, rows))
    np64 = lambda t: t.double().cpu().numpy()
    q, k, v, g, beta = (torch.as_tensor(np.asarray(t), device="cuda") for t in PK.delta_inputs(np64(x), np64(conv), np64(a_log), np64(dt_bias), H, G, d, e))
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    S, want = torch.zeros(H, d, e, dtype=torch.float64, device="cuda"), []
    for t in range(rows):
        S = S * g[t][:, None, None]
        S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t])))[:, None, :]
        want.append(torch.einsum("hde,hd->he", S, q[t]))
    off = [float((o - torch.stack(want)).norm() / torch.stack(want).norm()) for o in (scan, chunks)]
    # a warp's sums of four components a lane and a tree, against chains of eight to sixteen and pairs: some roundings more, 1.36 to 1.6 with
    # chains over all components
    assert off[1] <= 1.15 * off[0], off


def test_requests_in_any_order():
    """Requests listed in another order than their rows lie in, short ones between them: the same bits."""
    from kapel_b200 import kernels as K

    H, G, d, e, taps = 4, 2, 64, 32, 4
    sizes, order = (200, 1, 70, 192, 3, 65, 250), (5, 0, 6, 2, 4, 1, 3)      # `order`: the request that is listed at each place
    n, nv = G * d, H * e
    width, rows = 2 * n + nv + 2 * H, sum(sizes)
    gen = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=gen)
    ints = lambda x: torch.tensor(np.asarray(x), dtype=torch.int32, device="cuda")
    x, conv, a_log, dt_bias, start = rand(rows, width), rand(2 * n + nv, taps), rand(H), rand(H), rand(9, K.delta_state_floats(H, G, d, e, taps)) * 0.1
    first = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    out, states = [], []
    for listed in (tuple(range(7)), order):
        entry = np.zeros(rows, np.int32)
        for place, r in enumerate(listed):
            entry[first[r] : first[r] + sizes[r]] = place
        state = start.clone()
        out.append(K.delta_scan(x, 0, n, 2 * n, 2 * n + nv, 2 * n + nv + H, conv, a_log, dt_bias, state, ints(entry),
                                (ints([first[r] for r in listed]), ints([first[r] + sizes[r] for r in listed])), ints([r + 1 for r in listed]), 7,
                                H, G, d, e, taps, d ** -0.5, 1e-6, 250, 1))
        states.append(state)
    K.check_async_errors()
    assert torch.equal(out[0], out[1]) and torch.equal(states[0], states[1])
