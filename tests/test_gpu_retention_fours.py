"""Retention's inputs four components at a time, against the same columns one place further (which the general kernel reads): the memory has
the same bits, the read-outs differ by the order of one sum. Portions around the chunks' edges, memories around the tiles' edges."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,e,rotary,act", [(128, 128, 128, 1), (128, 64, 64, 0), (64, 132, 0, 1), (160, 36, 8, 1), (36, 4, 16, 0)])
@pytest.mark.parametrize("sizes", [(128,), (129, 64, 1), (65, 300, 192)])
def test_against_the_general_kernel(d, e, rotary, act, sizes):
    from kapel_b200 import kernels as K

    H, rows = 3, sum(sizes)
    g = torch.Generator(device="cuda").manual_seed(d + e + rows)
    nq, nv = H * d, H * e
    x = torch.randn(rows, 2 * nq + nv, device="cuda", generator=g)
    shifted = torch.zeros(rows, 2 * nq + nv + 4, device="cuda")
    shifted[:, 1:-3] = x
    entry = torch.tensor(np.repeat(np.arange(len(sizes)), sizes), dtype=torch.int32, device="cuda")
    slots = torch.arange(1, len(sizes) + 1, dtype=torch.int32, device="cuda")
    positions = torch.arange(rows, dtype=torch.int32, device="cuda")
    table = K.rope_table(positions, rotary, 70.0) if rotary else None
    decay = torch.tensor([0.99, 0.75, 0.0], device="cuda")
    start = torch.randn(len(sizes) + 1, nq * e, device="cuda", generator=g)
    got = []
    for src, off in ((x, 0), (shifted, 1)):
        state = start.clone()
        out = K.retention_scan(src, off, off + nq, off + 2 * nq, decay, table, rotary, d ** -0.5, state, K.entry_ranges(entry, len(sizes)), slots,
                               len(sizes), max(sizes), H, d, e, act="silu" if act else "none")
        got.append((out, state))
    assert torch.equal(got[0][1], got[1][1])
    # q.k is a sum of d products in another order: at most d roundings of 2^-24 of the products' sizes
    assert (got[0][0] - got[1][0]).abs().max() <= d * 2 ** -24 * got[1][0].abs().max()
