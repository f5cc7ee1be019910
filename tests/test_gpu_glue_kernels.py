"""The element-wise kernels around the quantized linears at sizes where their loops and look-ups turn."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one copy, an odd number of copies, more items than one step of the grid
@pytest.mark.parametrize("tokens, hidden, k", [(1, 8, 1), (7, 264, 2), (33, 4096, 3), (5, 1032, 5), (2222, 4096, 2), (4099, 4096, 1)])
def test_combine_adds_the_copies_in_their_order(tokens, hidden, k):
    from arcquant_b200 import ops

    torch.manual_seed(tokens)
    y = torch.randn(tokens * k + 3, hidden, device="cuda").bfloat16()
    pos = torch.randperm(tokens * k + 3, device="cuda")[:tokens * k].int().view(tokens, k)
    w = torch.rand(tokens, k, device="cuda").bfloat16()
    want = torch.zeros(tokens, hidden, dtype=torch.bfloat16, device="cuda")
    for j in range(k):
        want += y[pos[:, j].long()] * w[:, j:j + 1]
    assert torch.equal(ops.moe_combine(y, pos, w), want)


# one head, a row wider than its heads, tables shorter than the tokens, more items than one step of the grid
@pytest.mark.parametrize("tokens, heads, dim, extra, seq", [(1, 1, 16, 0, 1), (3, 5, 48, 8, 2), (130, 40, 128, 1024, 130), (9000, 40, 128, 1024, 1500)])
def test_rotary_embedding_in_place(tokens, heads, dim, extra, seq):
    from arcquant_b200 import ops

    torch.manual_seed(tokens)
    x = torch.randn(tokens, heads * dim + extra, device="cuda").bfloat16()
    c, s = torch.randn(seq, dim, device="cuda"), torch.randn(seq, dim, device="cuda")
    at = torch.arange(tokens, device="cuda") % seq
    a = x[:, :heads * dim].view(tokens, heads, dim).float()
    rotated = torch.cat((-a[..., dim // 2:], a[..., :dim // 2]), -1)
    want = x.clone()
    want[:, :heads * dim] = (a * c[at][:, None] + rotated * s[at][:, None]).bfloat16().view(tokens, -1)
    assert torch.equal(ops.rope_inplace(x, c, s, heads, dim), want)


# one run, runs without rows (the first, the last, all but one), 64 runs, rows of one vector, of fifteen, sixteen and seventeen times 32 and of a
# remainder; more rows than warps
@pytest.mark.parametrize("counts, k", [((1,), 8), ((0, 3, 0), 264), ((0, 0, 257, 1), 4096), ((5, 0) * 32, 3840), ((300, 257, 1, 0), 4352), ((7,) * 64, 2056),
                                       ((12000,), 64), ((255, 256, 4000, 9000, 0, 1), 136)])
@pytest.mark.parametrize("mapped", [False, True])
def test_maxima_of_the_runs(counts, k, mapped):
    from arcquant_b200 import ops

    torch.manual_seed(k)
    first, at = [], 0
    for c in counts:
        first.append(at)
        at += (c + 255) // 256 * 256
    at = max(at, 1)
    src = torch.randn(at, k, device="cuda").bfloat16()
    row_map = torch.randperm(at, device="cuda").int() if mapped else None
    rows = src[row_map.long()] if mapped else src
    for f, c in zip(first, counts):                    # the largest of a run is its last value, larger ones lie in the padding behind it
        rows[f + c:f + (c + 255) // 256 * 256] = 1e9
        if c:
            rows[f + c - 1, k - 1] = -50.0 - c
    if mapped:
        src[row_map.long()] = rows
    groups = torch.tensor(first + list(counts), dtype=torch.int32, device="cuda")
    got = ops.absmax_grouped(src, row_map, groups, len(counts))
    want = torch.stack([rows[f:f + c].abs().max().float() if c else torch.zeros((), device="cuda") for f, c in zip(first, counts)])
    assert torch.equal(got, want)
