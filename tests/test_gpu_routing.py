"""The routing kernel against its torch formulation (`route_top_k`), and the padded layout at the sizes where a warp's run
of slots changes length."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,experts,k", [(1, 8, 2), (37, 8, 2), (4096, 8, 2), (5, 1, 1), (130, 3, 3), (1000, 32, 4), (77, 17, 5)])
def test_route_topk_equals_softmax_topk(tokens, experts, k):
    from arcquant_b200 import ops

    g = torch.Generator().manual_seed(tokens + experts)
    logits = (4 * torch.randn((tokens, experts), generator=g)).to(torch.bfloat16).cuda()
    if experts > 3:
        logits[::7] = logits[::7].round()                          # ties
        logits[3::11, 1] = float("-inf")
    ids, w = ops.route_topk(logits, k)
    probs = torch.softmax(logits, 1, dtype=torch.float)
    pw, want = torch.topk(probs, k, dim=-1)
    assert ids.dtype == torch.int64 and int(ids.min()) >= 0 and int(ids.max()) < experts
    assert bool((ids.sort(1).values.diff(dim=1) > 0).all())        # all different
    # the same probabilities are selected, and of equal ones the earliest comes first; an fp32 sum in another order and
    # the division move a probability by a few 2^-24
    sel = probs.gather(1, ids)
    torch.testing.assert_close(sel, pw, rtol=1e-6, atol=0.0)
    for j in range(k - 1):
        eq = sel[:, j] == sel[:, j + 1]
        assert bool((ids[:, j][eq] < ids[:, j + 1][eq]).all())
    # bf16 weights: the fp32 quotient moves by some 2^-23, its rounding by one step at most
    ref = pw / pw.sum(-1, keepdim=True)
    assert bool(((w.float() - ref).abs() <= ref * 2.0 ** -8).all())


def test_route_topk_of_no_tokens_and_of_nan():
    from arcquant_b200 import ops

    ids, w = ops.route_topk(torch.empty((0, 8), dtype=torch.bfloat16, device="cuda"), 2)
    assert ids.shape == (0, 2) and w.shape == (0, 2)
    logits = torch.randn((4, 8), device="cuda").to(torch.bfloat16)
    logits[1, 3] = float("nan")
    logits[2] = float("-inf")
    ids, w = ops.route_topk(logits, 2)
    assert int(ids.min()) >= 0 and int(ids.max()) < 8 and bool(w[1:3].isnan().all()) and not bool(w[[0, 3]].isnan().any())
    with pytest.raises(RuntimeError):
        ops.route_topk(torch.zeros((4, 33), dtype=torch.bfloat16, device="cuda"), 2)


@pytest.mark.parametrize("n,e,div", [(1, 1, 1), (31, 8, 1), (74, 8, 2), (1024, 64, 2), (1025, 33, 3), (8192, 8, 2), (8193, 8, 1),
                                     (50001, 64, 2)])
def test_layout_kernel_against_the_tensor_formulation(n, e, div):
    from arcquant_b200.moe_block import padded_layout

    ids = torch.randint(0, e + 2, (n,), generator=torch.Generator().manual_seed(n))      # (>= e: nobody)
    want, got = padded_layout(ids, e, div=div), padded_layout(ids.cuda(), e, div=div)
    assert got[4] == want[4]
    for a, b in zip(want[:4], got[:4]):
        assert torch.equal(a.long(), b.cpu().long())
