"""RoutedExperts where two kernels could take a step: the block's result does not depend on which does.  Against a float64 restatement."""
import pytest
import torch

from mistralrs_b200 import mixers, seq_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [4, 7, 8, 32, 33])
def test_around_the_line_between_grouped_and_one_launch(cuda, tokens):
    E, top, W, ff = 16, 4, 2048, 2048
    g = torch.Generator(device=cuda).manual_seed(tokens)
    normal = lambda *s: torch.randn(s, device=cuda, generator=g)
    up, down = (normal(E, 2 * ff, W) * W ** -0.5).to(torch.bfloat16), (normal(E, W, ff) * ff ** -0.5).to(torch.bfloat16)
    router, x = (normal(E, W) * W ** -0.5).to(torch.bfloat16).float(), normal(tokens, W).to(torch.bfloat16)
    block = mixers.RoutedExperts(router, torch.zeros(E, device=cuda), up, down, top, 1, 1, seq_ops.ACT_SILU, renorm=True, renorm_eps=1e-20)
    assert block.groups_weights(tokens) == (tokens <= 7) and (tokens <= 7 or not block.streams_weights(tokens))
    got = block.forward(x).double()
    xd = x.double()
    score = torch.softmax(xd @ router.double().t(), -1)
    chosen = torch.topk(score, top, -1).indices
    weight = torch.gather(score, 1, chosen)
    weight = weight / weight.sum(-1, keepdim=True)
    want = torch.zeros_like(xd)
    for t in range(tokens):
        for j in range(top):
            gate, lift = (up[chosen[t, j]].double() @ xd[t]).chunk(2)
            want[t] += weight[t, j] * (down[chosen[t, j]].double() @ (gate * torch.sigmoid(gate) * lift))
    # bf16 hidden rows, expert outputs and result: three roundings of 2^-9 of values that add up at most in magnitude over `top` experts
    assert (got - want).abs().max().item() <= 3 * 2.0 ** -9 * top ** 0.5 * 2 * want.abs().max().item()


@pytest.mark.parametrize("dtype,width", [(torch.bfloat16, 64), (torch.bfloat16, 37), (torch.float32, 130)])
@pytest.mark.parametrize("tokens,top,n_experts", [(1, 1, 1), (1, 4, 40), (3, 2, 5), (32, 4, 16), (129, 2, 300), (512, 4, 8)])
def test_pairs_placed_in_one_launch(cuda, tokens, top, n_experts, dtype, width):
    """`moe_place` against a stable sort: rows, counts, and the row of each pair."""
    from mistralrs_b200 import seq_ops as K
    gen = torch.Generator(device=cuda).manual_seed(tokens + n_experts)
    experts = torch.randint(0, n_experts, (tokens, top), dtype=torch.int32, device=cuda, generator=gen)
    x = torch.randn(tokens, width, device=cuda, generator=gen).to(dtype)
    assert K.moe_place_fits(tokens * top, n_experts)
    rows, counts, inverse = K.moe_place(x, experts, n_experts)
    order = torch.argsort(experts.reshape(-1).long(), stable=True)
    assert torch.equal(counts.long(), torch.bincount(experts.reshape(-1).long(), minlength=n_experts))
    assert torch.equal(inverse.long()[order], torch.arange(tokens * top, device=cuda))
    assert torch.equal(rows, x[order // top])
    weights = torch.rand(tokens, top, device=cuda, generator=gen)
    assert torch.equal(K.moe_combine(rows, None, weights, inverse=inverse), K.moe_combine(rows, order.to(torch.int32), weights))
    assert not K.moe_place_fits(0, n_experts) and not K.moe_place_fits(2049, n_experts)
