"""RoutedExperts on both sides of the lines from which the one-launch products take a step: against a float64 restatement on either side."""
import pytest
import torch

from mistralrs_b200 import mixers, seq_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("E,top,tokens,one", [(8, 2, 9, False), (8, 2, 10, True), (16, 4, 7, False), (16, 4, 8, True), (32, 2, 15, False), (32, 2, 16, True),
                                              (5, 5, 3, False), (3, 2, 12, True)])
def test_both_sides_of_the_line(cuda, E, top, tokens, one, gated):
    W, ff = 256, 384
    g = torch.Generator(device=cuda).manual_seed(E + tokens)
    normal = lambda *s: torch.randn(s, device=cuda, generator=g)  # noqa: E731
    up, down = (normal(E, 2 * ff if gated else ff, W) * W ** -0.5).to(torch.bfloat16), (normal(E, W, ff) * ff ** -0.5).to(torch.bfloat16)
    router, x = (normal(E, W) * W ** -0.5).to(torch.bfloat16).float(), normal(tokens, W).to(torch.bfloat16)
    block = mixers.RoutedExperts(router, None, up, down, top, 1, 1, seq_ops.ACT_SILU if gated else seq_ops.ACT_RELU_SQ, renorm=True, gated=gated)
    assert block.outgrows_groups(tokens) == one and (not one or not (block.groups_weights(tokens) or block.streams_weights(tokens)))
    got = block.forward(x).double()
    xd = x.double()
    score = torch.softmax(xd @ router.double().t(), -1)
    chosen = torch.topk(score, top, -1).indices
    weight = torch.gather(score, 1, chosen)
    weight = weight / weight.sum(-1, keepdim=True)
    want, scale = torch.zeros_like(xd), torch.zeros_like(xd)
    for t in range(tokens):
        for j in range(top):
            e = chosen[t, j]
            z = up[e].double() @ xd[t]
            h = torch.nn.functional.silu(z[:ff]) * z[ff:] if gated else torch.clamp(z, min=0.0) ** 2
            want[t] += weight[t, j] * (down[e].double() @ h)
            scale[t] += weight[t, j] * (down[e].double().abs() @ h.abs())
    # hidden rows, expert outputs and the result are rounded to bf16: three relative errors of 2^-9 of at most `scale`
    assert ((got - want).abs() <= 3 * 2.0 ** -9 * scale + 1e-6).all()
