"""A routed-expert block behind one call against the calls it stands for: the same bits for every choice of products, rule and router."""
import pytest
import torch

from mistralrs_b200 import seq_ops as S

pytestmark = pytest.mark.gpu


def _calls(x, router, logits, correction, up, down, top, gated, act, route, products, rule):
    n, routes = up.shape[0], router.shape[0]
    if logits is None:
        logits = S.router_logits(x, router)
    if route == S.ROUTE_TOP_SOFTMAX:
        experts, weights = S.moe_route_top_softmax(logits, top)
    else:
        experts, weights = S.moe_route_scored(logits, correction, score_fn=S.SCORE_SIGMOID if route == S.ROUTE_SIGMOID else S.SCORE_SOFTMAX, top=top, **rule)
    if products == S.GROUPED:
        return S.moe_grouped(x, up, down, experts, weights, routes, act, gated)
    if products == S.STREAMED:
        return (S.moe_small if gated else S.moe_small_ungated)(x, up, down, experts, weights, act)
    rows, counts, inverse = S.moe_place(x, experts, routes)
    ys = S.moe_products(rows, up, down, counts, act, gated)
    return S.moe_combine(ys, None, weights, inverse=inverse, **({"experts": experts, "x": x, "n_ffn": n} if routes > n else {}))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("products", [S.ONE_LAUNCH, S.GROUPED, S.STREAMED])
@pytest.mark.parametrize("gated,identities", [(True, 0), (True, 3), (False, 0)])
@pytest.mark.parametrize("experts,top,tokens,given", [(1, 1, 1, False), (5, 2, 3, False), (8, 3, 33, False), (40, 4, 64, False), (8, 2, 65, True)])
def test_one_call_is_its_calls(experts, top, tokens, given, gated, identities, products, dtype):
    if products == S.ONE_LAUNCH and dtype == torch.float32:
        pytest.skip("bf16 products")
    cuda, W, ff = torch.device("cuda"), 136, 72
    g = torch.Generator(device=cuda).manual_seed(experts + tokens)

    def normal(*shape):
        return torch.randn(shape, device=cuda, generator=g)

    x, router = normal(tokens, W).to(dtype), normal(experts + identities, W) * W ** -0.5
    up, down = (normal(experts, 2 * ff if gated else ff, W) * W ** -0.5).to(dtype), (normal(experts, W, ff) * ff ** -0.5).to(dtype)
    correction = normal(experts + identities) * 0.1
    act = S.ACT_SILU if gated else S.ACT_RELU_SQ
    logits = S.router_logits(x, router).contiguous() if given else None
    for route, rule in ((S.ROUTE_SOFTMAX, dict(renorm=True, renorm_eps=1e-20)), (S.ROUTE_SIGMOID, dict(weight_scale=2.5)), (S.ROUTE_TOP_SOFTMAX, dict())):
        rule = dict(n_groups=1, keep_groups=1, **rule)
        want = _calls(x, router, logits, correction, up, down, top, gated, act, route, products, rule)
        got = S.moe_block(x, router, logits, correction, up, down, top, gated, act, route, products, **rule)
        assert torch.equal(got, want), (route, rule)
