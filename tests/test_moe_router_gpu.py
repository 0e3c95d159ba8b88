"""The router's product and the routing rule in one launch against the two launches it stands for: the same experts and weights, to the bit."""
import pytest
import torch

from mistralrs_b200 import seq_ops as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("width,n_experts", [(8, 1), (37, 5), (130, 9), (516, 16), (2048, 16), (2044, 12), (4096, 8)])
@pytest.mark.parametrize("n_tok", [1, 3, 64])
def test_one_launch_routes_as_two(n_tok, width, n_experts, dtype):
    cuda = torch.device("cuda")
    g = torch.Generator(device=cuda).manual_seed(width + n_tok)
    x = torch.randn(n_tok, width, device=cuda, generator=g).to(dtype)
    w = torch.randn(n_experts, width, device=cuda, generator=g) * width ** -0.5
    correction = torch.randn(n_experts, device=cuda, generator=g) * 0.1
    assert S.moe_router_fits(width, n_experts, n_tok)
    logits = S.router_logits(x, w)
    groups = 4 if n_experts % 4 == 0 else 1
    for correct, top, rule in ((correction, min(4, n_experts), dict(renorm=True, renorm_eps=1e-20)), (None, 1, dict()),
                               (correction, n_experts, dict(score_fn=S.SCORE_SIGMOID, group_top=2, weight_scale=2.5))):
        keep = max(1, groups // 2)
        got = S.moe_router(x, w, correct, groups, keep, top, **rule)
        want = S.moe_route_scored(logits, correct, groups, keep, top, **rule)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_sizes_beyond_it():
    assert not S.moe_router_fits(64, 17, 1) and not S.moe_router_fits(2048, 16, 65) and not S.moe_router_fits(4097, 8, 1)
