"""Both products of routed experts behind one call against the two calls it stands for: the same bits, whatever the rows of an expert (none, a few,
a tile, several), the columns and the length of the dots."""
import pytest
import torch

from mistralrs_b200 import seq_ops as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("counts", [[1], [0, 0], [15, 16, 17], [63, 0, 64, 65], [128, 3, 129, 0], [7] * 60])
@pytest.mark.parametrize("width,ff", [(8, 40), (264, 136), (512, 1024)])
def test_both_products_are_the_two_calls(gated, counts, width, ff):
    cuda = torch.device("cuda")
    g = torch.Generator(device=cuda).manual_seed(width + len(counts))
    n, e = sum(counts) + 5, len(counts)

    def normal(*shape):
        return torch.randn(shape, device=cuda, generator=g)

    rows = normal(n, width).to(torch.bfloat16)
    rows[n - 5:] = float("nan")                                             # behind the last expert: read by the boxes, used by no result
    up = (normal(e, 2 * ff if gated else ff, width) * width ** -0.5).to(torch.bfloat16)
    down = (normal(e, width, ff) * ff ** -0.5).to(torch.bfloat16)
    at = torch.tensor(counts, dtype=torch.int32, device=cuda)
    act = S.ACT_SILU if gated else S.ACT_RELU_SQ
    want = S.moe_gemm(S.moe_gemm(rows, up, at, act, gated), down, at)
    for _ in range(3):                                                      # one call's second launch runs into the next call's first
        got = S.moe_products(rows, up, down, at, act, gated)
    assert S.moe_gemm_timeouts() == 0
    assert torch.equal(got[:n - 5], want[:n - 5]) and not torch.isnan(got[:n - 5]).any()
    # against 64 bits: each product rounds its result to bf16 (2^-9) and sums in f32
    z = [rows[sum(counts[:i]):sum(counts[:i + 1])].double() @ up[i].double().T for i in range(e)]
    h = [torch.nn.functional.silu(a[:, :ff]) * a[:, ff:] if gated else torch.clamp(a, min=0.0) ** 2 for a in z]
    exact = torch.cat([a @ down[i].double().T for i, a in enumerate(h)])
    if exact.numel():
        scale = torch.cat([a.abs() @ down[i].double().abs().T for i, a in enumerate(h)])
        assert ((got[:n - 5].double() - exact).abs() <= 2 ** -8 * scale + 2 ** -8 * exact.abs() + 1e-6).all()
