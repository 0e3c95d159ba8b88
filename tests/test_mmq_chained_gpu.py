"""The dequantising GEMM, the GLU and the residual norm as links of a programmatic-dependent-launch chain against the same launches in plain order:
the same bits.  Each launch reads what the one before writes and the block's buffers are used again by its next turn."""
import pytest
import torch

from mistralrs_b200 import BLOCK_BYTES, BLOCK_ELEMS, mmq, ops, quant

pytestmark = pytest.mark.gpu

F16_AT = {"q4_k": (0, 2), "q5_k": (0, 2), "q6_k": (208,), "q8_0": (0,), "q4_0": (0,), "q2_k": (80, 82)}


def _matrix(kind, rows, cols, cuda, g):
    raw = torch.randint(0, 256, (rows * cols // BLOCK_ELEMS[kind], BLOCK_BYTES[kind]), dtype=torch.uint8, device=cuda, generator=g)
    for at in F16_AT[kind]:
        d = torch.rand(raw.shape[0], device=cuda, generator=g) * 1e-4
        raw[:, at:at + 2] = d.to(torch.float16).view(torch.uint8).view(-1, 2)
    return quant.QTensor(raw.view(-1), kind, (rows, cols))


@pytest.mark.parametrize("kind,down", [("q4_k", "q6_k"), ("q8_0", "q8_0"), ("q5_k", "q5_k"), ("q4_0", "q4_0"), ("q2_k", "q6_k")])
@pytest.mark.parametrize("tokens", [2, 9, 65, 300, 700])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_chained_block_is_the_plain_one(cuda, kind, down, tokens, dtype):
    g = torch.Generator(device=cuda).manual_seed(tokens)
    width, inner = 512, 1280
    gate, up, low = _matrix(kind, inner, width, cuda, g), _matrix(kind, inner, width, cuda, g), _matrix(down, width, inner, cuda, g)
    x = torch.randn(tokens, width, device=cuda, generator=g).to(dtype)
    norm = torch.rand(width, device=cuda, generator=g).to(dtype)

    def turns(chained):
        s, h = x, x
        for _ in range(6):
            a, b = mmq.forward_many([gate, up], h, chained=chained)
            if chained:
                d = mmq.forward_chained(low, ops.fused_glu_chained(a, b, 0))
                s, h = ops.add_rms_norm_chained(d, s, norm, 1e-5)
            else:
                d = mmq.forward(low, ops.fused_glu(a, b, 0))
                s, h = ops.add_rms_norm(d, s, norm, 1e-5)
        return s, h

    want, got = turns(False), turns(True)
    mmq.check_timeouts(cuda)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and bool(torch.isfinite(want[1].float()).all())


def test_links_refuse_what_their_kernels_do_not_take(cuda):
    x, w = torch.ones(40, 512, dtype=torch.float16, device=cuda), torch.ones(512, dtype=torch.float16, device=cuda)
    for a, b in ((x.float(), x.float()), (x, x.bfloat16()), (x, x[:2]), (x, x.cpu()), (x[:, ::2], x[:, ::2])):
        with pytest.raises(ValueError, match="fused_glu_chained"):
            ops.fused_glu_chained(a, b, 0)
        with pytest.raises(ValueError, match="add_rms_norm_chained"):
            ops.add_rms_norm_chained(a, b, w, 1e-5)
    for weight in (w.float(), w[:256], w.cpu(), torch.ones(1024, dtype=torch.float16, device=cuda)[::2]):
        with pytest.raises(ValueError, match="weight"):
            ops.add_rms_norm_chained(x, x, weight, 1e-5)
