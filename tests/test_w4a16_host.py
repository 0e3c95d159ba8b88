"""Int4 linears: what the C entry refuses before it touches a device (the addresses below are numbers that nothing reads)."""
import ctypes

import pytest

from mistralrs_b200 import lib

MISALIGNED = 716     # cudaErrorMisalignedAddress
X, W, SCALES, ZEROS, Y = (0x10000 * (i + 1) for i in range(5))


def _call(pdl, **kw):
    a = dict(x=X, w=W, scales=SCALES, qzeros=ZEROS, y=Y, M=4, K=256, N=64, group=64)
    a.update(kw)
    P, I = ctypes.c_void_p, ctypes.c_int
    args = [P(a["x"]), P(a["w"]), P(a["scales"]), P(a["qzeros"]), P(a["y"]), I(a["M"]), I(a["K"]), I(a["N"]), I(a["group"]), I(1), I(0)]
    return lib().mrs_w4a16_gemm_pdl(*args, I(1), P(0)) if pdl else lib().mrs_w4a16_gemm(*args, P(0))


@pytest.mark.parametrize("pdl", [False, True])
@pytest.mark.parametrize("kw", [dict(scales=SCALES + 2), dict(scales=SCALES + 8), dict(qzeros=ZEROS + 4), dict(qzeros=0, scales=SCALES + 2),
                                dict(x=X + 2), dict(w=W + 8)])
def test_operands_of_bulk_copies_start_on_16_bytes(pdl, kw):
    assert _call(pdl, **kw) == MISALIGNED


def test_no_rows_is_no_work():
    assert _call(False, M=0, scales=SCALES + 2) == 0
