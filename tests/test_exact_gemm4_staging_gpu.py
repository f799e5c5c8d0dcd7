"""GPU: the exact 4 x 4 product on both sides of the rule that stages its matrices in shared memory (real matrices of 8 to 16
limbs and complex ones up to 16), with spreads where neighbouring components sum in windows and by clusters, statuses, strides that
break 16-byte alignment and counts that leave a block short, against the oracle."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb
from test_exact_gemm4_gpu import shape_dict
from test_exact_gemm4_oracle import operands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [224, 256, 416, 512, 544])
@pytest.mark.parametrize("cx", [False, True])
def test_both_sides(engine, oracle, bits, cx):
    rng = np.random.default_rng(bits + cx)
    g = api.ExactGemm4(engine)
    for count, stride, span, accumulate in ((1, 16, 200, True), (9, 16, 150, True), (13, 17, 300, False), (6, 18, 1200, True)):
        n = stride * (count - 1) + 16
        A, B, Cm = (operands(bits, 2 * count, cx, rng, span)[:n] for _ in range(3))
        A[5, ..., :-1], A[5, ..., -1] = 0, nb.INVALID
        s = api.ExactGemm4Shape(count, stride, stride, stride, accumulate, True)
        want = oracle.exact_gemm4(bits, cx, shape_dict(s), A, B, Cm)
        got = Cm.copy()
        g.gemm(bits, cx, s, A, B, got)
        assert (got == want).all(), (count, stride, span)
