"""GPU: products of few outputs and long sums run a block per output; sums around the block's 256 threads, old entries,
statuses, empty sums and exponents beyond the block's window, against the oracle."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [64, 256, 544, 1024])
@pytest.mark.parametrize("m,n,k,span", [(1, 1, 128, 5), (3, 5, 255, 300), (2, 7, 257, 40), (4, 3, 600, 3000), (6, 6, 130, 20)])
def test_long_sums(engine, oracle, bits, m, n, k, span):
    rng = np.random.default_rng(bits + k)
    la = api.Linalg(engine, api.LinalgOptions(method=1))
    A = nb.random_numbers(rng, k * m, bits, span, zero_frac=0.1)
    B = nb.random_numbers(rng, k * n, bits, span, zero_frac=0.1)
    C0 = nb.random_numbers(rng, m * n, bits, span, zero_frac=0.2)
    if m > 2:
        A.reshape(k, m, -1)[:, 1] = 0                          # an empty sum: the old entry itself
        B[5, -1], B[5, :-1] = nb.INVALID, 0
    for subtract in (False, True):
        C = C0.copy()
        la.gemm(bits, True, A, B, m, n, k, C, subtract=subtract)
        assert (C == oracle.gemm(bits, True, A, B, m, n, k, C=C0 if subtract else None, subtract=subtract)).all(), subtract
    S = nb.random_numbers(rng, m * m, bits, span)
    C = S.copy()
    la.syrk(bits, A, k, m, C, lower_only=True, subtract=True)
    assert (C == oracle.syrk(bits, A, k, m, C=S, lower_only=True, subtract=True)).all()
