"""GPU: products whose exponents lie too far apart for the residue engine: windows as wide as the lines' spread, up to the
widest window and beyond it (the cluster method), against the oracle."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb

pytestmark = pytest.mark.gpu


# The spread of a line is at most 2 span; a window takes 2 spread + 64 limbs + log2 k bits in at most 2 limbs + 64 words: the
# last span that always fits is 510, and 1500 does not.
@pytest.mark.parametrize("bits", [64, 192, 544, 1024])
@pytest.mark.parametrize("m,n,k,span", [(9, 17, 5, 100), (25, 8, 33, 185), (24, 31, 20, 510), (24, 25, 40, 520), (30, 30, 9, 1500)])
def test_wide_products(engine, oracle, bits, m, n, k, span):
    rng = np.random.default_rng(bits + span)
    la = api.Linalg(engine)
    A = nb.random_numbers(rng, k * m, bits, span, zero_frac=0.05)
    B = nb.random_numbers(rng, k * n, bits, span, zero_frac=0.05)
    A.reshape(k, m, -1)[:, 2] = 0                              # an empty line
    B[1, -1], B[1, :-1] = nb.INVALID, 0
    C0 = nb.random_numbers(rng, m * n, bits, span, zero_frac=0.2)
    for subtract in (False, True):
        C = C0.copy()
        la.gemm(bits, True, A, B, m, n, k, C, subtract=subtract)
        assert (C == oracle.gemm(bits, True, A, B, m, n, k, C=C0 if subtract else None, subtract=subtract)).all(), subtract
    S = nb.random_numbers(rng, m * m, bits, span)
    C = S.copy()
    la.syrk(bits, A, k, m, C, lower_only=True, subtract=True)
    assert (C == oracle.syrk(bits, A, k, m, C=S, lower_only=True, subtract=True)).all()
