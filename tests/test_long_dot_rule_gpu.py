"""GPU: products that the residue engine refuses after its analysis (a line spans more than 192 bits), with long sums: output counts
and exponent spreads on both sides of the rule that gives an output a block of its own, old entries far from the products,
outputs that no window holds, a SYRK (one analysis for both sides); and the limb kernel asked for by name. Against the oracle."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb

pytestmark = pytest.mark.gpu


def lines(rng, count, k, bits, spread):
    """k x count entries whose every line spans exactly `spread` bits; an empty line, and a status in the last."""
    x = nb.random_numbers(rng, k * count, bits, 8, zero_frac=0.05).reshape(k, count, -1)
    N = bits // 32
    x[:, :, N] = np.where(x[:, :, N + 1] != 0, rng.integers(0, spread + 1, size=(k, count)), 0).astype(np.int32).view(np.uint32)
    x[:2] = nb.random_numbers(rng, 2 * count, bits, 0).reshape(2, count, -1)
    x[1, :, N] = spread
    if count > 4:
        x[:, 2] = 0
        x[5, -1, :N + 2], x[5, -1, N + 2] = 0, nb.INVALID
    return x.reshape(k * count, -1)


def old_entries(rng, count, bits, spread):
    c = nb.random_numbers(rng, count, bits, spread, zero_frac=0.1)
    far = rng.integers(0, 4, size=count)
    for kind, e in ((0, 6000), (1, -6000)):
        c[far == kind, bits // 32] = np.int32(e).view(np.uint32)
    c[nb.sign(c) == 0] = 0
    return c


# The block's window holds products that spread over less than 832 bits up to 16 limbs and 448 beyond.
@pytest.mark.parametrize("method,bits,m,n,k,spread", [
    (0, 256, 16, 32, 130, 205), (0, 256, 32, 64, 128, 409), (0, 256, 33, 63, 129, 300), (0, 256, 3, 7, 600, 420), (0, 512, 20, 30, 140, 500),
    (0, 544, 32, 64, 131, 205), (0, 544, 9, 11, 257, 230), (0, 1024, 16, 33, 128, 210), (0, 64, 5, 6, 300, 3000),
    (1, 64, 16, 32, 128, 400), (1, 256, 16, 32, 130, 3000), (1, 544, 8, 9, 150, 2000), (1, 1024, 6, 7, 128, 20)])
def test_rule(engine, oracle, method, bits, m, n, k, spread):
    rng = np.random.default_rng(bits + k + spread)
    la = api.Linalg(engine, api.LinalgOptions(method=method))
    A, B, C0 = lines(rng, m, k, bits, spread), lines(rng, n, k, bits, spread), old_entries(rng, m * n, bits, spread)
    for subtract in (False, True):
        C = C0.copy()
        la.gemm(bits, True, A, B, m, n, k, C, subtract=subtract)
        assert la.report()["method"] == 1
        assert (C == oracle.gemm(bits, True, A, B, m, n, k, C=C0 if subtract else None, subtract=subtract)).all(), subtract
    S = old_entries(rng, m * m, bits, spread)
    C = S.copy()
    la.syrk(bits, A, k, m, C, lower_only=True, subtract=True)
    assert (C == oracle.syrk(bits, A, k, m, C=S, lower_only=True, subtract=True)).all()
