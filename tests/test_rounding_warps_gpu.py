"""GPU: one warp of the residue engine's rounding holds outputs that leave it on every path (status, empty sum, an old entry
far above or below the product, the one-pass form, an exact cancellation), then writes its 32 entries together: products whose
neighbouring outputs differ in kind, against the oracle."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [64, 256, 544, 1024])
def test_mixed_outputs(engine, oracle, bits):
    m, n, k, N = 37, 41, 9, bits // 32
    rng = np.random.default_rng(bits)
    la = api.Linalg(engine, api.LinalgOptions(method=2))
    A = nb.random_numbers(rng, k * m, bits, 20, zero_frac=0.05)
    B = nb.random_numbers(rng, k * n, bits, 20, zero_frac=0.05)
    A.reshape(k, m, -1)[:, 3::11] = 0                          # empty lines on both sides
    B.reshape(k, n, -1)[:, 5::7] = 0
    B.reshape(k, n, -1)[2, 6::13, :N + 2] = 0
    B.reshape(k, n, -1)[2, 6::13, N + 2] = nb.INVALID
    C0 = np.zeros((m * n, N + 3), dtype=np.uint32)
    la.gemm(bits, True, A, B, m, n, k, C0)                     # entries that cancel where they are left as they are
    kind = rng.integers(0, 5, size=m * n)
    other = nb.random_numbers(rng, m * n, bits, 20)
    other[kind == 1, N] = np.int32(9 * bits).view(np.uint32)
    other[kind == 2, N] = np.int32(-9 * bits).view(np.uint32)
    other[kind == 3] = 0
    C0[kind > 0] = other[kind > 0]
    for subtract in (False, True):
        C = C0.copy()
        la.gemm(bits, True, A, B, m, n, k, C, subtract=subtract)
        assert la.report()["method"] == 2
        assert (C == oracle.gemm(bits, True, A, B, m, n, k, C=C0 if subtract else None, subtract=subtract)).all(), subtract
