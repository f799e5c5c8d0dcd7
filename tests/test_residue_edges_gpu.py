"""GPU: the residue engine at the edges of its tiles and tables, bit for bit against the limb kernel on the same data:
inner dimensions around one MMA step (32) and one K tile (128), output sizes around the 128 x 80 tile, modulus counts on both
sides of the digit table's copies (32 and 64) and of its second row tile (128), and old entries far above and far below the
product, which the rounding cannot take in one pass."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,m,n,k,span,lo,hi", [
    (64, 63, 64, 1, 4, 8, 16), (128, 65, 129, 31, 10, 17, 32), (192, 128, 79, 32, 8, 25, 32), (224, 127, 65, 33, 40, 33, 64),
    (256, 129, 130, 127, 20, 33, 64), (448, 64, 80, 128, 20, 57, 64), (512, 100, 81, 129, 40, 65, 128),
    (1024, 66, 161, 160, 2, 129, 160), (1024, 33, 35, 40, 60, 129, 160)])
def test_tile_and_table_edges(engine, bits, m, n, k, span, lo, hi):
    rng = np.random.default_rng(bits + k)
    residue, limb = (api.Linalg(engine, api.LinalgOptions(method=x)) for x in (2, 1))
    A = nb.random_numbers(rng, k * m, bits, span, zero_frac=0.02, sparse_frac=0.05)
    B = nb.random_numbers(rng, k * n, bits, span, zero_frac=0.02, sparse_frac=0.05)
    C0 = nb.random_numbers(rng, m * n, bits, span)
    far = rng.integers(0, 6, size=m * n)
    N = bits // 32
    C0[far == 0, N] = rng.integers(3 * bits, 9 * bits, size=int((far == 0).sum())).astype(np.int32).view(np.uint32)
    C0[far == 1, N] = rng.integers(-9 * bits, -2 * bits, size=int((far == 1).sum())).astype(np.int32).view(np.uint32)
    C0[far == 2] = 0
    C0[5 % (m * n), N:] = [0, 0, nb.INVALID]
    C0[5 % (m * n), :N] = 0
    for subtract in (False, True):
        x, y = C0.copy(), C0.copy()
        residue.gemm(bits, True, A, B, m, n, k, x, subtract=subtract)
        assert residue.report()["method"] == 2 and lo <= residue.report()["moduli"] <= hi
        limb.gemm(bits, True, A, B, m, n, k, y, subtract=subtract)
        assert (x == y).all(), subtract
        if subtract:                                        # C - A^T B = C exactly cancelled: old entries equal to the product
            residue.gemm(bits, True, A, B, m, n, k, y := np.zeros_like(C0))
            limb.gemm(bits, True, A, B, m, n, k, z := y.copy(), subtract=True)
            residue.gemm(bits, True, A, B, m, n, k, y, subtract=True)
            assert (y == z).all()
    x, y = C0[:m].copy().repeat(m, axis=0)[: m * m].copy(), None
    y = x.copy()
    residue.syrk(bits, A, k, m, x, lower_only=True, subtract=True)
    limb.syrk(bits, A, k, m, y, lower_only=True, subtract=True)
    assert (x == y).all()
