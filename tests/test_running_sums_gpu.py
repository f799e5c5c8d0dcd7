"""GPU: the triangular recurrences keep each entry's exact sum while its terms arrive, in a window placed by a guess.
Block sizes and line counts around a warp, and exponents that break the guess (far smaller and far larger terms than the
first entries suggest, zero right-hand sides that fill in, zero and status pivots), against the oracle."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb
from linalg_cases import rhs, spd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [64, 224, 256, 768, 800, 1024])
@pytest.mark.parametrize("n,nrhs,block,spread", [(1, 1, 32, 3), (31, 4, 32, 3), (33, 5, 32, 500), (40, 1, 13, 200), (34, 3, 31, 3000), (37, 2, 33, 40)])
def test_triangular_solves(engine, oracle, bits, n, nrhs, block, spread):
    la = api.Linalg(engine)
    rng = np.random.default_rng(bits + n)
    N = bits // 32
    L = nb.random_numbers(rng, n * n, bits, spread, zero_frac=0.1)
    diag = np.arange(n) * (n + 1)
    L[diag] = nb.random_numbers(rng, n, bits, spread // 2)
    for i in range(n):
        L[i * n + i + 1:(i + 1) * n] = 0
    if n > 35:
        L[diag[7]] = 0                                        # a zero pivot: division_by_zero from there on
    B = nb.random_numbers(rng, n * nrhs, bits, spread)
    B.reshape(n, nrhs, N + 3)[1:, 0] = 0                       # a unit right-hand side: every later entry fills in
    fo = api.FactorOptions(block=block)
    for passes in (1, 2):
        X = np.zeros_like(B)
        la.trsm(bits, passes == 2, L, n, B, nrhs, X, fo)
        assert (X == oracle.solve(bits, L, n, B, nrhs, block, passes)).all(), passes


@pytest.mark.parametrize("bits", [64, 256, 416, 768])
@pytest.mark.parametrize("kind,n,block", [("graded", 33, 32), ("wide", 45, 32), ("qsc", 64, 32), ("rank_deficient", 40, 32), ("moderate", 35, 17)])
def test_cholesky_blocks(engine, oracle, bits, kind, n, block):
    la = api.Linalg(engine)
    rng = np.random.default_rng(bits + n)
    A = spd(oracle, bits, n, kind, rng)
    if kind == "graded":                                      # rows scaled by powers of two hundreds of binades apart: still SPD
        s = rng.integers(-400, 401, size=n)
        e = nb.exponent(A).reshape(n, n) + s[:, None] + s[None, :]
        A[:, bits // 32] = np.where(nb.sign(A) != 0, e.ravel(), 0).astype(np.int32).view(np.uint32)
    L = np.zeros_like(A)
    info = la.cholesky(bits, A, n, L, api.FactorOptions(block=block))
    W, want = oracle.cholesky(bits, A, n, block)
    assert (info.pivot, info.pivot_sign, info.pivot_status) == want and (L == W).all()
    if info.pivot < n:
        return
    B = rhs(bits, n, 3, rng)
    X = np.zeros_like(B)
    la.cholesky_solve(bits, L, n, B, 3, X, api.FactorOptions(block=block))
    assert (X == oracle.solve(bits, L, n, B, 3, block, 3)).all()
