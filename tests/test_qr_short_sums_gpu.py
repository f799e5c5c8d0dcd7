"""GPU: the QR panel's four-lane sums (column reductions, short products between blocks) and the T and y entries that run side by
side, against the oracle at panel sizes around a warp and around the blocks' edges, with exponents too far apart for the
lanes' windows."""
import numpy as np
import pytest

from limbforge_b200 import api
from qr_cases import matrix, rhs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [96, 256, 544])
@pytest.mark.parametrize("kind,m,n,block", [("moderate", 5, 3, 32), ("extreme", 40, 34, 32), ("spread", 70, 33, 32), ("qsc", 131, 65, 32), ("wide", 50, 20, 7)])
def test_real(engine, oracle, bits, kind, m, n, block):
    rng = np.random.default_rng(bits + m)
    A, B = matrix(bits, m, n, kind, rng), rhs(bits, m, 2, rng)
    f = api.Linalg(engine).factor_qr(bits, A, m, n, api.QROptions(block=block))
    want = oracle.qr(bits, A, m, n, block)
    for got, name in ((f.r(), "R"), (f.v(), "V"), (f.tau(), "tau"), (f.t(), "T")):
        assert (got == want[name]).all(), name
    assert (f.solve(B, 2) == oracle.qr_solve(want, B, 2)).all()


@pytest.mark.parametrize("bits", [96, 256])
@pytest.mark.parametrize("kind,m,n", [("moderate", 4, 3), ("extreme", 36, 33), ("qsc", 70, 40)])
def test_complex(engine, oracle, bits, kind, m, n):
    rng = np.random.default_rng(bits + m)
    A = np.ascontiguousarray(np.stack([matrix(bits, m, n, kind, rng) for _ in range(2)], axis=1))
    f = api.Linalg(engine).factor_qr_complex(bits, A, m, n, api.QROptions(block=32))
    want = oracle.qr_complex(bits, A, m, n, 32)
    for got, name in ((f.r(), "R"), (f.v(), "V"), (f.tau(), "tau"), (f.t(), "T")):
        assert (got == want[name]).all(), name
