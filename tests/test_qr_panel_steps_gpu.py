"""GPU: in a QR panel's column step the last block to arrive forms its y entry from the T column that the other blocks have just
written: panels of one to 64 columns (one to 126 blocks a step), the same bits as the oracle every time."""
import numpy as np
import pytest

from limbforge_b200 import api
from qr_cases import matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,block,m,n", [(64, 64, 90, 64), (256, 64, 70, 66), (544, 33, 40, 34), (256, 2, 9, 7)])
def test_panel_steps(engine, oracle, bits, block, m, n):
    rng = np.random.default_rng(bits + block)
    la = api.Linalg(engine)
    A = matrix(bits, m, n, "qsc", rng)
    want = oracle.qr(bits, A, m, n, block)
    for _ in range(3):
        f = la.factor_qr(bits, A, m, n, api.QROptions(block=block))
        for got, name in ((f.t(), "T"), (f.tau(), "tau"), (f.r(), "R"), (f.v(), "V")):
            assert (got == want[name]).all(), name
