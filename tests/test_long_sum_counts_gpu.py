"""GPU: a block-wide exact sum of as many terms as an index can count: its window's headroom is found without overflow.  The
lines repeat one entry (inner stride 0), so the sum is the number of terms times one product."""
from fractions import Fraction

import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2**16 - 3, 2**24 + 1, 2**31 - 1])
def test_counts(engine, k):
    import torch
    bits = 64
    la = api.Linalg(engine, api.LinalgOptions(method=1))
    x, y, c = (nb.power(bits, e, s) for e, s in ((3, 1), (-7, -1), (11, 1)))
    x[0, 0], y[0, 1], c[0, 0] = 9, 0xf0000001, 77
    dev = [torch.from_numpy(v.view(np.int32).copy()).cuda() for v in (x, y, c)]
    for subtract in (False, True):
        out = dev[2].clone()
        torch.cuda.synchronize()
        la.dev_exact_product(bits, dev[0].data_ptr(), 1, 0, dev[1].data_ptr(), 1, 0, 1, 1, k, out.data_ptr(), 1, subtract=subtract)
        torch.cuda.synchronize()
        total = k * nb.to_fraction(x[0]) * nb.to_fraction(y[0])
        want = nb.to_fraction(c[0]) - total if subtract else total
        got = nb.to_fraction(out.cpu().numpy().view(np.uint32)[0])
        assert abs(got - want) <= abs(want) * Fraction(1, 2**64), subtract       # half a unit in the last place
