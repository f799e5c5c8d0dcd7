"""GPU: broadcast operands of the element-wise kernels, a row copied by its own thread: real, ternary and complex operations, both
operands broadcast alike, strides and periods that cut blocks, odd and even row lengths, short last blocks, against the oracle."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [64, 96, 256, 416, 1024])
@pytest.mark.parametrize("op", ["add", "div", "fma", "complex_add", "complex_div", "complex_fms"])
def test_broadcasts(engine, oracle, bits, op):
    op = api.Operation[op]
    cx, ternary = api.operation_is_complex(op), api.operation_is_ternary(op)
    rng = np.random.default_rng(bits + int(op))
    make = nb.random_complex if cx else nb.random_numbers
    for count, stride, period in ((1, 1, 1), (128, 1, 1), (129, 1, 7), (191, 3, 0), (300, 5, 4), (260, 1000, 0)):
        b = api.Broadcast(stride, period)
        n = api.broadcast_elements(count, b)
        x = make(rng, count, bits, 40, zero_frac=0.05)
        y, z = (make(rng, n, bits, 40, zero_frac=0.05) for _ in range(2))
        idx = np.arange(count) // stride
        idx = idx % period if period else idx
        bufs = [engine.make_buffer(len(v), bits, cx) for v in (x, y, z, x)]
        for buf, v in zip(bufs, (x, y, z)):
            buf.upload(v)
        batch = engine.batch()
        if ternary:
            batch.run(op, bufs[0], bufs[1], bufs[2], bufs[3], b_index=b, c_index=b)
        else:
            batch.run(op, bufs[0], bufs[1], None, bufs[3], b_index=b)
        batch.submit().wait()
        want = oracle.elementwise(bits, int(op), x, np.ascontiguousarray(y[idx]), np.ascontiguousarray(z[idx]) if ternary else None)
        assert (bufs[3].download() == want).all(), (count, stride, period)
