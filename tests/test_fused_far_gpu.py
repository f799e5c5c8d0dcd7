"""GPU: fused complex operations whose terms lie too far apart for one window (they sum by clusters), beside near ones in the same
block, at the widths around the kernels' shared-memory rule, against the oracle."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [64, 128, 160, 192, 224, 256, 384, 416, 1024])
@pytest.mark.parametrize("op", ["complex_fma", "complex_fms"])
def test_far_terms(engine, oracle, bits, op):
    op = api.Operation[op]
    rng = np.random.default_rng(bits + int(op))
    count = 1000
    ins = [nb.random_complex(rng, count, bits, span, zero_frac=0.02, sparse_frac=0.05) for span in (8, 3000, 300)]
    ins[1][::3] = nb.random_complex(rng, len(ins[1][::3]), bits, 8)
    out, _ = engine.run_ternary(bits, op, *ins)
    assert (out == oracle.elementwise(bits, int(op), *ins)).all()
    # a broadcast addend, and the result over the addend
    c = np.ascontiguousarray(ins[2][:7])
    bufs = [engine.make_buffer(len(v), bits, True) for v in (*ins[:2], c, ins[2])]
    for buf, v in zip(bufs, (*ins[:2], c, ins[2])):
        buf.upload(v)
    batch = engine.batch()
    batch.run(op, bufs[0], bufs[1], bufs[3], bufs[3])
    batch.submit().wait()
    assert (bufs[3].download() == out).all()
    batch = engine.batch()
    batch.run(op, bufs[0], bufs[1], bufs[2], bufs[3], b_index=api.Broadcast(1, 0), c_index=api.Broadcast(3, 7))
    batch.submit().wait()
    idx = np.arange(count) // 3 % 7
    assert (bufs[3].download() == oracle.elementwise(bits, int(op), ins[0], ins[1], np.ascontiguousarray(c[idx]))).all()
