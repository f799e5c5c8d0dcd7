"""GPU: operands that reach the rare branches of the limb arithmetic: quotient digits at their largest and one too large,
addition gaps at every word of the alignment, cancellation down to the last bits, products of all-ones rows; complex
operations, whose components run on two lanes, in place over each operand."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb

pytestmark = pytest.mark.gpu


def edge_numbers(rng, count, bits):
    n = bits // 32
    x = nb.random_numbers(rng, count, bits, 40)
    kind = rng.integers(0, 8, size=count)
    for i in np.nonzero(kind == 0)[0]:
        x[i, :n] = 0xFFFFFFFF
    for i in np.nonzero(kind == 1)[0]:
        x[i, :n - 1] = 0                                     # a word above zeros
    for i in np.nonzero(kind == 2)[0]:
        x[i, :n] = np.where(rng.integers(0, 2, size=n) == 1, 0xFFFFFFFF, 0)
    for i in np.nonzero(kind == 3)[0]:
        x[i, max(0, n - 2):n] = 0xFFFFFFFF                    # divisors and remainders with equal leading words
    x[:, n - 1] |= np.uint32(0x80000000)
    x[kind == 4, n] = rng.integers(-40 * n, 40 * n, size=int((kind == 4).sum())).astype(np.int32).view(np.uint32)
    return x


@pytest.mark.parametrize("bits", [64, 96, 128, 224, 256, 416, 512, 992, 1024])
def test_edge_operands(engine, oracle, bits):
    rng = np.random.default_rng(bits)
    count, n = 2000, bits // 32
    a, b, c = (edge_numbers(rng, count, bits) for _ in range(3))
    near = rng.integers(0, 4, size=count) == 0               # b = -a up to a few low bits: deep cancellation
    b[near] = nb.negate(a[near])
    b[near, 0] ^= rng.integers(0, 4, size=int(near.sum())).astype(np.uint32)
    for op in (api.Operation.add, api.Operation.sub, api.Operation.mul, api.Operation.div):
        got, _ = engine.run(bits, op, a, b)
        assert (got == oracle.elementwise(bits, int(op), a, b)).all(), op.name
    exact, _ = engine.run(bits, api.Operation.mul, a, c)      # quotients that are exact or one unit off
    got, _ = engine.run(bits, api.Operation.div, exact, c)
    assert (got == oracle.elementwise(bits, 3, exact, c)).all()
    got, _ = engine.run_ternary(bits, api.Operation.fma, a, b, c)
    assert (got == oracle.elementwise(bits, 9, a, b, c)).all()


@pytest.mark.parametrize("bits", [64, 160, 512, 1024])
def test_complex_in_place(engine, oracle, bits):
    rng = np.random.default_rng(bits + 1)
    count = 333
    x, y, z = (np.ascontiguousarray(np.stack([edge_numbers(rng, count, bits), edge_numbers(rng, count, bits)], axis=1)) for _ in range(3))
    for op in (api.Operation.complex_add, api.Operation.complex_mul, api.Operation.complex_div, api.Operation.complex_fma, api.Operation.complex_fms):
        ternary = api.operation_is_ternary(op)
        want = oracle.elementwise(bits, int(op), x, y, z if ternary else None)
        for target in range(3 if ternary else 2):
            bufs = [engine.make_buffer(count, bits, True) for _ in range(3)]
            for b, v in zip(bufs, (x, y, z)):
                b.upload(v)
            batch = engine.batch()
            args = bufs if ternary else bufs[:2]
            batch.run(op, *args, out=bufs[target])
            batch.submit().wait()
            assert (bufs[target].download() == want).all(), (op.name, target)
