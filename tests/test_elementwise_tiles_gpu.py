"""GPU: the element-wise kernels pass a block's 128 rows through shared memory; counts around whole blocks, arrays that do
not start on 16-byte boundaries, odd and even row lengths, broadcast operands and outputs over an input."""
import numpy as np
import pytest

from limbforge_b200 import api
from limbforge_b200 import numbers as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [64, 96, 256, 416, 928, 1024])
@pytest.mark.parametrize("shift", [0, 1])
def test_tiles(oracle, bits, shift):
    import torch
    rng = np.random.default_rng(bits + shift)
    E = bits // 32 + 3
    for count in (1, 63, 64, 65, 127, 128, 129, 300):
        for op in (api.Operation.mul, api.Operation.sqrt, api.Operation.fma, api.Operation.complex_mul, api.Operation.complex_fma):
            cx = api.operation_is_complex(op)
            make = nb.random_complex if cx else nb.random_numbers
            ins = [make(rng, count, bits, 30, zero_frac=0.05) for _ in range(3)]
            if op == api.Operation.sqrt:
                ins[0][ins[0][:, -2] != 0, -2] = 1
            used = 1 if api.operation_is_unary(op) else 3 if api.operation_is_ternary(op) else 2
            words = ins[0].size
            dev = [torch.zeros(words + 8, dtype=torch.int32, device="cuda") for _ in range(4)]
            for d, v in zip(dev, ins):
                d[shift:shift + words] = torch.from_numpy(v.view(np.int32).ravel()).cuda()
            torch.cuda.synchronize()
            want = oracle.elementwise(bits, int(op), ins[0], ins[1] if used > 1 else None, ins[2] if used > 2 else None)
            ptr = [d.data_ptr() + 4 * shift for d in dev]
            for out in (3, 0):                              # a buffer of its own, then over the first operand
                api.dev_elementwise(bits, op, ptr[0], ptr[1] if used > 1 else None, ptr[2] if used > 2 else None, ptr[out], count)
                torch.cuda.synchronize()
                got = dev[out][shift:shift + words].cpu().numpy().view(np.uint32).reshape(want.shape)
                assert (got == want).all(), (op.name, count, out)
                assert not dev[out][shift + words:].any()
    # broadcast operands: strides and periods that cut blocks
    a = nb.random_complex(rng, 300, bits, 30)
    b = nb.random_complex(rng, 100, bits, 30)
    da, db, do = (torch.from_numpy(v.view(np.int32)).cuda() for v in (a, b, np.zeros_like(a)))
    for stride, period in ((3, 0), (1, 7), (2, 5), (300, 0)):
        idx = np.arange(300) // stride
        idx = idx % period if period else idx
        api.dev_elementwise(bits, api.Operation.complex_mul, da.data_ptr(), db.data_ptr(), None, do.data_ptr(), 300,
                            api.Broadcast(stride, period))
        torch.cuda.synchronize()
        want = oracle.elementwise(bits, int(api.Operation.complex_mul), a, np.ascontiguousarray(b[idx]))
        assert (do.cpu().numpy().view(np.uint32) == want).all(), (stride, period)
