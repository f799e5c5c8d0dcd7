"""The timed cases: what users of limbforge_b200 have it do, at the sizes of its configurations, tests and benchmark.

Each case goes through a public entry point: Engine/CommandBatch for element-wise work, chains, 4x4 LU and exact 4x4
products; Linalg for exact products, Cholesky with solves and Householder QR; RaggedPlan for mixed-precision batches.
Data stay in device buffers, as a program that chains operations keeps them, except where the entry point takes host
arrays by its nature (complex QR).  Every result is a correctly rounded number, so outputs are compared bit for bit.
"""
import ctypes
import math

import numpy as np
import torch

from limbforge_b200 import api

OPS = {o.name: o for o in api.Operation}
_program = {}


def _engine():
    """The program's one engine and one Linalg: made at the first use and kept, as the API intends."""
    if not _program:
        _program["engine"] = api.Engine()
        _program["linalg"] = api.Linalg(_program["engine"])
        _program["abi"] = ctypes.CDLL(api.LIBRARY)      # the Buffer forms of Cholesky and its solves are C ABI calls
    return _program["engine"]


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1))


def _numbers(g, count, bits, lo, hi, zero=0.0, sparse=0.0):
    """Elements int32 [count, N + 3]: random significands, signs +-1, exponents uniform in [lo, hi]; shares of exact
    zeros and of significands with at most four set bits (exact results and ties)."""
    n = bits // 32
    x = torch.randint(-2**31, 2**31, (count, n + 3), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    if sparse:
        at = torch.nonzero(torch.rand(count, generator=g, device="cuda") < sparse)[:, 0]
        x[at, :n] = 0
        for _ in range(3):
            word = torch.randint(0, n, (len(at),), generator=g, device="cuda")
            bit = torch.randint(0, 32, (len(at),), generator=g, device="cuda")
            x[at, word] |= torch.where(bit < 31, 1 << bit, -2**31).to(torch.int32)
    x[:, n - 1] |= -2**31
    x[:, n] = torch.randint(lo, hi + 1, (count,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    x[:, n + 1] = 2 * torch.randint(0, 2, (count,), generator=g, device="cuda", dtype=torch.int32) - 1
    x[:, n + 2] = 0
    if zero:
        x[torch.rand(count, generator=g, device="cuda") < zero] = 0
    return x


def _uniform(g, count, bits):
    """Uniform in [-1, 1]: exponent -1 with probability 1/2, -2 with 1/4 and so on."""
    x = _numbers(g, count, bits, 0, 0)
    u = torch.rand(count, generator=g, device="cuda").clamp_min(2.0**-24)
    x[:, bits // 32] = (-torch.ceil(-torch.log2(u)).clamp_min(1)).to(torch.int32)
    return x


def _least_squares_matrix(g, m, n, bits):
    """Columns scaled by 2^[-60, 60], entries within 2^+-15 of their column's scale, a quarter of them zero, and in
    every 17th column one entry 2^-150 below the scale."""
    N = bits // 32
    x = _numbers(g, m * n, bits, -15, 15, zero=0.25).view(m, n, N + 3)
    scale = torch.randint(-60, 61, (n,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    live = x[:, :, N + 1] != 0
    x[:, :, N] = torch.where(live, x[:, :, N] + scale, 0)
    cols = torch.arange(5, n, 17, device="cuda")
    rows = torch.randint(0, m, (len(cols),), generator=g, device="cuda")
    far = torch.where(live[rows, cols], scale[cols] - 150, 0).to(torch.int32)
    x[rows, cols, N] = far
    return x.view(m * n, N + 3)


class _Words:
    """A buffer's device words for torch.as_tensor, which keeps this object, and so the buffer, as long as its tensor."""

    def __init__(self, buffer):
        self.buffer = buffer
        self.__cuda_array_interface__ = {"shape": (buffer.count * buffer.words,), "typestr": "<i4",
                                         "data": (buffer.device_pointer(), False), "version": 3}


def _view(buffer):
    """The buffer's device words as a tensor (no copy)."""
    return torch.as_tensor(_Words(buffer), device="cuda").view(buffer.count, buffer.words)


def _buffer(x, bits, complex_=False):
    b = _engine().make_buffer(len(x), bits, complex_)
    _view(b).copy_(x.reshape(len(x), -1))
    return b


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # one small call: what a caller waits for when few values are in hand
        {"name": "mul_256_1000", "kind": "elementwise", "bits": 256, "op": "mul", "count": 1000},
        # the 256-bit element-wise configuration
        {"name": "fma_256_65536", "kind": "elementwise", "bits": 256, "op": "fma", "count": 65536},
        # a large odd batch at a middle width
        {"name": "div_512_1000003", "kind": "elementwise", "bits": 512, "op": "div", "count": 1000003},
        # complex division at the largest width
        {"name": "cdiv_1024_65536", "kind": "elementwise", "bits": 1024, "op": "complex_div", "count": 65536},
        # the headline: products in sequence on resident values
        {"name": "chain_1024_65536x16", "kind": "chain", "bits": 1024, "count": 65536, "steps": 16},
        # the exact dense product C <- RN(C - A^T B)
        {"name": "gemm_512_1024", "kind": "product", "bits": 512, "m": 1024, "n": 1024, "k": 1024, "lower": False,
         "subtract": True, "span": 40},
        # normal equations: the lower triangle of A^T A, 2000 x 1000, sizes that fill no tile
        {"name": "syrk_256_1000x2000", "kind": "product", "bits": 256, "m": 1000, "n": 1000, "k": 2000, "lower": True,
         "subtract": False, "span": 10},
        # factor an SPD matrix and solve for 64 right-hand sides
        {"name": "spd_256_2048x64", "kind": "spd", "bits": 256, "n": 2048, "rhs": 64},
        # least squares by Householder QR
        {"name": "qr_256_2000x1000", "kind": "qr", "bits": 256, "m": 2000, "n": 1000, "rhs": 4, "complex": False, "pivot": False},
        # complex least squares from host arrays
        {"name": "cqr_256_800x400", "kind": "qr", "bits": 256, "m": 800, "n": 400, "rhs": 4, "complex": True, "pivot": False},
        # the exact 4x4 product
        {"name": "exact4_448_100000", "kind": "exact4", "bits": 448, "count": 100000, "complex": True, "accumulate": True},
        # mixed precisions and sizes in one launch, with the 4x4 LU job
        {"name": "ragged_20000", "kind": "ragged", "gemms": 20000, "lu": 200000, "complex": True, "fused": False},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["elementwise", "elementwise", "elementwise", "chain", "product", "product", "spd", "qr", "qr", "exact4", "lu4", "ragged"])
    bits = 32 * rng.randint(2, 32)
    if kind == "elementwise":
        op = rng.choice(sorted(OPS))
        return {"kind": kind, "bits": bits, "op": op, "count": _log(rng, 500, 1000000 if bits <= 512 else 300000)}
    if kind == "chain":
        return {"kind": kind, "bits": bits, "count": _log(rng, 1000, 200000), "steps": rng.randint(2, 32)}
    if kind == "product":
        bits = 32 * rng.randint(2, 24)
        wide = rng.random() < 0.2                      # exponents too far apart for the residue engine
        m, n, k = (_log(rng, 24, 300 if wide else 1200) for _ in range(3))
        lower = rng.random() < 0.4
        return {"kind": kind, "bits": bits, "m": m, "n": m if lower else n, "k": k, "lower": lower, "subtract": rng.random() < 0.5,
                "span": rng.randint(150, 400) if wide else rng.randint(4, 40)}
    if kind == "spd":
        return {"kind": kind, "bits": 32 * rng.randint(3, 12), "n": _log(rng, 60, 1200), "rhs": _log(rng, 1, 64)}
    if kind == "qr":
        cx, pivot = rng.random() < 0.3, rng.random() < 0.25
        n = _log(rng, 16, 200 if cx or pivot else 600)
        return {"kind": kind, "bits": 32 * rng.randint(4, 12), "m": int(n * rng.uniform(1.0, 2.5)) + 1, "n": n, "rhs": rng.randint(1, 8),
                "complex": cx, "pivot": pivot}
    if kind == "exact4":
        return {"kind": kind, "bits": bits, "count": _log(rng, 500, 60000), "complex": rng.random() < 0.5, "accumulate": rng.random() < 0.5}
    if kind == "lu4":
        inverse = rng.random() < 0.5
        return {"kind": kind, "bits": bits, "count": _log(rng, 500, 60000), "inverse": inverse, "rhs": 0 if inverse else rng.randint(1, 4),
                "fused": rng.random() < 0.3}
    return {"kind": kind, "gemms": _log(rng, 50, 4000), "lu": _log(rng, 500, 60000), "complex": rng.random() < 0.7, "fused": rng.random() < 0.3}


# ------------------------------------------------------------------------------------------------ prepare
def prepare(case, seed):
    eng, g = _engine(), _generator(seed)
    state = _PREPARE[case["kind"]](case, eng, g)
    state["case"] = case
    torch.cuda.synchronize()
    return state


def _prepare_elementwise(case, eng, g):
    bits, op, count = case["bits"], OPS[case["op"]], case["count"]
    cx = api.operation_is_complex(op)
    span = 8 if cx else 256
    inputs = 1 if api.operation_is_unary(op) else 3 if api.operation_is_ternary(op) else 2
    bufs = []
    for _ in range(inputs):
        x = _numbers(g, count * (2 if cx else 1), bits, -span, span, zero=0.01, sparse=0.02)
        bufs.append(_buffer(x.view(count, -1), bits, cx))
    return {"in": bufs, "out": eng.make_buffer(count, bits, cx), "op": op}


def _prepare_chain(case, eng, g):
    bits, count = case["bits"], case["count"]
    bufs = [_buffer(_numbers(g, count, bits, -8, 8, zero=0.01, sparse=0.02), bits) for _ in range(case["steps"] + 1)]
    return {"x": bufs[0], "factors": bufs[1:], "out": eng.make_buffer(count, bits)}


def _prepare_product(case, eng, g):
    bits, m, n, k, span = (case[f] for f in ("bits", "m", "n", "k", "span"))
    a = _numbers(g, k * m, bits, -span, span, zero=0.005)
    b = a if case["lower"] else _numbers(g, k * n, bits, -span, span, zero=0.005)
    return {"a": a, "b": b, "c": _numbers(g, m * n, bits, -span, span, zero=0.005)}


def _prepare_spd(case, eng, g):
    bits, n, rhs = case["bits"], case["n"], case["rhs"]
    gm = _uniform(g, n * n, bits)
    a = torch.zeros_like(gm)
    torch.cuda.synchronize()
    _program["linalg"].dev_exact_product(bits, gm.data_ptr(), 1, n, gm.data_ptr(), 1, n, n, n, n, a.data_ptr(), n)
    torch.cuda.synchronize()
    diag = a[:: n + 1].contiguous()
    shift = torch.zeros_like(diag)
    e = n.bit_length() - 1
    top = n << (31 - e)
    shift[:, bits // 32 - 1], shift[:, bits // 32], shift[:, bits // 32 + 1] = top - 2**32, e, 1
    api.dev_elementwise(bits, OPS["add"], diag.data_ptr(), shift.data_ptr(), None, diag.data_ptr(), n)
    a[:: n + 1] = diag
    return {"A": _buffer(a, bits), "L": eng.make_buffer(n * n, bits), "B": _buffer(_uniform(g, n * rhs, bits), bits),
            "X": eng.make_buffer(n * rhs, bits)}


def _prepare_qr(case, eng, g):
    bits, m, n, rhs = (case[f] for f in ("bits", "m", "n", "rhs"))
    if case["complex"]:
        a = torch.stack([_least_squares_matrix(g, m, n, bits) for _ in range(2)], dim=1)
        b = _numbers(g, 2 * m * rhs, bits, -8, 8, zero=0.09).view(m * rhs, 2, -1)
        return {"A": a.cpu().numpy().view(np.uint32), "B": b.cpu().numpy().view(np.uint32)}
    return {"A": _buffer(_least_squares_matrix(g, m, n, bits), bits), "B": _buffer(_numbers(g, m * rhs, bits, -8, 8, zero=0.09), bits),
            "X": eng.make_buffer(n * rhs, bits)}


def _prepare_exact4(case, eng, g):
    bits, count, cx = case["bits"], case["count"], case["complex"]
    parts = 2 if cx else 1
    bufs = [_buffer(_numbers(g, count * 16 * parts, bits, -30, 30, zero=0.01, sparse=0.05).view(count * 16, -1), bits, cx) for _ in range(3)]
    return {"bufs": bufs, "gemm4": api.ExactGemm4(eng),
            "shape": api.ExactGemm4Shape(count, 16, 16, 16, case["accumulate"], False)}


def _prepare_lu4(case, eng, g):
    bits, count, inverse = case["bits"], case["count"], case["inverse"]
    a = _buffer(_numbers(g, count * 32, bits, -32, 32).view(count * 16, -1), bits, True)
    cols = 4 if inverse else case["rhs"]
    b = None if inverse else _buffer(_numbers(g, count * 8 * cols, bits, -32, 32).view(count * 4 * cols, -1), bits, True)
    return {"A": a, "B": b, "X": eng.make_buffer(count * 4 * cols, bits, True), "det": eng.make_buffer(count, bits, True),
            "status": eng.make_buffer(count), "shape": api.Batched4(count, case["rhs"], inverse, True, case["fused"])}


def _prepare_ragged(case, eng, g):
    cx, count, lu_count = case["complex"], case["gemms"], case["lu"]
    parts = 2 if cx else 1
    sizes = np.random.default_rng([count, lu_count])       # the sizes are the case's, the values the seed's
    items = api.ragged_items(sizes.choice([128, 256, 512, 1024], size=count), *sizes.integers(4, 49, size=(3, count)))
    lu = api.RaggedLu4(512, api.Batched4(count=lu_count, rhs=1))
    total = api.ragged_pack(cx, items, lu)
    arena = torch.randint(-2**31, 2**31, (total // 4,), generator=g, device="cuda", dtype=torch.int32)

    def shape_elements(first_words, counts, bits):
        """Headers (top bit, exponent, sign, status) of runs of elements: run r starts at word first_words[r]."""
        n = bits // 32
        first, counts = (torch.as_tensor(np.asarray(v).astype(np.int64), device="cuda") for v in (first_words, counts))
        which = torch.repeat_interleave(torch.arange(len(counts), device="cuda"), counts)
        at = torch.arange(len(which), device="cuda") - (torch.cumsum(counts, 0) - counts)[which]
        at = first[which] + at * (n + 3)
        arena[at + n - 1] |= -2**31
        arena[at + n] = torch.randint(-32, 33, (len(at),), generator=g, device="cuda", dtype=torch.int32)
        arena[at + n + 1] = 2 * torch.randint(0, 2, (len(at),), generator=g, device="cuda", dtype=torch.int32) - 1
        arena[at + n + 2] = 0
    for bits in (128, 256, 512, 1024):
        t = items[items["bits"] == bits]
        m, n, k = (t[f].astype(np.int64) for f in "mnk")
        shape_elements(t["a"] // 4, m * k * parts, bits)
        shape_elements(t["b"] // 4, k * n * parts, bits)
    shape_elements([lu.A // 4], [lu_count * 32], 512)
    shape_elements([lu.B // 4], [lu_count * 8], 512)
    plan = api.RaggedPlan(eng, cx, case["fused"], items, total, lu)
    torch.cuda.synchronize()
    plan.tune(arena.data_ptr())
    return {"arena": arena, "plan": plan}


_PREPARE = {"elementwise": _prepare_elementwise, "chain": _prepare_chain, "product": _prepare_product, "spd": _prepare_spd,
            "qr": _prepare_qr, "exact4": _prepare_exact4, "lu4": _prepare_lu4, "ragged": _prepare_ragged}


# ------------------------------------------------------------------------------------------------ run
def run(state):
    return _RUN[state["case"]["kind"]](state)


def _run_elementwise(s):
    batch = _engine().batch()
    batch.run(s["op"], *s["in"], out=s["out"])
    batch.submit().wait()
    return _view(s["out"])


def _run_chain(s):
    batch = _engine().batch()
    x = s["x"]
    for f in s["factors"]:
        batch.run(OPS["mul"], x, f, None, s["out"])
        x = s["out"]
    batch.submit().wait()
    return _view(s["out"])


def _run_product(s):
    c = s["case"]
    m, n, k = c["m"], c["n"], c["k"]
    _program["linalg"].dev_exact_product(c["bits"], s["a"].data_ptr(), 1, m, s["b"].data_ptr(), 1, n, m, n, k, s["c"].data_ptr(), n,
                                         subtract=c["subtract"], lower=c["lower"])
    return s["c"]


def _run_spd(s):
    c, abi, la = s["case"], _program["abi"], ctypes.c_void_p(_program["linalg"].handle.value)
    bits, n, rhs = c["bits"], ctypes.c_size_t(c["n"]), ctypes.c_size_t(c["rhs"])
    api.check(abi.lf_linalg_cholesky_buffers(la, bits, s["A"].handle, n, s["L"].handle, None, None))
    api.check(abi.lf_linalg_solve_buffers(la, bits, 3, s["L"].handle, n, s["B"].handle, rhs, s["X"].handle, None, None))
    return _view(s["L"]), _view(s["X"])


def _run_qr(s):
    c, la = s["case"], _program["linalg"]
    options = api.QROptions(pivot=c["pivot"])
    if c["complex"]:
        f = la.factor_qr_complex(c["bits"], s["A"], c["m"], c["n"], options)
        return f.solve(s["B"], c["rhs"]).view(np.int32), f.tau().view(np.int32)
    f = la.factor_qr_buffer(s["A"], c["m"], c["n"], options)
    f.solve_buffers(s["B"], c["rhs"], s["X"])
    return _view(s["X"]), f.tau().view(np.int32)


def _run_exact4(s):
    batch = _engine().batch()
    s["gemm4"].encode(batch, s["shape"], *s["bufs"])
    batch.submit().wait()
    return _view(s["bufs"][2])


def _run_lu4(s):
    batch = _engine().batch()
    batch.lu4(s["shape"], s["A"], s["B"], s["X"], s["det"], s["status"])
    batch.submit().wait()
    return _view(s["X"]), _view(s["det"]), _view(s["status"])


def _run_ragged(s):
    s["plan"].run(s["arena"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    return s["arena"]


_RUN = {"elementwise": _run_elementwise, "chain": _run_chain, "product": _run_product, "spd": _run_spd, "qr": _run_qr,
        "exact4": _run_exact4, "lu4": _run_lu4, "ragged": _run_ragged}


# ------------------------------------------------------------------------------------------------ work, tolerance, exact
def work(case):
    """Each input read once and each output written once; two operations per 32 x 32-bit word product of the schoolbook
    form (quotients and roots count as one product)."""
    kind = case["kind"]
    if kind == "ragged":
        # the expected size of the draw: m, n, k uniform in 4..48 (mean 26), four widths
        parts, mean, mean_words = (2 if case["complex"] else 1), 26.0, (7 + 11 + 19 + 35) / 4
        products = 4 if case["complex"] else 1
        squares = (4**2 + 8**2 + 16**2 + 32**2) / 4
        return {"bytes": 4 * (case["gemms"] * 3 * mean**2 * parts * mean_words + case["lu"] * 24 * 2 * 19),
                "flops": 2 * (case["gemms"] * mean**3 * products * squares + case["lu"] * 46 * 4 * 16**2)}
    N = case["bits"] // 32
    E, P = 4 * (N + 3), N * N
    if kind == "elementwise":
        op = OPS[case["op"]]
        cx = api.operation_is_complex(op)
        arrays = 2 if api.operation_is_unary(op) else 4 if api.operation_is_ternary(op) else 3
        products = 0 if op in (0, 1, 4) else 8 if op == 6 else 4 if cx else 1
        return {"bytes": case["count"] * E * arrays * (2 if cx else 1), "flops": 2 * case["count"] * max(products * P, N)}
    if kind == "chain":
        return {"bytes": case["count"] * E * (case["steps"] + 2), "flops": 2 * case["count"] * case["steps"] * P}
    if kind == "product":
        m, n, k = case["m"], case["n"], case["k"]
        outputs = m * (m + 1) / 2 if case["lower"] else m * n
        operands = k * m if case["lower"] else k * (m + n)
        return {"bytes": E * (operands + outputs * (2 if case["subtract"] else 1)), "flops": 2 * outputs * k * P}
    if kind == "spd":
        n, rhs = case["n"], case["rhs"]
        return {"bytes": E * (n * n + 2 * n * rhs), "flops": 2 * P * (n**3 / 6 + n * n * rhs)}
    if kind == "qr":
        m, n, rhs, parts = case["m"], case["n"], case["rhs"], (2 if case["complex"] else 1)
        macs = m * n * n - n**3 / 3 + (2 * m * n + n * n / 2) * rhs
        return {"bytes": E * parts * (m * n + (m + n) * rhs), "flops": 2 * P * macs * parts**2}
    if kind == "exact4":
        parts = 2 if case["complex"] else 1
        return {"bytes": E * parts * case["count"] * 16 * (4 if case["accumulate"] else 3), "flops": 2 * P * case["count"] * 64 * parts**2}
    cols = 4 if case["inverse"] else case["rhs"]
    return {"bytes": case["count"] * (2 * E * (16 + 4 * cols + (0 if case["inverse"] else 4 * cols) + 1) + 4),
            "flops": 2 * P * case["count"] * 4 * (30 + 16 * cols)}


def tolerance(case):
    """Every result is the correctly rounded value of a fixed rounding sequence: one answer, bit for bit."""
    return "exact"


def exact(case, seed):
    """Results are 64..1024-bit integers in words, which 64-bit numbers cannot hold: they are compared bit for bit."""
    return None
