"""Timed cases of the GEMM backend, each one pass through a public call of
`ferray_b200` on operands that already lie in device memory.

A case is a dict of plain values:

* ``call``: "matmul" (NumPy-style product that returns a new array), "gemm"
  (the gemm_* call of the dtype, into a given C), "stacked"
  (gemm_batched_strided) or "ragged" (a prepared grouped plan);
* ``dtype``: f64, f32, c64 (two f64), c32 (two f32), i8, i16 or bf16;
* ``mode``: plain, split or split_f16;
* ``m``, ``n``, ``k``, and ``batch`` (stacked) or ``count`` and ``shapes``
  (ragged: the number of problems and the seed their sizes are drawn from);
* ``spread``: rows of A and columns of B are scaled by powers of ten from
  [-spread, spread] (split f64 / c64), 0 elsewhere.
"""
import math

import numpy as np
import torch

import ferray_b200 as fg

_NP = {"f64": np.float64, "f32": np.float32, "c64": np.complex128, "c32": np.complex64,
       "i8": np.int8, "i16": np.int16, "bf16": np.uint16}
_OUT = {"f64": np.float64, "f32": np.float32, "c64": np.complex128, "c32": np.complex64,
        "i8": np.int32, "i16": np.int32, "bf16": np.float32}
_ALIGN = 256  # bytes between the operands of a ragged batch, as separate device allocations have


def _case(call, dtype, mode, m=0, n=0, k=0, batch=1, count=0, shapes=0, spread=0, name=None):
    c = {"call": call, "dtype": dtype, "mode": mode, "m": m, "n": n, "k": k, "batch": batch, "count": count,
         "shapes": shapes, "spread": spread}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: an interactive product of two 100 x 100 matrices, all latency
        _case("matmul", "f64", "plain", 100, 100, 100, name="matmul_f64_100"),
        # a stack of small products in one call (batched linear algebra, attention-like heads)
        _case("stacked", "f32", "plain", 96, 80, 64, batch=512, name="stacked_f32_512"),
        # an ordinary dense SGEMM at the default (plain FP32) precision
        _case("gemm", "f32", "plain", 1536, 1536, 1536, name="sgemm_1536"),
        # the largest dense call: split SGEMM on the tensor cores
        _case("gemm", "f32", "split", 8192, 8192, 8192, name="sgemm_split_8192"),
        # a few rows against a large matrix (a decode step, a small batch of right-hand sides)
        _case("gemm", "f32", "plain", 32, 8192, 8192, name="sgemm_rows32"),
        _case("gemm", "f32", "split", 32, 8192, 8192, name="sgemm_split_rows32"),
        # an ordinary double-precision product, plain and emulated on the integer tensor cores
        _case("gemm", "f64", "plain", 1024, 1024, 1024, name="dgemm_1024"),
        _case("gemm", "f64", "split", 4096, 4096, 4096, spread=4, name="dgemm_split_4096"),
        # a complex product (signal processing): real and imaginary parts normal
        _case("gemm", "c32", "split", 4096, 4096, 4096, name="cgemm_split_4096"),
        # quantized integers and 16-bit floats, the two inference types
        _case("gemm", "i8", "plain", 4096, 4096, 4096, name="i8_4096"),
        _case("gemm", "bf16", "plain", 8192, 8192, 8192, name="bf16_8192"),
        # thousands of unrelated products of mixed sizes, one replayed plan
        _case("ragged", "f32", "plain", count=4096, shapes=42, name="ragged_f32_4096"),
    ]


def _log(rng, lo, hi):
    """An integer whose logarithm is uniform in [lo, hi]; half of them whole
    multiples of 16 where that is possible."""
    x = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if x >= 64 and rng.random() < 0.5:
        x = min(hi, (x + 8) // 16 * 16)
    return max(lo, min(hi, x))


# (dtype, mode, smallest, largest extent, most 2mnk of a drawn call)
_DENSE = [
    ("f32", "plain", 128, 4096, 6e10),
    ("f32", "split", 256, 8192, 8e11),
    ("f32", "split_f16", 256, 8192, 5e11),
    ("f64", "plain", 128, 4096, 3e10),
    ("f64", "split", 512, 4096, 1.3e11),
    ("c32", "split", 256, 4096, 1.3e11),
    ("c64", "split", 512, 2048, 1.7e10),
    ("i8", "plain", 256, 8192, 1.1e12),
    ("i16", "plain", 256, 8192, 1.1e12),
    ("bf16", "plain", 256, 8192, 1.1e12),
]
_SKINNY = [("f32", "plain"), ("f32", "split"), ("f64", "plain"), ("i8", "plain"), ("bf16", "plain")]


def draw(rng):
    kind = rng.choice(["small", "stacked", "dense", "dense", "dense", "dense", "rows", "rows", "ragged"])
    if kind == "small":
        dtype = rng.choice(["f64", "f32", "i8"])
        return _case("matmul", dtype, "plain", _log(rng, 10, 256), _log(rng, 10, 256), _log(rng, 10, 256))
    if kind == "stacked":
        dtype = rng.choice(["f32", "f64"])
        return _case("stacked", dtype, "plain", _log(rng, 16, 256), _log(rng, 16, 256), _log(rng, 16, 256),
                     batch=_log(rng, 16, 1024))
    if kind == "rows":
        dtype, mode = rng.choice(_SKINNY)
        return _case("gemm", dtype, mode, _log(rng, 2, 64), _log(rng, 1024, 8192), _log(rng, 1024, 8192))
    if kind == "ragged":
        dtype, mode = rng.choice([("f32", "plain"), ("f32", "split"), ("i8", "plain")])
        return _case("ragged", dtype, mode, count=_log(rng, 256, 4096), shapes=rng.randrange(1, 1 << 20))
    dtype, mode, lo, hi, most = rng.choice(_DENSE)
    while True:
        m, n, k = (_log(rng, lo, hi) for _ in range(3))
        if 2.0 * m * n * k <= most:
            break
    spread = rng.choice([0, 4, 8]) if mode == "split" and dtype in ("f64", "c64") else 0
    return _case("gemm", dtype, mode, m, n, k, spread=spread)


def _shapes(case):
    """(m, n, k) of every problem of a case."""
    if case["call"] == "ragged":
        rng = np.random.default_rng(case["shapes"])
        return np.rint(np.exp(rng.uniform(np.log(8), np.log(512), (case["count"], 3)))).astype(np.int64)
    return np.array([(case["m"], case["n"], case["k"])] * case["batch"], dtype=np.int64)


def work(case):
    d = _shapes(case).astype(np.float64)
    m, n, k = d[:, 0], d[:, 1], d[:, 2]
    e_in, e_out = np.dtype(_NP[case["dtype"]]).itemsize, np.dtype(_OUT[case["dtype"]]).itemsize
    flops = 8.0 if case["dtype"] in ("c64", "c32") else 2.0
    return {"bytes": float(((m * k + k * n) * e_in + m * n * e_out).sum()), "flops": float(flops * (m * n * k).sum())}


def _values(shape, dtype, gen):
    """Random operand values as a torch tensor: bf16 and f32 normal, f64
    uniform in [-1, 1), integers over their whole range."""
    if dtype == "f64":
        return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) * 2 - 1
    if dtype == "c64":
        return torch.randn(shape, generator=gen, device="cuda", dtype=torch.complex128)
    if dtype == "c32":
        return torch.randn(shape, generator=gen, device="cuda", dtype=torch.complex64)
    if dtype == "i8":
        return torch.randint(-128, 128, shape, generator=gen, device="cuda", dtype=torch.int8)
    if dtype == "i16":
        return torch.randint(-32768, 32768, shape, generator=gen, device="cuda", dtype=torch.int16)
    x = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)
    return x.bfloat16() if dtype == "bf16" else x


def _operands(case, seed):
    """A and B of a case (flat arenas for a ragged batch)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = case["dtype"]
    if case["call"] == "ragged":
        oa, ob, _, na, nb, _ = _arenas(case)
        return _values((na,), dtype, gen), _values((nb,), dtype, gen)
    m, n, k = case["m"], case["n"], case["k"]
    stack = (case["batch"],) if case["call"] == "stacked" else ()
    if case["spread"]:  # diag(10^(s u)) G diag(10^(s v)), G normal, u and v uniform in [-1, 1]
        def scaled(r, c):
            g = torch.randn((r, c), generator=gen, device="cuda",
                            dtype=torch.complex128 if dtype == "c64" else torch.float64)
            u, v = (torch.rand(x, generator=gen, device="cuda", dtype=torch.float64) * 2 - 1 for x in (r, c))
            return g * (10.0 ** (case["spread"] * u))[:, None] * (10.0 ** (case["spread"] * v))[None, :]
        return scaled(m, k), scaled(k, n)
    return _values(stack + (m, k), dtype, gen), _values(stack + (k, n), dtype, gen)


def _arenas(case):
    """Element offsets of every A, B and C of a ragged batch and the sizes of
    the three arenas they lie in."""
    d = _shapes(case)
    out = []
    for x, y, e in ((0, 2, _NP[case["dtype"]]), (2, 1, _NP[case["dtype"]]), (0, 1, _OUT[case["dtype"]])):
        step = _ALIGN // np.dtype(e).itemsize
        size = (d[:, x] * d[:, y] + step - 1) // step * step
        out.append(np.concatenate([[0], np.cumsum(size)]))
    return [o[:-1] for o in out] + [int(o[-1]) for o in out]


class _Cuda:
    """A DeviceArray as torch sees it; torch keeps this object, and so the
    array, alive."""

    def __init__(self, array, typestr):
        self.array = array
        self.__cuda_array_interface__ = {"shape": array.shape, "typestr": typestr, "data": (array.ptr, False),
                                         "version": 3, "strides": None}


def _view(array):
    """torch tensor over a DeviceArray (bf16 bit patterns as int16)."""
    typestr = "<i2" if array.dtype == np.uint16 else array.dtype.str
    return torch.as_tensor(_Cuda(array, typestr), device="cuda")


def _upload(x, dtype):
    d = fg.DeviceArray(tuple(x.shape), _NP[dtype])
    _view(d).copy_(x.view(torch.int16) if dtype == "bf16" else x)
    return d


class _Plan(fg.GroupedPlan):
    """A grouped plan that is given back with the state that holds it."""

    def __del__(self):
        self.close()


def prepare(case, seed):
    ta, tb = _operands(case, seed)
    a, b = _upload(ta, case["dtype"]), _upload(tb, case["dtype"])
    s = {"case": case, "a": a, "b": b}
    if case["call"] == "ragged":
        oa, ob, oc, _, _, nc = _arenas(case)
        c = fg.DeviceArray((nc,), _OUT[case["dtype"]])
        e_in, e_out = a.dtype.itemsize, c.dtype.itemsize
        problems = [(int(m), int(n), int(k), a.ptr + int(x) * e_in, b.ptr + int(y) * e_in, c.ptr + int(z) * e_out)
                    for (m, n, k), x, y, z in zip(_shapes(case), oa, ob, oc)]
        s["plan"] = _Plan(problems, dtype=_NP[case["dtype"]], mode=case["mode"])
    elif case["call"] != "matmul":
        stack = (case["batch"],) if case["call"] == "stacked" else ()
        c = fg.DeviceArray(stack + (case["m"], case["n"]), _OUT[case["dtype"]])
    if case["call"] != "matmul":
        s["c"], s["out"] = c, _view(c)
        s["out"].zero_()
    torch.cuda.synchronize()
    return s


def run(s):
    case, a, b = s["case"], s["a"], s["b"]
    m, n, k, mode = case["m"], case["n"], case["k"], case["mode"]
    if case["call"] == "matmul":
        return _view(fg.matmul(a, b, mode=mode))
    if case["call"] == "ragged":
        s["plan"].run()
        return s["out"]
    if case["call"] == "stacked":
        fg.gemm_batched_strided(_NP[case["dtype"]], case["batch"], m, n, k, a, m * k, b, k * n, s["c"], m * n,
                                mode=mode)
        return s["out"]
    dtype = case["dtype"]
    if dtype == "f64":
        fg.gemm_f64(m, n, k, 1.0, a, b, 0.0, s["c"], mode=mode)
    elif dtype == "f32":
        fg.gemm_f32(m, n, k, 1.0, a, b, 0.0, s["c"], mode=mode)
    elif dtype == "c64":
        fg.gemm_c64(m, n, k, 1.0, 0.0, a, b, 0.0, 0.0, s["c"], mode=mode)
    elif dtype == "c32":
        fg.gemm_c32(m, n, k, 1.0, 0.0, a, b, 0.0, 0.0, s["c"], mode=mode)
    elif dtype == "i8":
        fg.gemm_i8_signed(m, n, k, a, b, s["c"])
    elif dtype == "i16":
        fg.gemm_i16(m, n, k, a, b, s["c"])
    else:
        fg.gemm_bf16_f32(m, n, k, a, b, s["c"])
    return s["out"]


def exact(case, seed):
    if case["dtype"] in ("i8", "i16"):
        return None
    a, b = _operands(case, seed)
    wide = torch.complex128 if case["dtype"] in ("c64", "c32") else torch.float64
    a, b = a.to(wide), b.to(wide)
    if case["call"] != "ragged":
        return a @ b
    oa, ob, oc, _, _, nc = _arenas(case)
    c = torch.zeros(nc, dtype=wide, device="cuda")
    for (m, n, k), x, y, z in zip(_shapes(case).tolist(), oa.tolist(), ob.tolist(), oc.tolist()):
        torch.mm(a[x:x + m * k].view(m, k), b[y:y + k * n].view(k, n), out=c[z:z + m * n].view(m, n))
    return c
