"""The calls this framework's speed is judged by: convolutions, broadcast expressions and matrix products as a user's program
issues them, through the Function / Tensor layer (`Function.of(...)`, `@`, `backward`) or, where a program keeps its own result
buffers as the JVM host does, through the C ABI (`nk_conv` into a drain that exists already).

A case is a dict of plain values; shapes are texts such as "8x32x512x512". Inputs are made on the GPU from a seed.
"""
from __future__ import annotations

import ctypes as C
import math

import torch

from neureka_b200 import _lib as L
from neureka_b200.device import CudaDevice
from neureka_b200.functions import Function
from neureka_b200.ndconf import NDConfiguration
from neureka_b200.tensor import Tensor

_TORCH = {"float32": torch.float32, "float64": torch.float64}
_NK = {"float32": L.NK_F32, "float64": L.NK_F64}
_BYTES = {"float32": 4, "float64": 8}

CHAIN = "tanh(i0*i1+i1)"
VIEWS = "i0*i1+i2"


def listed():
    return [
        # one small image and one filter: the cost of a call
        {"name": "conv_image_small", "op": "conv", "dtype": "float32", "image": "256x256", "kernel": "5x5"},
        # a multi-channel plane collapsed to one output, e.g. a spectral cube or a layer's single feature
        {"name": "conv_channels", "op": "conv_into", "dtype": "float32", "image": "64x512x512", "kernel": "64x3x3"},
        # a batch of large multi-channel images, result buffer kept by the program
        {"name": "conv_batch_large", "op": "conv_into", "dtype": "float32", "image": "8x32x2048x2048", "kernel": "1x32x5x5"},
        # the backward pass of such a batch: gradients of image and kernel into kept buffers
        {"name": "conv_batch_gradients", "op": "conv_gradients", "dtype": "float32", "image": "8x32x512x2048", "kernel": "1x32x5x5"},
        # a training step on a batch of small images of odd width
        {"name": "conv_train_ragged", "op": "conv_train", "dtype": "float32", "image": "16x16x131x127", "kernel": "1x16x3x3"},
        # a training step on a volume in double precision
        {"name": "conv_train_volume_f64", "op": "conv_train", "dtype": "float64", "image": "128x128x128", "kernel": "7x7x7"},
        # a broadcast expression op by op, its sum, and the gradients of that sum for both operands
        {"name": "chain_train", "op": "chain_train", "dtype": "float32", "rows": 256, "cols": 256, "inner": 1024},
        # the same kind of expression as one compiled operation, forward and backward, at odd extents
        {"name": "fused_train_ragged", "op": "fused_train", "dtype": "float32", "expr": "silu(i0*i1+i1)", "rows": 100, "cols": 333, "inner": 777},
        # a dense layer's product and both of its gradients
        {"name": "matmul_train_large", "op": "matmul_train", "dtype": "float32", "m": 4096, "k": 4096, "n": 4096},
        # a product of odd sizes in double precision
        {"name": "matmul_ragged_f64", "op": "matmul", "dtype": "float64", "m": 777, "k": 1023, "n": 515},
        # activation of a small layer's output plus its bias
        {"name": "layer_epilogue_small", "op": "epilogue", "dtype": "float32", "fun": "gelu", "rows": 64, "inner": 1000},
        # slices, a transposed operand and a row vector in one expression
        {"name": "views_expression", "op": "views", "dtype": "float32", "rows": 4093, "inner": 4099},
    ]


def _log(rng, lo, hi):
    """an integer spread over the logarithm of its range, odd values as likely as even ones"""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    op = rng.choice(["conv", "conv_into", "conv_gradients", "conv_train", "chain_train", "fused_train", "matmul_train", "matmul", "epilogue", "views"])
    dtype = rng.choice(["float32", "float32", "float32", "float64"])
    case = {"op": op, "dtype": dtype}
    if op.startswith("conv"):
        most = (1 << 28 if op in ("conv_into", "conv_gradients") else 1 << 24) // (2 if dtype == "float64" else 1)
        window = rng.choice([3, 5, 7]) if dtype == "float64" else rng.choice([3, 5])
        kind = rng.choice(["plane", "channels", "batch", "volume"])
        while True:
            h, w = _log(rng, 64, 2048), _log(rng, 64, 2048)
            c, b = _log(rng, 3, 64), _log(rng, 1, 16)
            if kind == "plane":
                image, kernel = [h, w], [window, window]
            elif kind == "channels":
                image, kernel = [c, h, w], [c, window, window]
            elif kind == "batch":
                image, kernel = [b, c, h, w], [1, c, window, window]
            else:
                d = _log(rng, 16, 160)
                image, kernel = [d, h, w], [window, window, window]
            if math.prod(image) <= most:
                break
        case["image"], case["kernel"] = "x".join(map(str, image)), "x".join(map(str, kernel))
    elif op in ("chain_train", "fused_train"):
        while True:
            case["rows"], case["cols"], case["inner"] = _log(rng, 8, 512), _log(rng, 8, 512), _log(rng, 32, 2048)
            if case["rows"] * case["cols"] * case["inner"] <= (1 << 26) // (2 if dtype == "float64" else 1):
                break
        if op == "fused_train":
            case["expr"] = rng.choice(["silu(i0*i1+i1)", "i0*i1+i1"])
    elif op.startswith("matmul"):
        most = 4096 if dtype == "float32" else 1536
        case["m"], case["k"], case["n"] = (_log(rng, 64, most) for _ in range(3))
    elif op == "epilogue":
        case["fun"] = rng.choice(["gelu", "relu", "tanh", "sig"])
        case["rows"], case["inner"] = _log(rng, 16, 4096), _log(rng, 32, 4096)
    else:
        case["rows"], case["inner"] = _log(rng, 64, 4096), _log(rng, 64, 4096)
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------
class _DevicePointer:
    """a tensor's memory as torch sees it (no copy); keeps the tensor alive"""

    def __init__(self, tensor, shape, dtype):
        ptr = C.c_void_p()
        L.check(L.lib.nk_buf_info(tensor._data.buf, C.byref(ptr), None, None))
        self.tensor = tensor
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4" if dtype == "float32" else "<f8", "data": (ptr.value, False), "version": 3}


def _as_torch(tensor):
    return torch.as_tensor(_DevicePointer(tensor, tensor.shape, tensor.dtype.name), device="cuda")


def _stored(device, dtype, values):
    """a tensor on the device holding the given torch values"""
    t = Tensor.of(dtype, tuple(values.shape), 0).to(device).set_is_virtual(False)
    device.sync()
    _as_torch(t).copy_(values)
    return t


class _Buffer:
    """a program's own device memory as the C ABI takes it, with its view descriptor"""

    def __init__(self, device, values, dtype):
        self.values, self.device = values, device
        self.handle = C.c_void_p()
        L.check(L.lib.nk_wrap(device.ctx, _NK[dtype], C.c_void_p(values.data_ptr()), values.numel(), C.byref(self.handle)), device.ctx)
        self._inline = NDConfiguration.of_shape(tuple(values.shape)).as_inline_array()
        self.cfg = self._inline.ctypes.data_as(C.POINTER(C.c_int32))

    def __del__(self):
        L.lib.nk_free(self.device.ctx, self.handle)


_FUSED = {}


def _fused(device, expr):
    """a program compiles its operation once and keeps it"""
    if expr not in _FUSED:
        _FUSED[expr] = device.optimized_operation_of(Function.of(expr), "cases")
    return _FUSED[expr]


def _conv_shapes(case):
    image, kernel = ([int(s) for s in case[k].split("x")] for k in ("image", "kernel"))
    return image, kernel, [a - b + 1 for a, b in zip(image, kernel)]


def prepare(case, seed):
    device = CudaDevice.get(0)
    op, dtype = case["op"], case["dtype"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    td = _TORCH[dtype]

    def uniform(lo, hi, *shape):
        return torch.empty(shape, dtype=td, device="cuda").uniform_(lo, hi, generator=g)

    def normal(std, *shape):
        return torch.empty(shape, dtype=td, device="cuda").normal_(0.0, std, generator=g)

    s = {"op": op, "device": device, "nk": _NK[dtype]}
    if op.startswith("conv"):
        image, kernel, out = _conv_shapes(case)
        taps = math.prod(kernel)
        a, k = uniform(0.0, 1.0, *image), normal(1.0 / math.sqrt(taps), *kernel)   # pixel values; filter weights of unit gain
        if op in ("conv", "conv_train"):
            s["a"], s["k"] = _stored(device, dtype, a), _stored(device, dtype, k)
            s["f"] = Function.of("i0 x i1")
            if op == "conv_train":
                s["e"] = _stored(device, dtype, normal(1.0, *out))
                s["a"].set_rqs_gradient(True)
                s["k"].set_rqs_gradient(True)
        else:
            s["rank"] = len(image)
            s["a"], s["k"] = _Buffer(device, a, dtype), _Buffer(device, k, dtype)
            if op == "conv_into":
                s["y"] = _Buffer(device, torch.empty(out, dtype=td, device="cuda"), dtype)
            else:
                s["e"] = _Buffer(device, normal(1.0, *out), dtype)
                s["ga"], s["gk"] = _Buffer(device, torch.empty_like(a), dtype), _Buffer(device, torch.empty_like(k), dtype)
    elif op in ("chain_train", "fused_train"):
        n, m, k = case["rows"], case["cols"], case["inner"]
        s["a"], s["b"] = _stored(device, dtype, uniform(-2.0, 2.0, n, 1, k)), _stored(device, dtype, uniform(-2.0, 2.0, 1, m, k))
        s["a"].set_rqs_gradient(True)
        s["b"].set_rqs_gradient(True)
        if op == "chain_train":
            s["f"], s["sum"] = Function.of(CHAIN), Function.of("sumItems(i0)")
        else:
            s["f"], s["e"] = _fused(device, case["expr"]), _stored(device, dtype, normal(1.0, n, m, k))
    elif op.startswith("matmul"):
        m, k, n = case["m"], case["k"], case["n"]
        s["a"], s["b"] = _stored(device, dtype, normal(1.0, m, k)), _stored(device, dtype, normal(1.0 / math.sqrt(k), k, n))
        s["f"] = Function.of("i0 @ i1")
        if op == "matmul_train":
            s["e"] = _stored(device, dtype, normal(1.0, m, n))
            s["a"].set_rqs_gradient(True)
            s["b"].set_rqs_gradient(True)
    elif op == "epilogue":
        s["a"], s["b"] = _stored(device, dtype, normal(1.0, case["rows"], case["inner"])), _stored(device, dtype, normal(1.0, 1, case["inner"]))
        s["f"] = Function.of(case["fun"] + "(i0+i1)")
    else:
        n, m = case["rows"], case["inner"]
        s["a"], s["b"], s["c"] = (_stored(device, dtype, normal(1.0, *shape)) for shape in ((n + 3, m + 5), (m, n), (1, m)))
        s["f"] = Function.of(VIEWS)
    torch.cuda.synchronize()
    return s


def run(s):
    op = s["op"]
    if op == "conv_into":
        d = s["device"]
        L.check(L.lib.nk_conv(d.ctx, s["nk"], s["rank"], s["y"].handle, s["y"].cfg, s["a"].handle, s["a"].cfg, s["k"].handle, s["k"].cfg, -1), d.ctx)
        return s["y"].values
    if op == "conv_gradients":   # the drain, then the operands in the order of XConvRight after its rearrangement
        d, a, k, e, ga, gk = s["device"], s["a"], s["k"], s["e"], s["ga"], s["gk"]
        L.check(L.lib.nk_conv(d.ctx, s["nk"], s["rank"], ga.handle, ga.cfg, k.handle, k.cfg, e.handle, e.cfg, 0), d.ctx)
        L.check(L.lib.nk_conv(d.ctx, s["nk"], s["rank"], gk.handle, gk.cfg, a.handle, a.cfg, e.handle, e.cfg, 0), d.ctx)
        return [ga.values, gk.values]
    if op == "conv":
        return _as_torch(s["f"](s["a"], s["k"]))
    if op in ("matmul", "epilogue"):
        return _as_torch(s["f"](s["a"], s["b"]))
    if op == "views":
        return _as_torch(s["f"](s["a"][3:, 5:], s["b"].permute(1, 0), s["c"]))
    a, b = s["a"], s["k" if op == "conv_train" else "b"]
    a.gradient = b.gradient = None   # a new step
    y = s["f"](a, b)
    if op == "chain_train":
        loss = s["sum"](y)
        loss.backward()
        return [_as_torch(t) for t in (y, loss, a.gradient, b.gradient)]
    y.backward(s["e"])
    return [_as_torch(t) for t in (y, a.gradient, b.gradient)]


def work(case):
    op, size = case["op"], _BYTES[case["dtype"]]
    if op.startswith("conv"):
        image, kernel, out = _conv_shapes(case)
        a, k, y = math.prod(image), math.prod(kernel), math.prod(out)
        fma = 2.0 * y * k
        passes, moved = {"conv": (1, a + k + y), "conv_into": (1, a + k + y), "conv_gradients": (2, 2 * a + 2 * k + y),
                         "conv_train": (3, 2 * a + 2 * k + 2 * y)}[op]
        return {"bytes": size * moved, "flops": passes * fma}
    if op in ("chain_train", "fused_train"):
        n, m, k = case["rows"], case["cols"], case["inner"]
        full = n * m * k
        moved = 2 * (n + m) * k + (full if op == "chain_train" else 2 * full)   # fused: the error is an input
        return {"bytes": size * moved, "flops": 10.0 * full}
    if op.startswith("matmul"):
        m, k, n = case["m"], case["k"], case["n"]
        if op == "matmul":
            return {"bytes": size * (m * k + k * n + m * n), "flops": 2.0 * m * k * n}
        return {"bytes": size * 2 * (m * k + k * n + m * n), "flops": 6.0 * m * k * n}
    if op == "epilogue":
        n, m = case["rows"], case["inner"]
        return {"bytes": size * (2 * n * m + m), "flops": 2.0 * n * m}
    n, m = case["rows"], case["inner"]
    return {"bytes": size * (3 * n * m + m), "flops": 2.0 * n * m}


def tolerance(case):
    """About four times what the path differs by from the same result computed in 64 bits (for float64: in another order)."""
    op, double = case["op"], case["dtype"] == "float64"
    if op in ("epilogue", "views"):   # one rounding per operation; the functions to one unit in the last place
        return {"rel": 1e-15, "max": 4e-15} if double else {"rel": 1.3e-7, "max": 7e-7}
    if double:
        return {"rel": 1e-14, "max": 5e-14}
    if op == "conv_into" or op == "conv":   # seen: 2.2e-7
        return {"rel": 1e-6, "max": 6e-6}
    if op.startswith("conv"):   # kernel gradients are sums over whole images; seen: 1.6e-6
        return {"rel": 6e-6, "max": 3e-5}
    return {"rel": 4e-6, "max": 2e-5}   # products and reduced gradients; seen: 9.2e-7
