"""The operators' two host paths, without a GPU: csrc/native.cpp takes a call only where ops.py would make the same one.

Both run against a library that records its calls (ctypes callbacks) and accepts what the real one accepts of a quantization.
"""
import ctypes as C
import gc
import random

import numpy as np
import pytest

import nuvec_b200 as nv
from nuvec_b200 import _ffi, ops

FLOATS, DTYPES = [nv.F16, nv.BF16, nv.F32], [nv.F16, nv.BF16, nv.F32, nv.U32, nv.I32, nv.U8]


class Recorder:
    """Every function of the library: notes its name and arguments and succeeds."""

    def __init__(self):
        self.calls, self.kept, self.at, self.refuse = [], [], 0x10000000, False
        for name, (res, args) in _ffi.SIGNATURES.items():
            self._add(name, res, args)

    def _add(self, name, res, args):
        def call(*got):
            if name == "nvc_alloc":
                if self.refuse:
                    return -3
                self.at += 4096 + int(got[1])
                C.cast(got[2], C.POINTER(C.c_void_p))[0] = self.at
                return 0
            if name == "nvc_free":
                return 0
            plain = []
            for a in got:
                if isinstance(a, C.POINTER(_ffi.Quant)):
                    q = a.contents
                    a = ("quant", q.mode, q.group_size, q.bits)
                    try:
                        nv.Quant(list(nv.QuantMode)[q.mode], q.group_size, q.bits).checked("t")
                    except nv.InvalidArgument:
                        return -1
                plain.append(a)
            self.calls.append((name, *plain))
            return 0
        # (an error of the real library, worded by nvc_last_error)
        if name == "nvc_last_error":
            call = lambda buf, n: 0
        fn = C.CFUNCTYPE(res, *args)(call)
        self.kept.append(fn)
        setattr(self, name, fn)

    def bound(self):
        return {name: C.cast(getattr(self, name), C.c_void_p).value for name in _ffi.SIGNATURES}


class Declines:
    """The native module with every operator declining."""

    def __getattr__(self, name):
        return lambda *a: None


@pytest.fixture
def lib(monkeypatch):
    real = _ffi.lib()
    rec = Recorder()
    _ffi.native.bind(rec.bound())
    monkeypatch.setattr(_ffi, "_lib", rec)
    dev = nv.Device.__new__(nv.Device)
    dev._h, dev.ordinal = C.c_void_p(0x1234), 0
    dev._set_handle(0x1234)
    rec.dev = dev
    yield rec
    dev._set_handle(None)
    dev._h = None
    gc.collect()
    _ffi.native.bind({name: C.cast(getattr(real, name), C.c_void_p).value for name in _ffi.SIGNATURES})


# ── calls of the usual form, and what may be off about them ──────────────────────────────────
def some_quant(r):
    mode = r.choice([nv.QuantMode.AFFINE] * 3 + list(nv.QuantMode))
    if mode == nv.QuantMode.AFFINE:
        return nv.Quant.affine(r.choice([32, 64, 128]), r.choice([1, 2, 3, 4, 5, 6, 8]))
    return nv.Quant.new(mode)


def packed(r, dev, q, lead, cols, dtype):
    codes = dev.empty((*lead, cols * q.bits // 32), nv.U32)
    affine = q.mode == nv.QuantMode.AFFINE
    groups = (*lead, cols // q.group_size)
    scales = dev.empty(groups, dtype if affine else nv.U8)
    return nv.Quantized(codes, scales, dev.empty(groups, dtype) if affine else None, q)


def spoil_array(r, a):
    kind = r.randrange(4)
    if kind == 0:
        return a.dev.empty(a.shape, r.choice(DTYPES))
    if kind == 1 and a.ndim:
        i = r.randrange(a.ndim)
        return a.dev.empty(a.shape[:i] + (r.choice([0, 1, a.shape[i] + 1, 2 * a.shape[i]]),) + a.shape[i + 1:], a.dtype)
    if kind == 2 and a.ndim:
        return a.dev.empty(a.shape[1:], a.dtype)
    return a.dev.empty((1, *a.shape), a.dtype)


def spoil(r, v):
    """The same argument with one thing off, sometimes something that is allowed."""
    if isinstance(v, nv.Array):
        return None if r.random() < 0.15 else spoil_array(r, v)
    if isinstance(v, nv.Quantized):
        field = r.choice(["weight", "scales", "biases", "quant", "global_scale"])
        now = getattr(v, field)
        if field == "quant":
            new = r.choice([some_quant(r), nv.Quant.affine(64, 7), nv.Quant.affine(16, 4), nv.Quant(nv.QuantMode.NVFP4, 32, 4)])
        elif now is None:
            new = v.weight.dev.empty(r.choice([(), (1,), v.weight.shape[:-2], v.scales.shape]), r.choice([nv.F32, nv.BF16]))
        else:
            new = None if r.random() < 0.2 and field != "weight" and field != "scales" else spoil_array(r, now)
        return ops.replace(v, **{field: new})
    if isinstance(v, bool):
        return not v
    if isinstance(v, int):
        return r.choice([0, -1, v + 1, 1000, np.int64(v)])
    if isinstance(v, float):
        return r.choice([0, 3, np.float32(0.5), float("inf")])
    return v


def cases(r, dev):
    f, q = r.choice(FLOATS), some_quant(r)
    pick = lambda *n: r.choice(n)
    rows, cols, lead = pick(1, 5, 32), 128 * pick(1, 2), tuple(pick(1, 2, 3) for _ in range(r.randrange(3)))
    E, T, k = pick(1, 4), pick(1, 3), pick(1, 2)
    fp4 = nv.Quant.new(pick(nv.QuantMode.MXFP4, nv.QuantMode.NVFP4))
    xq = nv.BF16 if q.mode != nv.QuantMode.AFFINE and r.random() < 0.5 else f
    kvq = nv.Quant.affine(pick(32, 64), pick(3, 4, 8))
    kv = lambda: packed(r, dev, kvq, (lead[0] if lead else 1, 2, 7), 128, f)
    scaled = nv.Quant.new(nv.QuantMode.NVFP4)
    yield nv.quantize, [dev.empty((*lead, rows, cols), f), q]
    yield nv.dequantize, [packed(r, dev, q, (*lead, rows), cols, f)]
    yield nv.quantized_embedding, [packed(r, dev, q, (rows,), cols, f), dev.empty(lead, nv.U32)]
    yield nv.sorted_offsets, [dev.empty((rows,), nv.U32), E]
    yield nv.moe_route, [dev.empty((*lead, 4), f), pick(1, 2, 4), pick(True, False)]
    yield nv.weighted_sum, [dev.empty((*lead, k, cols), f), dev.empty((*lead, k), f)]
    yield nv.expert_bias_add, [dev.empty((rows, cols), f), dev.empty((E, cols), f), dev.empty((rows,), nv.U32)]
    yield nv.moe_sort, [dev.empty((*lead, k), nv.U32), E]
    yield nv.take_rows, [dev.empty((rows, *lead), pick(*DTYPES)), dev.empty(lead, nv.U32)]
    yield nv.rms_norm, [dev.empty((*lead, cols), f), pick(None, dev.empty((cols,), f)), 1e-5]
    yield nv.add_rms_norm, [dev.empty((*lead, cols), f), dev.empty((*lead, cols), f), pick(None, dev.empty((cols,), f)), 1e-6]
    yield nv.swiglu, [dev.empty((*lead, cols), f), dev.empty((*lead, cols), f)]
    yield nv.swiglu_oai, [dev.empty((*lead, cols), f), dev.empty((*lead, cols), f), 1.702, 7.0]
    yield nv.qqmm, [dev.empty((*lead, cols), nv.BF16), packed(r, dev, fp4, (rows,), cols, f), pick(None, dev.empty((512,), nv.U8))]
    yield nv.quantized_attention, [dev.empty((lead[0] if lead else 1, 4, pick(1, 3), 128), f), kv(), kv(), 0.125, pick(None, dev.empty((4,), f)), pick(None, 5), pick(True, False)]
    yield nv.quantized_matmul, [dev.empty((*lead, rows, cols), xq), packed(r, dev, q, (6,), cols, f), True]
    yield nv.quantized_matmul, [dev.empty((6,), xq), packed(r, dev, q, (6,), cols, f), False]
    yield nv.quantized_matmul, [dev.empty((rows, cols), f), ops.replace(packed(r, dev, scaled, (6,), cols, f), global_scale=dev.empty((1,), nv.F32)), True]
    options = nv.GatherQmm(sorted_indices=pick(True, False))
    yield nv.gather_qmm, [dev.empty((T * k, 1, cols), xq), packed(r, dev, q, (E, 6), cols, f), None, dev.empty((T * k,), pick(nv.U32, nv.I32)), options,
                          pick(None, dev.empty((E,), nv.I32))]
    yield nv.gather_qmm, [dev.empty((T, 1, cols), xq), packed(r, dev, q, (E, 6), cols, f), dev.empty((T, k), nv.U32), dev.empty((T, k), nv.U32), options, None]
    yield nv.gather_qmm, [dev.empty((T, 2, 6), xq), packed(r, dev, q, (E, 6), cols, f), dev.empty((T,), nv.U32), dev.empty((T,), nv.U32), nv.GatherQmm(False), None]
    yield nv.gather_qmm, [dev.empty((T, 1, cols), f), ops.replace(packed(r, dev, scaled, (E, 6), cols, f), global_scale=dev.empty((E,), nv.F32)), None, dev.empty((T,), nv.U32)]


def described(result):
    if isinstance(result, nv.Quantized):
        return ["Quantized", result.quant, *map(described, (result.weight, result.scales, result.biases))]
    if isinstance(result, nv.Array):
        return (type(result), result.shape, result.dtype, result._address)
    return [described(x) for x in result] if isinstance(result, tuple) else result


def made(lib, fn, args):
    """What the call returned and asked of the library, or the error; addresses as if nothing had been allocated before."""
    lib.calls, lib.at = [], 0x70000000
    try:
        got = described(fn(*args))
    except Exception as e:  # noqa: BLE001
        got = type(e)
    return got, lib.calls


@pytest.mark.parametrize("seed", range(8))
def test_the_native_path_makes_the_calls_of_the_python_path(lib, monkeypatch, seed):
    r = random.Random(seed)
    taken, declined = {}, 0
    for _ in range(60):
        for fn, args in cases(r, lib.dev):
            for spoiled in (False, True, True, True):
                these = list(args)
                if spoiled:
                    i = r.randrange(len(these))
                    these[i] = spoil(r, these[i])
                name = {"swiglu_oai": "swiglu"}.get(fn.__name__, fn.__name__)
                heard = []
                native = getattr(_ffi.native, name)

                class Listens:
                    def __getattr__(self, other):
                        assert other == name or other in ("quantized_matmul", "dequantize")
                        inner = getattr(_ffi.native, other)
                        return lambda *a: heard.append(inner(*a)) or heard[-1]
                monkeypatch.setattr(ops, "_native", Listens())
                if fn is nv.gather_qmm and these[3] is None and these[2] is None or native is None:
                    continue
                with_native = made(lib, fn, these)
                accepted = any(x is not None for x in heard)
                if not accepted:
                    declined += 1
                    continue
                monkeypatch.setattr(ops, "_native", Declines())
                alone = made(lib, fn, these)
                assert with_native == alone, (fn.__name__, [described(a) for a in these])
                taken[fn.__name__] = taken.get(fn.__name__, 0) + 1
    assert len(taken) == 17 and min(taken.values()) > 20 and declined > 500, (taken, declined)


def test_a_refused_allocation_is_an_error_on_both_paths(lib):
    x = lib.dev.empty((2, 128), nv.BF16)
    lib.refuse = True
    with pytest.raises(nv.OutOfMemory):
        nv.rms_norm(x)
    assert not lib.calls


# ── arrays ───────────────────────────────────────────────────────────────────────────────────
@pytest.mark.parametrize("dtype", [99, 0, -1, 2])
def test_unknown_dtype_codes_are_refused_before_anything_is_allocated(lib, dtype):
    at = lib.at
    with pytest.raises(KeyError):
        lib.dev.empty((1024,), dtype)
    a = lib.dev.empty((4,), nv.F32)
    with pytest.raises(KeyError):
        nv.Array(lib.dev, (4,), dtype, a, 0)
    assert lib.at == at + 4096 + 16


def test_impossible_shapes_are_refused(lib):
    at = lib.at
    for shape, error in (((-1, 4), ValueError), ((-2, -3), ValueError), ((1 << 40, 1 << 40), OverflowError), ((1 << 62,), OverflowError), ((1 << 70,), OverflowError)):
        with pytest.raises(error):
            lib.dev.empty(shape, nv.F32)
    assert lib.at == at
    assert lib.dev.empty((0, 5), nv.F32).nbytes == 0 and lib.dev.empty((), nv.U8).nbytes == 1
