"""nuvec_b200: a B200 (sm_100a) backend for nuvec's quantized-matmul path.

The computation lives in ``libnuvec_cuda.so`` (hand-written CUDA behind the C ABI of
``include/nuvec_cuda.h``); this package is the host-side mirror of the reference's operator
interface.  Build the library with ``python -m nuvec_b200.build``.

The operators (``ops.py``) are loaded with the first name that is asked for: they stand on compiled code, and
``nuvec_b200.build``, which compiles it, lives in this package.
"""
import importlib
import importlib.util

_DTYPES = ("BF16", "F16", "F32", "I32", "U8", "U32")


def __getattr__(name):
    if name.startswith("__") and name != "__all__":
        raise AttributeError(f"module {__name__!r} has no attribute {name!r}")
    if name != "__all__" and importlib.util.find_spec(f"{__name__}.{name}") is not None:
        return importlib.import_module(f"{__name__}.{name}")
    ops = importlib.import_module(f"{__name__}.ops")
    public = [*ops.__all__, *_DTYPES]
    globals().update({n: getattr(ops, n) for n in public}, __all__=public)
    if name not in globals():
        raise AttributeError(f"module {__name__!r} has no attribute {name!r}")
    return globals()[name]


def __dir__():
    return sorted({*globals(), *__getattr__("__all__")})
