"""ctypes loader for the in-tree native libraries.

The kernels library is required on any machine with a CUDA device: :func:`kernels` raises a
``RuntimeError`` instead of silently falling back when the shared object is missing, so a GPU run
can never pass on a PyTorch fallback by accident.
"""
from __future__ import annotations

import ctypes
import importlib.util
import os
import sysconfig
import threading
import warnings
from pathlib import Path
from types import SimpleNamespace

import torch

_PKG_LIBDIR = Path(__file__).resolve().parent.parent / "lib"
_LIBDIR = Path(os.environ.get("LLMQ_LIB_DIR") or _PKG_LIBDIR)      # LLMQ_LIB_DIR: another build of the libraries
_lock = threading.Lock()
_kernels = None
_rt = None
_binding = None            # the extension module, False when it was not built
_calls = None

DT_BF16, DT_E4M3, DT_E5M2, DT_FP32, DT_FP16, DT_INT32, DT_INT8 = range(7)

_TORCH2CODE = {
    torch.bfloat16: DT_BF16,
    torch.float8_e4m3fn: DT_E4M3,
    torch.float8_e5m2: DT_E5M2,
    torch.float32: DT_FP32,
    torch.float16: DT_FP16,
    torch.int32: DT_INT32,
    torch.int8: DT_INT8,
}


def dtype_code(dt: torch.dtype) -> int:
    try:
        return _TORCH2CODE[dt]
    except KeyError:
        raise TypeError(f"unsupported dtype {dt}") from None


def _load(name: str):
    path = _LIBDIR / name
    if not path.exists():
        raise RuntimeError(
            f"native library {path} is missing; run `python -m llmq_b200.build` (needs nvcc, no GPU required)")
    return ctypes.CDLL(str(path))


def kernels():
    """Returns the CUDA kernels library (loads it on first use)."""
    global _kernels
    if _kernels is None:
        with _lock:
            if _kernels is None:
                lib = _load("libllmq_b200_kernels.so")
                lib.llmq_gemm_splitk_floats.restype = ctypes.c_longlong
                _kernels = lib
    return _kernels


# Arguments of the entry points in calls(), without the stream: p pointer (tensor, address or None), i int, u unsigned, l long long, f float, d double
SIGNATURES = {
    "llmq_gemm_ready": "ppppiiiiiiillliiippfppipuidpl", "llmq_gemm_split_mode": "piiiilii", "llmq_rmsnorm_forward": "pppppppfiiippp", "llmq_rmsnorm_backward": "pppppppiiipiip",
    "llmq_swiglu_forward": "pppliipppi", "llmq_swiglu_backward": "pppliipi", "llmq_rope": "pppiiiiiiipi",
    "llmq_attention_forward": "pppiiiiipp", "llmq_attention_backward": "ppppppiiiiip", "llmq_bias_backward": "pppliippiii", "llmq_abs_max": "pplii",
    "llmq_quantize": "ppppliii", "llmq_quantize_transpose": "pppppiiii", "llmq_transpose": "ppppiiii", "llmq_fused_classifier": "ppppffiilii",
    "llmq_norm_squared": "pplii", "llmq_deterministic_sum": "ppi", "llmq_norm_sum_finish": "ppifp", "llmq_norm_finish": "pfp", "llmq_adamw_hyper": "ppppplfffiffppuliiiiip",
}
_CTYPES = {"p": ctypes.c_void_p, "i": ctypes.c_int, "u": ctypes.c_uint, "l": ctypes.c_longlong, "f": ctypes.c_float, "d": ctypes.c_double}


# Name of the extension module for this interpreter
BINDING_FILE = "llmq_b200_binding" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so")


def _load_binding(path: Path):
    """The extension module at ``path``; ImportError where it is not one for this torch and these entry points.

    It reads tensors through torch's inline accessors and calls the C functions with the argument types it was compiled with, so it is
    used with the very torch that it was compiled against and with the entry points of SIGNATURES, or not at all."""
    spec = importlib.util.spec_from_file_location("llmq_b200_binding", path)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    if module.torch_version != str(torch.__version__):
        raise ImportError(f"compiled against torch {module.torch_version}, this is {torch.__version__}")
    if module.signatures() != SIGNATURES:
        raise ImportError("its entry points are not those of this package")
    return module


def binding():
    """The extension module of ``csrc/py/binding.cpp``, or None where there is none that loads (it needs the headers of torch and Python, and fits one
    interpreter and one torch); the same kernels are then called through ctypes."""
    global _binding
    if _binding is None:
        with _lock:
            if _binding is None:
                found = False
                for path in dict.fromkeys((_LIBDIR / BINDING_FILE, _PKG_LIBDIR / BINDING_FILE)):
                    if not path.exists():
                        continue
                    try:
                        found = _load_binding(path)
                        break
                    except (ImportError, OSError, AttributeError) as e:
                        warnings.warn(f"{path} is not used, calls go through ctypes: {e}; run `python -m llmq_b200.build`", RuntimeWarning, stacklevel=2)
                _binding = found
    return _binding or None


def _through_ctypes(fn, codes):
    fn.argtypes = [_CTYPES[c] for c in codes] + [ctypes.c_void_p]
    take = [{"p": lambda a: a.data_ptr() if isinstance(a, torch.Tensor) else a, "f": float, "d": float}.get(c, int) for c in codes]

    def call(*args):
        return fn(*[t(a) for t, a in zip(take, args, strict=True)], raw_stream())
    return call


def calls():
    """The entry points of SIGNATURES as functions of tensors and numbers that launch on the current stream and return the C function's code:
    those of :func:`binding`, or slower ones of the same kernels through ctypes."""
    global _calls
    if _calls is None:
        lib, b = kernels(), binding()
        if b is not None:
            for name in SIGNATURES:
                b.bind(name, ctypes.cast(getattr(lib, name), ctypes.c_void_p).value)
            _calls = b
        else:
            _calls = SimpleNamespace(**{name: _through_ctypes(getattr(lib, name), codes) for name, codes in SIGNATURES.items()})
    return _calls


def runtime():
    """Returns the host runtime library (data loader, safetensors writer, arena)."""
    global _rt
    if _rt is None:
        with _lock:
            if _rt is None:
                _rt = _load("libllmq_b200_rt.so")
    return _rt


def have_kernels() -> bool:
    return (_LIBDIR / "libllmq_b200_kernels.so").exists()


def ptr(t):
    """Device/host address of a tensor (``None`` -> NULL)."""
    if t is None:
        return ctypes.c_void_p(0)
    return ctypes.c_void_p(t.data_ptr())


def raw_stream() -> int:
    """Handle of the current stream of the current device (3 us less host time than a Stream object)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def stream_ptr(stream=None):
    return ctypes.c_void_p(stream.cuda_stream if stream is not None else raw_stream())


class KernelError(RuntimeError):
    pass


# Number of device kernels launched through this module (each entry point knows how many it launches; small bias gradients take one instead of two).
_EXTRA_LAUNCHES = {"rmsnorm_backward": 1, "bias_backward": 1, "attention_backward": 1, "encoder_backward": 1}
launch_count = 0


def check(rc: int, what: str):
    global launch_count
    if rc != 0:
        raise KernelError(f"{what} failed with code {rc}")
    launch_count += 1 + _EXTRA_LAUNCHES.get(what, 0)
