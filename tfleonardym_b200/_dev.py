"""Device plumbing: torch CUDA tensors in, raw pointers and the current stream out."""
import ctypes

import torch

from . import _lib

_Tensor, _C128 = torch.Tensor, torch.complex128  # looked up once: as_c128 runs several times a call


def require_cuda():
    if not torch.cuda.is_available():
        raise RuntimeError("tfleonardym_b200 needs a CUDA device (sm_100a); there is no CPU fallback")


def stream():
    # the handle of torch.cuda.current_stream() without the object around it (0.3 us instead of 3.3)
    return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(torch.cuda.current_device()))


def as_c128(t, name="tensor"):
    """Return a contiguous complex128 CUDA tensor view/copy of ``t`` (DLPack producers accepted).

    Its memory holds its values: a lazy conjugate or sign, which torch keeps as a flag that
    contiguous() passes on, is written out (into a copy; without a flag nothing is copied)."""
    if not isinstance(t, _Tensor):
        t = torch.from_dlpack(t)
    if not t.is_cuda:
        raise ValueError(f"{name} must be a CUDA tensor")
    if t.dtype is not _C128:
        t = t.to(_C128)
    t = t.contiguous()
    if t.is_conj() or t.is_neg():  # two flags to test cost half of what the two calls below do
        t = t.resolve_conj().resolve_neg()
    return t


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def cdot(a, b):
    """sum conj(a) b as a Python complex (synchronises the current stream)."""
    a = as_c128(a)
    b = as_c128(b)
    if a.shape != b.shape:
        raise RuntimeError("Incompatible vector shapes!")
    out = (ctypes.c_double * 2)()
    _lib.check(_lib.lib().lym_cdot(a.numel(), ptr(a), ptr(b), out, stream()), "lym_cdot")
    return complex(out[0], out[1])


def axpby(a, x, b, y):
    """Return a*x + b*y (complex scalars) as a new tensor, computed by the lym kernel."""
    x = as_c128(x)
    y = as_c128(y)
    if x.shape != y.shape:
        raise RuntimeError("Incompatible vector shapes!")
    out = y.clone()
    ca = (ctypes.c_double * 2)(complex(a).real, complex(a).imag)
    cb = (ctypes.c_double * 2)(complex(b).real, complex(b).imag)
    _lib.check(_lib.lib().lym_caxpby(x.numel(), ca, ptr(x), cb, ptr(out), stream()), "lym_caxpby")
    return out


def axpby_(a, x, b, y):
    """y <- a*x + b*y in place."""
    ca = (ctypes.c_double * 2)(complex(a).real, complex(a).imag)
    cb = (ctypes.c_double * 2)(complex(b).real, complex(b).imag)
    _lib.check(_lib.lib().lym_caxpby(x.numel(), ca, ptr(x), cb, ptr(y), stream()), "lym_caxpby")
    return y
