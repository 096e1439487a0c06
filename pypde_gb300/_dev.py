"""Device-tensor helpers: every field lives in a float64 CUDA tensor."""
import numpy as np
import torch

from . import _lib

DTYPE = torch.float64


def device():
    if not torch.cuda.is_available():
        raise _lib.PgxError("pypde_gb300 needs a CUDA GPU (GB300, sm_103a); no CPU fallback exists")
    return torch.device("cuda", torch.cuda.current_device())


def to_dev(x):
    """float64 CUDA tensor view of x (numpy array, scalar or tensor)."""
    if isinstance(x, torch.Tensor):
        if x.is_cuda and x.dtype == DTYPE:
            return x
        return x.to(device=device(), dtype=DTYPE)
    return torch.as_tensor(np.asarray(x, dtype=np.float64), device=device())


def to_host(x):
    if isinstance(x, torch.Tensor):
        return x.detach().cpu().numpy()
    return np.asarray(x)


# The public call builds a Stream object on the way to the handle: 2.8 us a call against 0.3 on the GB300's host,
# where an operator of a small field is 4 us of launch.
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def stream():
    """Handle of the current stream of the current device, asked anew on every call."""
    if _raw_stream is None:
        return torch.cuda.current_stream().cuda_stream
    return _raw_stream(torch.cuda.current_device())


def geom(t, axis):
    """(ptr, s0, s1, n_axis, nlines) for a 1-D or 2-D tensor seen along ``axis``.

    A 1-D tensor is an (n, 1) array: one line along axis 0.
    """
    if t.dim() == 2:
        s0, s1 = t.stride()
        shape = t.shape
        return t.data_ptr(), s0, s1, shape[axis], shape[1 - axis]
    if t.dim() == 1:
        if axis != 0:
            raise ValueError("axis must be 0 for a 1-D array")
        return t.data_ptr(), t.stride(0), 1, t.shape[0], 1
    raise NotImplementedError("ndim must be less than 3")


def new_along(t, axis, n):
    """A new row-major tensor shaped like the 1-D or 2-D ``t`` with extent n along axis, and its (ptr, s0, s1)."""
    if t.dim() == 1:
        out = torch.empty((n,), dtype=DTYPE, device=t.device)
        return out, out.data_ptr(), 1, 1
    shape = (n, t.shape[1]) if axis == 0 else (t.shape[0], n)
    out = torch.empty(shape, dtype=DTYPE, device=t.device)
    return out, out.data_ptr(), max(shape[1], 1), 1
