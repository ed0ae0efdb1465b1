"""Device-array plumbing for the drop-in API.

Public functions accept numpy arrays (the reference's types) or torch tensors.
Numpy inputs are copied to the current CUDA device and results come back as
numpy float64 arrays in C order, like the reference returns; torch inputs stay
on the device and results are returned as torch tensors with no host copy.
"""
import numpy as np
import torch

from . import _lib

# bytes moved between host and device by the numpy-in / numpy-out paths
transfer_bytes = {"h2d": 0, "d2h": 0}


# What follows runs several times in each call of the drop-in API, and the small
# calls (a 401 x 201 FTLE field: 8 us of kernel) take as long as their host code:
# so the device is looked for until it has been found, the raw stream is read
# without a Stream object, new arrays go to the unindexed (current) device, and
# pointers are passed as the ints that ctypes takes.
_CUDA = torch.device("cuda")
_found = False


def require_cuda():
    global _found
    if _found:
        return
    if not torch.cuda.is_available():
        raise RuntimeError("numbacs_gb300 needs a CUDA device (no CPU fallback)")
    _lib.load()
    torch.cuda.init()
    _found = True


def is_torch(*arrays):
    return any(isinstance(a, torch.Tensor) for a in arrays if a is not None)


def device():
    return torch.device("cuda", torch.cuda.current_device())


def stream_ptr():
    """The current stream of the current device (None: the default stream)."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device()) or None


def to_dev(a, dtype=torch.float64):
    """Contiguous CUDA tensor of `dtype` holding `a` (no copy if already so)."""
    if a is None:
        return None
    if isinstance(a, torch.Tensor):
        t = a
        if not t.is_cuda:
            t = t.to(device())
        if t.dtype != dtype:
            t = t.to(dtype)
        return t.contiguous()
    arr = np.ascontiguousarray(np.asarray(a), dtype=_np_dtype(dtype))
    transfer_bytes["h2d"] += arr.nbytes
    return torch.from_numpy(arr).to(device(), non_blocking=False)


def mask_to_dev(mask):
    if mask is None:
        return None
    if isinstance(mask, torch.Tensor):
        return to_dev(mask.to(torch.bool), torch.uint8)
    return to_dev(np.asarray(mask, dtype=bool).astype(np.uint8), torch.uint8)


def _np_dtype(dtype):
    return {torch.float64: np.float64, torch.float32: np.float32, torch.uint8: np.uint8,
            torch.int32: np.int32, torch.int64: np.int64}[dtype]


def ptr(t):
    return (t.data_ptr() or None) if t is not None else None


def empty(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, device=_CUDA)


def readback(shape, dtype):
    """Page-locked host array that a kernel writes and the host reads after
    synchronize(): a small result without a device-to-host copy behind the
    kernel (7 us less per call).  Synchronize before it goes out of scope, also
    where the call that may have launched the kernel raises: the allocator hands
    the memory out again at once."""
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def synchronize():
    torch.cuda.current_stream().synchronize()


def finish(t, as_torch):
    """Return a device tensor as-is (torch callers) or as a numpy array."""
    if as_torch:
        return t
    transfer_bytes["d2h"] += t.numel() * t.element_size()
    return t.cpu().numpy()
