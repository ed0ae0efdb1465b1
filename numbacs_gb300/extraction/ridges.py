"""FTLE ridge extraction: drop-in for src/numbacs/extraction/ridges.py.

``ftle_ridge_pts`` (ridges.py:9-76) and the ``_ftle_ridges`` mask
(ridges.py:79-154) run as one percentile-selection + stencil + order-preserving
compaction pipeline on the GPU (csrc/ridges.cu).  The threshold is the
reference's ``np.percentile(f, percentile)`` as numba evaluates it, or 0 when
``percentile == 0``.
"""
import torch

from .. import _device as D
from .. import _lib


def _inputs(f, eigvec_max, x, y):
    fd = D.to_dev(f)
    ev = D.to_dev(eigvec_max)
    xd, yd = D.to_dev(x), D.to_dev(y)
    if fd.dim() != 2:
        raise ValueError("f must have shape (nx, ny)")
    nx, ny = fd.shape
    if tuple(ev.shape) != (nx, ny, 2):
        raise ValueError("eigvec_max must have shape (nx, ny, 2)")
    return fd, ev, xd, yd


# The bit pattern of nbcs_percentile's answer when its launch gave up (nbcs.h)
_PERCENTILE_FAILED = 0x7ff800000000dead


def _count(n_out):
    """The number of ridge points of a launch that has ended; of one that gave up
    waiting for its blocks an error."""
    k = int(n_out)
    if k < 0:
        raise RuntimeError("ridge extraction: the launch did not finish")
    return k


def _run(f, eigvec_max, x, y, sdd_thresh, percentile, f_min=None, dxdy=None, full_mask=False):
    """Ridge points (k, 2), or with full_mask (points or zeros (nx*ny, 2), mask
    (nx, ny), count), which are not waited for: the caller that waits passes the
    count to _count (of a launch that gave up the points are NaN, the mask 1)."""
    D.require_cuda()
    fd, ev, xd, yd = _inputs(f, eigvec_max, x, y)
    nx, ny = fd.shape
    L = _lib.load()
    nbytes = L.nbcs_ridge_scratch_bytes(nx, ny)
    scratch = torch.empty(max(nbytes, 1), dtype=torch.uint8, device=fd.device)
    mask = D.empty((nx, ny), torch.uint8) if full_mask else None
    full = D.empty((nx * ny, 2)) if full_mask else None
    pts = D.empty((nx * ny, 2))
    n_out = D.empty((1,), torch.int64) if full_mask else D.readback((1,), torch.int64)
    try:
        if f_min is None:
            _lib.check(L.nbcs_ridge_pts(D.ptr(fd), D.ptr(ev), D.ptr(xd), nx, D.ptr(yd), ny,
                                        float(sdd_thresh), float(percentile), D.ptr(mask),
                                        D.ptr(full), D.ptr(pts), D.ptr(n_out), D.ptr(scratch),
                                        nbytes, D.stream_ptr()))
        else:
            _lib.check(L.nbcs_ridge_pts_fmin(D.ptr(fd), D.ptr(ev), D.ptr(xd), nx, D.ptr(yd), ny,
                                             float(dxdy[0]), float(dxdy[1]), float(sdd_thresh),
                                             float(f_min), D.ptr(mask), D.ptr(full), D.ptr(pts),
                                             D.ptr(n_out), D.ptr(scratch), nbytes,
                                             D.stream_ptr()))
    finally:
        if not full_mask:
            D.synchronize()  # n_out is page-locked: also when the call raised
    if full_mask:
        return full, mask, n_out
    return pts[:_count(n_out)]


def ridge_pts_fmin(f, eigvec_max, x, y, dx, dy, sdd_thresh, f_min):
    """ftle_ridge_pts with the threshold f_min and the spacing dx, dy given (a
    row block of a field sharded over several GPUs: the global threshold and
    spacing) -> ridge points (k, 2), row-major."""
    as_torch = D.is_torch(f, eigvec_max)
    pts = _run(f, eigvec_max, x, y, sdd_thresh, 0, f_min=f_min, dxdy=(dx, dy))
    return D.finish(pts, as_torch)


def percentile(f, q):
    """np.percentile(f, q) as the reference's numba code evaluates it (float)."""
    D.require_cuda()
    fd = D.to_dev(f).reshape(-1)
    L = _lib.load()
    nbytes = L.nbcs_percentile_scratch_bytes(fd.numel())
    scratch = torch.empty(max(nbytes, 1), dtype=torch.uint8, device=fd.device)
    out = D.readback((1,), torch.float64)
    try:
        _lib.check(L.nbcs_percentile(D.ptr(fd), fd.numel(), float(q), D.ptr(out), D.ptr(scratch),
                                     nbytes, D.stream_ptr()))
    finally:
        D.synchronize()
    if int(out.view(torch.int64)) == _PERCENTILE_FAILED:
        raise RuntimeError("percentile: the launch did not finish")
    return float(out)


def ftle_ridge_pts(f, eigvec_max, x, y, sdd_thresh=0.0, percentile=0):
    """Sub-pixel ridge points (k, 2), in row-major grid order."""
    as_torch = D.is_torch(f, eigvec_max)
    return D.finish(_run(f, eigvec_max, x, y, sdd_thresh, percentile), as_torch)


def _ftle_ridges(f, eigvec_max, x, y, sdd_thresh=0.0, percentile=0, *, wait=False):
    """(r_pts (nx*ny, 2) zero off the ridge, ridge_bool (nx, ny), nx, ny).  Torch
    callers are not waited for unless they say so (a launch that gave up then raises,
    as for numpy callers)."""
    as_torch = D.is_torch(f, eigvec_max)
    full, mask, n_out = _run(f, eigvec_max, x, y, sdd_thresh, percentile, full_mask=True)
    if wait or not as_torch:
        _count(n_out)
    nx, ny = mask.shape
    return D.finish(full, as_torch), D.finish(mask.to(torch.bool), as_torch), nx, ny


def label8(mask):
    """8-connected component labels of a (nx, ny) mask on the GPU, numbered
    1..n by first pixel in row-major order (scipy.ndimage.label with a 3x3
    structure).  Returns (labels int32 CUDA tensor, n)."""
    D.require_cuda()
    m = D.mask_to_dev(mask)
    nx, ny = m.shape
    L = _lib.load()
    nbytes = L.nbcs_label8_scratch_bytes(nx, ny)
    scratch = torch.empty(max(nbytes, 1), dtype=torch.uint8, device=m.device)
    labels = D.empty((nx, ny), torch.int32)
    n = D.empty((1,), torch.int32)
    _lib.check(L.nbcs_label8(D.ptr(m), nx, ny, D.ptr(labels), D.ptr(n), D.ptr(scratch), nbytes,
                             D.stream_ptr()))
    k = int(n.item())
    if k < 0:
        raise RuntimeError("label8: union-find did not converge")
    return labels, k


def ftle_ridges(f, eigvec_max, x, y, sdd_thresh=0.0, percentile=0, min_ridge_pts=3):
    """Connected ridges: list of (m, 2) point arrays, one per 8-connected
    component of the ridge mask with at least ``min_ridge_pts`` points,
    components ordered by their first grid point in row-major order and
    points within a ridge in row-major order (ridges.py:186-229).

    Ridge points, components and their order are computed on the GPU in two
    launches (csrc/ridges.cu) for up to 8192 ridge points; beyond, the mask is
    labelled (csrc/label.cu) and the points sorted by label.
    """
    D.require_cuda()
    as_torch = D.is_torch(f, eigvec_max)
    fd, ev, xd, yd = _inputs(f, eigvec_max, x, y)
    nx, ny = fd.shape
    if nx * ny > 0x7fffffff:
        raise ValueError("grids of more than 2^31 - 1 points are not supported")
    L = _lib.load()
    nbytes = L.nbcs_ridge_scratch_bytes(nx, ny)
    scratch = torch.empty(max(nbytes, 1), dtype=torch.uint8, device=fd.device)
    mask = D.empty((nx, ny), torch.uint8)
    pts = D.empty((nx * ny, 2))
    index = D.empty((nx * ny,), torch.int32)
    n_out = D.empty((1,), torch.int64)
    cap = _lib.RIDGE_COMPONENTS_MAX
    comp = D.empty((cap, 2))
    head = D.readback((cap + 2,), torch.int32)
    try:
        _lib.check(L.nbcs_ridge_components(D.ptr(fd), D.ptr(ev), D.ptr(xd), nx, D.ptr(yd), ny,
                                           float(sdd_thresh), float(percentile), D.ptr(mask),
                                           D.ptr(pts), D.ptr(index), D.ptr(n_out), D.ptr(comp),
                                           D.ptr(head), D.ptr(scratch), nbytes, D.stream_ptr()))
    finally:
        D.synchronize()
    head = head.numpy()
    n, ncomp = int(head[0]), int(head[1])
    _count(n)
    if ncomp >= 0:
        counts = head[2:2 + ncomp].tolist()
        pts = comp[:n]
    else:
        n = int(n_out.item())
        labels, ncomp = label8(mask)
        labs = labels.view(-1).index_select(0, index[:n].long()).long()
        order = torch.sort(labs, stable=True).indices
        pts = pts.index_select(0, order)
        counts = torch.bincount(labs, minlength=ncomp + 1)[1:].tolist()
    if not as_torch:
        pts = pts.cpu().numpy()  # one copy for all ridges
    ridges, start = [], 0
    for c in counts:
        if c >= min_ridge_pts:
            ridges.append(pts.narrow(0, start, c) if as_torch else pts[start:start + c].copy())
        start += c
    return ridges
