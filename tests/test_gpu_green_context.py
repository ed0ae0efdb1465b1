"""Ridge calls on a stream whose context owns a part of the device's SMs (a green
context): the launch, whose blocks wait for one another, has to fit there."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SM = 1  # CU_DEV_RESOURCE_TYPE_SM


@pytest.fixture
def small_stream(nb):
    """(stream, its number of SMs) of a green context with 16 SMs or the fewest
    that the device gives"""
    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    torch.zeros(1, device="cuda")
    dev = ctypes.c_int(torch.cuda.current_device())
    # CUdevResource: type, 92 bytes, then the SM count; 144 bytes
    whole, part, rest = (ctypes.create_string_buffer(256) for _ in range(3))
    desc, ctx, stream = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    groups = ctypes.c_uint(1)
    for call, args in (("cuDeviceGetDevResource", (dev, whole, SM)),
                       ("cuDevSmResourceSplitByCount", (part, ctypes.byref(groups), whole, rest,
                                                        ctypes.c_uint(0), ctypes.c_uint(16))),
                       ("cuDevResourceGenerateDesc", (ctypes.byref(desc), part, ctypes.c_uint(1))),
                       ("cuGreenCtxCreate", (ctypes.byref(ctx), desc, dev, ctypes.c_uint(1))),
                       ("cuGreenCtxStreamCreate", (ctypes.byref(stream), ctx, ctypes.c_uint(1), 0))):
        if getattr(cu, call)(*args):
            pytest.skip("%s: not available" % call)
    sms = ctypes.c_uint.from_buffer(part, 96).value
    assert 1 <= sms < torch.cuda.get_device_properties(dev.value).multi_processor_count
    yield torch.cuda.ExternalStream(stream.value), sms
    torch.cuda.synchronize()
    cu.cuStreamDestroy(stream)
    cu.cuGreenCtxDestroy(ctx)


def test_ridges_on_a_part_of_the_device(nb, small_stream):
    import torch
    from numbacs_gb300.extraction import ftle_ridge_pts, ftle_ridges
    from numbacs_gb300.extraction.ridges import percentile
    stream, _ = small_stream
    rng = np.random.default_rng(1)
    nx, ny = 901, 600                      # blocks for the whole device
    f = torch.from_numpy(rng.standard_normal((nx, ny)) + 5.0).cuda()
    a = rng.uniform(-1.5, 1.5, (nx, ny))
    e = torch.from_numpy(np.stack([np.cos(a), np.sin(a)], -1)).cuda()
    x, y = np.arange(nx) * 0.5, np.arange(ny) * 0.25
    want = (percentile(f, 90.0), ftle_ridge_pts(f, e, x, y, 0.0, 90), ftle_ridges(f, e, x, y, 0.0, 98))
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        assert percentile(f, 90.0) == want[0]
        assert torch.equal(ftle_ridge_pts(f, e, x, y, 0.0, 90), want[1])
        got = ftle_ridges(f, e, x, y, 0.0, 98)
    assert len(got) == len(want[2]) > 0
    assert all(torch.equal(g, w) for g, w in zip(got, want[2]))
