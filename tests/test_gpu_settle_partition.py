"""A call on a stream that owns a part of the GPU (a green context) gives what it
gives on the whole one: the grid's team takes the SMs that the stream has."""
import ctypes as C

import numpy as np
import pytest

from hbtg import abi, synthetic
from hbtg.gpu import DeviceBatch

pytestmark = pytest.mark.gpu

SM = 1  # CU_DEV_RESOURCE_TYPE_SM


class Resource(C.Structure):
    _fields_ = [("type", C.c_int), ("pad", C.c_ubyte * 92), ("sm_count", C.c_uint), ("rest", C.c_ubyte * 44)]


@pytest.fixture()
def part_of_the_gpu():
    import torch
    torch.zeros(1, device="cuda")
    try:
        cu = C.CDLL("libcuda.so.1")
        cu.cuDevSmResourceSplitByCount
    except (OSError, AttributeError):
        pytest.skip("no green contexts")
    whole, part, rest = Resource(), Resource(), Resource()
    groups, desc, ctx, stream = C.c_uint(1), C.c_void_p(), C.c_void_p(), C.c_void_p()

    def ok(rc):
        if rc != 0:
            pytest.skip("green contexts: error %d" % rc)
    ok(cu.cuDeviceGetDevResource(0, C.byref(whole), SM))
    ok(cu.cuDevSmResourceSplitByCount(C.byref(part), C.byref(groups), C.byref(whole), C.byref(rest), 0, 48))
    ok(cu.cuDevResourceGenerateDesc(C.byref(desc), C.byref(part), 1))
    ok(cu.cuGreenCtxCreate(C.byref(ctx), desc, 0, 1))
    ok(cu.cuGreenCtxStreamCreate(C.byref(stream), ctx, 1, 0))
    # the stream says which part it has: the library asks the same way
    again, of_ctx = C.c_void_p(), Resource()
    ok(cu.cuStreamGetGreenCtx(stream, C.byref(again)))
    assert again.value
    ok(cu.cuGreenCtxGetDevResource(again, C.byref(of_ctx), SM))
    assert 0 < of_ctx.sm_count == part.sm_count < whole.sm_count
    yield stream.value
    torch.cuda.synchronize()
    cu.cuStreamDestroy_v2(stream)
    cu.cuGreenCtxDestroy(ctx)


@pytest.mark.parametrize("sizes", [(46_000,), (21_000, 12_000, 900)])
def test_same_results(unbinder, part_of_the_gpu, sizes):
    import torch
    prm = abi.parity_params(dm_only=1, box_size=500.0)
    parts = [synthetic.stripped(n_sub=1, seed=1 + k, nmin=n, nmax=n + 1) for k, n in enumerate(sizes)]
    cat = lambda k: np.concatenate([getattr(p, k) for p in parts])  # noqa: E731
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    inp = abi.Inputs(off, cat("pos"), cat("vel"), cat("mass"), np.arange(off[-1]) + 5, None, None, cat("ref_pos"),
                     cat("ref_vel"), cat("mostbound_pos"), cat("mostbound_vel"), cat("most_bound_id"))
    outs = []
    for stream in (0, part_of_the_gpu):
        db = DeviceBatch(inp)
        db.reset_inout()
        torch.cuda.synchronize()
        unbinder.unbind_device(prm, db.c, stream)
        torch.cuda.synchronize()
        outs.append(db.outputs())
    a, b = outs
    assert a.nbound.min() > 0
    for k in ("nbound", "mbound", "ref_pos", "ref_vel", "iterations", "status", "order"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
