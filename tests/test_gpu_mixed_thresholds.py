"""GPU test of a mixed-form call with other thresholds while the one before is still queued.

The calls run on a stream that synchronous copies do not wait for, behind work that keeps the device
busy while the second call is prepared; each must give what it gives alone, bit for bit.
"""
import ctypes

import pytest

from gbasis_b200 import _engine
from gbasis_b200.synthetic import make_workload

pytestmark = pytest.mark.gpu


def test_other_thresholds_leave_the_queued_call_alone():
    import torch
    db = _engine.DeviceBasis(make_workload("large64")[:40])
    db.set_fp32_lists(1, 1 << 30)  # every block's FP32 quartets get their own launch
    n = db.nbf ** 4
    st = torch.cuda.Stream()
    sp = ctypes.c_void_p(st.cuda_stream)
    forms = [(1e-11, 1e-5), (1e-11, 1e-300)]  # many FP32 lists, none

    def call(out, mixed):
        db.full_device(out.data_ptr(), stream=sp, mixed=mixed)
    ref = []
    for mixed in forms:
        ref.append(torch.zeros(n, dtype=torch.float64, device="cuda"))
        torch.cuda.synchronize()
        call(ref[-1], mixed)
        torch.cuda.synchronize()
    assert not torch.equal(*ref)
    busy = torch.ones((4096, 4096), device="cuda")
    for _ in range(3):
        got = [torch.zeros_like(r) for r in ref]
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            for _ in range(20):
                busy @ busy
        for out, mixed in zip(got, forms):
            call(out, mixed)
        torch.cuda.synchronize()
        for g, r in zip(got, ref):
            assert torch.equal(g, r)
    db.close()
