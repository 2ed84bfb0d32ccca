"""A call that fails with work on its streams gives back a workspace that the next call can use."""
import ctypes

import pytest

from helpers import scalar

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_workspace_is_idle_after_a_failed_call(gpu, oracle, kind):
    idle = ctypes.c_int32(-1)
    fn = gpu.lib().cubbs_bbs_gpu_failed_call_for_test_v2
    fn.restype, fn.argtypes = ctypes.c_int32, [ctypes.c_int32, ctypes.c_void_p]
    assert fn(kind, ctypes.byref(idle)) == 0 and idle.value == 1
    p1, gens = oracle.generators(8)
    pts = ([p1] + gens)[:8]
    msms = [(pts, [scalar(b"failed", b"%d" % i, k) for k in range(8)]) for i in range(33)]
    assert gpu.g1_msm_batch(msms) == [(0, oracle.g1_msm(p, s)) for p, s in msms]
