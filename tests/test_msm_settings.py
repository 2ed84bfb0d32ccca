"""Which way an uneven MSM batch takes: split windows while no caller has made settings, the persistent engine under
settings whatever their values, and what the settings and the autotuner report."""
import ctypes

import pytest

from conftest import load_package

INITIAL = ([8, 16, 32, 32], [4] * 4, [0] * 4)
SPLIT = [2] * 4


def plan(K, settings=None, sms=152):
    """(window of split windows or 0, terms of the largest chunk, chunks, engine units, ...)"""
    pkg = load_package()
    pkg.build()
    fn = pkg.lib().cubbs_bbs_gpu_msm_plan_for_test_v2
    fn.restype = ctypes.c_int32
    fn.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int32] + [ctypes.c_void_p] * 4
    arrs = [(ctypes.c_uint32 * 4)(*v) for v in settings] if settings else [None] * 3
    out = (ctypes.c_uint64 * 8)()
    rc = fn((ctypes.c_uint32 * len(K))(*K), len(K), sms, *arrs, out)
    if rc:
        raise ValueError(rc)
    return list(out)


@pytest.mark.parametrize("settings,split", [(None, True), (([1] * 4, [1] * 4, SPLIT), True), (INITIAL, False),
                                            (([8] * 4, [4] * 4, [0] * 4), False), (([8] * 4, [9] * 4, [1] * 4), False)])
def test_way_taken(settings, split):
    c, _, chunks, units, *_ = plan([2 + i % 256 for i in range(1024)], settings)
    assert chunks > 0 or settings[2][0] == 1
    assert (3 <= c <= 5 and units == 0) if split else (c == 0 and units > 0)


@pytest.mark.parametrize("mode", [[2, 2, 2, 0], [2, 0, 0, 0], [3] * 4])
def test_mixed_modes_are_refused(mode):
    with pytest.raises(ValueError):
        plan([8] * 32, ([8] * 4, [4] * 4, mode))


@pytest.mark.gpu
def test_settings_in_force(gpu):
    saved = gpu.msm_tuning()
    try:
        assert gpu.msm_tuning([8] * 4, [4] * 4, SPLIT)[2] == SPLIT
        assert gpu.msm_uneven_bench(n_msms=256, tune=False, warmup=0, steps=1)["mode"] == SPLIT
        assert gpu.msm_tuning(*INITIAL) == INITIAL  # the initial values too select the engine
        r = gpu.msm_uneven_bench(n_msms=256, tune=False, warmup=0, steps=1)
        assert (r["chunk"], r["window"], r["mode"]) == INITIAL and r["mismatch"] == 0
        r = gpu.msm_uneven_bench(n_msms=256, k_min=2, k_max=40, tune=True, warmup=0, steps=1)
        assert r["mismatch"] == 0 and (r["chunk"], r["window"], r["mode"]) == gpu.msm_tuning()
        assert r["mode"] == SPLIT or 2 not in r["mode"]
        with pytest.raises(ValueError):
            gpu.msm_tuning([8] * 4, [4] * 4, [2, 2, 2, 0])
    finally:
        assert gpu.msm_tuning(*saved) == saved
