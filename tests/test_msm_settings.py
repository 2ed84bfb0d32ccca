"""Which way an uneven MSM batch takes: split windows while no caller has made settings, the persistent engine under
settings whatever their values, and what the settings and the autotuner report."""
import ctypes
import random

import pytest

from conftest import load_package
from helpers import R_MOD

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


@pytest.mark.parametrize("longest", [8, 257, 4096, 524288])
def test_long_msm_among_short_ones(longest):
    """No lane adds many chunks one after another, however long one MSM is: at most 8, or a 32nd of them."""
    c, t, _, _, lanes, *_ = plan([longest] + [8] * 39)
    chunks = -(-longest // t)
    assert c and lanes in (1, 2, 4, 8, 16, 32) and -(-chunks // lanes) <= max(8, -(-chunks // 32))


def test_plan_is_for_the_devices_sms():
    """On fewer SMs the same batch fills the GPU earlier, so its MSMs are cut into fewer chunks."""
    K = [2 + (i * 7919) % 256 for i in range(700)]
    assert plan(K, sms=16)[1] > plan(K, sms=152)[1] > plan(K, sms=1000)[1]


@pytest.mark.parametrize("settings", [None, INITIAL])
@pytest.mark.parametrize("n,hi", [(32, 8), (1024, 257), (16384, 257), (40, 20000)])
def test_pinned_bytes_are_those_uploaded(n, hi, settings):
    """A call page-locks what it copies (points, scalars, indexes, chunks), not the plan's device buffers."""
    K = [2 + (i * 7919) % (hi - 1) for i in range(n)]
    _, _, chunks, units, _, pinned, *_ = plan(K, settings)
    terms = sum(K)
    copied = (48 + 32 + 4 + 1) * terms + 16 * chunks + 8 * units + 16 * (n + 1)
    assert copied <= pinned <= copied + 70000


@pytest.mark.gpu
@pytest.mark.parametrize("longest", [63, 70, 130, 260, 520, 1100, 2100])
def test_joined_chunks(gpu, oracle, longest):
    """One long MSM among short ones, in chunks joined by 1, 2, .. 32 lanes: equal, opposite and identity points."""
    rng = random.Random(longest)
    p1, gens = oracle.generators(5)
    base = [p1] + list(gens)
    base += [bytes([p[0] ^ 0x20]) + p[1:] for p in base[:2]] + [bytes([0xC0]) + bytes(47)]
    sizes = [8] * 40
    sizes[7], sizes[9], sizes[11] = longest, 0, 40
    msms = [([rng.choice(base) for _ in range(k)], [rng.randrange(R_MOD).to_bytes(32, "big") for _ in range(k)])
            for k in sizes]
    # one MSM of the long one's points and summed scalars: at most nine terms
    total = {}
    for p, k in zip(*msms[7]):
        total[p] = (total.get(p, 0) + int.from_bytes(k, "big")) % R_MOD
    want = [oracle.g1_msm(*m) if i != 7 else oracle.g1_msm(list(total), [v.to_bytes(32, "big") for v in total.values()])
            for i, m in enumerate(msms)]
    assert gpu.g1_msm_batch(msms) == [(0, w) for w in want]


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
