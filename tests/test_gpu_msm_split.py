"""Uneven variable-base MSMs split over lanes by window and chunk."""
import random

import pytest

from helpers import R_MOD as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lo,hi", [(32, 8, 8), (33, 1, 30), (40, 0, 300), (700, 8, 24), (64, 120, 140)])
def test_split_windows(gpu, oracle, n, lo, hi):
    """MSMs split over lanes by window and chunk (the way of a batch without settings of its own): every window width,
    one and several chunks, empty MSMs, identity points, equal and opposite points, scalars 0, 1, r - 1; against the
    persistent engine, and against the oracle for some of the rows."""
    p1, gens = oracle.generators(6)
    base = [p1] + list(gens)
    base += [bytes([p[0] ^ 0x20]) + p[1:] for p in base[:3]] + [bytes([0xC0]) + bytes(47)]
    rng = random.Random(repr((n, lo, hi)))
    ks = [rng.choice([0, 1, R - 1]) if rng.random() < 0.1 else rng.randrange(R) for _ in range(50)]
    sizes = [lo + (i * 7919) % (hi - lo + 1) for i in range(n)]
    sizes[-1], sizes[n // 2] = hi, lo
    msms = [([rng.choice(base) for _ in range(k)], [rng.choice(ks).to_bytes(32, "big") for _ in range(k)]) for k in sizes]
    got = gpu.g1_msm_batch(msms)
    saved = gpu.msm_tuning()
    try:
        gpu.msm_tuning([8, 8, 8, 8], [4, 5, 5, 5], [0, 0, 0, 0])
        assert gpu.g1_msm_batch(msms) == got
    finally:
        gpu.msm_tuning(*saved)
    for i in (0, 1, n // 2, n - 1):
        if sizes[i] <= 40:
            assert got[i] == (0, oracle.g1_msm(*msms[i]))
