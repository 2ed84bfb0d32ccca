"""Pairing checks whose cyclotomic squarings share their products between two warps, and those that do not."""
import pytest

from helpers import keypair, scalar

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 304, 305])
def test_pairing_eq(gpu, oracle, n):
    """Up to two checks an SM, and one more: equal and unequal pairs, scaled points, and identity points."""
    p1, _ = oracle.generators(1)
    inf = bytes([0xC0]) + bytes(47)
    pks = [keypair(oracle, b"halves", i)[1] for i in range(3)]
    a = [oracle.g1_mul(p1, scalar(b"halves", b"a", i)) for i in range(4)]
    kinds = [(a[0], pks[0], a[0], pks[0], True), (a[0], pks[0], a[1], pks[0], False),
             (a[2], pks[1], a[2], pks[2], False), (inf, pks[0], inf, pks[1], True), (a[3], pks[2], a[3], pks[2], True),
             (inf, pks[0], a[1], pks[0], False), (a[1], pks[1], a[1], pks[1], True)]
    items = [kinds[i % 7] for i in range(n)]
    assert gpu.pairing_eq_batch([k[:4] for k in items]) == [(0, k[4]) for k in items]
