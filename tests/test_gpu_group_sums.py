"""Group sums of the aggregated checks: eight-lane ladders up to 1216 items, buckets or lane pairs beyond."""
import pytest

from helpers import drbg, keypair, messages

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(16, 17, 18, 19, 60), (1216,), (1217,), (200,) * 6 + (33,), (16,) * 77])
def test_verify_groups(gpu, oracle, sizes):
    """Keys with these many items each: groups that end inside a warp's four items, one group of every warp, and one
    item more than the ladders take; then with one failing item in the first and the last group, and with one
    signature twice in a group."""
    reqs = []
    for k, n in enumerate(sizes):
        sk, pk = keypair(oracle, b"sums", k)
        some = [messages(b"sums-%d" % k, i, 2, 16) for i in range(6)]
        sigs = [s for _, s in gpu.sign_batch([(sk, pk, b"h", m) for m in some])]
        reqs += [(pk, sigs[i % 6], b"h", some[i % 6]) for i in range(n)]
    assert [v for _, v in gpu.verify_batch(reqs)] == [True] * len(reqs)
    bad = {3, len(reqs) - 2}
    for i in bad:
        pk, sig, hdr, msgs = reqs[i]
        reqs[i] = (pk, sig, hdr, [msgs[1], msgs[0]])
    assert [v for _, v in gpu.verify_batch(reqs)] == [i not in bad for i in range(len(reqs))]
