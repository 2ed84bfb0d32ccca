"""The launches that a ProofGen step reports: the products with A and those with B apart up to 292 items, one launch of
both beyond."""
import pytest

from helpers import drbg, keypair, messages

pytestmark = pytest.mark.gpu


def test_proof_gen_launches(gpu, oracle):
    sk, pk = keypair(oracle, b"launches")
    msgs = messages(b"launches", 0, 2, 16)
    sig = oracle.sign(sk, pk, b"h", msgs)[0]
    seeds = [drbg(b"launches", b"seed", 0, 32)] * 293
    counts = [gpu.bench_device_steps(gpu.OP_PROOF_GEN, [(pk, sig, b"h", b"p", msgs, [0])] * n, 0, 1, seeds=seeds[:n])[1]
              for n in (292, 293)]
    # hash, decode, membership check, two launches of scalars, domain, two times rows and MSM, jobs of A and of B, the
    # prefix of the challenge, finish, responses; and the terms, in two launches or one
    assert counts == [15 + 2, 15 + 1]
