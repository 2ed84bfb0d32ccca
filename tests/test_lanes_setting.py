"""CUBBS_BBS_VAR_LANES forces the lanes of ProofGen's membership check at every batch size (the setting is read once per
process, so each value runs in a child process)."""
import json
import os
import pathlib
import subprocess
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]

RULE = r"""
import ctypes, json, sys
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[1] + "/tests")
from tests.conftest import load_package
pkg = load_package(); pkg.build()
fn = pkg.lib().cubbs_bbs_gpu_proof_gen_check_lanes_for_test_v2
fn.argtypes, fn.restype = [ctypes.c_size_t], ctypes.c_int32
print(json.dumps([fn(n) for n in (1, 512, 513, 4096, 19457)]))
"""

# 600 items: damaged points, a point outside G1 and good signatures, compared byte for byte
CALL = r"""
import json, sys
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[1] + "/tests")
from tests.conftest import load_package
from oracle import oracle_ctypes as O
from helpers import drbg, keypair, messages
from tests.test_gpu_parity import _on_curve_outside_g1
pkg = load_package(); pkg.build()
sk, pk = keypair(O, b"lanes-many")
reqs, seeds = [], []
some = [(messages(b"lanes-many", i, 3, 32)) for i in range(5)]
sigs = [O.sign(sk, pk, b"h", m)[0] for m in some]
for i in range(600):
    sig = sigs[i % 5]
    if i % 100 == 7: sig = _on_curve_outside_g1(O, b"lanes-many") + sig[48:]
    if i % 100 == 9: sig = bytes([sig[0] & 0x7f]) + sig[1:]
    reqs.append((pk, sig, b"h", b"p", some[i % 5], [i % 3]))
    seeds.append(drbg(b"lanes-many", b"seed", i % 15, 32))
got = pkg.proof_gen_batch(reqs, seeds=seeds)
bad = {i for i in range(600) if i % 100 in (7, 9)}
want = {k: O.proof_gen(*reqs[15 + k], seed=seeds[15 + k]) for k in range(15)}
print(json.dumps(all((c != 0) if i in bad else (c == 0 and p == want[i % 15]) for i, (c, p) in enumerate(got))))
"""


def _child(code, lanes):
    env = {k: v for k, v in os.environ.items() if k != "CUBBS_BBS_VAR_LANES"}
    if lanes:
        env["CUBBS_BBS_VAR_LANES"] = str(lanes)
    out = subprocess.run([sys.executable, "-c", code, str(ROOT)], env=env, capture_output=True, text=True, timeout=900)
    assert out.returncode == 0, out.stderr[-3000:]
    return json.loads(out.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("lanes,want", [(0, [8, 8, 2, 2, 2]), (1, [1] * 5), (2, [2] * 5), (4, [4] * 5), (8, [8] * 5)])
def test_setting_reaches_every_size(lanes, want):
    assert _child(RULE, lanes) == want


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [0, 1, 4, 8])
def test_proof_gen_of_many(lanes):
    assert _child(CALL, lanes) is True
