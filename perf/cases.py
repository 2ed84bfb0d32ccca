"""Timed cases: what programs have the library do, through its C ABI.

A case is a dict of plain values; `prepare` builds the host buffers that a caller
holds before the call (the ABI's item arrays over contiguous bytes), `run` makes
the ABI call or calls and returns result codes, verdicts and output bytes.  The
prepared state of the library (generator table, key lines) is built by the first
call that needs it and kept for the process, as in a service.

Kinds:
  trip      sign -> verify -> proof_gen -> proof_verify of n credentials, one call each
  sign, verify, proof_gen, proof_verify   one batch call over n items
  mixed     one batch call per operation over a mix of sizes and keys
  fixed_msm common-points MSM: `rows` rows over the first `terms` generators
  msm       n variable-base MSMs of 2..kmax terms
"""
import ctypes
import importlib.util
import json
import math
import pathlib
import sys

import numpy as np

ROOT = pathlib.Path(__file__).resolve().parents[1]
ABI = 2
R_MOD = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
SHA, SHAKE = 0, 1


def _package():
    if "cubbs_gb300" not in sys.modules:
        path = ROOT / "cubbs-cred_gb300"
        spec = importlib.util.spec_from_file_location("cubbs_gb300", path / "__init__.py",
                                                      submodule_search_locations=[str(path)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["cubbs_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["cubbs_gb300"]


def _golden(name):
    return json.loads((ROOT / "tests" / "golden" / name).read_text())


_KEYS = None


def _keys():
    """256 key pairs as two byte matrices (32 and 96 bytes a row)."""
    global _KEYS
    if _KEYS is None:
        ks = _golden("keypairs256.json")
        _KEYS = (np.frombuffer(b"".join(bytes.fromhex(k["sk"]) for k in ks), np.uint8).reshape(-1, 32).copy(),
                 np.frombuffer(b"".join(bytes.fromhex(k["pk"]) for k in ks), np.uint8).reshape(-1, 96).copy())
    return _KEYS


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a wallet or a demo: one credential, issued, checked, presented, checked (latency of the smallest calls)
        {"name": "trip_1_L10", "kind": "trip", "n": 1, "L": 10, "R": 5, "keys": 1, "msg": 32, "suite": SHA},
        # an issuer's and a relying party's small batches
        {"name": "sign_64_L10", "kind": "sign", "n": 64, "L": 10, "keys": 1, "msg": 64, "suite": SHA},
        {"name": "verify_64_L10", "kind": "verify", "n": 64, "L": 10, "keys": 1, "msg": 64, "suite": SHA,
         "bad": "message"},
        # bulk issuance
        {"name": "sign_4096_L30", "kind": "sign", "n": 4096, "L": 30, "keys": 8, "msg": 64, "suite": SHA},
        # re-checking a store of credentials of one issuer; a few records are damaged
        {"name": "verify_1000_L20", "kind": "verify", "n": 1000, "L": 20, "keys": 1, "msg": 64, "suite": SHA,
         "bad": "encoding"},
        # the headline pair: presentations of 50 of 100 messages
        {"name": "proof_gen_1024_L100", "kind": "proof_gen", "n": 1024, "L": 100, "R": 50, "keys": 1, "msg": 64,
         "suite": SHA},
        {"name": "proof_verify_1024_L100", "kind": "proof_verify", "n": 1024, "L": 100, "R": 50, "keys": 1, "msg": 64,
         "suite": SHA, "bad": "presentation"},
        # a verifier that serves many issuers
        {"name": "proof_verify_1024_64keys", "kind": "proof_verify", "n": 1024, "L": 100, "R": 50, "keys": 64,
         "msg": 64, "suite": SHA, "bad": "presentation"},
        # a small odd batch under the other ciphersuite
        {"name": "proof_verify_37_shake", "kind": "proof_verify", "n": 37, "L": 30, "R": 11, "keys": 3, "msg": 50,
         "suite": SHAKE, "bad": "presentation"},
        # a batch window of a service: 40/40/10/10 of the four operations, L in 5..200, 256 keys
        {"name": "mixed_256", "kind": "mixed", "n": 256, "L": 200, "keys": 256, "msg": 64, "suite": SHA,
         "bad": "message"},
        # the primitives: fixed-base rows, and MSMs of uneven length over points given by the caller
        {"name": "fixed_msm_4096x12", "kind": "fixed_msm", "rows": 4096, "terms": 12},
        {"name": "msm_1024_K257", "kind": "msm", "n": 1024, "kmax": 257},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["trip", "sign", "verify", "verify", "proof_gen", "proof_gen", "proof_verify", "proof_verify",
                       "proof_verify", "mixed", "fixed_msm", "msm"])
    if kind == "fixed_msm":
        return {"kind": kind, "rows": log(3, 4096), "terms": rng.randint(2, 12)}
    if kind == "msm":
        return {"kind": kind, "n": log(8, 1000), "kmax": log(3, 257)}
    suite = SHAKE if rng.random() < 0.2 else SHA
    if kind == "mixed":
        return {"kind": kind, "n": log(40, 256), "L": rng.choice([20, 50, 100, 200]), "keys": rng.choice([1, 16, 256]),
                "msg": 64, "suite": SHA, "bad": "message"}
    L = log(1, 100)
    n = log(1, 31) if kind == "trip" else log(16, 4096) if kind == "sign" else log(33, 1024)
    case = {"kind": kind, "n": n, "L": L, "keys": min(n, rng.choice([1, 1, 8, 64])), "msg": log(16, 128),
            "suite": suite}
    if kind in ("trip", "proof_gen", "proof_verify"):
        case["R"] = rng.randint(0, L)
    if kind == "verify":
        case["bad"] = rng.choice(["message", "encoding"]) if n < 128 or case["keys"] > 1 else "encoding"
    if kind == "proof_verify":
        case["bad"] = "presentation"
    return case


# ------------------------------------------------------------------ buffers
def _ptr(a):
    return a.ctypes.data


class _Messages:
    """Ragged message lists: `counts[i]` messages of `size` bytes for item i, and the ABI's slices of them."""

    def __init__(self, rng, counts, size):
        self.counts = np.asarray(counts, np.int64)
        self.first = np.concatenate([[0], np.cumsum(self.counts)])
        self.bytes = rng.integers(0, 256, (max(1, int(self.first[-1])), size), dtype=np.uint8)
        self._slices()

    def _slices(self):
        m, size = self.bytes.shape
        self.table = np.empty((m, 2), np.uint64)
        self.table[:, 0] = _ptr(self.bytes) + np.arange(m, dtype=np.uint64) * np.uint64(size)
        self.table[:, 1] = size

    def pointers(self):
        return np.uint64(_ptr(self.table)) + self.first[:-1].astype(np.uint64) * np.uint64(16)

    def picked(self, lists):
        """The messages at `lists[i]` of every item, as another ragged list."""
        out = object.__new__(_Messages)
        out.counts = np.array([len(x) for x in lists], np.int64)
        out.first = np.concatenate([[0], np.cumsum(out.counts)])
        at = [self.first[i] + np.asarray(x, np.int64) for i, x in enumerate(lists)]
        at = np.concatenate(at) if len(at) else np.zeros(0, np.int64)
        out.bytes = self.bytes[at] if len(at) else self.bytes[:1].copy()
        out._slices()
        return out


def _rows(a):
    """Addresses of a matrix's rows."""
    return np.uint64(_ptr(a)) + np.arange(len(a), dtype=np.uint64) * np.uint64(a.strides[0])


class _Call:
    """One batch entry point with its item array, results and output rows; keeps every buffer alive."""

    def __init__(self, name, suite, items, keep, out=None, seeds=None):
        lib = _package().lib()
        self.items, self.keep, self.out, self.seeds = items, keep, out, seeds
        n = len(items)
        self.raw = np.zeros((n, 16), np.uint8)  # CuBbsBbsGpuResult
        self.codes = self.raw[:, :4].view(np.int32)[:, 0]
        self.values = self.raw[:, 4]
        args = [ABI, _ptr(items), n] + ([_ptr(seeds)] if seeds is not None else []) + [_ptr(self.raw)]
        if suite != SHA:
            name = name.replace("_batch_v2", "_batch_cs_v2")
            args.insert(1, suite)
        self.name, self.fn, self.args = name, getattr(lib, name), args

    def __call__(self):
        rc = self.fn(*self.args)
        if rc:
            raise RuntimeError("%s returned %d" % (self.name, rc))
        return [self.codes, self.values] + ([self.out] if self.out is not None else [])


def _sign(suite, sk, pk, hdr, msgs):
    n = len(pk)
    out = np.zeros((n, 80), np.uint8)
    it = np.zeros((n, 11), np.uint64)
    it[:, 0], it[:, 1], it[:, 2], it[:, 3] = _rows(sk), 32, _rows(pk), 96
    it[:, 4], it[:, 5], it[:, 6], it[:, 7] = _rows(hdr), hdr.shape[1], msgs.pointers(), msgs.counts
    it[:, 8], it[:, 9] = _rows(out), 80
    return _Call("cubbs_bbs_gpu_sign_batch_v2", suite, it, (sk, pk, hdr, msgs), out)


def _verify(suite, pk, sig, hdr, msgs):
    it = np.zeros((len(pk), 8), np.uint64)
    it[:, 0], it[:, 1], it[:, 2], it[:, 3] = _rows(pk), 96, _rows(sig), 80
    it[:, 4], it[:, 5], it[:, 6], it[:, 7] = _rows(hdr), hdr.shape[1], msgs.pointers(), msgs.counts
    return _Call("cubbs_bbs_gpu_verify_batch_v2", suite, it, (pk, sig, hdr, msgs))


def _index_lists(lists):
    flat = np.array([j for x in lists for j in x] or [0], np.uint64)
    first = np.concatenate([[0], np.cumsum([len(x) for x in lists])])[:-1].astype(np.uint64)
    return flat, np.uint64(_ptr(flat)) + first * np.uint64(8)


def _proof_gen(suite, pk, sig, hdr, ph, msgs, lists, seeds):
    n = len(pk)
    R = np.array([len(x) for x in lists], np.int64)
    out = np.zeros((n, 272 + 32 * int(msgs.counts.max())), np.uint8)  # room for any disclosure
    flat, at = _index_lists(lists)
    it = np.zeros((n, 15), np.uint64)
    it[:, 0], it[:, 1], it[:, 2], it[:, 3] = _rows(pk), 96, _rows(sig), 80
    it[:, 4], it[:, 5], it[:, 6], it[:, 7] = _rows(hdr), hdr.shape[1], _rows(ph), ph.shape[1]
    it[:, 8], it[:, 9], it[:, 10], it[:, 11] = msgs.pointers(), msgs.counts, at, R
    it[:, 12], it[:, 13] = _rows(out), out.shape[1]
    return _Call("cubbs_bbs_gpu_proof_gen_seeded_batch_v2", suite, it, (pk, sig, hdr, ph, msgs, flat), out, seeds)


def _proof_verify(suite, pk, proof, hdr, ph, msgs, lists):
    shown = msgs.picked(lists)
    flat, at = _index_lists(lists)
    it = np.zeros((len(pk), 13), np.uint64)
    size = 272 + 32 * (msgs.counts - shown.counts)
    it[:, 0], it[:, 1], it[:, 2], it[:, 3] = _rows(pk), 96, _rows(proof), size
    it[:, 4], it[:, 5], it[:, 6], it[:, 7] = _rows(hdr), hdr.shape[1], _rows(ph), ph.shape[1]
    it[:, 8], it[:, 9], it[:, 10], it[:, 11] = shown.pointers(), shown.counts, at, shown.counts
    it[:, 12] = msgs.counts
    return _Call("cubbs_bbs_gpu_proof_verify_batch_v2", suite, it, (pk, proof, hdr, ph, shown, flat))


class _Items:
    """n credentials: keys, headers, messages, disclosed indexes, blinding seeds."""

    def __init__(self, rng, n, lengths, disclosed, keys, size, suite):
        sks, pks = _keys()
        which = np.arange(n) % keys
        rng.shuffle(which)
        self.n, self.suite, self.rng = n, suite, rng
        self.sk, self.pk = sks[which], pks[which]
        self.hdr = rng.integers(0, 256, (n, 64), dtype=np.uint8)
        self.ph = rng.integers(0, 256, (n, 64), dtype=np.uint8)
        self.seeds = rng.integers(0, 256, (n, 32), dtype=np.uint8)
        self.msgs = _Messages(rng, lengths, size)
        self.lists = [sorted(rng.permutation(int(L))[:int(R)].tolist()) for L, R in zip(lengths, disclosed)]

    def sign(self):
        return _sign(self.suite, self.sk, self.pk, self.hdr, self.msgs)

    def verify(self, sig, msgs=None):
        return _verify(self.suite, self.pk, sig, self.hdr, msgs or self.msgs)

    def proof_gen(self, sig):
        return _proof_gen(self.suite, self.pk, sig, self.hdr, self.ph, self.msgs, self.lists, self.seeds)

    def proof_verify(self, proof, ph=None):
        return _proof_verify(self.suite, self.pk, proof, self.hdr, self.ph if ph is None else ph, self.msgs, self.lists)

    def some(self):
        """A few items that get something wrong, as in a store or a stream of requests: one in 64 on average."""
        n = self.n
        return self.rng.permutation(n)[:int(self.rng.integers(1, max(2, n // 32) + 1))]

    def spoiled(self, kind, sig=None, proof=None):
        """The verifying call with a few items spoiled: another message, a damaged encoding, another presentation."""
        at = self.some()
        if proof is not None:
            ph = self.ph.copy()
            ph[at, 5] ^= 1
            return self.proof_verify(proof, ph)
        if kind == "encoding":
            sig = sig.copy()
            sig[at, 0] &= 0x7F
            return self.verify(sig)
        msgs = object.__new__(_Messages)
        msgs.counts, msgs.first, msgs.bytes = self.msgs.counts, self.msgs.first, self.msgs.bytes.copy()
        msgs.bytes[self.msgs.first[at], 0] ^= 1
        msgs._slices()
        return self.verify(sig, msgs)


def _first_generators(terms):
    g = _golden("cfrg_bls12381_sha256.json")["generators"]
    pts = [bytes.fromhex(x) for x in [g["P1"], g["Q1"]] + g["MsgGenerators"]][:terms]
    return np.frombuffer(b"".join(pts), np.uint8).reshape(-1, 48).copy()


def _scalars(rng, n):
    """n canonical scalars, uniform below 2^254 (all below the group order), big-endian."""
    s = rng.integers(0, 256, (n, 32), dtype=np.uint8)
    s[:, 0] &= 0x3F
    return s


def _common_rows(points, scalars, rows):
    """The common-points call over `rows` packed scalar rows."""
    terms = len(points)
    pts = np.zeros((terms, 2), np.uint64)
    pts[:, 0], pts[:, 1] = _rows(points), 48
    out = np.zeros((rows, 48), np.uint8)
    outs = np.zeros((rows, 3), np.uint64)
    outs[:, 0], outs[:, 1] = _rows(out), 48
    item = np.array([[_ptr(pts), terms, 0, _ptr(scalars), 32 * terms, rows, _ptr(outs)]], np.uint64)
    call = _Call("cubbs_bbs_gpu_g1_msm_common_points_batch_v2", SHA, item, (points, scalars, pts, outs), out)
    call.raw = np.zeros((rows, 16), np.uint8)  # one result per row of the item
    call.codes, call.values = call.raw[:, :4].view(np.int32)[:, 0], call.raw[:, 4]
    call.args[-1] = _ptr(call.raw)
    return call


# ------------------------------------------------------------------ the four functions over a case
def prepare(case, seed):
    rng = np.random.default_rng(int(seed))
    kind = case["kind"]
    if kind == "fixed_msm":
        return [_common_rows(_first_generators(case["terms"]), _scalars(rng, case["rows"] * case["terms"]),
                             case["rows"])]
    if kind == "msm":
        K = rng.integers(2, case["kmax"] + 1, case["n"])
        total, first = int(K.sum()), np.concatenate([[0], np.cumsum(K)])[:-1].astype(np.uint64)
        made = _common_rows(_first_generators(1), _scalars(rng, total), total)
        points, scalars = made()[2], _scalars(rng, total)
        ps, ss = np.zeros((total, 2), np.uint64), np.zeros((total, 2), np.uint64)
        ps[:, 0], ps[:, 1], ss[:, 0], ss[:, 1] = _rows(points), 48, _rows(scalars), 32
        out = np.zeros((case["n"], 48), np.uint8)
        it = np.zeros((case["n"], 6), np.uint64)
        it[:, 0] = np.uint64(_ptr(ps)) + first * np.uint64(16)
        it[:, 1] = np.uint64(_ptr(ss)) + first * np.uint64(16)
        it[:, 2], it[:, 3], it[:, 4] = K, _rows(out), 48
        return [_Call("cubbs_bbs_gpu_g1_msm_batch_v2", SHA, it, (points, scalars, ps, ss), out)]
    n, suite = case["n"], case["suite"]
    if kind == "mixed":
        share = [2 * n // 5, 2 * n // 5, n // 10]
        share.append(n - sum(share))
        sets = []
        for m in share:
            L = rng.choice([x for x in (5, 10, 20, 50, 100, 200) if x <= case["L"]], m)
            L[0] = case["L"]
            R = np.maximum(1, np.round(rng.uniform(0.1, 0.9, m) * L)).astype(int)
            sets.append(_Items(rng, m, L, R, case["keys"], case["msg"], suite))
        sigs = [None] + [s.sign()()[2] for s in sets[1:]]
        proof = sets[3].proof_gen(sigs[3])()[2]
        return [sets[0].sign(), sets[1].spoiled(case["bad"], sig=sigs[1]), sets[2].proof_gen(sigs[2]),
                sets[3].proof_verify(proof)]
    it = _Items(rng, n, [case["L"]] * n, [case.get("R", 0)] * n, case["keys"], case["msg"], suite)
    sign = it.sign()
    if kind == "sign":
        return [sign]
    sig = sign()[2]
    if kind == "verify":
        return [it.spoiled(case["bad"], sig=sig)]
    gen = it.proof_gen(sig)
    if kind == "proof_gen":
        return [gen]
    proof = gen()[2]
    if kind == "proof_verify":
        return [it.spoiled(case["bad"], proof=proof)]
    # trip: every call reads what the one before it wrote
    return [sign, it.verify(sig), gen, it.proof_verify(proof)]


def run(state):
    return [call() for call in state]


# 381-bit Montgomery products (M) that the group operations need: a fixed-base term of 13 mixed additions, a GLV
# term of 128 doublings and 50 mixed additions with its table, a square root, the 64-bit batch coefficient of one
# point (8-bit windows), a pairing check; and 600 32-bit integer operations per product (300 multiply-adds).
_FIXED, _VAR, _SQRT, _BATCH, _PAIRING, _OPS = 130, 1800, 450, 80, 16470, 600


def _one(kind, n, L, R, keys, msg):
    """(bytes, M) of n items of one operation."""
    given = n * (L * msg + 64 + 96)
    if kind == "sign":
        return given + n * (32 + 80), n * (L + 2) * _FIXED
    if kind == "verify":
        return given + n * 80, n * ((L + 2) * _FIXED + _VAR + _SQRT + 2 * _BATCH) + min(n, keys) * _PAIRING
    proof = 272 + 32 * (L - R)
    if kind == "proof_gen":
        return given + n * (64 + 80 + 32 + 8 * R + proof), n * ((2 * L + 3 - R) * _FIXED + 7 * _VAR + _SQRT)
    return (n * (R * (msg + 8) + 64 + 64 + 96 + proof),
            n * ((L + 2) * _FIXED + 4 * _VAR + 3 * _SQRT + 2 * _BATCH) + min(n, keys) * _PAIRING)


def work(case):
    kind = case["kind"]
    if kind == "fixed_msm":
        n = case["rows"]
        return {"bytes": n * (32 * case["terms"] + 48), "flops": n * case["terms"] * _FIXED * _OPS}
    if kind == "msm":
        terms = case["n"] * (2 + case["kmax"]) / 2
        return {"bytes": terms * 80 + case["n"] * 48, "flops": terms * (_SQRT + 32 * 2 * 10) * _OPS}
    if kind == "mixed":
        Ls = [x for x in (5, 10, 20, 50, 100, 200) if x <= case["L"]]
        L = sum(Ls) / len(Ls)
        parts = [_one(k, case["n"] * share, L, L / 2, case["keys"], case["msg"])
                 for k, share in (("sign", .4), ("verify", .4), ("proof_gen", .1), ("proof_verify", .1))]
    else:
        kinds = ("sign", "verify", "proof_gen", "proof_verify") if kind == "trip" else (kind,)
        parts = [_one(k, case["n"], case["L"], case.get("R", 0), case["keys"], case["msg"]) for k in kinds]
    return {"bytes": sum(b for b, _ in parts), "flops": sum(m for _, m in parts) * _OPS}


def exact(case, seed):
    """Every output is a whole number (codes, verdicts, encoded bytes): none is a rounded value."""
    return None
