"""The work that a user of this framework has it do, as cases that can be timed.

Every case goes through the package's public entry points, as the prover
(gb_prover.plonk), a proof server or a host program on the C ABI calls them.
Sizes are those of this repository's workloads: a 2^20-point commitment and
16 transforms of 2^20, a proof of 2^16 rows, 64 multiexps of 2^10..2^18
points with transforms of the matching sizes, and a stream of proofs of
2^12..2^18 rows, most of them small.  All results are field elements, points
or bytes, exact whole numbers, so there is no 64-bit floating value to hold
them against.
"""
import ctypes
import hashlib
import os
import sys

import numpy as np
import torch

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(REPO, "midnight-ledger-cuda_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import gb_prover as gb  # noqa: E402
from gb_prover import plonk  # noqa: E402
from gb_prover.kzg import CircuitTranscript, ParamsKZG, affine_from_projective_batch  # noqa: E402
from gb_prover.rng import ChaCha20Rng, ints_to_mont  # noqa: E402

TAU = 0x5EED0F7A0


def listed():
    return [
        # one short polynomial committed against the resident SRS: the
        # smallest call, launches and latency
        {"name": "commit_2p10", "kind": "commit", "log_ctx": 10, "n": 1 << 10, "count": 1},
        # the commitments of one round of a proof of 2^16 rows
        {"name": "commit_3x2p16", "kind": "commit", "log_ctx": 16, "n": 1 << 16, "count": 3},
        # the commitment of one polynomial of 2^20 coefficients
        {"name": "commit_2p20", "kind": "commit", "log_ctx": 20, "n": 1 << 20, "count": 1},
        # 64 multiexps of uneven sizes in one batch, a fifth of the scalars
        # below 2^64 and a tenth of them zero
        {"name": "multiexp_ragged_64", "kind": "ragged", "log_ctx": 18, "count": 64, "lo": 10, "hi": 18},
        # one multiexp over bases and scalars in host memory, nothing kept:
        # the drop-in call of a program without resident bases
        {"name": "multiexp_host_2p16", "kind": "host", "n": 1 << 16},
        # the transforms of 16 polynomials of 2^20 values
        {"name": "ntt_16x2p20", "kind": "ntt", "log_n": 20, "count": 16, "inverse": False},
        # one column of a small proof to coefficients: a transform's latency
        {"name": "intt_2p12", "kind": "ntt", "log_n": 12, "count": 1, "inverse": True},
        # 64 transforms of uneven sizes in one call
        {"name": "ntt_ragged_64", "kind": "ntt_ragged", "count": 64, "lo": 10, "hi": 18, "inverse": False},
        # coefficients to the extended coset, 8 columns of 2^18 rows, blowup 4
        {"name": "lde_8x2p18", "kind": "lde", "log_n": 18, "log_ext": 20, "count": 8},
        # the permutation grand products of a proof of 2^16 rows
        {"name": "products_2p16", "kind": "products", "log_n": 16, "columns": 3},
        # a whole proof of the server's most frequent request
        {"name": "proof_2p12", "kind": "proof", "k": 12, "advice": 3, "degree": 3, "lookups": 0},
        # a whole proof: 2^16 rows, 3 advice columns, 2^14 copies, one lookup
        {"name": "proof_2p16", "kind": "proof", "k": 16, "advice": 3, "degree": 3, "lookups": 1},
    ]


def draw(rng):
    kind = rng.choice(["commit", "commit", "ragged", "host", "ntt", "ntt_ragged", "lde", "products", "proof"])
    if kind == "commit":
        # polynomials of any length up to the SRS's; a round commits a few
        n = int(2 ** rng.uniform(8, 20))
        count = 1 if n > 1 << 18 else rng.randint(1, 5)
        return {"kind": kind, "log_ctx": max(8, (n - 1).bit_length()), "n": n, "count": count}
    if kind == "ragged":
        return {"kind": kind, "log_ctx": rng.randint(16, 18), "count": rng.randint(4, 64), "lo": rng.randint(6, 11),
                "hi": rng.randint(13, 16)}
    if kind == "host":
        return {"kind": kind, "n": int(2 ** rng.uniform(6, 17))}
    if kind == "ntt":
        log_n = rng.randint(6, 20)
        return {"kind": kind, "log_n": log_n, "count": rng.randint(1, min(32, 1 << (24 - log_n))),
                "inverse": rng.random() < 0.5}
    if kind == "ntt_ragged":
        return {"kind": kind, "count": rng.randint(3, 64), "lo": rng.randint(3, 11), "hi": rng.randint(12, 18),
                "inverse": rng.random() < 0.5}
    if kind == "lde":
        log_n = rng.randint(8, 19)
        return {"kind": kind, "log_n": log_n, "log_ext": log_n + rng.randint(1, 3),
                "count": rng.randint(1, min(12, 1 << (21 - log_n)))}
    if kind == "products":
        return {"kind": kind, "log_n": rng.randint(8, 18), "columns": rng.randint(1, 8)}
    return {"kind": kind, "k": rng.randint(9, 14), "advice": rng.randint(3, 6), "degree": rng.randint(3, 5),
            "lookups": rng.randint(0, 2)}


# ---------------------------------------------------------------- inputs

ONE = ints_to_mont([1])[0]
_KEPT = {}


def _keep(key, make):
    """what a program makes once and keeps: the resident SRS by its size"""
    if key not in _KEPT:
        _KEPT[key] = make()
    return _KEPT[key]


def _context(log_n):
    """resident bases [r_i] G, 2^log_n of them"""
    def make():
        vec, _ = gb.fr_random_chacha20(hashlib.sha256(b"bases").digest(), 0, 1 << log_n)
        return gb.Bls12_381G1MsmContext(gb.g1_generator_mul(vec.download()))
    return _keep(("context", log_n), make)


def _params(k):
    return _keep(("params", k), lambda: ParamsKZG.unsafe_setup(k, plonk.fr_mont(TAU)))


def _uniform(tag, seed, n):
    """n uniform field elements, resident"""
    return gb.fr_random_chacha20(hashlib.sha256(("%s %d" % (tag, seed)).encode()).digest(), 0, n)[0]


def _sizes(case):
    """the uneven sizes of a ragged case: 2^u, u uniform between lo and hi"""
    rng = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    return [int(round(2 ** u)) for u in rng.uniform(case["lo"], case["hi"], size=case["count"])]


class _Values:
    """the resident values of a device vector, for a tensor that views them"""

    def __init__(self, vec):
        self.vec = vec
        address = ctypes.c_uint64.from_address(vec.raw.value).value  # the handle begins with its values' address
        self.__cuda_array_interface__ = {"shape": (vec.len, 4), "typestr": "<i8", "data": (address, False),
                                         "version": 3}


def _view(vec):
    return torch.as_tensor(_Values(vec), device="cuda")


def _points(jacobian):
    """projective results as a commitment's user reads them: affine"""
    return affine_from_projective_batch(jacobian).view(np.int64)


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "commit":
        st["context"] = _context(case["log_ctx"])
        st["scalars"] = _uniform("commit", seed, case["n"] * case["count"])
    elif kind == "ragged":
        # 70% uniform, 20% uniform below 2^64, 10% zero
        sizes = [min(n, 1 << case["log_ctx"]) for n in _sizes(case)]
        total = sum(sizes)
        rng = np.random.default_rng([seed, 1])
        values = _uniform("ragged", seed, total).download()
        u = rng.random(total)
        small = np.nonzero((u >= 0.7) & (u < 0.9))[0]
        limbs = np.zeros((len(small), 4), dtype=np.uint64)
        limbs[:, 0] = rng.integers(0, 2**64, size=len(small), dtype=np.uint64)
        if len(small):
            r2 = ints_to_mont([pow(2, 256, plonk.R)])
            values[small] = gb.bls12_381_fr_poly_lincomb(limbs[None], r2)
        values[u >= 0.9] = 0
        st["context"] = _context(case["log_ctx"])
        st["scalars"] = gb.Bls12_381FrDeviceVec.upload(values)
        st["slices"] = [(int(o), 0, n) for o, n in zip(np.concatenate([[0], np.cumsum(sizes)[:-1]]), sizes)]
    elif kind == "host":
        st["points"] = gb.g1_generator_mul(_uniform("points", seed, case["n"]).download())
        st["scalars"] = _uniform("host", seed, case["n"]).download()
    elif kind == "ntt":
        st["vec"] = _uniform("ntt", seed, case["count"] << case["log_n"])
        st["view"] = _view(st["vec"])
    elif kind == "ntt_ragged":
        st["logs"] = sorted(((n - 1).bit_length() for n in _sizes(case)), reverse=True)
        st["offsets"] = np.concatenate([[0], np.cumsum([1 << lg for lg in st["logs"]])[:-1]]).astype(np.uint64)
        st["vec"] = _uniform("ntt_ragged", seed, sum(1 << lg for lg in st["logs"]))
        st["view"] = _view(st["vec"])
    elif kind == "lde":
        st["vec"] = _uniform("lde", seed, case["count"] << case["log_n"])
        st["backend"] = plonk.GpuBackend(None)
    elif kind == "products":
        n, m = 1 << case["log_n"], case["columns"]
        st["columns"], st["sigma"] = _uniform("columns", seed, m * n), _uniform("sigma", seed, m * n)
        st["beta"], st["gamma"] = _uniform("challenges", seed, 2).download()
        st["deltas"] = ints_to_mont([pow(plonk.DELTA, j, plonk.R) for j in range(m)])
        st["omega"] = ints_to_mont([plonk.omega_for(case["log_n"])])[0]
        st["blinds"] = _uniform("blinds", seed, 5 * m).download()
    else:
        k = case["k"]
        c = plonk.SyntheticCircuit(k, advice=case["advice"], degree=case["degree"], lookups=case["lookups"],
                                   copies=1 << (k - 2), table_log=min(12, k - 3), label="circuit")
        fixed, advice, copies = c.synthesize("circuit %d" % seed)
        st["params"] = _params(k)
        st["backend"] = plonk.GpuBackend(st["params"])
        st["key"] = plonk.keygen(st["params"], c, st["backend"], fixed, copies)
        st["advice"] = ints_to_mont([v for col in advice for v in col])
        st["seed"] = seed
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "commit":
        return _points(st["context"].device_batch(st["scalars"], 0, case["n"], case["count"]))
    if kind == "ragged":
        return _points(st["context"].device_ragged(st["scalars"], st["slices"]))
    if kind == "host":
        return _points(gb.bls12_381_g1_msm(st["points"], st["scalars"]))
    if kind == "ntt":
        st["vec"].ntt_zeta_batch(case["log_n"], case["count"], case["inverse"], ONE, ONE, ONE)
        return st["view"]
    if kind == "ntt_ragged":
        st["vec"].ntt_ragged(st["offsets"], st["logs"], case["inverse"], ONE, ONE, ONE)
        return st["view"]
    if kind == "lde":
        return _view(st["backend"].coeff_to_extended(st["vec"], case["log_n"], case["count"], case["log_ext"]))
    if kind == "products":
        m, chunk = case["columns"], 3
        sets = -(-m // chunk)
        return _view(gb.fr_permutation_products_device(st["columns"], st["sigma"], 1 << case["log_n"], m, chunk,
                                                       st["beta"], st["gamma"], st["omega"], st["deltas"],
                                                       st["blinds"][:5 * sets], 5))
    proof = plonk.create_proof(st["params"], st["key"], st["advice"], st["backend"], CircuitTranscript(),
                               ChaCha20Rng.from_label("proof %d" % st["seed"]))
    return np.frombuffer(proof, dtype=np.uint8)


# ---------------------------------------------------------------- work

# 32-bit multiply-adds, two operations each, of one product in either field
_FP, _FR = 2 * 300, 2 * 136


def _multiexp(n, resident=True):
    """(bytes, operations): each scalar and base read once; 10 products a
    mixed addition, 14 a bucket addition, at the best window of 8..20 bits"""
    best = min(10 * n * (254 // c + 1) + 14 * (1 if resident else 254 // c + 1) * (1 << c) for c in range(8, 21))
    return n * (32 + 96) + 96, best * _FP


def _transform(log_n, count):
    return (64 << log_n) * count, (log_n << log_n) // 2 * count * _FR


def work(case):
    kind = case["kind"]
    if kind in ("commit", "ragged", "host"):
        if kind == "commit":
            parts = [_multiexp(case["n"])] * case["count"]
        elif kind == "ragged":
            mid = 2 ** case["hi"] / (case["hi"] - case["lo"]) * 1.4427  # mean of 2^u, u uniform in lo..hi
            parts = [_multiexp(int(mid), False)] * case["count"]
        else:
            parts = [_multiexp(case["n"], False)]
        b, f = (sum(p[i] for p in parts) for i in (0, 1))
    elif kind == "ntt":
        b, f = _transform(case["log_n"], case["count"])
    elif kind == "ntt_ragged":
        logs = [case["lo"] + (case["hi"] - case["lo"]) * (i + 0.5) / case["count"] for i in range(case["count"])]
        parts = [_transform(int(lg) + 1, 1) for lg in logs]
        b, f = (sum(p[i] for p in parts) for i in (0, 1))
    elif kind == "lde":
        f = _transform(case["log_ext"], case["count"])[1]
        b = 32 * case["count"] * ((1 << case["log_n"]) + (1 << case["log_ext"]))
    elif kind == "products":
        n, m = 1 << case["log_n"], case["columns"]
        sets = -(-m // 3)
        b, f = 32 * n * (2 * m + sets), n * (4 * m + 6 * sets) * _FR
    else:
        # the multiexps of its commitments and the transforms of its columns
        k, m, d, lk = case["k"], case["advice"], case["degree"], case["lookups"]
        pieces = max(d, 5 if lk else 4) - 1
        ext = k + (pieces - 1).bit_length()
        sets = -(-m // 3)
        columns = m + 3 * lk + sets
        commits = m + 2 * lk + sets + lk + 1 + pieces + 2
        b = 32 * (m + columns + pieces) << k
        f = commits * _multiexp(1 << k)[1] + _transform(k, columns + 1)[1] + _transform(ext, columns + 1)[1]
    return {"bytes": float(b), "flops": float(f)}


def exact(case, seed):
    return None  # whole numbers and bytes: every output is exact
