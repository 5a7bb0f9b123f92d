"""The work a user has this library do, as cases that can be timed and compared.

Every case goes through the Python binding of the C ABI (bend-groth16_gb300/bendg.py), as a
program would call it: the primitives on device-resident or host buffers, and whole Groth16
proofs of SquareChain(2^K) circuits against a resident key, from uploaded files, and in a batch.
A prover keeps its circuit's proving key and proves many assignments, so a case's key belongs to
the process (one per K, from a fixed seed) and its witness and randomness come from the seed.
"""
import os
import shutil
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "bend-groth16_gb300"))
import bendg  # noqa: E402

R = 21888242871839275222246405745257275088548364400416034343698204186575808495617  # Fr
Q = 21888242871839275222246405745257275088696311157297823662689037894645226208583  # Fq
R256 = 1 << 256
ROOT_2_28 = 19103219067921713944291392827692070036145651957329286315305642004821462161904
G2_X = (10857046999023057135944570762232829481370756359578518086990519993285655852781,
        11559732032986387107991004021392285783925812861821192530917403151452391805634)
G2_Y = (8495653923123431417604973247489272438418190587263600148770280649306958101930,
        4082367875863433681332203403145435568316851327593401208105741076214120093531)
KEY_SEED = 18181818
MODES = {"forward": bendg.NTT_FORWARD, "inverse": bendg.NTT_INVERSE, "coset_forward": bendg.NTT_COSET_FORWARD,
         "coset_inverse": bendg.NTT_COSET_INVERSE}
LANES = 8


def listed():
    return [
        # latency of the smallest call: a commitment to a thousand values already on the device
        {"name": "msm_g1_1000", "kind": "msm", "curve": 1, "n": 1000, "where": "device"},
        # the seam call of the prover (host buffers in the wire layout), a ragged size
        {"name": "msm_g1_host_50021", "kind": "msm", "curve": 1, "n": 50021, "where": "host"},
        # the standalone primitives of the benchmark
        {"name": "msm_g1_2e20", "kind": "msm", "curve": 1, "n": 1 << 20, "where": "device"},
        {"name": "msm_g2_2e18", "kind": "msm", "curve": 2, "n": 1 << 18, "where": "device"},
        {"name": "ntt_2e20", "kind": "ntt", "log2n": 20, "mode": "forward"},
        # the QAP seam call on host buffers, a mid-size circuit's domain
        {"name": "qap_host_2e15", "kind": "qap", "log2d": 15},
        # proofs against a resident key: a small circuit (latency), a mid-size one, the headline
        # size and the largest of the benchmark
        {"name": "prove_2e10", "kind": "prove", "log2k": 10, "proofs": 1},
        {"name": "prove_2e14", "kind": "prove", "log2k": 14, "proofs": 1},
        {"name": "prove_2e18", "kind": "prove", "log2k": 18, "proofs": 1},
        {"name": "prove_2e20", "kind": "prove", "log2k": 20, "proofs": 1},
        # one proof with every file uploaded (what a process that proves once does)
        {"name": "oneshot_2e18", "kind": "oneshot", "log2k": 18},
        # many proofs of mixed size at once, K drawn by the benchmark's weights
        {"name": "batch_16", "kind": "batch", "ks": "10 10 10 10 10 12 12 12 12 14 14 14 16 16 16 18"},
    ]


def _log_int(rng, lo, hi):
    """an integer of [lo, hi], uniform over its logarithm"""
    return min(hi, max(lo, int(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choices(["msm", "ntt", "qap", "prove", "oneshot", "batch"], [8, 2, 1, 3, 1, 4])[0]
    if kind == "msm":
        curve = rng.choice([1, 2])
        n = _log_int(rng, 300, (1 << 20) if curve == 1 else (1 << 18))
        return {"kind": kind, "curve": curve, "n": n, "where": rng.choice(["device", "host"])}
    if kind == "ntt":
        return {"kind": kind, "log2n": rng.randint(8, 21), "mode": rng.choice(sorted(MODES))}
    if kind == "qap":
        return {"kind": kind, "log2d": rng.choice([8, 9, 10, 11, 12, 13, 14, 16, 17, 18])}
    if kind == "batch":
        ks = rng.choices([10, 12, 14, 16, 18], [0.3, 0.25, 0.2, 0.15, 0.1], k=rng.randint(4, 16))
        return {"kind": kind, "ks": " ".join(str(k) for k in sorted(ks))}
    if kind == "oneshot":
        return {"kind": kind, "log2k": rng.randint(8, 17)}
    k = rng.choice([8, 9, 11, 12, 13, 15, 16, 17, 19])
    # one assignment after another against the same key
    return {"kind": kind, "log2k": k, "proofs": 1 if k == 19 else rng.randint(1, 4)}


# ---------------------------------------------------------------- inputs
_ctx = None
_files, _keys = {}, {}


def _context():
    global _ctx
    if _ctx is None:
        _ctx = bendg.Context(0)
    return _ctx


def _key_files(k):
    """the .bin files of one SquareChain(2^k) instance, in pinned host memory"""
    if k not in _files:
        path = tempfile.mkdtemp(prefix="bendg_cases_")
        try:
            _context().synth_square_chain(k, KEY_SEED + k, path)
            _files[k] = bendg.HostFiles(path, pinned=True)
        finally:
            shutil.rmtree(path, ignore_errors=True)
    return _files[k]


def _resident_key(k):
    if k not in _keys:
        _keys[k] = _context().pk_upload(_key_files(k))
    return _keys[k]


def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0xFFFFFFFF, int(case.get("n", case.get("log2k", 0)))])


def _scalars(rng, n):
    """n values uniform below 0x3064 2^240 < r (all but one in 40000 of the field), 16-bit words"""
    w = rng.integers(0, 1 << 16, size=(n, 16), dtype=np.uint32)
    w[:, 15] = rng.integers(0, 0x3064, size=n, dtype=np.uint32)
    return w


def _mont_words(vals, p):
    return bendg.ints_to_wire([v * R256 % p for v in vals]).reshape(-1)


def _points(rng, curve, n):
    """n seeded random multiples of the curve's generator (wire layout), and the multipliers"""
    g = _mont_words((1, 2) if curve == 1 else G2_X + G2_Y, Q)
    k = _scalars(rng, n)
    c = bendg.CURVE_G1 if curve == 1 else bendg.CURVE_G2
    return _context().curve_op(c, bendg.COP_MUL, np.broadcast_to(g, (n, g.size)), k16=k).reshape(n, -1), k


def _pack(words):
    """wire words (16-bit limbs) to the device's packed layout (32-bit limbs), on the device"""
    w = np.ascontiguousarray(words).reshape(-1, 2)
    return torch.from_numpy((w[:, 0] | (w[:, 1] << 16)).view(np.int32)).cuda()


def _pinned(words):
    """a copy in pinned host memory, where a prover's program keeps what it uploads"""
    t = torch.empty(words.size, dtype=torch.int32, pin_memory=True)
    t.numpy()[:] = words.reshape(-1).view(np.int32)
    return t


def _witness(rng, k):
    """z = [1, x_N, x_0 .. x_{N-1}] of SquareChain(2^k) for a seeded x_0, and r and s (Montgomery)"""
    rinv = pow(R256, -1, R)
    x = int.from_bytes(_scalars(rng, 1).astype("<u2").tobytes(), "little")
    chain = []
    for _ in range((1 << k) + 1):
        chain.append(x)
        x = x * x % R * rinv % R  # squares in Montgomery form
    z = bendg.ints_to_wire([R256 % R, chain[-1]] + chain[:-1])
    return _pinned(z), _pinned(_scalars(rng, 2))


def prepare(case, seed):
    rng, kind = _rng(case, seed), case["kind"]
    if kind == "msm":
        pts, _ = _points(rng, case["curve"], case["n"])
        sc = _scalars(rng, case["n"])
        if case["where"] == "device":
            pts, sc = _pack(pts), _pack(sc)
        return {"case": case, "points": pts, "scalars": sc}
    if kind == "ntt":
        return {"case": case, "data": _pack(_scalars(rng, 1 << case["log2n"]))}
    if kind == "qap":
        return {"case": case, "abc": [_scalars(rng, 1 << case["log2d"]) for _ in range(3)]}
    if kind == "batch":
        ks = [int(k) for k in case["ks"].split()]
        ws = [_witness(rng, k) for k in ks]
        return {"case": case, "keys": [_resident_key(k) for k in ks], "wit": ws}
    k = case["log2k"]
    if kind == "prove":
        return {"case": case, "key": _resident_key(k), "wit": [_witness(rng, k) for _ in range(case["proofs"])]}
    z, rs = _witness(rng, k)
    files = _key_files(k)
    inputs = bendg.Inputs.from_buffer_copy(files.inputs)  # the key's files with this witness
    inputs.witness, inputs.rs = z.data_ptr(), rs.data_ptr()
    return {"case": case, "inputs": inputs, "keep": (files, z, rs)}


# ---------------------------------------------------------------- one pass
def _proof_arrays(p):
    return {name: np.ctypeslib.as_array(getattr(p, name)).view(np.int32).copy() for name in ("a", "b", "c")}


def run(state):
    case, ctx = state["case"], _context()
    kind = case["kind"]
    if kind == "msm":
        p, s, n = state["points"], state["scalars"], case["n"]
        if case["where"] == "device":
            f = ctx.msm_g1_dev if case["curve"] == 1 else ctx.msm_g2_dev
            return f(p.data_ptr(), s.data_ptr(), n).view(np.int32)
        return (ctx.msm_g1 if case["curve"] == 1 else ctx.msm_g2)(p, s, n).view(np.int32)
    if kind == "ntt":
        ctx.ntt_dev(state["data"].data_ptr(), case["log2n"], MODES[case["mode"]])  # in place
        return state["data"]
    if kind == "qap":
        return ctx.qap_h(*state["abc"], case["log2d"]).view(np.int32)
    if kind == "prove":
        return [_proof_arrays(state["key"].prove(z.numpy().view(np.uint32), rs.numpy().view(np.uint32))[0])
                for z, rs in state["wit"]]
    if kind == "oneshot":
        proof, _ = ctx.prove_inputs(state["inputs"])
        return _proof_arrays(proof)
    proofs, _, statuses = ctx.prove_batch(state["keys"], [z.data_ptr() for z, _ in state["wit"]],
                                          [rs.data_ptr() for _, rs in state["wit"]], lanes=LANES)
    return {name: np.stack([_proof_arrays(p)[name] for p in proofs]) for name in ("a", "b", "c")} | {
        "status": np.array(statuses, dtype=np.int32)}


# ---------------------------------------------------------------- what a pass cannot do without
FQ_MUL = 2 * 136  # operations of one modular product: 64 limb products, 64 + 8 for its reduction
ADD_G1, ADD_G2 = 10 * FQ_MUL, 30 * FQ_MUL  # one point addition


def _msm_work(curve, n):
    """points and scalars read once; every scalar's windows (about log2 n bits) one addition each"""
    c = max(4, n.bit_length() - 1)
    return n * ((64 if curve == 1 else 128) + 32), n * -(-254 // c) * (ADD_G1 if curve == 1 else ADD_G2)


def _ntt_work(lg):
    return 64 << lg, (lg << lg) // 2 * FQ_MUL


def _proof_work(k, host):
    n, parts = 1 << k, []
    for curve, m in ((1, n + 2), (1, n + 2), (2, n + 2), (1, 2 * n - 1), (1, n)):
        parts.append(_msm_work(curve, m))
    parts += [_ntt_work(k + 1)] * 7
    scale = 2 if host else 1  # the files hold 16-bit limbs in 32-bit words
    return sum(b for b, _ in parts) * scale, sum(f for _, f in parts)


def work(case):
    kind = case["kind"]
    if kind == "msm":
        b, f = _msm_work(case["curve"], case["n"])
        b *= 2 if case["where"] == "host" else 1
    elif kind == "ntt":
        b, f = _ntt_work(case["log2n"])
    elif kind == "qap":
        lg = case["log2d"]
        b, f = 4 * (64 << lg), 7 * _ntt_work(lg)[1]
    elif kind == "batch":
        got = [_proof_work(int(k), False) for k in case["ks"].split()]
        b, f = sum(x for x, _ in got), sum(x for _, x in got)
    else:
        b, f = (x * case.get("proofs", 1) for x in _proof_work(case["log2k"], kind == "oneshot"))
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- plain integers, without the library
def _ints(words):
    raw = words.astype("<u2").tobytes()
    return [int.from_bytes(raw[i: i + 32], "little") for i in range(0, len(raw), 32)]


class _Fq2:
    """just enough of Fq[u]/(u^2 + 1) for an affine addition"""

    @staticmethod
    def mul(a, b):
        return ((a[0] * b[0] - a[1] * b[1]) % Q, (a[0] * b[1] + a[1] * b[0]) % Q)

    @staticmethod
    def sub(a, b):
        return ((a[0] - b[0]) % Q, (a[1] - b[1]) % Q)

    @staticmethod
    def inv(a):
        d = pow(a[0] * a[0] + a[1] * a[1], -1, Q)
        return (a[0] * d % Q, -a[1] * d % Q)


def _add(p, q):
    if p is None or q is None:
        return q if p is None else p
    f = _Fq2
    if p[0] == q[0]:
        if p[1] != q[1]:
            return None
        x2 = f.mul(p[0], p[0])
        lam = f.mul(f.mul((3, 0), x2), f.inv(f.mul((2, 0), p[1])))
    else:
        lam = f.mul(f.sub(q[1], p[1]), f.inv(f.sub(q[0], p[0])))
    x = f.sub(f.sub(f.mul(lam, lam), p[0]), q[0])
    return x, f.sub(f.mul(lam, f.sub(p[0], x)), p[1])


def _times(p, k):
    acc = None
    for bit in bin(k)[2:]:
        acc = _add(acc, acc)
        if bit == "1":
            acc = _add(acc, p)
    return acc


def _fft(a, w):
    """sum_j a_j w^(ij), radix 2"""
    n = len(a)
    if n == 1:
        return a
    e, o = _fft(a[0::2], w * w % R), _fft(a[1::2], w * w % R)
    out, t = [0] * n, 1
    for i in range(n // 2):
        u = t * o[i] % R
        out[i], out[i + n // 2] = (e[i] + u) % R, (e[i] - u) % R
        t = t * w % R
    return out


def _ntt(a, mode):
    n = len(a)
    w = pow(ROOT_2_28, (1 << 28) // n, R)
    if mode.startswith("coset") and mode.endswith("forward"):
        g = 1
        for j in range(n):
            a[j], g = a[j] * g % R, g * 5 % R
    if mode.endswith("forward"):
        return _fft(a, w)
    out = [x * pow(n, -1, R) % R for x in _fft(a, pow(w, -1, R))]
    if mode.startswith("coset"):
        gi, g = pow(5, -1, R), 1
        for j in range(n):
            out[j], g = out[j] * g % R, g * gi % R
    return out


def exact(case, seed):
    """the same outputs from Python integers; None for whole proofs (a pairing-free restatement of
    the prover would be another prover) and for transforms too long for plain Python"""
    rng, kind = _rng(case, seed), case["kind"]
    if kind == "msm":
        k, sc = _scalars(rng, case["n"]), _scalars(rng, case["n"])
        total = sum(a * b for a, b in zip(_ints(k), _ints(sc))) % R
        g1 = case["curve"] == 1
        p = _times(((1, 0), (2, 0)) if g1 else (G2_X, G2_Y), total)
        xy = [p[0][0], p[1][0]] if g1 else [*p[0], *p[1]]
        words = _mont_words(xy, Q)
        if case["where"] == "host":  # Jacobian with z = 1
            return np.concatenate([words, _mont_words([1] if g1 else [1, 0], Q)]).view(np.int32)
        return (words[0::2] | (words[1::2] << 16)).view(np.int32)
    if kind == "ntt" and case["log2n"] <= 16:  # the transform is linear: Montgomery form passes through
        words = bendg.ints_to_wire(_ntt(_ints(_scalars(rng, 1 << case["log2n"])), case["mode"])).reshape(-1)
        return torch.from_numpy((words[0::2] | (words[1::2] << 16)).view(np.int32))
    if kind == "qap" and case["log2d"] <= 14:
        rinv = pow(R256, -1, R)
        a, b, c = ([x * rinv % R for x in _ints(_scalars(rng, 1 << case["log2d"]))] for _ in range(3))
        a, b, c = (_ntt(_ntt(v, "inverse"), "coset_forward") for v in (a, b, c))
        zinv = pow(pow(5, len(a), R) - 1, -1, R)
        h = _ntt([(x * y - z) * zinv % R for x, y, z in zip(a, b, c)], "coset_inverse")
        return bendg.ints_to_wire([v * R256 % R for v in h]).reshape(-1).view(np.int32)
    return None
