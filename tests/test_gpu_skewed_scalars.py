"""Scalars of a few bits, as most of a circuit's assignment has: they leave all but a few hundred buckets
empty and put many pieces into each of those (k_bucket_heavy's limit, msm.cu).  Results are checked
through the discrete logarithms, and proofs against the same proof by another route."""
import numpy as np
import pytest

import bendg
import bn254_ref as o
from gpu_helpers import g1_from_jac_wire, g2_from_jac_wire, scalars_wire
from test_gpu_batch import rs_words
from test_gpu_msm import gpu_points

pytestmark = pytest.mark.gpu


def few_bits(rng, n, bits, spread):
    """n scalars below 2^bits, `spread` of them uniform over the field"""
    return [int.from_bytes(rng.bytes(32), "little") % o.P_FR if u < spread else int(v)
            for u, v in zip(rng.random(n), rng.integers(0, 1 << bits, size=n))]


def msm(ctx, curve, pts, words, n):
    if curve == bendg.CURVE_G1:
        return g1_from_jac_wire(ctx.msm_g1(pts, words, n))
    return g2_from_jac_wire(ctx.msm_g2(pts, words, n))


@pytest.mark.parametrize("bits,spread", [(1, 0.0), (4, 0.0), (8, 0.0), (8, 0.5), (11, 0.0)])
@pytest.mark.parametrize("n", [5000, 131072])
@pytest.mark.parametrize("curve", [bendg.CURVE_G1, bendg.CURVE_G2])
def test_dense_buckets(ctx, curve, n, bits, spread):
    rng = np.random.default_rng(600 + bits + n)
    ks = [int.from_bytes(rng.bytes(32), "little") % o.P_FR for _ in range(4096)]
    reps = -(-n // len(ks))
    pts = np.tile(np.asarray(gpu_points(ctx, curve, ks)).reshape(len(ks), -1), (reps, 1))[:n]
    sc = few_bits(rng, n, bits, spread)
    c = o.G1 if curve == bendg.CURVE_G1 else o.G2
    want = c.mul(c.gen, sum(ks[i % len(ks)] * s for i, s in enumerate(sc)) % o.P_FR)
    assert msm(ctx, curve, pts, scalars_wire(sc), n) == want


@pytest.mark.parametrize("curve", [bendg.CURVE_G1, bendg.CURVE_G2])
def test_scalars_of_8_bits_take_no_longer_than_uniform_ones(ctx, curve):
    """a tenth of the entries: the buckets that hold them must not become one thread's chain"""
    n = 131072
    rng = np.random.default_rng(640)
    ks = [int.from_bytes(rng.bytes(32), "little") % o.P_FR for _ in range(4096)]
    pts = np.tile(np.asarray(gpu_points(ctx, curve, ks)).reshape(len(ks), -1), (n // len(ks), 1))
    run, g = (ctx.msm_g1, "g1") if curve == bendg.CURVE_G1 else (ctx.msm_g2, "g2")
    times = {}
    for name, bits in (("few", 8), ("uniform", 62)):
        words = scalars_wire(few_bits(rng, n, bits, 1.0 if name == "uniform" else 0.0))
        got = []
        for _ in range(5):  # the buckets' kernels on the device
            ctx.profile(True)
            run(pts, words, n)
            got.append(sum(ctx.kernel_stats(k + g)[1] for k in ("msm_bucket_acc_", "msm_heavy_", "msm_reduce_")))
            ctx.profile(False)
        times[name] = min(got)
    assert 0 < times["few"] < times["uniform"], times


@pytest.mark.parametrize("bits,spread", [(1, 0.0), (8, 0.1)])
def test_few_bit_witness_through_pair_rounds_over_tables(ctx, tmp_path, bits, spread):
    """window tables of 2^18 points and up take pair rounds; the same proof without tables takes
    none (the prover does not ask whether the assignment satisfies the circuit)"""
    k = 18
    ctx.synth_square_chain(k, 618, str(tmp_path))
    files = bendg.HostFiles(str(tmp_path))
    rng = np.random.default_rng(650 + bits)
    z = few_bits(rng, (1 << k) + 2, bits, spread)
    w = bendg.ints_to_wire([v * (1 << 256) % o.P_FR for v in z]).reshape(-1)
    rs = rs_words(11, 12)
    key = ctx.pk_upload(files)
    got, _ = key.prove(w, rs)
    key.release()
    inputs = bendg.Inputs.from_buffer_copy(files.inputs)
    inputs.witness, inputs.rs = w.ctypes.data, np.ascontiguousarray(rs).ctypes.data
    want, _ = ctx.prove_inputs(inputs)
    assert ctx.proof_text(got) == ctx.proof_text(want)
