"""Proof inputs whose words lie at or above their modulus stand for the residue: the proof is the one
that the reduced words give."""
import os

import numpy as np
import pytest

import bendg
import bn254_ref as o
from conftest import GOLDEN

pytestmark = pytest.mark.gpu


def lifted(words, p):
    """the largest 256-bit representative of each 16-word element"""
    vals = bendg.wire_to_ints(words)
    return bendg.ints_to_wire([v + (2**256 - 1 - v) // p * p if v else 0 for v in vals]).reshape(words.shape)


@pytest.mark.parametrize("log2n", [0, 1, 5, 9, 13, 16])
@pytest.mark.parametrize("mode", [bendg.NTT_FORWARD, bendg.NTT_INVERSE, bendg.NTT_COSET_FORWARD,
                                  bendg.NTT_COSET_INVERSE])
def test_ntt_of_lifted_words(ctx, log2n, mode):
    rng = np.random.default_rng(60 + log2n)
    vals = [int.from_bytes(rng.bytes(32), "little") % o.P_FR for _ in range(1 << log2n)]
    words = bendg.ints_to_wire(vals)
    up = lifted(words.reshape(-1), o.P_FR).reshape(words.shape)
    some = np.where(rng.random(len(vals))[:, None] < 0.5, up, words)
    want = ctx.ntt(words.reshape(-1), log2n, mode)
    for w in (up, some):
        got = ctx.ntt(np.ascontiguousarray(w).reshape(-1), log2n, mode)
        if log2n:
            assert np.array_equal(got, want)
        else:  # nothing is computed: the word comes back
            assert bendg.wire_to_ints(got)[0] % o.P_FR == bendg.wire_to_ints(want)[0]


@pytest.mark.parametrize("log2d", [1, 7, 14, 15])
def test_qap_of_lifted_words(ctx, log2d):
    rng = np.random.default_rng(61 + log2d)
    abc = [bendg.ints_to_wire([int.from_bytes(rng.bytes(32), "little") % o.P_FR for _ in range(1 << log2d)]).reshape(-1)
           for _ in range(3)]
    want = ctx.qap_h(*abc, log2d)
    assert np.array_equal(ctx.qap_h(*[lifted(v, o.P_FR) for v in abc], log2d), want)


def test_blinding_words_and_key_points(ctx, tmp_path):
    import shutil
    d = os.path.join(GOLDEN, "k4")
    want = open(os.path.join(d, "proof_ref.txt")).read()
    for f in os.listdir(d):
        shutil.copy(os.path.join(d, f), tmp_path / f)
    for f, p in (("rs.bin", o.P_FR), ("pk_g1.bin", o.P_FQ), ("pk_g2.bin", o.P_FQ)):
        w = np.fromfile(tmp_path / f, dtype="<u4")
        lifted(w, p).astype("<u4").tofile(tmp_path / f)
    files = bendg.HostFiles(str(tmp_path))
    proof, _ = ctx.prove_host(files)
    assert ctx.proof_text(proof) == want
    key = ctx.pk_upload(files)
    proof, _ = key.prove(files.words("witness"), files.words("rs"))
    key.release()
    assert ctx.proof_text(proof) == want
